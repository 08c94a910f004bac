// Grouped expert GEMV for decode / batched decode: streams only the routed experts' quantised rows from HBM through
// a shared-memory ring filled by 1-D bulk async copies (TMA), integer dot products against the reference's int8
// activation grid, and fp32 accumulation in EXACTLY the order of the reference's AVX2 kernels, so every dot product
// is bit-identical to the CPU path (and with it every later re-quantisation of activations).
//
// How the reference sums (ggml-cpu/arch/x86/quants.c, AVX2 branches): eight fp32 lanes; lane L collects, block after
// block, fma(scale, (float) p_L, acc_L) where p_L is the integer dot of a fixed group of 4 elements per 32
// (NVFP4: group L of each Q8_0 block; Q3_K: elements 4L..4L+3 of every 32-group of the super-block, scale-weighted and
// summed over the super-block first); the eight lanes are folded at the end as ((a0+a4)+(a2+a6))+((a1+a5)+(a3+a7)).
// Here 8 GPU lanes play the 8 AVX lanes of one weight row (4 rows per warp), each running its chain over K in
// order; three xor-shuffles reproduce the fold.
//
// One kernel template serves
//   DUAL = true : gate and up projections of the same rows + SwiGLU epilogue  -> hidden[row][n_out]
//   DUAL = false: one indexed matmul (ggml MUL_MAT_ID semantics)               -> dst[row][n_out]
// "row" is a routed row: token*n_ids + slot.
//
// Work distribution: the rows of all active experts form one flat list (active expert a, output row r); every CTA of
// the persistent grid takes a contiguous span of equal WORK (rows x passes over the expert's routed rows).  A span is
// walked in chunks of at most ROWS_PER_STAGE rows of one expert; chunk c lives in ring stage c % STAGES.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "formats.cuh"
#include "router.cuh"

namespace b200moe {

struct GemvParams {
    const uint8_t * w0;   // DUAL: gate experts; else the expert tensor  [n_as][n_out][row_bytes]
    const uint8_t * w1;   // DUAL: up experts
    const float * scale0; // per-expert fp32 scale applied to w0's result (or null)
    const float * scale1;
    ActQuant act;         // quantised activation planes, row index = (row / n_ids) * ne11 + (row % n_ids) % ne11
    const float * act_f32; // or: the fp32 activations [rows][K], quantised (Q8_0 or Q8_K) while they are staged (act unused)
    const int * offsets;  // [n_as + 1]
    const int * perm;     // [rows]
    const int * active;   // [n_as]
    const int * meta;     // meta[0] = number of active experts
    const int * cost;     // work prefixes (see Groups::cost)
    float * out;          // [rows][n_out]
    int n_out;
    int n_ids;
    int ne11;
    int n_as;
    float * comb_out;     // one-or-two-token kernel only, or null: the weighted sum over a token's rows goes here ([tokens][n_out])
    const float * comb_w; // [rows] combine weights
    int * comb_cnt;       // [tokens][n_out / 16] rows of `out` finished so far, cleared by the grouping
    int w_stride;         // rows between consecutive experts' matrices: n_out, or 0 when every group uses the same matrix
    int * err;
};

template <int WT, int K, int NW = 8>
struct GemvCfg {
    static constexpr int LPR = 8;            // lanes per row = the reference's 8 SIMD lanes
    static constexpr int RPP = 4;            // rows per warp pass
    static constexpr int ROW_BYTES = WT == TYPE_NVFP4 ? K / 64 * 36 : K / 256 * 110;
    static constexpr int GRAN = (ROW_BYTES % 16 == 0) ? 1 : 8;  // span granularity in rows (16-byte rule of bulk copies)
    static constexpr int NWARPS = NW;        // 8; 4 for the one-or-two-token kernel (several small CTAs per SM)
    // passes per warp per stage chosen so a (single-tensor) stage is roughly 12-40 KB
    static constexpr int PASSES = (ROW_BYTES * RPP * NWARPS >= 12288) ? 1 : (ROW_BYTES * RPP * NWARPS >= 6144) ? 2 : 4;
    static constexpr int ROWS_PER_STAGE = NWARPS * RPP * PASSES;
    static constexpr int TENSOR_STAGE_BYTES = ROWS_PER_STAGE * ROW_BYTES;
    static_assert(TENSOR_STAGE_BYTES % 16 == 0, "stage must keep 16-byte alignment");
    // activations of one token in shared memory: K int8, then the block scales as floats (padded to 16 bytes)
    static constexpr int ACT_D = WT == TYPE_NVFP4 ? K / 32 : K / 256;
    static constexpr int ACT_TOKEN_BYTES = K + ((ACT_D * 4 + 15) / 16) * 16;
};

__device__ __forceinline__ uint32_t lds_u32_a2(const uint8_t * p) {  // 2-byte aligned 32-bit load from shared memory
    const uint16_t * h = reinterpret_cast<const uint16_t *>(p);
    return (uint32_t) h[0] | ((uint32_t) h[1] << 16);
}

// One SIMD lane (L = 0..7) of the reference's dot product of one weight row with NT activation rows.
//   row   : the quantised weight row in shared memory
//   acts  : the activations of NTS rows, token-interleaved: words [K/4][NTS] of int8x4, then block scales [ACT_D][NTS];
//           the first NT of the NTS rows are used
template <int N, typename T>
__device__ __forceinline__ void load_vec(T (&dst)[N], const T * src) {
    static_assert(sizeof(T) == 4, "32-bit elements");
    if (N == 4) {
        const uint4 v = *reinterpret_cast<const uint4 *>(src);
        memcpy(&dst[0], &v, 16);
    } else if (N == 2) {
        const uint2 v = *reinterpret_cast<const uint2 *>(src);
        memcpy(&dst[0], &v, 8);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) dst[i] = src[i];
    }
}

template <int WT, int K, int NT, int NTS>
__device__ __forceinline__ void lane_chain(const uint8_t * __restrict__ row, int L, const uint8_t * __restrict__ acts,
                                           const float * __restrict__ ue_tab, float (&acc)[NT]) {
    using C = GemvCfg<WT, K>;
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t] = 0.0f;
    if (WT == TYPE_NVFP4) {
        // lane L: sub-block (L>>2) of each half block, elements 4*(L&3) .. +3 of it = the low (L&3 < 2) or high nibbles of
        // one qs word; they meet word L of the Q8_0 block.  ggml_vec_dot_nvfp4_q8_0, ggml-cpu/arch/x86/quants.c:1004-1062.
        const int sub_in_half = L >> 2, mp = L & 3;
        const int word_off = 4 + 8 * sub_in_half + 4 * (mp & 1);
        const int nib_shift = 4 * (mp >> 1);
#pragma unroll 2
        for (int b = 0; b < K / 64; ++b) {
            const uint8_t * blk = row + b * NVFP4_BLOCK_BYTES;
            const uint32_t dw = *reinterpret_cast<const uint32_t *>(blk);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const uint32_t w = *reinterpret_cast<const uint32_t *>(blk + 16 * hf + word_off);
                const uint32_t t4 = (w >> nib_shift) & 0x0f0f0f0fu;          // four codes, one per byte
                const uint32_t u = t4 | (t4 >> 4);
                const uint32_t sel = byte_perm(u, 0u, 0x4420u);              // the four codes packed into 16 bits (bytes 0 and 2 of u)
                const uint32_t pos = byte_perm(FP4_MAG_LO, FP4_MAG_HI, sel);
                const uint32_t neg = byte_perm(FP4_MAG_LO, FP4_MAG_HI, sel ^ 0x8888u);
                // signed bytes: a byte of `neg` is a magnitude 0..12, 0x80 - it never borrows, the xor drops the guard bit
                const uint32_t code = pos | ((0x80808080u - neg) ^ 0x80808080u);
                const float sw = ue_tab[(dw >> (8 * (2 * hf + sub_in_half))) & 0xff];
                const int unit = 2 * b + hf;
                // activations are stored [unit][lane word][token] and [unit][token]: one vector load serves all NT rows
                uint32_t aw[NT];
                float dy[NT];
                load_vec<NT>(aw, reinterpret_cast<const uint32_t *>(acts) + (size_t) (unit * 8 + L) * NTS);
                load_vec<NT>(dy, reinterpret_cast<const float *>(acts + (size_t) K * NTS) + (size_t) unit * NTS);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const int p = dot4((int) code, (int) aw[t], 0);
                    acc[t] = __fmaf_rn(__fmul_rn(sw, dy[t]), small_int_to_float(p), acc[t]);
                }
            }
        }
    } else {
        // lane L: byte columns 4L..4L+3 of every super-block; integer sum over the super-block with the signed 6-bit
        // sub-block scales, then one fma with d_w*d_x.  ggml_vec_dot_q3_K_q8_K, ggml-cpu/arch/x86/quants.c:1766-1880.
        const int hi = L >= 4 ? 1 : 0;
#pragma unroll 1
        for (int sb = 0; sb < K / 256; ++sb) {
            const uint8_t * blk = row + sb * Q3K_BLOCK_BYTES;  // 2-byte aligned
            const uint32_t hm = lds_u32_a2(blk + 4 * L);
            const uint32_t qs0 = lds_u32_a2(blk + 32 + 4 * L);
            const uint32_t qs1 = lds_u32_a2(blk + 64 + 4 * L);
            uint32_t sc[4];
            q3k_unpack_scales(lds_u32_a2(blk + 96), lds_u32_a2(blk + 100), lds_u32_a2(blk + 104), sc);
            const float dw = __half2float(*reinterpret_cast<const __half *>(blk + 108));
            int sumi[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) sumi[t] = 0;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint32_t w = j ? qs1 : qs0;
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const int bit = 4 * j + s;
                    const uint32_t lo2 = (w >> (2 * s)) & 0x03030303u;
                    const uint32_t hb4 = bit >= 2 ? ((hm >> (bit - 2)) & 0x04040404u) : ((hm << (2 - bit)) & 0x04040404u);
                    // codes 0..7 -> signed -4..3 in every byte without borrows between bytes
                    const uint32_t code = (((lo2 | hb4) | 0x80808080u) - 0x04040404u) ^ 0x80808080u;
                    const int scale = q3k_scale_at(sc, 8 * j + 2 * s + hi);
                    uint32_t aw[NT];
                    load_vec<NT>(aw, reinterpret_cast<const uint32_t *>(acts) + (size_t) (sb * 64 + 8 * (4 * j + s) + L) * NTS);
#pragma unroll
                    for (int t = 0; t < NT; ++t) sumi[t] += scale * dot4((int) code, (int) aw[t], 0);
                }
            }
            float dx[NT];
            load_vec<NT>(dx, reinterpret_cast<const float *>(acts + (size_t) K * NTS) + (size_t) sb * NTS);
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[t] = __fmaf_rn(__fmul_rn(dx[t], dw), small_int_to_float(sumi[t]), acc[t]);
        }
    }
    // hsum_float_8: (a4+a0, a5+a1, a6+a2, a7+a3) -> (r0+r2, r1+r3) -> s0+s1
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        float v = acc[t];
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
        acc[t] = v;
    }
}

// decode of four NVFP4 codes (one per byte of t4's nibbles) to signed int8 (twice the E2M1 value)
__device__ __forceinline__ uint32_t nvfp4_codes_to_s8(uint32_t w, int nib_shift) {
    const uint32_t t4 = (w >> nib_shift) & 0x0f0f0f0fu;          // four codes, one per byte
    const uint32_t u = t4 | (t4 >> 4);
    const uint32_t sel = byte_perm(u, 0u, 0x4420u);              // the four codes packed into 16 bits (bytes 0 and 2 of u)
    const uint32_t pos = byte_perm(FP4_MAG_LO, FP4_MAG_HI, sel);
    const uint32_t neg = byte_perm(FP4_MAG_LO, FP4_MAG_HI, sel ^ 0x8888u);
    // signed bytes: a byte of `neg` is a magnitude 0..12, 0x80 - it never borrows, the xor drops the guard bit
    return pos | ((0x80808080u - neg) ^ 0x80808080u);
}

// lane_chain<TYPE_NVFP4> for TWO weight rows against the same activations (the gate row and the up row of a feature): the two
// chains are independent, so running them in one loop doubles the work in flight per lane - and each activation word and block
// scale is fetched once for both.  Every chain keeps its own order of operations: the results are those of two lane_chain calls.
template <int K, int NT, int NTS>
__device__ __forceinline__ void lane_chain_pair(const uint8_t * __restrict__ row0, const uint8_t * __restrict__ row1, int L,
                                                const uint8_t * __restrict__ acts, const float * __restrict__ ue_tab, float (&acc0)[NT],
                                                float (&acc1)[NT]) {
#pragma unroll
    for (int t = 0; t < NT; ++t) acc0[t] = acc1[t] = 0.0f;
    const int sub_in_half = L >> 2, mp = L & 3;
    const int word_off = 4 + 8 * sub_in_half + 4 * (mp & 1);
    const int nib_shift = 4 * (mp >> 1);
#pragma unroll 2
    for (int b = 0; b < K / 64; ++b) {
        const uint8_t * blk0 = row0 + b * NVFP4_BLOCK_BYTES, * blk1 = row1 + b * NVFP4_BLOCK_BYTES;
        const uint32_t dw0 = *reinterpret_cast<const uint32_t *>(blk0), dw1 = *reinterpret_cast<const uint32_t *>(blk1);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const uint32_t code0 = nvfp4_codes_to_s8(*reinterpret_cast<const uint32_t *>(blk0 + 16 * hf + word_off), nib_shift);
            const uint32_t code1 = nvfp4_codes_to_s8(*reinterpret_cast<const uint32_t *>(blk1 + 16 * hf + word_off), nib_shift);
            const float sw0 = ue_tab[(dw0 >> (8 * (2 * hf + sub_in_half))) & 0xff], sw1 = ue_tab[(dw1 >> (8 * (2 * hf + sub_in_half))) & 0xff];
            const int unit = 2 * b + hf;
            uint32_t aw[NT];
            float dy[NT];
            load_vec<NT>(aw, reinterpret_cast<const uint32_t *>(acts) + (size_t) (unit * 8 + L) * NTS);
            load_vec<NT>(dy, reinterpret_cast<const float *>(acts + (size_t) K * NTS) + (size_t) unit * NTS);
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                acc0[t] = __fmaf_rn(__fmul_rn(sw0, dy[t]), small_int_to_float(dot4((int) code0, (int) aw[t], 0)), acc0[t]);
                acc1[t] = __fmaf_rn(__fmul_rn(sw1, dy[t]), small_int_to_float(dot4((int) code1, (int) aw[t], 0)), acc1[t]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        float v = acc0[t], w = acc1[t];
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
        w = __fadd_rn(w, __shfl_xor_sync(0xffffffffu, w, 4));
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
        w = __fadd_rn(w, __shfl_xor_sync(0xffffffffu, w, 2));
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
        w = __fadd_rn(w, __shfl_xor_sync(0xffffffffu, w, 1));
        acc0[t] = v;
        acc1[t] = w;
    }
}

// ---- two SIMD lanes per thread ---------------------------------------------------------------------------------------------
// The low nibbles of a qs word belong to one lane of the reference and its high nibbles to another (lanes 4 sub + w and 4 sub + w + 2 of
// sub-block `sub`, word w), so four threads can play the eight lanes of a row: a thread takes word m = 2 sub + w of every half-block, looks
// all eight codes up at once and shares the block scale between its two chains.  That is 13 instructions of decode for eight codes where a
// lane by itself spends 10 on four and throws the other nibbles away, and half the loads of words, scales and table entries.
// `lo` and `hi`: four signed bytes each (twice the E2M1 values), in the order of the lane's activation word.
__device__ __forceinline__ void nvfp4_word_to_s8(uint32_t w, uint32_t & lo, uint32_t & hi) {
    const uint32_t wn = w ^ 0x88888888u;
    const uint32_t pa = byte_perm(FP4_MAG_LO, FP4_MAG_HI, w), pb = byte_perm(FP4_MAG_LO, FP4_MAG_HI, w >> 16);
    const uint32_t na = byte_perm(FP4_MAG_LO, FP4_MAG_HI, wn), nb = byte_perm(FP4_MAG_LO, FP4_MAG_HI, wn >> 16);
    // signed bytes: a byte of `n` is a magnitude 0..12, 0x80 - it never borrows, the xor drops the guard bit
    const uint32_t a = pa | ((0x80808080u - na) ^ 0x80808080u);   // low, high nibble of byte 0, low, high nibble of byte 1
    const uint32_t b = pb | ((0x80808080u - nb) ^ 0x80808080u);   // the same of bytes 2 and 3
    lo = byte_perm(a, b, 0x6420);
    hi = byte_perm(a, b, 0x7531);
}
// Two fp32 values in one register pair: sm_100's packed instructions round each half as the scalar ones do.
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f32x2_halves(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// two integer dots as floats: the constant 1.5 * 2^23 rides in the accumulator of dp4a (see small_int_to_float)
__device__ __forceinline__ uint64_t dots_to_f32x2(uint32_t code0, uint32_t act0, uint32_t code1, uint32_t act1) {
    return add_f32x2(f32x2(__int_as_float(dot4((int) code0, (int) act0, 0x4B400000)), __int_as_float(dot4((int) code1, (int) act1, 0x4B400000))),
                     f32x2(-12582912.0f, -12582912.0f));
}
// hsum_float_8 of a row whose lanes L0 = 4 (m >> 1) + (m & 1) and L0 + 2 thread m holds: (a0+a4), (a2+a6) / (a1+a5), (a3+a7) across the
// threads of a word, (r0+r2) / (r1+r3) inside the thread, then the two words.  The result is valid in all four threads.
__device__ __forceinline__ float hsum_two_lanes(float lo, float hi) {
    lo = __fadd_rn(lo, __shfl_xor_sync(0xffffffffu, lo, 2));
    hi = __fadd_rn(hi, __shfl_xor_sync(0xffffffffu, hi, 2));
    lo = __fadd_rn(lo, hi);
    return __fadd_rn(lo, __shfl_xor_sync(0xffffffffu, lo, 1));
}
// where the word of SIMD lane L of a 32-unit lies in activations staged for these chains: the two lanes of thread m are neighbours
__host__ __device__ __forceinline__ constexpr int act_slot(int L) { return (L & 4) | ((L & 1) << 1) | ((L >> 1) & 1); }

// The chains of NROW weight rows against NT activation rows (1, 2 or 4) as pairs of accumulators: of two tokens' same lane, or, for one
// token, of its two lanes.
template <int NROW, int NT>
struct TwoLaneAcc {
    static constexpr int N = NT == 1 ? 1 : NT;
    uint64_t v[NROW][N];                                       // [row][lane lo: token pairs, lane hi: token pairs]
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int r = 0; r < NROW; ++r)
#pragma unroll
            for (int i = 0; i < N; ++i) v[r][i] = f32x2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void lanes(int r, int t, float & lo, float & hi) const {
        if (NT == 1) {
            const float2 a = f32x2_halves(v[r][0]);
            lo = a.x; hi = a.y;
        } else {
            const float2 a = f32x2_halves(v[r][t / 2]), b = f32x2_halves(v[r][(N / 2 + t / 2) % N]);
            lo = t & 1 ? a.y : a.x; hi = t & 1 ? b.y : b.x;
        }
    }
};

// 256 elements (four blocks) of the weight rows: the chains go on in acc.
//   blk[r]: first byte of the four blocks of row r; acts: the words of these eight units, [unit][act_slot][NTS]; dy: [unit][NTS]
template <int NROW, int NT, int NTS>
__device__ __forceinline__ void two_lane_chains(const uint8_t * const (&blk)[NROW], int m, const uint32_t * __restrict__ acts, const float * __restrict__ dy,
                                                const float * __restrict__ ue_tab, TwoLaneAcc<NROW, NT> & acc) {
    const int sub = m >> 1;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        uint32_t dw[NROW];
#pragma unroll
        for (int r = 0; r < NROW; ++r) dw[r] = *reinterpret_cast<const uint32_t *>(blk[r] + b * NVFP4_BLOCK_BYTES) >> (8 * sub);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int unit = 2 * b + hf;
            uint32_t alo[NT], ahi[NT];
            float d[NT];
            const uint32_t * aw = acts + (unit * 8 + 2 * m) * NTS;
            load_vec<NT>(alo, aw);
            load_vec<NT>(ahi, aw + NTS);
            load_vec<NT>(d, dy + unit * NTS);
#pragma unroll
            for (int r = 0; r < NROW; ++r) {
                uint32_t lo, hi;
                nvfp4_word_to_s8(*reinterpret_cast<const uint32_t *>(blk[r] + b * NVFP4_BLOCK_BYTES + 4 + 16 * hf + 4 * m), lo, hi);
                const float sw = ue_tab[(dw[r] >> (16 * hf)) & 0xff];
                if constexpr (NT == 1) {
                    const float s = __fmul_rn(sw, d[0]);
                    acc.v[r][0] = fma_f32x2(f32x2(s, s), dots_to_f32x2(lo, alo[0], hi, ahi[0]), acc.v[r][0]);
                } else {
                    const uint64_t sw2 = f32x2(sw, sw);
#pragma unroll
                    for (int t = 0; t < NT; t += 2) {
                        const uint64_t s = mul_f32x2(sw2, f32x2(d[t], d[t + 1]));
                        acc.v[r][t / 2] = fma_f32x2(s, dots_to_f32x2(lo, alo[t], lo, alo[t + 1]), acc.v[r][t / 2]);
                        acc.v[r][NT / 2 + t / 2] = fma_f32x2(s, dots_to_f32x2(hi, ahi[t], hi, ahi[t + 1]), acc.v[r][NT / 2 + t / 2]);
                    }
                }
            }
        }
    }
}

// The chains of one weight row in shared memory against ONE activation row whose int8 values (q, K bytes) and block scales (d, K/32
// floats, 8-byte aligned) lie in separate arrays in global memory.  The result is valid in the row's four threads.
template <int K>
__device__ __forceinline__ float two_lane_chain_split(const uint8_t * __restrict__ row, int m, const uint8_t * __restrict__ q, const float * __restrict__ d,
                                                      const float * __restrict__ ue_tab) {
    const int sub = m >> 1;
    const uint32_t * qw = reinterpret_cast<const uint32_t *>(q) + 4 * sub + (m & 1);
    uint64_t acc = f32x2(0.0f, 0.0f);
#pragma unroll 8
    for (int b = 0; b < K / 64; ++b) {
        const float2 dy = __ldg(reinterpret_cast<const float2 *>(d) + b);
        const uint8_t * const blk = row + b * NVFP4_BLOCK_BYTES;
        const uint32_t dw = *reinterpret_cast<const uint32_t *>(blk) >> (8 * sub);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            uint32_t lo, hi;
            nvfp4_word_to_s8(*reinterpret_cast<const uint32_t *>(blk + 4 + 16 * hf + 4 * m), lo, hi);
            const float s = __fmul_rn(ue_tab[(dw >> (16 * hf)) & 0xff], hf ? dy.y : dy.x);
            acc = fma_f32x2(f32x2(s, s), dots_to_f32x2(lo, __ldg(qw + (2 * b + hf) * 8), hi, __ldg(qw + (2 * b + hf) * 8 + 2)), acc);
        }
    }
    const float2 a = f32x2_halves(acc);
    return hsum_two_lanes(a.x, a.y);
}

// Distance of staged weight rows that the two-lane chains read: eight rows of a warp, four words of each, then fall on different banks.
__host__ __device__ constexpr int two_lane_pitch(int row_bytes) { return row_bytes % 32 ? row_bytes : row_bytes + 16; }

// The same chain run by a whole warp for ONE row: the four 8-lane groups split the half-blocks between them (group rg takes
// units rg, rg + 4, ...), every lane fetches and decodes its share with all loads in flight at once, and the fp32 chain - which
// must stay sequential to keep the reference's bits - then collects scale and dot product of every unit in order through
// shuffles.  All four groups end with the same eight partial sums; the result is valid in every lane.
template <int K>
__device__ __forceinline__ float lane_chain_warp(const uint8_t * __restrict__ row, int lane, const uint8_t * __restrict__ q,
                                                 const float * __restrict__ d, const float * __restrict__ ue_tab) {
    constexpr int UNITS = K / 32, UPL = UNITS / 4;       // half-blocks in the row, and per lane
    constexpr int BATCH = UPL < 8 ? UPL : 8;             // fetched and decoded at a time (bounds the registers)
    static_assert(UNITS % 4 == 0 && UPL % BATCH == 0, "half-blocks must split over four lane groups in whole batches");
    const int L = lane & 7, rg = lane >> 3;
    const int sub_in_half = L >> 2, mp = L & 3;
    const int word_off = 4 + 8 * sub_in_half + 4 * (mp & 1);
    const int nib_shift = 4 * (mp >> 1);
    float a = 0.0f;
#pragma unroll 1
    for (int i0 = 0; i0 < UPL; i0 += BATCH) {
        uint32_t w[BATCH], aw[BATCH], dw[BATCH];
        float dy[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int u = 4 * (i0 + i) + rg, b = u >> 1, hf = u & 1;
            const uint8_t * blk = row + b * NVFP4_BLOCK_BYTES;
            dw[i] = *reinterpret_cast<const uint32_t *>(blk);
            w[i] = *reinterpret_cast<const uint32_t *>(blk + 16 * hf + word_off);
            aw[i] = reinterpret_cast<const uint32_t *>(q)[u * 8 + L];
            dy[i] = d[u];
        }
        float sd[BATCH], pf[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int hf = rg & 1;                       // u = 4 (i0 + i) + rg
            const uint32_t t4 = (w[i] >> nib_shift) & 0x0f0f0f0fu;
            const uint32_t u8 = t4 | (t4 >> 4);
            const uint32_t sel = byte_perm(u8, 0u, 0x4420u);
            const uint32_t pos = byte_perm(FP4_MAG_LO, FP4_MAG_HI, sel);
            const uint32_t neg = byte_perm(FP4_MAG_LO, FP4_MAG_HI, sel ^ 0x8888u);
            const uint32_t code = pos | ((0x80808080u - neg) ^ 0x80808080u);
            const float sw = ue_tab[(dw[i] >> (8 * (2 * hf + sub_in_half))) & 0xff];
            sd[i] = __fmul_rn(sw, dy[i]);
            pf[i] = small_int_to_float(dot4((int) code, (int) aw[i], 0));
        }
#pragma unroll
        for (int u = 0; u < 4 * BATCH; ++u) {            // units 4 i0 .. 4 (i0 + BATCH) - 1, in order
            const int src = (u & 3) * 8 + L;
            const float sv = __shfl_sync(0xffffffffu, sd[u >> 2], src), pv = __shfl_sync(0xffffffffu, pf[u >> 2], src);
            a = __fmaf_rn(sv, pv, a);
        }
    }
    a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 4));
    a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 2));
    a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, 1));
    return a;
}

// chunk walker shared by the producer thread and the consumers
struct Chunk {
    int a;      // index into active[]
    int r0;     // first output row
    int n;      // rows
};
struct ChunkWalker {
    int u, u_end, units_per_expert, gran, max_rows;
    __device__ __forceinline__ bool next(Chunk & c) {
        if (u >= u_end) return false;
        const int a = u / units_per_expert;
        const int uu = u - a * units_per_expert;
        int n_units = min(u_end - u, units_per_expert - uu);
        n_units = min(n_units, max_rows / gran);
        c.a = a;
        c.r0 = uu * gran;
        c.n = n_units * gran;
        u += n_units;
        return true;
    }
};

// A CTA's part of the work: items (active expert a, pass ps over PT of its routed rows, chunk ch of its weight rows), chunks fastest.
template <int PT>
struct PassSpan {
    int a, ps, ch;          // next item
    int a1, ps1, ch1;       // the next CTA's first
    int chunks;             // of an expert
    __device__ __forceinline__ bool more() const { return a < a1 || (a == a1 && (ps < ps1 || (ps == ps1 && ch < ch1))); }
    __device__ __forceinline__ void next(int n_e) {          // n_e: routed rows of expert a
        if (++ch < chunks) return;
        ch = 0;
        if (PT * ++ps < n_e) return;
        ps = 0;
        ++a;
    }
};
// Boundary i sits at work i / grid of the total; both neighbours compute it the same way, so the spans tile exactly.  cw: prefix over the
// active experts of the work per chunk: FULL for each pass, what is left of it for the last one.  The whole block looks for its two experts
// at once.
template <int THREADS, int PT, int FULL>
__device__ __forceinline__ PassSpan<PT> pass_span(const int * __restrict__ cw, int n_active, int chunks) {
    __shared__ int s_at[2];
    const long long work = n_active ? (long long) cw[n_active] * chunks : 0;
    const long long c[2] = { work * blockIdx.x / gridDim.x, work * (blockIdx.x + 1) / gridDim.x };
    if (threadIdx.x < 2) s_at[threadIdx.x] = n_active;
    __syncthreads();
    for (int i = threadIdx.x; i < n_active; i += THREADS) {
        const long long here = (long long) cw[i] * chunks, next = (long long) cw[i + 1] * chunks;
        if (here <= c[0] && c[0] < next) s_at[0] = i;
        if (here <= c[1] && c[1] < next) s_at[1] = i;
    }
    __syncthreads();
    int at[2][3] = { { n_active, 0, 0 }, { n_active, 0, 0 } };
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int a = s_at[k];
        if (a == n_active) continue;                         // the end of the list
        const int w = cw[a + 1] - cw[a];
        const long long left = c[k] - (long long) cw[a] * chunks;
        at[k][0] = a;
        at[k][1] = (int) (left / (FULL * chunks));
        at[k][2] = (int) (left - (long long) at[k][1] * FULL * chunks) / min(FULL, w - FULL * at[k][1]);
    }
    return PassSpan<PT>{ at[0][0], at[0][1], at[0][2], at[1][0], at[1][1], at[1][2], chunks };
}

template <int WT, int K, bool DUAL, int NT, int STAGES, int NW = 8>
constexpr size_t gemv_smem_bytes() {
    return (size_t) STAGES * GemvCfg<WT, K, NW>::TENSOR_STAGE_BYTES * (DUAL ? 2 : 1) + NT * GemvCfg<WT, K, NW>::ACT_TOKEN_BYTES + STAGES * 8 +
           256 * 4 + 64;
}

// CTAs per SM: the kernel waits on the latency of its own lane chains, so two CTAs (16 warps) beat one with a deeper ring; two
// whenever two stages and the activations fit twice.  Ring depth: what fits then, up to four stages.
template <int WT, int K, bool DUAL, int NT>
constexpr int gemv_ctas() { return 2 * (gemv_smem_bytes<WT, K, DUAL, NT, 2>() + 1024 + 128) <= 228 * 1024 ? 2 : 1; }
template <int WT, int K, bool DUAL, int NT>
constexpr int gemv_stages() {
    if (gemv_ctas<WT, K, DUAL, NT>() == 2)
        return 2 * (gemv_smem_bytes<WT, K, DUAL, NT, 4>() + 1024 + 128) <= 228 * 1024 ? 4 : 2 * (gemv_smem_bytes<WT, K, DUAL, NT, 3>() + 1024 + 128) <= 228 * 1024 ? 3 : 2;
    constexpr int stage = GemvCfg<WT, K>::TENSOR_STAGE_BYTES * (DUAL ? 2 : 1);
    return (4 * stage <= 190 * 1024) ? 4 : (3 * stage <= 190 * 1024) ? 3 : 2;
}

template <int WT, int K, bool DUAL, int NT, int STAGES, int NW = 8>
__global__ void __launch_bounds__(NW * 32, NW == 8 ? gemv_ctas<WT, K, DUAL, NT>() : 4) expert_gemv_kernel(const GemvParams p) {
    using C = GemvCfg<WT, K, NW>;
    constexpr int NTENS = DUAL ? 2 : 1;
    constexpr int STAGE_BYTES = C::TENSOR_STAGE_BYTES * NTENS;
    constexpr int NTHREADS = C::NWARPS * 32;

    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t * ring = smem;                                                        // STAGES * STAGE_BYTES
    uint8_t * acts = smem + STAGES * STAGE_BYTES;                                 // NT * ACT_TOKEN_BYTES (16-byte aligned)
    uint64_t * full = reinterpret_cast<uint64_t *>(acts + NT * C::ACT_TOKEN_BYTES);  // STAGES barriers
    float * ue_tab = reinterpret_cast<float *>(full + STAGES);                    // 256 floats (NVFP4 only)
    __shared__ int s_abort, s_last;
    __shared__ int s_span[2];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int L = lane & 7;       // SIMD lane of the reference this thread plays
    const int rgrp = lane >> 3;   // which of the 4 rows of a warp pass

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
        mbar_fence_init();
        s_abort = 0;
    }
    if (WT == TYPE_NVFP4)
        for (int i = tid; i < 256; i += NTHREADS) ue_tab[i] = ue4m3_half_to_f32(i);
    __syncthreads();
    pdl_wait();                 // programmatic dependent launch: everything before this ran alongside the previous kernel's tail
    pdl_launch_dependents();

    const int n_active = p.meta[0];
    const int upe = p.n_out / C::GRAN;                       // span units per expert
    const long long total = (long long) n_active * upe;
    // Span boundaries balance WORK, not rows: a weight row of an expert with n routed rows costs 3 per pass (decode) + 2 per routed row.
    // Boundary i sits at work i/grid of the total; both neighbours compute it the same way, so spans tile exactly.
    if (NW != 8) {
        // one-or-two-token kernel: CTA b owns stage-sized chunk b of the flat row list - no search, no dependent loads
        if (tid < 2) {
            const long long u = (long long) (blockIdx.x + tid) * (C::ROWS_PER_STAGE / C::GRAN);
            s_span[tid] = (int) (u < total ? u : total);
        }
    } else if (tid < 2) {
        const int * cw = p.cost + (NT == 1 ? 0 : 2) * (p.n_as + 1);
        const long long total_work = (long long) cw[n_active] * upe;
        const long long c = total_work * (blockIdx.x + tid) / gridDim.x;
        int lo = 0, hi = n_active;  // largest a with cw[a]*upe <= c
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((long long) cw[mid] * upe <= c) lo = mid; else hi = mid;
        }
        int u;
        if (n_active == 0) u = 0;
        else if (blockIdx.x + tid == gridDim.x) u = (int) total;
        else {
            const int per = max(cw[lo + 1] - cw[lo], 1);
            const long long uu = (c - (long long) cw[lo] * upe) / per;
            u = lo * upe + (int) (uu < (long long) upe ? uu : (long long) upe);
        }
        s_span[tid] = u;
    }
    __syncthreads();
    ChunkWalker cons, prod;
    cons.u = s_span[0];
    cons.u_end = s_span[1];
    cons.units_per_expert = upe;
    cons.gran = C::GRAN;
    cons.max_rows = C::ROWS_PER_STAGE;
    prod = cons;

    auto issue = [&](const Chunk & c, int stage) {
        const int e = p.active[c.a];
        const uint32_t bytes = (uint32_t) c.n * C::ROW_BYTES;
        uint8_t * dst = ring + (size_t) stage * STAGE_BYTES;
        mbar_arrive_expect_tx(&full[stage], bytes * NTENS);
        const size_t off = ((size_t) e * p.w_stride + c.r0) * C::ROW_BYTES;
        bulk_g2s(dst, p.w0 + off, bytes, &full[stage]);
        if (DUAL) bulk_g2s(dst + C::TENSOR_STAGE_BYTES, p.w1 + off, bytes, &full[stage]);
    };

    int issued = 0;
    if (tid == 0) {
        Chunk c;
        for (int s = 0; s < STAGES; ++s)
            if (prod.next(c)) { issue(c, s); ++issued; }
    }

    int loaded_e = -1, loaded_tc = -1;
    Chunk ck;
    int ci = 0;
    bool failed = false;
    while (cons.next(ck)) {
        const int stage = ci % STAGES;
        const uint32_t parity = (uint32_t) (ci / STAGES) & 1u;
        bool landed = false;    // the weights are waited for behind the loads of the first pass's activations

        const int e = p.active[ck.a];
        const int row_beg = p.offsets[e], n_e = p.offsets[e + 1] - row_beg;
        const uint8_t * st = ring + (size_t) stage * STAGE_BYTES;
        // A warp without rows leaves a pass out: with two CTAs on the SM its idle chains would hold up the other's (8 experts, 256 -> 512, 400
        // rows each: 1020 us with them, 547 without; one CTA per SM 906 and 547).  The chunks of the few-row kernel are whole at the widths of a layer.
        const int first_row = warp * C::RPP, pass_rows = C::NWARPS * C::RPP;
        const int my_passes = NW != 8 ? C::PASSES : ck.n > first_row ? (ck.n - first_row + pass_rows - 1) / pass_rows : 0;
        const int se = p.w_stride ? e : 0;      // every group of a dense product has the one matrix and its scale
        const float sc0 = p.scale0 ? p.scale0[se] : 1.0f;
        const float sc1 = (DUAL && p.scale1) ? p.scale1[se] : 1.0f;

        // Routed rows of this expert are taken NT at a time; a remainder of 1 or 2 runs the narrower chains instead of
        // padding to NT (the weight decode is shared by the rows of a pass, the per-row work is not).
        for (int t0 = 0, tc = 0; t0 < n_e; ++tc) {
            const int left = n_e - t0;
            const int ntc = (NT >= 4 && left >= 3) ? 4 : (NT >= 2 && left >= 2) ? 2 : 1;
            int rows[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int i = t0 + t;
                rows[t] = (t < ntc && i < n_e) ? p.perm[row_beg + i] : -1;
            }
            if (loaded_e != e || loaded_tc != tc) {
                // the activation rows of this pass into shared memory (all warps use the same ones)
                __syncthreads();
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    if (t >= ntc) break;
                    const int r = rows[t];
                    const int arow = r >= 0 ? (r / p.n_ids) * p.ne11 + (r % p.n_ids) % p.ne11 : 0;
                    uint32_t * dq = reinterpret_cast<uint32_t *>(acts);
                    float * dd = reinterpret_cast<float *>(acts + (size_t) K * NT);
                    if (WT == TYPE_NVFP4 && p.act_f32) {
                        // Q8_0 on the fly, the arithmetic of quantize_q8_0_block: 8 lanes hold one block of 32 (4 values each)
                        const float4 * src = reinterpret_cast<const float4 *>(p.act_f32 + (size_t) arow * K);
                        for (int i0 = 0; i0 < K / 4; i0 += NTHREADS) {
                            const int i = i0 + tid;
                            const bool in = i < K / 4;
                            const float4 v = (in && r >= 0) ? __ldg(src + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
                            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
                            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
                            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
                            const float id = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
                            const uint32_t q = ((uint32_t) __float2int_rn(__fmul_rn(v.x, id)) & 0xffu) |
                                               (((uint32_t) __float2int_rn(__fmul_rn(v.y, id)) & 0xffu) << 8) |
                                               (((uint32_t) __float2int_rn(__fmul_rn(v.z, id)) & 0xffu) << 16) |
                                               (((uint32_t) __float2int_rn(__fmul_rn(v.w, id)) & 0xffu) << 24);
                            if (in) {
                                dq[(size_t) i * NT + t] = q;
                                if ((i & 7) == 0) dd[(size_t) (i >> 3) * NT + t] = __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
                            }
                        }
                    } else if (WT == TYPE_Q3_K && p.act_f32) {
                        for (int b = warp; b < K / 256; b += C::NWARPS) {      // a warp quantises one 256-block
                            uint32_t q[2] = { 0u, 0u };
                            float d = 0.0f;
                            if (r >= 0) q8_K_words(p.act_f32 + (size_t) arow * K + b * 256 + lane * 8, lane, q, d);
                            dq[(size_t) (b * 64 + lane * 2) * NT + t] = q[0];
                            dq[(size_t) (b * 64 + lane * 2 + 1) * NT + t] = q[1];
                            if (lane == 0) dd[(size_t) b * NT + t] = d;
                        }
                    } else {
                        const uint32_t * srcq = reinterpret_cast<const uint32_t *>(p.act.q + (size_t) arow * K);
                        for (int i = tid; i < K / 4; i += NTHREADS) dq[(size_t) i * NT + t] = r >= 0 ? __ldg(srcq + i) : 0u;
                        for (int i = tid; i < C::ACT_D; i += NTHREADS) dd[(size_t) i * NT + t] = r >= 0 ? __ldg(p.act.d + (size_t) arow * C::ACT_D + i) : 0.0f;
                    }
                }
                __syncthreads();
                loaded_e = e;
                loaded_tc = tc;
            }
            if (!landed) {
                if (!mbar_wait_bounded(&full[stage], parity)) {
                    report_error(p.err, DEV_ERR_BARRIER_TIMEOUT);
                    s_abort = 1;
                }
                if (__syncthreads_or(s_abort)) { failed = true; break; }
                landed = true;
            }
#pragma unroll 1
            for (int ps = 0; ps < C::PASSES; ++ps) {
                if (ps >= my_passes) break;
                const int lr = (ps * C::NWARPS + warp) * C::RPP + rgrp;  // row within the stage
                const bool row_ok = lr < ck.n;
                const uint8_t * wrow = st + (size_t) (row_ok ? lr : 0) * C::ROW_BYTES;
                float g[NT], uacc[NT];
                auto run = [&](auto ntag) {
                    constexpr int NTC = decltype(ntag)::value;
                    float gg[NTC], uu[NTC];
                    if constexpr (DUAL && WT == TYPE_NVFP4) {
                        lane_chain_pair<K, NTC, NT>(wrow, wrow + C::TENSOR_STAGE_BYTES, L, acts, ue_tab, gg, uu);
                    } else {
                        lane_chain<WT, K, NTC, NT>(wrow, L, acts, ue_tab, gg);
                        if (DUAL) lane_chain<WT, K, NTC, NT>(wrow + C::TENSOR_STAGE_BYTES, L, acts, ue_tab, uu);
                    }
#pragma unroll
                    for (int t = 0; t < NTC; ++t) { g[t] = gg[t]; uacc[t] = DUAL ? uu[t] : 0.0f; }
                };
                if (NT >= 4 && ntc == 4) run(std::integral_constant<int, (NT >= 4 ? 4 : 1)>{});
                else if (NT >= 2 && ntc == 2) run(std::integral_constant<int, (NT >= 2 ? 2 : 1)>{});
                else run(std::integral_constant<int, 1>{});
                if (row_ok && L == 0) {
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        const int r = rows[t];
                        if (t < ntc && r >= 0) {
                            float v = __fmul_rn(g[t], sc0);
                            if (DUAL) v = __fmul_rn(ggml_silu(v), __fmul_rn(uacc[t], sc1));
                            p.out[(size_t) r * p.n_out + ck.r0 + lr] = v;
                        }
                    }
                }
            }
            t0 += ntc;
        }
        if (failed) break;
        if (NW != 8 && !DUAL && p.comb_out) {
            // The rows of this chunk are finished for every routed row of this expert.  The CTA that finishes the last of a token's
            // rows sums them - in slot order, so which CTA that is does not show - and saves the combine its launch.
            __threadfence();
            __syncthreads();
            for (int i = 0; i < n_e; ++i) {
                const int tok = p.perm[row_beg + i] / p.n_ids;
                if (tid == 0) s_last = atomicAdd(&p.comb_cnt[tok * (p.n_out / 16) + ck.r0 / 16], 1) == p.n_ids - 1;
                __syncthreads();
                if (s_last) {
                    __threadfence();
                    const float * wr = p.comb_w + (size_t) tok * p.n_ids;
                    for (int j = tid; j < ck.n; j += NTHREADS) {
                        const float * y = p.out + (size_t) tok * p.n_ids * p.n_out + ck.r0 + j;
                        float a = 0.0f;
                        for (int s0 = 0; s0 < p.n_ids; s0 += 8) {          // eight rows' loads in flight, added in slot order
                            float v[8], w[8];
#pragma unroll
                            for (int s = 0; s < 8; ++s) {
                                const bool in = s0 + s < p.n_ids;
                                v[s] = in ? __ldcg(y + (size_t) (s0 + s) * p.n_out) : 0.0f;
                                w[s] = in ? wr[s0 + s] : 0.0f;
                            }
#pragma unroll
                            for (int s = 0; s < 8; ++s)
                                if (s0 + s < p.n_ids) a = s0 + s == 0 ? __fmul_rn(v[s], w[s]) : __fadd_rn(a, __fmul_rn(v[s], w[s]));
                        }
                        p.comb_out[(size_t) tok * p.n_out + ck.r0 + j] = a;
                    }
                }
                __syncthreads();
            }
        }
        __syncthreads();  // everyone is done reading this stage
        if (tid == 0) {
            Chunk c;
            if (prod.next(c)) { issue(c, stage); ++issued; }
        }
        ++ci;
    }

    if (failed && tid == 0) {
        // bounded drain of copies still in flight before the block (and its shared memory) goes away
        for (int k = ci; k < issued; ++k) mbar_wait_bounded(&full[k % STAGES], (uint32_t) (k / STAGES) & 1u, 200000000ull);
    }
}

// ---- weighted combine: out[t][i] = sum over slots in slot order of y[t*k+s][i] * w[t][s] (forward.cpp:308-310)
__global__ void __launch_bounds__(256) combine_kernel(const float * __restrict__ y, const float * __restrict__ w, float * __restrict__ out,
                                                     int n, int k, int T) {
    pdl_wait();
    pdl_launch_dependents();

    const int i4 = blockIdx.x * blockDim.x + threadIdx.x;  // float4 index within a token row
    const int t = blockIdx.y;
    if (i4 * 4 >= n || t >= T) return;
    const float4 * yr = reinterpret_cast<const float4 *>(y + (size_t) t * k * n) + i4;
    const float * wr = w + (size_t) t * k;
    float4 a = yr[0];
    const float w0 = wr[0];
    a.x = __fmul_rn(a.x, w0); a.y = __fmul_rn(a.y, w0); a.z = __fmul_rn(a.z, w0); a.w = __fmul_rn(a.w, w0);
    for (int s = 1; s < k; ++s) {
        const float4 b = yr[(size_t) s * (n / 4)];
        const float ws = wr[s];
        a.x = __fadd_rn(a.x, __fmul_rn(b.x, ws));
        a.y = __fadd_rn(a.y, __fmul_rn(b.y, ws));
        a.z = __fadd_rn(a.z, __fmul_rn(b.z, ws));
        a.w = __fadd_rn(a.w, __fmul_rn(b.w, ws));
    }
    reinterpret_cast<float4 *>(out + (size_t) t * n)[i4] = a;
}

}  // namespace b200moe
