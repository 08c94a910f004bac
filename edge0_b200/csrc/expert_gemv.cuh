// The integer chains of the reference's dot products and the kernel of one or two tokens built on them.
//
// How the reference sums (ggml-cpu/arch/x86/quants.c, AVX2 branches): eight fp32 lanes; lane L collects, block after
// block, fma(scale, (float) p_L, acc_L) where p_L is the integer dot of a fixed group of 4 elements per 32
// (NVFP4: group L of each Q8_0 block; Q3_K: elements 4L..4L+3 of every 32-group of the super-block, scale-weighted and
// summed over the super-block first); the eight lanes are folded at the end as ((a0+a4)+(a2+a6))+((a1+a5)+(a3+a7)).
// Integer partial sums are exact in any order and the fp32 chains run in the reference's, so every dot product is bit-identical to
// the CPU path (and with it every later re-quantisation of activations).
//
// Shared by the integer kernels (this file, expert_gemv_nvfp4.cuh, expert_mma_q3k.cuh, requant_fixup.cuh):
//   DUAL = true : gate and up projections of the same rows + SwiGLU epilogue  -> hidden[row][n_out]
//   DUAL = false: one indexed matmul (ggml MUL_MAT_ID semantics)               -> dst[row][n_out]
// "row" is a routed row: token*n_ids + slot.
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
    const int32_t * ids;  // expert of routed row r at [r / n_ids * ids_stride + r % n_ids] (the kernel of one or two tokens, which needs no groups)
    int64_t ids_stride;
    int allow_empty;      // ids of -1 mark rows that do not exist
    float * out;          // [rows][n_out]
    int n_out;
    int n_ids;
    int ne11;
    int n_as;
    float * comb_out;     // one-or-two-token kernel only, or null: the weighted sum over a token's rows goes here ([tokens][n_out])
    const float * comb_w; // [rows] combine weights
    int * comb_cnt;       // [tokens][n_out / 16] rows of `out` finished so far, cleared by the routing
    int w_stride;         // rows between consecutive experts' matrices: n_out, or 0 when every group uses the same matrix
    int * err;
};

__device__ __forceinline__ uint32_t lds_u32_a2(const uint8_t * p) {  // 2-byte aligned 32-bit load from shared memory
    const uint16_t * h = reinterpret_cast<const uint16_t *>(p);
    return (uint32_t) h[0] | ((uint32_t) h[1] << 16);
}

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

// Integer part of SIMD lane L (0..7) of a super-block: the signed 6-bit sub-block scales times the dots of byte columns 4L..4L+3
// (ggml_vec_dot_q3_K_q8_K, ggml-cpu/arch/x86/quants.c:1766-1880).  blk: 2-byte aligned; acts: the 256 activations of the super-block.
__device__ __forceinline__ int q3k_lane_sum(const uint8_t * __restrict__ blk, int L, const uint32_t * __restrict__ acts) {
    const int hi = L >= 4 ? 1 : 0;
    const uint32_t hm = lds_u32_a2(blk + 4 * L);
    const uint32_t qs0 = lds_u32_a2(blk + 32 + 4 * L);
    const uint32_t qs1 = lds_u32_a2(blk + 64 + 4 * L);
    uint32_t sc[4];
    q3k_unpack_scales(lds_u32_a2(blk + 96), lds_u32_a2(blk + 100), lds_u32_a2(blk + 104), sc);
    int sum = 0;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int bit = 4 * j + s;
            const uint32_t lo2 = ((j ? qs1 : qs0) >> (2 * s)) & 0x03030303u;
            const uint32_t hb4 = bit >= 2 ? ((hm >> (bit - 2)) & 0x04040404u) : ((hm << (2 - bit)) & 0x04040404u);
            // codes 0..7 -> signed -4..3 in every byte without borrows between bytes
            const uint32_t code = (((lo2 | hb4) | 0x80808080u) - 0x04040404u) ^ 0x80808080u;
            sum += q3k_scale_at(sc, 8 * j + 2 * s + hi) * dot4((int) code, (int) acts[8 * bit + L], 0);
        }
    return sum;
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
__device__ __forceinline__ float two_lane_chain_split(const uint8_t * row, int m, const uint8_t * q, const float * d,
                                                      const float * __restrict__ ue_tab) {
    const int sub = m >> 1;
    const uint32_t * qw = reinterpret_cast<const uint32_t *>(q) + 4 * sub + (m & 1);
    uint64_t acc = f32x2(0.0f, 0.0f);
#pragma unroll 8
    for (int b = 0; b < K / 64; ++b) {
        const float2 dy = reinterpret_cast<const float2 *>(d)[b];
        const uint8_t * const blk = row + b * NVFP4_BLOCK_BYTES;
        const uint32_t dw = *reinterpret_cast<const uint32_t *>(blk) >> (8 * sub);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            uint32_t lo, hi;
            nvfp4_word_to_s8(*reinterpret_cast<const uint32_t *>(blk + 4 + 16 * hf + 4 * m), lo, hi);
            const float s = __fmul_rn(ue_tab[(dw >> (16 * hf)) & 0xff], hf ? dy.y : dy.x);
            acc = fma_f32x2(f32x2(s, s), dots_to_f32x2(lo, qw[(2 * b + hf) * 8], hi, qw[(2 * b + hf) * 8 + 2]), acc);
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
__device__ __forceinline__ float lane_chain_warp(const uint8_t * row, int lane, const uint8_t * q,
                                                 const float * d, const float * __restrict__ ue_tab) {
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
// a / b of what is as a rule small: a division of 64 bits is a subroutine
__device__ __forceinline__ long long span_div(long long a, int b) {
    return a >> 32 ? a / b : (long long) ((uint32_t) a / (uint32_t) b);
}
// Boundary i sits at work i / grid of the total; both neighbours compute it the same way, so the spans tile exactly.  cw: prefix over the
// active experts of the work per chunk: FULL for each pass, what is left of it for the last one.  Half of the block looks for either end of
// the span, and the thread that finds its expert works the rest out: a call of a few microseconds waits for three divisions in a row where
// every thread on its own had seven and two more loads (227 rows of 256, Q3_K: 2270 cycles of the kernel's 10,000, so 1880).
template <int THREADS, int PT, int FULL>
__device__ __forceinline__ PassSpan<PT> pass_span(const int * cw, int n_active, int chunks) {
    constexpr int HALF = THREADS / 64 * 32, BATCH = 4;
    __shared__ int s_at[2][3];
    const int end = threadIdx.x >= HALF ? 1 : 0, step = end ? THREADS - HALF : HALF;
    const long long work = n_active ? (long long) cw[n_active] * chunks : 0;
    const long long c = span_div(work * (blockIdx.x + end), gridDim.x);
    if (threadIdx.x < 2) {
        s_at[threadIdx.x][0] = n_active;                     // the end of the list
        s_at[threadIdx.x][1] = s_at[threadIdx.x][2] = 0;
    }
    __syncthreads();
    for (int i0 = threadIdx.x - end * HALF; i0 < n_active; i0 += BATCH * step) {
        int here[BATCH], next[BATCH];
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            const int i = min(i0 + j * step, n_active - 1);
            here[j] = cw[i];
            next[j] = cw[i + 1];
        }
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            const long long left = c - (long long) here[j] * chunks;
            if (i0 + j * step >= n_active || left < 0 || c >= (long long) next[j] * chunks) continue;
            const int ps = (int) span_div(left, FULL * chunks);
            s_at[end][0] = i0 + j * step;
            s_at[end][1] = ps;
            s_at[end][2] = (int) (left - (long long) ps * FULL * chunks) / min(FULL, next[j] - here[j] - FULL * ps);
        }
    }
    __syncthreads();
    return PassSpan<PT>{ s_at[0][0], s_at[0][1], s_at[0][2], s_at[1][0], s_at[1][1], s_at[1][2], chunks };
}

// ---- one or two tokens -------------------------------------------------------------------------------------------------
// The whole call is a few thousand weight rows, so its time is what one row takes: a CTA has 8 features of gate and up (or 32 rows of one
// tensor) for one routed row, reads their expert straight from the ids, and cuts every row's K into SEG segments of a warp each.  All the
// integer work and the products of the scales run at once; only the fp32 chains, a few steps to a segment, go from segment to segment.
//   NVFP4: four threads to a weight row, two SIMD lanes each; Q3_K: a thread per SIMD lane; either way two rows to a thread (gate and up of a
//   feature), which share the activations and the thread's fixed work.
// A chain per thread over the whole K, 16 rows to a four-warp CTA, chunks looked up in the group tables: one token, 2048 -> 768, top-8
// of 128, gate/up and down 12.1 and 9.8 us (Q3_K 9.9 and 8.6), so 10.4 and 8.3 (8.8 and 8.3).  16 features of gate and up to a CTA 11.1, eight
// segments 12.1 (and of K = 4096, whose four leave a thread 255 registers and none spilled: 1024 features, 8 rows 15.3 and 13.8, 2048 27.5 and
// 24.4); a segment's bytes behind a barrier of their own gained nothing.
template <int WT, int K, bool DUAL>
struct FewCfg {
    static constexpr int PAIRS = DUAL ? 8 : 16;               // row pairs of a CTA
    static constexpr int FEAT = DUAL ? PAIRS : 2 * PAIRS;     // its features
    static constexpr int ROW_BYTES = WT == TYPE_NVFP4 ? K / 64 * NVFP4_BLOCK_BYTES : K / 256 * Q3K_BLOCK_BYTES;
    static constexpr int PITCH = WT == TYPE_NVFP4 ? two_lane_pitch(ROW_BYTES) : ROW_BYTES;
    static constexpr int TPR = WT == TYPE_NVFP4 ? 4 : 8;      // threads of a row pair
    static constexpr int GROUPS = PAIRS * TPR / 32;           // warps of a segment
    static constexpr int STEPS = WT == TYPE_NVFP4 ? K / 32 : K / 256;   // of a chain
    static constexpr int SEG = WT == TYPE_NVFP4 ? 4 : STEPS == 8 ? 4 : STEPS;
    static constexpr int U = STEPS / SEG;                     // steps of a segment
    static constexpr int THREADS = GROUPS * SEG * 32;
    static constexpr int ACT_D = WT == TYPE_NVFP4 ? K / 32 : K / 256;
    static constexpr size_t WBYTES = (size_t) 2 * PAIRS * PITCH;
    static constexpr size_t SMEM = WBYTES + K + (ACT_D * 4 + 15) / 16 * 16;
    static_assert(U * SEG == STEPS && (WT != TYPE_NVFP4 || U % 2 == 0), "segments hold whole blocks");
    static_assert(8 * ROW_BYTES % 16 == 0 && WBYTES % 16 == 0, "bulk copies move multiples of 16 bytes");
};

// ue4m3_half_to_f32 of every byte
struct UeTable {
    float v[256];
    constexpr UeTable() : v() {
        for (int x = 0; x < 256; ++x) {
            const int exp = (x >> 3) & 0xf, man = x & 7;
            float f = exp ? 1.0f + man * 0.125f : man * 0.125f;
            for (int e = exp ? exp : 1; e < 8; ++e) f *= 0.5f;          // 2^(exp - 7) / 2
            for (int e = 8; e < exp; ++e) f *= 2.0f;
            v[x] = x == 0 || x == 0x7f ? 0.0f : f;
        }
    }
};
__device__ __align__(16) const UeTable g_ue_table = UeTable();

template <int WT, int K, bool DUAL>
__global__ void __launch_bounds__(FewCfg<WT, K, DUAL>::THREADS) expert_few_rows_kernel(const GemvParams p) {
    using C = FewCfg<WT, K, DUAL>;
    extern __shared__ __align__(128) uint8_t few_smem[];
    uint8_t * const wrows = few_smem;                         // [2 * PAIRS][PITCH]; DUAL: gate rows, then up rows
    uint32_t * const acts = reinterpret_cast<uint32_t *>(few_smem + C::WBYTES);
    float * const act_d = reinterpret_cast<float *>(acts + K / 4);
    __shared__ uint64_t full;
    __shared__ float ue_tab[WT == TYPE_NVFP4 ? 256 : 4];
    __shared__ float s_val[2 * C::PAIRS];
    __shared__ float s_acc[2][2][C::PAIRS][C::TPR];                 // [row of the pair][SIMD lane of the thread][pair][thread]
    __shared__ int s_last;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) { mbar_init(&full, 1); mbar_fence_init(); }
    if (WT == TYPE_NVFP4)
        for (int i = tid; i < 256; i += C::THREADS) ue_tab[i] = g_ue_table.v[i];
    __syncthreads();
    pdl_wait();                 // programmatic dependent launch: everything before this ran alongside the previous kernel's tail
    pdl_launch_dependents();

    const int r = blockIdx.y, f0 = blockIdx.x * C::FEAT, n = min(C::FEAT, p.n_out - f0);
    const int tok = r / p.n_ids, slot = r - tok * p.n_ids;
    const int e = p.ids ? p.ids[(size_t) tok * p.ids_stride + slot] : 0;   // (a dense product has one matrix)
    if (e < 0 || e >= p.n_as) {                               // the whole block; nothing is addressed with it
        if (tid == 0 && !(p.allow_empty && e == -1)) report_error(p.err, DEV_ERR_BAD_EXPERT_ID);
        return;
    }
    const size_t off = ((size_t) e * p.w_stride + f0) * C::ROW_BYTES;
    if (warp == 0) {
        if (lane == 0) mbar_arrive_expect_tx(&full, (uint32_t) (n * C::ROW_BYTES * (DUAL ? 2 : 1)));
        __syncwarp();
        if (C::PITCH == C::ROW_BYTES) {                       // rows stay as they lie
            if (lane == 0) bulk_g2s(wrows, p.w0 + off, n * C::ROW_BYTES, &full);
            if (DUAL && lane == 1) bulk_g2s(wrows + C::PAIRS * C::PITCH, p.w1 + off, n * C::ROW_BYTES, &full);
        } else if (DUAL) {
            const int i = lane % C::PAIRS;
            if (i < n && lane < 2 * C::PAIRS) bulk_g2s(wrows + lane * C::PITCH, (lane < C::PAIRS ? p.w0 : p.w1) + off + (size_t) i * C::ROW_BYTES, C::ROW_BYTES, &full);
        } else if (lane < n) {
            bulk_g2s(wrows + lane * C::PITCH, p.w0 + off + (size_t) lane * C::ROW_BYTES, C::ROW_BYTES, &full);
        }
    }
    // the routed row's activations meanwhile
    const size_t arow = (size_t) tok * p.ne11 + slot % p.ne11;
    if (WT == TYPE_NVFP4 && p.act_f32) {
        // Q8_0 on the fly, the arithmetic of quantize_q8_0_block: 8 lanes hold one block of 32 (4 values each)
        const float4 * src = reinterpret_cast<const float4 *>(p.act_f32 + arow * K);
        for (int i0 = 0; i0 < K / 4; i0 += C::THREADS) {
            const int i = i0 + tid;
            const bool in = i < K / 4;
            const float4 v = in ? src[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
            const float id = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
            if (in) {
                acts[i] = ((uint32_t) __float2int_rn(__fmul_rn(v.x, id)) & 0xffu) | (((uint32_t) __float2int_rn(__fmul_rn(v.y, id)) & 0xffu) << 8) |
                          (((uint32_t) __float2int_rn(__fmul_rn(v.z, id)) & 0xffu) << 16) | (((uint32_t) __float2int_rn(__fmul_rn(v.w, id)) & 0xffu) << 24);
                if ((i & 7) == 0) act_d[i >> 3] = __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
            }
        }
    } else if (WT == TYPE_Q3_K && p.act_f32) {
        for (int b = warp; b < K / 256; b += C::THREADS / 32) {               // a warp quantises one 256-block
            uint32_t q[2] = { 0u, 0u };
            float d = 0.0f;
            q8_K_words(p.act_f32 + arow * K + b * 256 + lane * 8, lane, q, d);
            acts[b * 64 + lane * 2] = q[0];
            acts[b * 64 + lane * 2 + 1] = q[1];
            if (lane == 0) act_d[b] = d;
        }
    } else {
        const uint4 * src = reinterpret_cast<const uint4 *>(p.act.q + arow * K);
        for (int i = tid; i < K / 16; i += C::THREADS) reinterpret_cast<uint4 *>(acts)[i] = src[i];
        for (int i = tid; i < C::ACT_D; i += C::THREADS) act_d[i] = p.act.d[arow * C::ACT_D + i];
    }
    const float sc0 = p.scale0 ? p.scale0[p.w_stride ? e : 0] : 1.0f, sc1 = DUAL && p.scale1 ? p.scale1[p.w_stride ? e : 0] : 1.0f;
    const bool landed = mbar_wait_bounded(&full, 0);
    if (!landed) report_error(p.err, DEV_ERR_BARRIER_TIMEOUT);
    if (__syncthreads_or(!landed)) {                          // bounded drain before the block (and its shared memory) goes away
        if (tid == 0) mbar_wait_bounded(&full, 0, 200000000ull);
        __syncthreads();
        return;
    }

    const int seg = warp / C::GROUPS, pair = (warp % C::GROUPS) * (32 / C::TPR) + lane / C::TPR, m = lane % C::TPR;
    const uint8_t * wrow[2];                                  // where the segment's bytes of the pair lie
#pragma unroll
    for (int r = 0; r < 2; ++r)
        wrow[r] = wrows + (pair + r * C::PAIRS) * C::PITCH + (WT == TYPE_NVFP4 ? C::U / 2 * NVFP4_BLOCK_BYTES : C::U * Q3K_BLOCK_BYTES) * seg;
    if constexpr (WT == TYPE_NVFP4) {
        float s[2][C::U];
        uint64_t dots[2][C::U];
        const uint32_t * aw = acts + seg * C::U * 8 + 4 * (m >> 1) + (m & 1);
#pragma unroll
        for (int b = 0; b < C::U / 2; ++b) {
            const int at = b * NVFP4_BLOCK_BYTES;
            const float2 d = *reinterpret_cast<const float2 *>(act_d + seg * C::U + 2 * b);
            uint32_t dw[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) dw[r] = *reinterpret_cast<const uint32_t *>(wrow[r] + at) >> (8 * (m >> 1));
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int u = 2 * b + hf;
                const uint32_t alo = aw[u * 8], ahi = aw[u * 8 + 2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    uint32_t lo, hi;
                    nvfp4_word_to_s8(*reinterpret_cast<const uint32_t *>(wrow[r] + at + 4 + 16 * hf + 4 * m), lo, hi);
                    s[r][u] = __fmul_rn(ue_tab[(dw[r] >> (16 * hf)) & 0xff], hf ? d.y : d.x);
                    dots[r][u] = dots_to_f32x2(lo, alo, hi, ahi);
                }
            }
        }
#pragma unroll 1
        for (int g = 0; g < C::SEG; ++g) {
            if (seg == g) {
                uint64_t acc[2] = { f32x2(0.0f, 0.0f), f32x2(0.0f, 0.0f) };
                if (g > 0) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) acc[r] = f32x2(s_acc[r][0][pair][m], s_acc[r][1][pair][m]);
                }
#pragma unroll
                for (int u = 0; u < C::U; ++u)
#pragma unroll
                    for (int r = 0; r < 2; ++r) acc[r] = fma_f32x2(f32x2(s[r][u], s[r][u]), dots[r][u], acc[r]);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 a = f32x2_halves(acc[r]);
                    if (g < C::SEG - 1) {
                        s_acc[r][0][pair][m] = a.x;
                        s_acc[r][1][pair][m] = a.y;
                    } else {
                        const float v = hsum_two_lanes(a.x, a.y);
                        if (m == 0) s_val[pair + C::PAIRS * r] = v;
                    }
                }
            }
            __syncthreads();
        }
    } else {
        float s[2][C::U], sums[2][C::U];
#pragma unroll
        for (int u = 0; u < C::U; ++u) {
            const int sb = seg * C::U + u;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint8_t * blk = wrow[r] + u * Q3K_BLOCK_BYTES;
                sums[r][u] = small_int_to_float(q3k_lane_sum(blk, m, acts + sb * 64));
                s[r][u] = __fmul_rn(act_d[sb], __half2float(*reinterpret_cast<const __half *>(blk + 108)));
            }
        }
#pragma unroll 1
        for (int g = 0; g < C::SEG; ++g) {
            if (seg == g) {
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float acc = g > 0 ? s_acc[r][0][pair][m] : 0.0f;
#pragma unroll
                    for (int u = 0; u < C::U; ++u) acc = __fmaf_rn(s[r][u], sums[r][u], acc);
                    if (g < C::SEG - 1) {
                        s_acc[r][0][pair][m] = acc;
                    } else {                                  // hsum_float_8: (a4+a0, a5+a1, a6+a2, a7+a3) -> (r0+r2, r1+r3) -> s0+s1
                        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 4));
                        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 2));
                        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 1));
                        if (m == 0) s_val[pair + C::PAIRS * r] = acc;
                    }
                }
            }
            __syncthreads();
        }
    }
    if (tid < n) {
        float v = __fmul_rn(s_val[tid], sc0);
        if (DUAL) v = __fmul_rn(ggml_silu(v), __fmul_rn(s_val[C::PAIRS + tid], sc1));
        p.out[(size_t) r * p.n_out + f0 + tid] = v;
    }
    if (!DUAL && p.comb_out) {
        // The CTA that finishes the last of a token's rows sums them - in slot order, so which CTA that is does not show - and saves the
        // combine its launch.
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(&p.comb_cnt[tok * (p.n_out / 16) + blockIdx.x], 1) == p.n_ids - 1;
        __syncthreads();
        if (s_last && tid < n) {
            __threadfence();
            const float * wr = p.comb_w + (size_t) tok * p.n_ids;
            const float * y = p.out + (size_t) tok * p.n_ids * p.n_out + f0 + tid;
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
            p.comb_out[(size_t) tok * p.n_out + f0 + tid] = a;
        }
    }
}

// ---- weighted combine: out[t][i] = sum over slots in slot order of y[t*k+s][i] * w[t][s] (forward.cpp:308-310)
__global__ void __launch_bounds__(256) combine_kernel(const float * y, const float * w, float * __restrict__ out,
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
