// Grouped expert GEMM on the block-scaled FP4 tensor-core instruction (tcgen05.mma kind::mxf4nvf4, one UE4M3 scale per 16
// elements, fp32 accumulators in tensor memory) for NVFP4 experts in batched decode and prefill.
//
// Why it fits: ggml's block_nvfp4 IS the operand format of that instruction - E2M1 codes, one UE4M3 scale per 16 elements
// (ggml-common.h:221-227; the doubled code table and the halved scale decode of ggml-impl.h:514-527 cancel).  A weight row
// needs no arithmetic at all before the MMA: the 4 scale bytes in front of every 32 code bytes are stripped while the row moves
// from the raw TMA stage into the 128B-swizzled K-major operand tile, and go to tensor memory as the instruction's scale
// factors.  Element order inside a 16-block does not matter as long as both operands agree on it, so the
// activations are simply stored in ggml's nibble order (byte j = elements j and j+8 of the block).
//
// Activations stay on the reference's int8 grid (q * d with d an fp16 number per 32 elements, the Q8_0 rows the CPU path
// multiplies with).  With d = M * 2^e (M an 11-bit integer) the product q * M is an integer of at most 127 * 2047 = 259969; its six balanced
// radix-9 digits (each in [-4, 4], all E2M1 values; six reach 265720) are six "planes" of one routed row, and 2^e - relative to the row's
// largest block exponent - is a power of two that UE4M3 holds exactly.  So
//     x_hat[k] = 2^(E_row - 8) * sum_p 9^p * digit_p[k] * sf[k / 16]
// is exact (blocks more than 17 binades below the row's largest flush to zero: a relative 2^-17 of the row's unit), every
// product inside the tensor core is exact, and the result differs from the integer path only by fp32 accumulation.
//
// Operand roles: D[feature, plane] = W[feature, k] * P[plane, k].  M = 128 weight rows, N = 6 planes x up to 14 routed rows
// (N = 8 .. 88; prefill: up to 27 rows, N = 168), K = 64 per instruction.  The six plane columns of a routed row sit next to each other in
// one lane of tensor memory, so the epilogue recombines them with a Horner chain in registers and stores 32 consecutive features per warp.
// Two weight tiles are in flight per stage with an accumulator each (gate and up rows of the same 128 features, or two
// consecutive 128-row tiles of `down`): dependent MMAs on one accumulator issue every ~190-230 cycles, MMAs that alternate
// between two accumulators every ~116 (measured with the probe kernel in fp4_probe.cuh).
//
// Roles (every wait bounded, as in expert_gemm.cuh):
//   warp 0       raw-weight producer: tiled TMA of [128 rows][144 bytes] boxes (K = 256 per row) of both tiles
//   warp 1       activation producer: tiled TMA boxes of the plane rows (128 bytes each) of four routed rows + one bulk copy of the rows'
//                scales, into a ring of its own that runs three stages ahead (the planes come from L2 with about a microsecond of latency)
//   warp 2       MMA issuer: two tcgen05.mma per K = 64 step
//   warp 3       owns tensor memory
//   warps 4-7, 20-23  epilogue
//   warps 8-15   repack: thread = one weight row of one tile; 9 x 16-byte loads, 8 x 16-byte stores, the row's scale words set aside
//   warps 16-19  scale factors: from shared memory through registers into tensor memory (tcgen05.st)
// The scales go through registers because a tcgen05.cp holds its issuing thread ~80 cycles: twelve per stage in front of the MMAs cost
// 15-20 % of the kernel, and from a thread of their own an instruction now and then read a scale that was not in place.  The exchange
// between rows and lanes and the waits of tcgen05.st have warps of their own because the repack warps' chain is the longest of a stage: with
// both in the repack warps gate/up of 64 tokens over 512 experts (1024 -> 1024) took 107 us, like this 98; sixteen repack warps
// that take the stages in turn gained nothing more and cost the prefill tile its registers (4096 tokens: 481 -> 685 us).
// 24 warps leave a thread 80 registers (see the register split in the kernel).  What a stage takes is the hand-over between the roles: repack,
// scale factors and MMAs each keep busy for some 1,150 cycles of its 1,500 to 2,200.  One weight tile against two token tiles in a stage
// (half the weight bytes through shared memory) took as long to a stage and twice as many of them below 27 rows an expert; scale words
// through a buffer of their own or warps of their own for either operand's scales gained nothing or lost.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "expert_gemm.cuh"
#include "expert_mma.cuh"
#include "formats.cuh"

namespace b200moe {

constexpr int FP4_PLANES = 6;
// Routed rows per token tile: 14 for few rows per expert (two accumulator buffers, so the epilogue runs beside the next unit), 27 for
// more (N = 168, one buffer; a weight tile is repacked and fetched half as often per routed row).
constexpr int FP4_RPT_SMALL = TOKEN_TILE_SMALL, FP4_RPT_LARGE = TOKEN_TILE_LARGE;
constexpr int FP4_THREADS = 768;

__device__ __forceinline__ void umma_fp4(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                         bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %7, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], da, db, %4, [%5], [%6], p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(sfa), "r"(sfb), "r"((uint32_t) accumulate)
        : "memory");
}
// shared memory -> tensor memory: 32 rows x 16 bytes, replicated to the four lane quarters (the layout the MMA reads scales from)
__device__ __forceinline__ void tmem_cp_sf(uint32_t taddr, uint32_t smem_addr) {
    // matrix descriptor without swizzle: 8-row groups of 16-byte rows, 128 bytes apart
    const uint64_t desc = (uint64_t) ((smem_addr >> 4) & 0x3fff) | ((uint64_t) (128 >> 4) << 32) | ((uint64_t) 1 << 46);
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
// tensor memory <- registers: thread i of the warp writes N consecutive 32-bit columns of lane (its quarter's base + i)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint4 (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0].x),
                 "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w), "r"(v[2].x), "r"(v[2].y), "r"(v[2].z),
                 "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// instruction descriptor: E2M1 x E2M1, UE4M3 scales, both operands K-major, M = 128, N = n (a multiple of 8)
__host__ __device__ constexpr uint32_t umma_idesc_fp4(int n) { return (1u << 7) | (1u << 10) | ((uint32_t) (n >> 3) << 17) | ((128u >> 4) << 24); }
// byte offset of the 4 scale bytes of row r (0..127) inside the 512-byte scale tile of one K = 64 step
__host__ __device__ constexpr uint32_t sf_tile_offset(int r) { return (uint32_t) ((r & 31) * 16 + (r >> 5) * 4); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- activation planes ---------------------------------------------------------------------------------------------------
// Expert-sorted routed row i -> six plane rows 6i .. 6i+5 of `planes` (K/2 bytes each, ggml nibble order inside every
// 16-block), its scale bytes, which its planes have in common, and the power of two the epilogue multiplies with.
struct PlaneOut {
    uint8_t * planes;       // [rows * 6][K / 2]
    uint8_t * sf;           // [K / 256][rows][16]: scale of every 16-block
    float *   row_scale;    // [rows] by sorted position
    int4 *    tiles;        // [tiles] of every token tile: expert, first sorted row, routed rows
    int       rpt;          // routed rows per token tile
    int       rows;
};

// E2M1 codes of the balanced radix-9 digits of 0 .. 728, less four each: lowest digit in byte 0, highest in byte 2
__device__ __forceinline__ uint32_t digit_codes(int v) {
    uint32_t w = 0;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const int d = v % 9 - 4;
        v /= 9;
        w |= (((0x65420u >> (4 * abs(d))) & 0xfu) | (d < 0 ? 8u : 0u)) << (8 * p);
    }
    return w;
}

// K / 16 threads per ACTIVATION row, a thread for a 16-block (a block of threads holds 256 * 16 / K rows).  The digits of a row are worked
// out once and stored for each of the n_ids / ne11 routed rows that read it (gate/up: the k experts of a token).
// SRC_F32 = false: the row's activations are already quantised (ActQuant planes, Q8_0).
// SRC_F32 = true: they are fp32 (`src`, rows `src_stride` floats apart) and are quantised here exactly as quantize_q8_0_block
// does it (d = half(amax / 127), q = rint(v * (127 / amax))), which saves the separate quantisation pass; `emit`, when it has
// planes, receives that quantised form as well (row index as in `src`).
// Three digits at a time come from a table, a byte each, so eight of them merge into a word of one plane by byte permutes: some 10 instructions
// a value where dividing out digit by digit took 40.  Bound by the stores: 3 bytes per routed value, 8 of them at a time.
// 4096 tokens top-8, K = 2048: 94 us with seven planes, scales per plane and digits one by one, so 39; fp32 rows of K = 768: 104 us, so 48.
template <bool SRC_F32>
__global__ void __launch_bounds__(256) act_planes_kernel(ActQuant act, const float * src, int64_t src_stride,
                                                        const int * pos, const int32_t * ids,
                                                        const int * offsets, const int * tile_of_expert,
                                                        int act_rows, int K, int n_ids, int ne11, int n_as, PlaneOut out, ActQuant emit) {
    constexpr int MAX_ROWS = 16;             // K = 256
    __shared__ uint32_t s_digits[729];
    __shared__ int s_E[MAX_ROWS];
    __shared__ int s_at[MAX_ROWS][32];       // sorted position of every routed row of a block row
    const int tid = threadIdx.x, lane = tid & 31;
    const int tpr = K / 16, rpb = 256 / tpr;
    const int lrow = tid / tpr, g = tid % tpr;
    const int arow = blockIdx.x * rpb + lrow;
    const int n_dst = n_ids / ne11;
    const int dst_step = gridDim.y, dst0 = blockIdx.y;    // few rows: the blocks of a column store every dst_step-th routed row each
    for (int i = tid; i < 729; i += 256) s_digits[i] = digit_codes(i);
    if (tid < MAX_ROWS) s_E[tid] = -1000;
    pdl_wait();                              // the table is made while the previous kernel ends
    pdl_launch_dependents();
    const bool live = lrow < rpb && arow < act_rows;   // threads beyond the block's last whole row idle (K = 768)
    for (int j = g; live && j < n_dst; j += tpr) {
        const int r = (arow / ne11) * n_ids + arow % ne11 + ne11 * j;
        const int e = ids[r];
        int at = -1;                                   // an id of -1 is an empty slot; other bad ids were reported by the grouping kernels
        if (e >= 0 && e < n_as) {
            const int in_e = pos[r];
            at = offsets[e] + in_e;
            if (in_e % out.rpt == 0) out.tiles[tile_of_expert[e] + in_e / out.rpt] = make_int4(e, at, min(out.rpt, offsets[e + 1] - at), 0);
        }
        s_at[lrow][j] = at;
    }
    // the block's values in order and its scale's bits
    int v[16];
    uint32_t dbits = 0;
    if (SRC_F32) {
        float x[16];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const float4 f = live ? reinterpret_cast<const float4 *>(src + (size_t) arow * src_stride + 16 * g)[m] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            x[4 * m] = f.x; x[4 * m + 1] = f.y; x[4 * m + 2] = f.z; x[4 * m + 3] = f.w;
        }
        float amax = fabsf(x[0]);                      // NaN only for a block of nothing else
#pragma unroll
        for (int m = 1; m < 16; ++m) amax = fmaxf(amax, fabsf(x[m]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));   // the 32-block's other half: the neighbour (an even number of threads to a row)
        const float d = __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
        const float id = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = __float2int_rn(__fmul_rn(x[m], id));
        dbits = __float_as_uint(d);
        if (emit.q && blockIdx.y == 0 && live) {
            uint32_t w[4];
#pragma unroll
            for (int m = 0; m < 4; ++m)
                w[m] = (uint32_t) (v[4 * m] & 0xff) | ((uint32_t) (v[4 * m + 1] & 0xff) << 8) | ((uint32_t) (v[4 * m + 2] & 0xff) << 16) |
                       ((uint32_t) (v[4 * m + 3] & 0xff) << 24);
            *reinterpret_cast<uint4 *>(emit.q + (size_t) arow * K + 16 * g) = make_uint4(w[0], w[1], w[2], w[3]);
            if ((g & 1) == 0) emit.d[(size_t) arow * (K / 32) + (g >> 1)] = d;
        }
    } else {
        const uint4 f = live ? *reinterpret_cast<const uint4 *>(act.q + (size_t) arow * K + 16 * g) : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t w[4] = { f.x, f.y, f.z, f.w };
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = (int) (int8_t) (w[m >> 2] >> (8 * (m & 3)));
        if (live) dbits = __float_as_uint(act.d[(size_t) arow * (K / 32) + (g >> 1)]);
    }
    // d is an fp16 number: d = M * 2^(exp8 - 137) with M the top 11 bits of the significand
    const bool nz = (dbits & 0x7fffffffu) != 0;
    const int e8 = nz && live ? (int) ((dbits >> 23) & 0xff) - 137 : -1000;
    __syncthreads();
    // the row's largest exponent; sixteen threads never belong to two rows
    const int emax = __reduce_max_sync(0xffffu << (lane & 16), e8);
    if ((lane & 15) == 0 && live) atomicMax(&s_E[lrow], emax);
    __syncthreads();
    if (!live) return;
    const int E_row = s_E[lrow];
    for (int j = g; j < n_dst; j += tpr)
        if (s_at[lrow][j] >= 0)
            // 2^(E_row - 8): far from the fp32 limits.  A block scale that is infinite or NaN has no digits: the row's results are NaN, which is
            // what 0 * inf makes of them on the other engines (and in the reference).
            out.row_scale[s_at[lrow][j]] = E_row == 255 - 137 ? __uint_as_float(0x7fc00000u) : E_row > -1000 ? __uint_as_float((uint32_t) (E_row - 8 + 127) << 23) : 0.0f;
    const int s = nz ? e8 - E_row + 8 : -100;                                           // scale exponent, at most 8
    const int M = s >= -9 ? (int) (((dbits & 0x7fffffu) | 0x800000u) >> 13) : 0;        // flushed blocks contribute nothing
    // the scale's UE4M3 byte: normal for s >= -6, the three power-of-two subnormals below, zero when flushed
    const uint8_t sb = (uint8_t) (s >= -6 ? (uint32_t) (s + 7) << 3 : s == -7 ? 4u : s == -8 ? 2u : s == -9 ? 1u : 0u);
    // digits: elements m and m + 8 of the block share byte m, low and high nibble.  An out-of-range v (a block of infinities) must not leave
    // the table: its row is NaN whatever its digits are.
    uint32_t words[FP4_PLANES][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t lo3[4], hi3[4];                       // bytes: planes 0 .. 2 and 3 .. 5 of byte 4h + m
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            uint32_t c[2][2];
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const uint32_t u = min((uint32_t) (v[4 * h + m + 8 * n] * M + 265720), 531440u);
                const uint32_t up = u / 729u;
                c[n][0] = s_digits[u - up * 729u];
                c[n][1] = s_digits[up];
            }
            lo3[m] = c[0][0] | (c[1][0] << 4);
            hi3[m] = c[0][1] | (c[1][1] << 4);
        }
        auto planes3 = [&](const uint32_t (&t)[4], int p) {
            const uint32_t a = __byte_perm(t[0], t[1], 0x5140), b = __byte_perm(t[2], t[3], 0x5140);
            words[p][h] = __byte_perm(a, b, 0x5410);
            words[p + 1][h] = __byte_perm(a, b, 0x7632);
            words[p + 2][h] = __byte_perm(__byte_perm(t[0], t[1], 0x0062), __byte_perm(t[2], t[3], 0x0062), 0x5410);
        };
        planes3(lo3, 0);
        planes3(hi3, 3);
    }
    for (int j = dst0; j < n_dst; j += dst_step) {
        const int at = s_at[lrow][j];
        if (at < 0) continue;
        uint2 * pw = reinterpret_cast<uint2 *>(out.planes + (size_t) at * FP4_PLANES * (K / 2)) + g;
#pragma unroll
        for (int p = 0; p < FP4_PLANES; ++p) pw[(size_t) p * (K / 16)] = make_uint2(words[p][0], words[p][1]);
        out.sf[((size_t) (g >> 4) * out.rows + at) * 16 + (g & 15)] = sb;
    }
}

// Development builds (-DB200MOE_FP4_PROF) record, per CTA, the cycles each role spends waiting on each of its barriers.
#ifdef B200MOE_FP4_PROF
#define FP4_PROF_T0() const long long prof_t0_ = clock64()
#define FP4_PROF_ADD(slot) prof_[slot] += clock64() - prof_t0_
#define FP4_PROF_DECL() long long prof_[4] = {0, 0, 0, 0}; const long long prof_beg_ = clock64()
#define FP4_PROF_STORE(base, n) do { if (p.prof) { for (int i_ = 0; i_ < n; ++i_) p.prof[blockIdx.x * 24 + base + i_] = prof_[i_]; p.prof[blockIdx.x * 24 + base + n] = clock64() - prof_beg_; } } while (0)
#else
#define FP4_PROF_T0()
#define FP4_PROF_ADD(slot)
#define FP4_PROF_DECL()
#define FP4_PROF_STORE(base, n)
#endif

struct Fp4Params {
    const float * scale0;   // per-expert fp32 scale of tile 0's tensor (or null)
    const float * scale1;
    const uint8_t * sf;     // activation scales [K / 256][sf_rows][16]
    const float * row_scale;
    const int * perm;       // [rows]
    const int * tile_of_expert;   // [n_as + 1]: first token tile of every expert, total number of tiles at the end
    const int4 * tiles;           // [tiles]: see PlaneOut
    float * out;            // [rows][n_out] indexed by routed row
    int n_out;
    int n_as;
    int sf_rows;
    int * err;
    long long * prof;       // development builds only
};

template <int K, int RPT>
struct Fp4Cfg {
    static constexpr bool LARGE = RPT == FP4_RPT_LARGE;
    static constexpr int NROW = FP4_PLANES * RPT;                    // plane rows of a token tile (84, 162)
    static constexpr int NCOL = (NROW + 7) / 8 * 8;                  // accumulator columns per weight tile: N of the instruction is a multiple of 8
    static constexpr int NACC = LARGE ? 1 : 2;                        // accumulator buffers
    static constexpr int NBLK = (NROW + 127) / 128;                  // blocks of 128 plane rows in the scale factors
    static constexpr int A_TILE = 128 * 128;                         // 128 weight rows x 256 K as fp4
    // Routed rows whose planes one tiled copy brings: four (24 x 128 bytes, whole swizzle atoms) where a tile holds few of its rows, all of
    // them where it is mostly full (seven boxes to a stage instead of one: gate/up of 4096 tokens 433 us and 511).
    static constexpr int BOX_ROWS = LARGE ? RPT : 4;
    static constexpr int BOX_BYTES = BOX_ROWS * FP4_PLANES * 128;
    static constexpr int B_TILE = ((RPT + BOX_ROWS - 1) / BOX_ROWS * BOX_BYTES + 1023) / 1024 * 1024;   // (rows beyond the tile's are read by the instruction: columns nobody uses)
    static constexpr int SFB = 1024;                                 // room for the rows' scales, 16 bytes each
    static constexpr int STAGE = 2 * A_TILE;                         // repacked weights of both tiles
    static constexpr int ACT_STAGE = B_TILE + SFB;                   // digit planes, then their scales
    static constexpr int RAW_STAGE = 256 * GEMM_RAW_ROW;
    static constexpr int RS = LARGE ? 2 : 3, TS = 2;
    static constexpr int AS = 3;                                      // plane tiles come from L2 with ~1 us latency: fetched three stages ahead
    static constexpr uint32_t TMEM_COLS = 512;                        // NACC buffers x 2 accumulators, then two sets of scale factors
    static constexpr uint32_t SF_COL = NACC * 2 * NCOL;
    static constexpr uint32_t SF_SET = 32 + 16 * NBLK;                // [tile 0][tile 1][planes]: 4 columns per K = 64 step and 128 rows
    static_assert(SF_COL + TS * SF_SET <= TMEM_COLS, "accumulators and one scale-factor set per operand stage fit tensor memory");
    static_assert(NCOL * 128 <= B_TILE && RPT * 16 <= SFB, "operand rows and scales fit their room");
    static_assert(BOX_ROWS == RPT || BOX_BYTES % 1024 == 0, "boxes start on a swizzle atom");
    static_assert(STAGE % 1024 == 0 && ACT_STAGE % 1024 == 0, "stages keep the 1024-byte alignment of swizzled tiles");
    static_assert(K % GEMM_RAW_K == 0, "K must be a multiple of 256");
    static constexpr size_t SMEM = (size_t) TS * STAGE + (size_t) AS * ACT_STAGE + (size_t) RS * RAW_STAGE + 1024;
};
// DUAL: tile 0 = gate rows f .. f+127, tile 1 = up rows of the same features; epilogue = SwiGLU; 128 features per item.
// single: tiles 0 and 1 = 256 consecutive rows of the one tensor; 256 features per item.
template <int K, bool DUAL, int RPT>
__global__ void __launch_bounds__(FP4_THREADS, 1)
expert_gemm_fp4_kernel(const Fp4Params p, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1,
                       const __grid_constant__ CUtensorMap map_planes) {
    using C = Fp4Cfg<K, RPT>;
    constexpr int TS = C::TS, RS = C::RS, AS = C::AS, NACC = C::NACC;
    constexpr int KC = K / GEMM_RAW_K;
    constexpr int FEAT = DUAL ? 128 : 256;

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t * tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    uint8_t * acts = tiles + (size_t) TS * C::STAGE;
    uint8_t * raws = acts + (size_t) AS * C::ACT_STAGE;
    __shared__ uint64_t raw_full[RS], raw_empty[RS], tile_full[TS], tile_empty[TS], act_full[AS], act_empty[AS], acc_full[NACC], acc_empty[NACC], sf_ready[RS];
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < RS; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4); mbar_init(&sf_ready[i], 8); }
        for (int i = 0; i < TS; ++i) { mbar_init(&tile_full[i], 256 + 4); mbar_init(&tile_empty[i], 1); }
        for (int i = 0; i < AS; ++i) { mbar_init(&act_full[i], 1); mbar_init(&act_empty[i], 1); }
        for (int i = 0; i < NACC; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        mbar_fence_init();
        s_abort = 0;
    }
    if (warp == 3) {
        tmem_alloc(&s_tmem, C::TMEM_COLS);
        tmem_relinquish();
    }
    if (tid == 32) {   // the first use of a tensor map otherwise pays for its fetch
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w0) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w1) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_planes) : "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    // Work unit = (token tile of an expert, feature tile): every role walks the same units, blockIdx.x, blockIdx.x + gridDim.x, ...
    // Feature tiles of one token tile are neighbours in that order, so they find the tile's planes in L2; token tiles of one
    // expert follow each other, so a second pass over an expert's weights comes from L2 as well.
    const int f_tiles = p.n_out / FEAT;
    const int n_units = p.tile_of_expert[p.n_as] * f_tiles;
    struct Unit { int e, ft, row0, nt; };
    auto unit_at = [&](int u) {
        const int tile = u / f_tiles;
        const int4 t = __ldg(p.tiles + tile);
        return Unit{ t.x, u - tile * f_tiles, t.y, t.z };
    };
    const int my_stages = n_units > (int) blockIdx.x ? (n_units - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x * KC : 0;
    // weight stage: [A0][A1]; activation stage: [B][SFB]
    constexpr uint32_t OFF_A1 = C::A_TILE, OFF_SFB = C::B_TILE;
    // 768 threads leave 80 registers to a thread.  With the small tile producers and issuer give theirs to the epilogue, which spilled without (4 to 8 bytes are left)
    // (40 + 2 x 104 + 3 x 72 = 464 of the launch's 480 per 128 threads; 64 tokens over 128 experts: gate/up 51.7 us, so 49.9, down 29.4 and 27.0).
    // The large one loses with it (4096 tokens, down: 244 us, 283 so); what kept a short K from spilling there is that the loops over
    // K = 256 pieces stay loops (K = 512, 1024 tokens x 32768 features: 111 us unrolled, so 98).
    if (warp < 4) {
        if constexpr (!C::LARGE) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ raw weight producer
            Ring raw;
            FP4_PROF_DECL();
            for (int u = blockIdx.x; u < n_units && !s_abort; u += gridDim.x) {
                const Unit w = unit_at(u);
                const int row0 = w.e * p.n_out + w.ft * FEAT;
#pragma unroll 1
                for (int kc = 0; kc < KC; ++kc) {
                    FP4_PROF_T0();
                    if (!wait_or_abort<40>(&raw_empty[raw.stage], raw.phase ^ 1u, &s_abort, p.err)) break;
                    FP4_PROF_ADD(0);
                    uint8_t * dst = raws + (size_t) raw.stage * C::RAW_STAGE;
                    mbar_arrive_expect_tx(&raw_full[raw.stage], C::RAW_STAGE);
                    tma_load_2d(dst, &map_w0, kc * GEMM_RAW_ROW, row0, &raw_full[raw.stage]);
                    if (DUAL) tma_load_2d(dst + 128 * GEMM_RAW_ROW, &map_w1, kc * GEMM_RAW_ROW, row0, &raw_full[raw.stage]);
                    else tma_load_2d(dst + 128 * GEMM_RAW_ROW, &map_w0, kc * GEMM_RAW_ROW, row0 + 128, &raw_full[raw.stage]);
                    raw.template advance<RS>();
                }
            }
            FP4_PROF_STORE(0, 1);
        } else if (warp == 1 && lane == 0) {
            // ------------------------------------------------------------ activation producer
            Ring act;
            FP4_PROF_DECL();
            for (int u = blockIdx.x; u < n_units && !s_abort; u += gridDim.x) {
                const Unit w = unit_at(u);
                const uint8_t * sfr = p.sf + (size_t) w.row0 * 16;
                const int boxes = (w.nt + C::BOX_ROWS - 1) / C::BOX_ROWS;
#pragma unroll 1
                for (int kc = 0; kc < KC; ++kc) {
                    FP4_PROF_T0();
                    if (!wait_or_abort<40>(&act_empty[act.stage], act.phase ^ 1u, &s_abort, p.err)) break;
                    FP4_PROF_ADD(0);
                    uint8_t * st = acts + (size_t) act.stage * C::ACT_STAGE;
                    mbar_arrive_expect_tx(&act_full[act.stage], (uint32_t) (boxes * C::BOX_BYTES + w.nt * 16));
                    for (int b = 0; b < boxes; ++b)
                        tma_load_2d(st + b * C::BOX_BYTES, &map_planes, kc * 128, FP4_PLANES * (w.row0 + C::BOX_ROWS * b), &act_full[act.stage]);
                    bulk_g2s(st + OFF_SFB, sfr + (size_t) kc * p.sf_rows * 16, (uint32_t) w.nt * 16, &act_full[act.stage]);
                    act.template advance<AS>();
                }
            }
            FP4_PROF_STORE(2, 1);
        } else if (warp == 2 && lane == 0) {
            // ------------------------------------------------------------ MMA issuer
            Ring tile, act, acc;
            FP4_PROF_DECL();
            for (int u = blockIdx.x; u < n_units && !s_abort; u += gridDim.x) {
                const uint32_t idesc = umma_idesc_fp4((FP4_PLANES * unit_at(u).nt + 7) & ~7);
                {
                    FP4_PROF_T0();
                    if (!wait_or_abort<40>(&acc_empty[acc.stage], acc.phase ^ 1u, &s_abort, p.err)) break;
                    FP4_PROF_ADD(0);
                }
                tc_fence_after();
                const uint32_t d0 = tmem + (uint32_t) acc.stage * (2 * C::NCOL), d1 = d0 + C::NCOL;
                bool ok = true;
#pragma unroll 1
                for (int kc = 0; kc < KC; ++kc) {
                    {
                        FP4_PROF_T0();
                        if (!(ok = wait_or_abort<20>(&act_full[act.stage], act.phase, &s_abort, p.err))) break;
                        FP4_PROF_ADD(1);
                    }
                    {
                        FP4_PROF_T0();
                        if (!(ok = wait_or_abort<20>(&tile_full[tile.stage], tile.phase, &s_abort, p.err))) break;
                        FP4_PROF_ADD(2);
                    }
                    tc_fence_after();
                    const uint32_t sbase = smem_u32(tiles + (size_t) tile.stage * C::STAGE);
                    const uint32_t abase = smem_u32(acts + (size_t) act.stage * C::ACT_STAGE);
                    const uint32_t da = DESC_LO | (sbase >> 4), db = DESC_LO | (abase >> 4);
                    const uint32_t sf_set = tmem + C::SF_COL + C::SF_SET * (uint32_t) tile.stage;   // [tile 0][tile 1][planes]
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {   // 4 x K64 = 256; 32 bytes (2 units) further along the 128-byte row each
                        const uint32_t t_sfa0 = sf_set + 4 * kk, t_sfa1 = t_sfa0 + 16, t_sfb = sf_set + 32 + 4 * C::NBLK * kk;
                        const bool accum = kc != 0 || kk != 0;
                        umma_fp4(d0, da + 2 * kk, db + 2 * kk, DESC_HI, idesc, t_sfa0, t_sfb, accum);
                        umma_fp4(d1, da + (OFF_A1 >> 4) + 2 * kk, db + 2 * kk, DESC_HI, idesc, t_sfa1, t_sfb, accum);
                    }
                    umma_commit(&tile_empty[tile.stage]);   // frees both operand stages when these MMAs have read them
                    umma_commit(&act_empty[act.stage]);
                    tile.template advance<TS>();
                    act.template advance<AS>();
                }
                if (!ok) break;
                umma_commit(&acc_full[acc.stage]);
                acc.template advance<NACC>();
            }
            FP4_PROF_STORE(4, 3);
        }
    } else if (warp < 8 || warp >= 20) {
        // ---------------------------------------------------------------- epilogue
        if constexpr (!C::LARGE) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        Ring acc;
        FP4_PROF_DECL();
        const int q = warp & 3;                 // TMEM lane quarter this warp may read
        // two warps per quarter: the first takes the tile's first rows, the second the rest.  Routed rows to a tensor memory load of 32 columns: five
        // fill it, four cost a tile of few rows less, and the large tile where five spill (one tensor, K = 256: 33 tokens x 32768 features 8.8 us,
        // so 8.4; elsewhere four spill and five do not: K = 512, 1024 x 32768 115 and 98; 768, 512 x 32768 67.4 and 65.7).
        constexpr int FOLD = C::LARGE && (DUAL || K > 256) ? 5 : 4, HALF = (RPT + 2 * FOLD - 1) / (2 * FOLD) * FOLD;
        const int first = warp >= 20 ? HALF : 0;
        for (int u = blockIdx.x; u < n_units && !s_abort; u += gridDim.x) {
            const Unit w = unit_at(u);
            const float sc0 = p.scale0 ? __ldg(p.scale0 + w.e) : 1.0f;
            const float sc1 = DUAL ? (p.scale1 ? __ldg(p.scale1 + w.e) : 1.0f) : sc0;
            // lane i holds the routed row and the power of two of the tile's row i (a tile has at most 27)
            const int my_row = lane < w.nt ? __ldg(p.perm + w.row0 + lane) : 0;
            const float my_rs = lane < w.nt ? __ldg(p.row_scale + w.row0 + lane) : 0.0f;
            // lanes leave the polling loop one by one: the vote reconverges the warp (tcgen05.ld below needs all of it)
            {
                FP4_PROF_T0();
                if (!__all_sync(0xffffffffu, wait_or_abort<200>(&acc_full[acc.stage], acc.phase, &s_abort, p.err))) break;
                FP4_PROF_ADD(0);
            }
            tc_fence_after();
            const uint32_t d0 = tmem + (uint32_t) acc.stage * (2 * C::NCOL) + ((uint32_t) (q * 32) << 16);
            // The planes of every routed row are folded first and the accumulators given back before anything else is done with the
            // sums: with a single accumulator buffer the next unit's instructions wait for this loop.
            float x0[HALF], x1[HALF];
#pragma unroll
            for (int j = 0; j < HALF; j += FOLD)          // (the last load may read past the tile's columns)
                if (first + j < w.nt) {
                    auto fold = [&](uint32_t col, float * x) {
                        float v[32];
                        tmem_ld32(col, v);
#pragma unroll
                        for (int rr = 0; rr < FOLD; ++rr) {
                            float a = v[FP4_PLANES * rr + FP4_PLANES - 1];     // sum_p 9^p * plane_p, highest plane first
#pragma unroll
                            for (int pl = FP4_PLANES - 2; pl >= 0; --pl) a = __fmaf_rn(a, 9.0f, v[FP4_PLANES * rr + pl]);
                            x[rr] = a;
                        }
                    };
                    fold(d0 + FP4_PLANES * (first + j), x0 + j);
                    fold(d0 + C::NCOL + FP4_PLANES * (first + j), x1 + j);
                }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc.stage]);
            acc.template advance<NACC>();
            const int feature = w.ft * FEAT + q * 32 + lane;
#pragma unroll
            for (int i = 0; i < HALF; ++i)
                if (first + i < w.nt) {
                    const float rs = __shfl_sync(0xffffffffu, my_rs, first + i);
                    float * orow = p.out + (size_t) __shfl_sync(0xffffffffu, my_row, first + i) * p.n_out;
                    const float v0 = __fmul_rn(__fmul_rn(x0[i], rs), sc0), v1 = __fmul_rn(__fmul_rn(x1[i], rs), sc1);
                    if (DUAL) orow[feature] = __fmul_rn(ggml_silu(v0), v1);
                    else { orow[feature] = v0; orow[feature + 128] = v1; }
                }
        }
        if (warp == 4 && lane == 0) FP4_PROF_STORE(8, 1);
    } else if (warp < 16) {
        // ---------------------------------------------------------------- repack: strip the scale bytes, keep everything else
        if constexpr (!C::LARGE) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        const int dq = tid - 256;
        const int trow = dq & 127, tsel = dq >> 7;
        const uint32_t a_off = tsel * C::A_TILE + sw128_offset(trow, 0);   // 16-byte chunk c of the row lies at a_off ^ (16 c)
        const uint32_t raw_off = (uint32_t) dq * GEMM_RAW_ROW;
        Ring raw, tile;
        FP4_PROF_DECL();
        for (int i = 0; i < my_stages && !s_abort; ++i) {
            {
                FP4_PROF_T0();
                if (!__all_sync(0xffffffffu, wait_or_abort(&raw_full[raw.stage], raw.phase, &s_abort, p.err))) break;
                FP4_PROF_ADD(0);
            }
            uint4 * const src = reinterpret_cast<uint4 *>(raws + (size_t) raw.stage * C::RAW_STAGE + raw_off);
            uint32_t R[36];                // 4 blocks of [scale word][8 code words]
#pragma unroll
            for (int j = 0; j < 9; ++j) {
                const uint4 v = src[j];
                R[4 * j] = v.x; R[4 * j + 1] = v.y; R[4 * j + 2] = v.z; R[4 * j + 3] = v.w;
            }
            // the row's four scale words, for the scale warps, into the first 16 bytes of the raw row, which this thread has just read
            uint32_t S[4];
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                // The reference reads scale bytes through ggml_ue4m3_to_fp32: bit 7 ignored, 0x7f decodes to zero; to the tensor
                // core 0x7f is NaN.  Clear bit 7 and turn 0x7f into 0 (t <= 0x7f per byte, so t + 1 carries into bit 7 only
                // for 0x7f and never into the next byte).
                const uint32_t t = R[9 * kb] & 0x7f7f7f7fu;
                const uint32_t nan1 = ((t + 0x01010101u) >> 7) & 0x01010101u;
                S[kb] = t & ~((nan1 << 7) - nan1);
            }
            *src = make_uint4(S[0], S[1], S[2], S[3]);
            __syncwarp();
            if (lane == 0) mbar_arrive(&sf_ready[raw.stage]);
            raw.template advance<RS>();
            {
                FP4_PROF_T0();
                if (!__all_sync(0xffffffffu, wait_or_abort(&tile_empty[tile.stage], tile.phase ^ 1u, &s_abort, p.err))) break;
                FP4_PROF_ADD(1);
            }
            uint8_t * st = tiles + (size_t) tile.stage * C::STAGE;
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                *reinterpret_cast<uint4 *>(st + (a_off ^ (32 * kb))) = make_uint4(R[9 * kb + 1], R[9 * kb + 2], R[9 * kb + 3], R[9 * kb + 4]);
                *reinterpret_cast<uint4 *>(st + (a_off ^ (32 * kb + 16))) = make_uint4(R[9 * kb + 5], R[9 * kb + 6], R[9 * kb + 7], R[9 * kb + 8]);
            }
            // every writer orders its own stores against the tensor core's (async proxy) reads and then arrives itself
            fence_async_smem();
            mbar_arrive(&tile_full[tile.stage]);
            tile.template advance<TS>();
        }
        if (tid == 256) FP4_PROF_STORE(10, 2);
    } else {
        // ---------------------------------------------------------------- scale factors: registers -> tensor memory
        // One warp per lane quarter of tensor memory; each writes all of a stage's scales to its quarter.  Lane l holds those of rows l,
        // l + 32, l + 64 and l + 96 of a weight tile (what tcgen05.cp 32x128b.warpx4 would put there) and of a block of planes.
        if constexpr (!C::LARGE) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        const uint32_t quarter = (uint32_t) ((warp & 3) * 32) << 16;
        Ring raw, tile, act;
        FP4_PROF_DECL();
        for (int i = 0; i < my_stages && !s_abort; ++i) {
            {
                FP4_PROF_T0();
                if (!__all_sync(0xffffffffu, wait_or_abort<20>(&sf_ready[raw.stage], raw.phase, &s_abort, p.err))) break;
                FP4_PROF_ADD(0);
            }
            const uint8_t * rows = raws + (size_t) raw.stage * C::RAW_STAGE + lane * GEMM_RAW_ROW;
            uint4 a[2][4];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                uint4 r[4];                // [row l + 32 j][K = 64 step]
#pragma unroll
                for (int j = 0; j < 4; ++j) r[j] = *reinterpret_cast<const uint4 *>(rows + (128 * t + 32 * j) * GEMM_RAW_ROW);
                a[t][0] = make_uint4(r[0].x, r[1].x, r[2].x, r[3].x);
                a[t][1] = make_uint4(r[0].y, r[1].y, r[2].y, r[3].y);
                a[t][2] = make_uint4(r[0].z, r[1].z, r[2].z, r[3].z);
                a[t][3] = make_uint4(r[0].w, r[1].w, r[2].w, r[3].w);
            }
            fence_async_smem();            // the next copy into this stage comes behind the words written to it
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[raw.stage]);
            raw.template advance<RS>();
            {
                FP4_PROF_T0();
                if (!__all_sync(0xffffffffu, wait_or_abort<20>(&tile_empty[tile.stage], tile.phase ^ 1u, &s_abort, p.err))) break;
                FP4_PROF_ADD(2);
            }
            tc_fence_after();
            const uint32_t sf_set = tmem + C::SF_COL + C::SF_SET * (uint32_t) tile.stage + quarter;
            tmem_st16(sf_set, a[0]);
            tmem_st16(sf_set + 16, a[1]);
            {
                FP4_PROF_T0();
                if (!__all_sync(0xffffffffu, wait_or_abort<20>(&act_full[act.stage], act.phase, &s_abort, p.err))) break;
                FP4_PROF_ADD(1);
            }
            // plane rows l + 32 j of a block of 128 read the scales of their routed row (behind the stores of the weights' scales: there is no
            // room for both in the registers)
            const uint8_t * sfb = acts + (size_t) act.stage * C::ACT_STAGE + OFF_SFB;
            uint4 b[C::NBLK][4];           // in memory order: [K = 64 step][block]
            auto put = [&](int step, int n, const uint4 & v) { b[(step * C::NBLK + n) >> 2][(step * C::NBLK + n) & 3] = v; };
#pragma unroll
            for (int n = 0; n < C::NBLK; ++n) {
                uint4 r[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) r[j] = *reinterpret_cast<const uint4 *>(sfb + min((128 * n + 32 * j + lane) / FP4_PLANES, RPT - 1) * 16);
                put(0, n, make_uint4(r[0].x, r[1].x, r[2].x, r[3].x));
                put(1, n, make_uint4(r[0].y, r[1].y, r[2].y, r[3].y));
                put(2, n, make_uint4(r[0].z, r[1].z, r[2].z, r[3].z));
                put(3, n, make_uint4(r[0].w, r[1].w, r[2].w, r[3].w));
            }
#pragma unroll
            for (int n = 0; n < C::NBLK; ++n) tmem_st16(sf_set + 32 + 16 * n, b[n]);
            act.template advance<AS>();
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tile_full[tile.stage]);
            tile.template advance<TS>();
        }
        if (tid == 512) FP4_PROF_STORE(13, 3);
    }

    // ---- teardown: everyone meets here (all waits above are bounded), then tensor memory goes back
    if (s_abort) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 1000000ull) { }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 3) tmem_dealloc(tmem, C::TMEM_COLS);
}

}  // namespace b200moe
