// Grouped Q3_K expert matmul on the int8 matrix instruction, bit-identical to the reference: every call but one or two tokens' (those take
// expert_few_rows_kernel).
//
// Why a matrix instruction can keep the reference's bits: ggml_vec_dot_q3_K_q8_K (ggml-cpu/arch/x86/quants.c:1766-1880) sums
// INTEGERS over a whole super-block in every one of its eight SIMD lanes - lane L collects scale * code * activation over byte
// columns 4L..4L+3 of the eight 32-groups - and only then runs one fma(d_w * d_x, (float) sum_L, acc_L).  Those 32 products are
// one K = 32 step of mma.m16n8k32 (s8 x s8 -> s32, exact): one instruction per lane and super-block for 16 weight rows x 8 routed
// rows, whose accumulators come out as the lane sums, followed by the reference's fp32 chain in registers.  The folded weight
// scale * code lies in -128..128; its negative (-128..124) fits int8, so the operand holds -scale * code and the sum is negated,
// exactly, on its way to fp32 (|sum| <= 32 * 128 * 128 < 2^22).
//
// Why mma.sync and not tcgen05 (kind::i8): every accumulator is read after ONE K = 32 step.  With accumulators in tensor memory
// each of those reads is a tcgen05.ld and a conversion more; here they are already in the registers of the thread that runs the chain.
//
// A warp owns 16 weight rows (8 features of gate and up, or 16 rows of one tensor) and up to 32 routed rows.  It decodes the weights
// straight into the instruction's operand: thread (row g, quarter q) holds 32-groups q and q + 4 of rows g and g + 8, so one funnel shift
// brings the two low code bits of its group in place, one the high bits of both groups, and a byte permute picks four of the eight products
// of a (row, sub-block) by the codes packed to a selector.  No operand tile in shared memory, no barrier between super-blocks: a warp fetches
// its own raw rows and meets the others only when the routed rows change.  The code is separate for each number of token groups: with a test
// between them nothing was scheduled across (1001 tokens, gate/up: 430 us, then 308).
// What bounds it is the half-rate integer unit and, with 32 routed rows to a pass, its own dependences at two warps per scheduler (255
// registers, a few values spilled beside the loops; IPC 0.56 per scheduler).  Decoding 64 x 64 tiles through shared memory, a barrier to a super-block (IPC 0.32), and a thread per
// reference lane with dp4a took, 2048 -> 768 of 128 experts, us: gate/up of 32 tokens 130 and of 1001 tokens 537, down 71 and 311; so 75 and
// 289, 42 and 174.
// Activation rows are K + 16 bytes apart, which makes the 16-byte fragment loads conflict-free.
#pragma once
#include "common.cuh"
#include "expert_gemm.cuh"
#include "expert_gemv.cuh"
#include "formats.cuh"
#include "router.cuh"

namespace b200moe {

// Routed rows per expert (on average) from which a pass is 32 routed rows instead of 16.  Whole calls, us, 16 and 32: 128 experts, 2048 -> 768,
// 5 rows 64 and 65, 9 rows 69 and 70, 12 rows 75 and 74, 16 rows 89 and 80, 48 rows 168 and 146; 256 -> 512: 5 rows 27 and 27, 24 rows 37 and 34.
constexpr int Q3K_MMA_MIN_ROWS = 12;

template <int K, bool DUAL, int NTG>
struct Q3kCfg {
    static constexpr int TOK = 8 * NTG;                       // routed rows of a pass: NTG token groups
    static constexpr int ROW_BYTES = K / 256 * Q3K_BLOCK_BYTES;
    static constexpr int FEAT = DUAL ? 8 : 16;                // features of a warp's tile
    static constexpr int TILE = 16 * ROW_BYTES;
    static constexpr int WARPS = 8;
    static constexpr int STAGES = K == 2048 ? 1 : 2;          // raw tiles of a warp
    static constexpr int THREADS = WARPS * 32;
    static constexpr int PITCH = K + 16;                      // of an activation row
    static constexpr int SB = K / 256;
    static constexpr int FULL = 4 + NTG;       // work of a full pass (q3k_work)
    // A pass's activation rows come by bulk copies, one to a row; rows of up to 512 bytes by the threads, whose loads do not queue up: 256 -> 256,
    // 50 rows to each of 16 experts, 18.4 us with copies and 16.5 without (whole call), 512 -> 768, 8000 rows over 128 experts 70 and 68; pieces of
    // 768 do not divide by the threads.
    static constexpr bool WIDE_ACTS = K > 512;
    static constexpr size_t SMEM = (size_t) WARPS * STAGES * TILE + (size_t) TOK * PITCH;
    static_assert(TILE % 32 == 0 && PITCH % 128 == 16, "halves of a tile are multiples of 16 bytes; fragment loads fall on different banks");
    static_assert(WIDE_ACTS || (THREADS % (K / 16) == 0 && TOK % (THREADS / (K / 16)) == 0), "every thread moves as many pieces of the activation rows");
    static_assert(SMEM + 4096 <= 227 * 1024, "one CTA fits an SM");
};

__device__ __forceinline__ void mma_s8_16832(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c));
}
template <int K, bool DUAL, int NTG>
__device__ __forceinline__ void q3k_mma_body(const GemvParams & p) {
    using C = Q3kCfg<K, DUAL, NTG>;
    constexpr int SB = C::SB, RB = C::ROW_BYTES;
    constexpr int MAGIC = 0x4B400000;                         // bits of 1.5 * 2^23: see small_int_to_float
    extern __shared__ __align__(128) uint8_t q3k_smem[];
    uint8_t * const acts = q3k_smem;                          // [TOK][PITCH]
    uint8_t * const tiles = acts + (size_t) C::TOK * C::PITCH;   // [WARPS][STAGES][16 rows]
    __shared__ uint2 s_prod[64];                              // six-bit scale v -> bytes (32 - v) * (c - 4), c = 0..7
    __shared__ float s_dx[C::TOK][SB];
    __shared__ int s_row[C::TOK];                             // the pass's routed rows
    __shared__ uint64_t full[C::WARPS][C::STAGES], act_full;
    __shared__ volatile int s_abort;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int w = 0; w < C::WARPS; ++w)
            for (int s = 0; s < C::STAGES; ++s) mbar_init(&full[w][s], 1);
        mbar_init(&act_full, 1);
        mbar_fence_init();
        s_abort = 0;
    }
    if (tid < 64) {
        const int s = tid - 32;
        auto b = [&](int c) { return (uint32_t) ((s * (4 - c)) & 0xff); };
        s_prod[tid] = make_uint2(b(0) | b(1) << 8 | b(2) << 16 | b(3) << 24, b(4) | b(5) << 8 | b(6) << 16 | b(7) << 24);
    }
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();

    const int n_active = p.meta[0];
    const int * const cw = p.cost + (NTG < 4 ? 0 : 2) * (p.n_as + 1);
    // a tile for each warp to a chunk; while there are items for less than every CTA, as few as leaves one to a CTA
    const int n_tiles = (p.n_out + C::FEAT - 1) / C::FEAT;
    const long long passes = (cw[n_active] + 4) / 5;
    int log_per = 0;
    while (C::WARPS >> log_per > 1 && passes * ((n_tiles + (1 << log_per) - 1) >> log_per) > gridDim.x) ++log_per;
    const int per = 1 << log_per;
    auto span = pass_span<C::THREADS, C::TOK, C::FULL>(cw, n_active, (n_tiles + per - 1) >> log_per);

    // raw rows of the warp's tile of an item, if it has one
    auto has_tile = [&](int ch) { return warp < per && ch * per + warp < n_tiles; };
    uint8_t * const my_tiles = tiles + (size_t) warp * C::STAGES * C::TILE;
    auto pre = span;
    int pre_stage = 0;
    auto fetch = [&] {                                        // of the next item that has one
        while (pre.more()) {
            // (asked for again for every item: held in registers they spilled the chains, 2048 -> 768, 1001 tokens, whole layer 545 us, so 526)
            const int pre_e = p.active[pre.a], pre_n = p.offsets[pre_e + 1] - p.offsets[pre_e];
            const int ch = pre.ch;
            pre.next(pre_n);
            if (!has_tile(ch)) continue;
            const int f0 = (ch * per + warp) * C::FEAT;
            if (lane == 0) {
                uint8_t * dst = my_tiles + (size_t) pre_stage * C::TILE;
                uint64_t * bar = &full[warp][pre_stage];
                const size_t off = ((size_t) pre_e * p.w_stride + f0) * RB;
                const uint32_t bytes = DUAL ? C::TILE : (uint32_t) min(16, p.n_out - f0) * RB;
                mbar_arrive_expect_tx(bar, bytes);
                if (DUAL) {
                    bulk_g2s(dst, p.w0 + off, C::TILE / 2, bar);
                    bulk_g2s(dst + C::TILE / 2, p.w1 + off, C::TILE / 2, bar);
                } else {
                    bulk_g2s(dst, p.w0 + off, bytes, bar);
                }
            }
            pre_stage = pre_stage + 1 == C::STAGES ? 0 : pre_stage + 1;
            return;
        }
    };
    for (int s = 0; s < C::STAGES; ++s) fetch();

    const int g = lane >> 2, q = lane & 3;
    const uint64_t minus_one = f32x2(-1.0f, -1.0f), magic2 = f32x2(12582912.0f, 12582912.0f);
    int at = -1, row_beg = 0, n_e = 0, loaded = -1;           // of the expert; the pass whose activations are in place
    float sc0 = 1.0f, sc1 = 1.0f;
    uint32_t act_parity = 0;
    Ring st;
    for (; span.more(); span.next(n_e)) {
        if (span.a != at) {
            at = span.a;
            const int e = p.active[at], se = p.w_stride ? e : 0;         // every group of a dense product has the one matrix and its scale
            row_beg = p.offsets[e];
            n_e = p.offsets[e + 1] - row_beg;
            if (p.scale0) sc0 = p.scale0[se];
            if (DUAL && p.scale1) sc1 = p.scale1[se];
            loaded = -1;
        }
        const int t0 = C::TOK * span.ps, n = min(C::TOK, n_e - t0);
        if (loaded != span.ps) {
            auto act_row = [&](int r) { return (int) ((r / p.n_ids) * p.ne11 + (r % p.n_ids) % p.ne11); };
            const int * const rows = p.perm + row_beg + t0;
            if constexpr (C::WIDE_ACTS) {
                __syncthreads();                              // everybody is done with the rows that give way
                if (warp == 0) {
                    if (lane == 0) mbar_arrive_expect_tx(&act_full, (uint32_t) (n * K));
                    __syncwarp();
                    if (lane < n) {
                        const int r = rows[lane];
                        bulk_g2s(acts + (size_t) lane * C::PITCH, p.act.q + (size_t) act_row(r) * K, K, &act_full);
                    }
                }
                if (tid < n) s_row[tid] = rows[tid];
                for (int i = tid; i < n * SB; i += C::THREADS) s_dx[i / SB][i % SB] = p.act.d[(size_t) act_row(rows[i / SB]) * SB + i % SB];
                wait_or_abort(&act_full, act_parity, &s_abort, p.err);
                act_parity ^= 1u;
            } else {
                constexpr int PIECES = K / 16, STEP = C::THREADS / PIECES;     // a thread moves its piece of every STEP-th row
                const int piece = tid % PIECES, first = tid / PIECES;
                uint4 v[C::TOK / STEP];
                int r[C::TOK / STEP];
                float d[C::TOK / STEP];
#pragma unroll
                for (int i = 0; i < C::TOK / STEP; ++i) r[i] = rows[min(first + i * STEP, n - 1)];
#pragma unroll
                for (int i = 0; i < C::TOK / STEP; ++i) {
                    const size_t row = act_row(r[i]);
                    v[i] = reinterpret_cast<const uint4 *>(p.act.q + row * K)[piece];
                    d[i] = p.act.d[row * SB + piece / 16];
                }
                __syncthreads();                              // everybody is done with the rows that give way
#pragma unroll
                for (int i = 0; i < C::TOK / STEP; ++i) {
                    const int t = first + i * STEP;
                    reinterpret_cast<uint4 *>(acts + (size_t) t * C::PITCH)[piece] = v[i];
                    if (piece % 16 == 0) s_dx[t][piece / 16] = d[i];
                    if (piece == 0) s_row[t] = r[i];
                }
            }
            __syncthreads();
            loaded = span.ps;
        }
        if (!has_tile(span.ch)) continue;
        const bool ok = __all_sync(0xffffffffu, wait_or_abort(&full[warp][st.stage], st.phase, &s_abort, p.err));
        if (!ok) continue;                                    // the barriers above still see this warp
        const uint8_t * const tile = my_tiles + (size_t) st.stage * C::TILE;

        auto run = [&](auto gtag) {                           // token groups that exist: no branch between them
            constexpr int G = decltype(gtag)::value;
            uint64_t acc[G][8][2];                              // [token group][SIMD lane][row g, g + 8]: routed rows 2q and 2q + 1 of the group
#pragma unroll
            for (int i = 0; i < G; ++i)
#pragma unroll
                for (int L = 0; L < 8; ++L) acc[i][L][0] = acc[i][L][1] = f32x2(0.0f, 0.0f);
#pragma unroll 1
            for (int sb = 0; sb < SB; ++sb) {
                const uint32_t * hw[2];                           // aligned words of the block of rows g and g + 8
                int sh[2];                                        // a block starts on a 2-byte boundary
                uint32_t sc[2];
                uint64_t s2[G][2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t off = (uint32_t) ((r * 8 + g) * RB + sb * Q3K_BLOCK_BYTES);
                    const uint8_t * blk = tile + off;
                    hw[r] = reinterpret_cast<const uint32_t *>(tile + (off & ~3u));
                    sh[r] = (int) (off & 2u) * 8;
                    // scales of sub-blocks 8j + 2q and 8j + 2q + 1: nibble j of bytes 2q, 2q + 1, two more bits from the last four bytes
                    const uint32_t lo4 = *reinterpret_cast<const uint16_t *>(blk + 96 + 2 * q);
                    const uint32_t hi2 = (uint32_t) *reinterpret_cast<const uint16_t *>(blk + 104 + (2 * q & 2)) >> (q & 2);
                    sc[r] = (lo4 & 0x0f0fu) + (lo4 & 0xf0f0u) * 4096u + (hi2 & 0x0303u) * 16u + (hi2 & 0x3030u) * 65536u;   // byte 2j + hf
                    const float dw = __half2float(*reinterpret_cast<const __half *>(blk + 108));
#pragma unroll
                    for (int i = 0; i < G; ++i) s2[i][r] = mul_f32x2(f32x2(s_dx[8 * i + 2 * q][sb], s_dx[8 * i + 2 * q + 1][sb]), f32x2(dw, dw));
                }
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {                  // lanes 4 hf .. 4 hf + 3, which have their sub-blocks' scales in common
                    uint2 prod[2][2];                             // [row][j]
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int j = 0; j < 2; ++j) prod[r][j] = s_prod[(sc[r] >> (16 * j + 8 * hf)) & 0xffu];
                    uint4 b[G][2];
#pragma unroll
                    for (int i = 0; i < G; ++i)
#pragma unroll
                        for (int j = 0; j < 2; ++j)
                            b[i][j] = *reinterpret_cast<const uint4 *>(acts + (size_t) (8 * i + g) * C::PITCH + sb * 256 + j * 128 + q * 32 + 16 * hf);
                    auto word = [](const uint4 & v, int l) { return l == 0 ? v.x : l == 1 ? v.y : l == 2 ? v.z : v.w; };
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        const int L = 4 * hf + l;
                        uint32_t a[4];                            // [row g, g + 8] of group q, then of group q + 4
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const uint32_t hb = __funnelshift_r(hw[r][L], hw[r][L + 1], sh[r] + q);          // bit 0: group q, bit 4: group q + 4
                            const uint32_t q0 = __funnelshift_r(hw[r][8 + L], hw[r][9 + L], sh[r] + 2 * q) & 0x03030303u;
                            const uint32_t q1 = __funnelshift_r(hw[r][16 + L], hw[r][17 + L], sh[r] + 2 * q) & 0x03030303u;
                            // Codes c = 4 hb + q, 0..7, one per byte; c * 272 is c in the high nibble of its byte and in the low nibble of
                            // the next, so bytes 1 and 3 hold the selector of the four products.  (Multiplications: the integer unit is the busy one.)
                            const uint32_t u0 = (hb & 0x01010101u) * 1088u + q0 * 272u, u1 = (hb & 0x10101010u) * 68u + q1 * 272u;
                            a[r] = __byte_perm(prod[r][0].x, prod[r][0].y, __byte_perm(u0, 0u, 0x4431));
                            a[2 + r] = __byte_perm(prod[r][1].x, prod[r][1].y, __byte_perm(u1, 0u, 0x4431));
                        }
#pragma unroll
                        for (int i = 0; i < G; ++i) {
                                int d[4];
                                mma_s8_16832(d, a, word(b[i][0], l), word(b[i][1], l), MAGIC);
#pragma unroll
                                for (int r = 0; r < 2; ++r) {
                                    const uint64_t sum = fma_f32x2(f32x2(__int_as_float(d[2 * r]), __int_as_float(d[2 * r + 1])), minus_one, magic2);
                                    acc[i][L][r] = fma_f32x2(s2[i][r], sum, acc[i][L][r]);
                                }
                            }
                    }
                }
            }
            __syncwarp();                                         // all lanes are done with the raw rows
            fetch();
            st.template advance<C::STAGES>();

            // hsum_float_8 of every value, scales, SwiGLU, scatter
            const int f0 = (span.ch * per + warp) * C::FEAT;
#pragma unroll
            for (int i = 0; i < G; ++i) {
                float v[2][2];                                    // [row][routed row]
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    uint64_t s4[4];
#pragma unroll
                    for (int l = 0; l < 4; ++l) s4[l] = add_f32x2(acc[i][l][r], acc[i][l + 4][r]);
                    const float2 s = f32x2_halves(add_f32x2(add_f32x2(s4[0], s4[2]), add_f32x2(s4[1], s4[3])));
                    v[r][0] = s.x;
                    v[r][1] = s.y;
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int t = 8 * i + 2 * q + c;
                    if (t >= n) continue;
                    float * orow = p.out + (size_t) s_row[t] * p.n_out + f0;
                    if (DUAL) {
                        orow[g] = __fmul_rn(ggml_silu(__fmul_rn(v[0][c], sc0)), __fmul_rn(v[1][c], sc1));
                    } else {
                        orow[g] = __fmul_rn(v[0][c], sc0);
                        if (f0 + 8 < p.n_out) orow[g + 8] = __fmul_rn(v[1][c], sc0);
                    }
                }
            }
        };
        const int groups = (n + 7) / 8;
        if (groups == 1) run(std::integral_constant<int, 1>{});
        else if (NTG == 2 || groups == 2) run(std::integral_constant<int, 2>{});
        else if (groups == 3) run(std::integral_constant<int, NTG == 2 ? 1 : 3>{});
        else run(std::integral_constant<int, NTG>{});
    }
    if (s_abort) {   // copies still in flight land before the block (and its shared memory) goes away
        const uint64_t t = global_timer_ns();
        while (global_timer_ns() - t < 1000000ull) { }
    }
    __syncthreads();
}

// passes of 16 routed rows, for few rows per expert, and of 32 (Q3K_MMA_MIN_ROWS)
template <int K, bool DUAL>
__global__ void __launch_bounds__(Q3kCfg<K, DUAL, 2>::THREADS, 1) q3k_expert_gemv_kernel(const GemvParams p) {
    q3k_mma_body<K, DUAL, 2>(p);
}
template <int K, bool DUAL>
__global__ void __launch_bounds__(Q3kCfg<K, DUAL, 4>::THREADS, 1) expert_mma_q3k_kernel(const GemvParams p) {
    q3k_mma_body<K, DUAL, 4>(p);
}

}  // namespace b200moe
