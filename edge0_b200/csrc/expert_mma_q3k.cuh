// Grouped Q3_K expert matmul for prefill on the int8 matrix instruction, bit-identical to the reference.
//
// Why a matrix instruction can keep the reference's bits: ggml_vec_dot_q3_K_q8_K (ggml-cpu/arch/x86/quants.c:1766-1880) sums
// INTEGERS over a whole super-block in every one of its eight SIMD lanes - lane L collects scale * code * activation over byte
// columns 4L..4L+3 of the eight 32-groups - and only then runs one fma(d_w * d_x, (float) sum_L, acc_L).  Those 32 products are
// one K = 32 step of mma.m16n8k32 (s8 x s8 -> s32, exact): one instruction per lane and super-block for 16 weight rows x 8 routed
// rows, whose accumulators come out as the lane sums, followed by the reference's fp32 chain in registers.  The folded weight
// scale * code lies in -128..128; its negative (-128..124) fits int8, so the tiles hold -scale * code and the sum is negated,
// exactly, on its way to fp32 (|sum| <= 32 * 128 * 128 < 2^22).
//
// Why mma.sync and not tcgen05 (kind::i8): every accumulator is read after ONE K = 32 step.  With accumulators in tensor memory
// each of those reads is a tcgen05.ld and a conversion more; here they are already in the registers of the thread that runs the chain, and
// what bounds the kernel is that chain (per lane sum one add that converts and one fma) and the decode, not the matrix pipe.
//
// A CTA (8 warps) takes units of 64 weight rows (32 features of gate and up each, or 64 rows of one tensor) x up to 64 routed rows of
// one expert.  A warp owns 32 weight rows x 16 routed rows: 128 fp32 chains per thread.  A weight is decoded once per unit:
// one table look-up per (row, sub-block) gives the eight possible products as 8 bytes and one byte permute picks four of
// them.  Decode of step s + 1 and the copies of its activations run beside the matrix work of step s (two operand buffers, one
// barrier per super-block); the raw rows of the next unit arrive by bulk copy meanwhile.
// What it waits for is its own decode and shared memory at two warps per scheduler (0.32 instructions per cycle); sixteen warps of half
// the tile were no faster (581 against 537 us), the A fragments then being read twice as often.  1001 tokens, 128 experts: gate/up
// 2823 -> 537 us, down 1986 -> 305 us.
// Operand rows are 272 bytes apart (256 + 16), which makes the 16-byte fragment loads conflict-free.
#pragma once
#include "common.cuh"
#include "expert_gemv.cuh"
#include "formats.cuh"
#include "router.cuh"

namespace b200moe {

// Routed rows per expert (on average) from which this kernel replaces the GEMV, whose time grows with them while this one's does not up
// to 64.  Gate/up (2048 -> 768), 128 experts: 4 rows GEMV 217 us, this 357; 8 rows 369 and 366; 16 rows 741 and 362; 63 rows 2825 and 537.
// 16 experts: 8 rows 76 and 110 us, 16 rows 135 and 110.
constexpr int Q3K_MMA_MIN_ROWS = 12;

template <int K, bool DUAL>
struct Q3kMmaCfg {
    static constexpr int ROWS = 64, TOK = 64, PITCH = 272;
    static constexpr int FEAT = DUAL ? 32 : 64;               // features of a unit
    static constexpr int ROW_BYTES = K / 256 * Q3K_BLOCK_BYTES;
    static constexpr int RAW = ROWS * ROW_BYTES + 128;        // the last decode of a row may look past it by a word
    static constexpr int TILE = ROWS * PITCH;
    static constexpr size_t SMEM = 2 * (size_t) RAW + 4 * (size_t) TILE;
    static_assert(RAW % 128 == 0 && TILE % 16 == 0 && ROWS == TOK, "buffers stay aligned for bulk copies");
    static_assert((8 * ROW_BYTES) % 16 == 0, "a multiple of eight rows is a multiple of 16 bytes");
};

__device__ __forceinline__ void mma_s8_16832(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void cp_async4(void * smem, const void * gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}

template <int K, bool DUAL>
__global__ void __launch_bounds__(256, 1) expert_mma_q3k_kernel(const GemvParams p) {
    using C = Q3kMmaCfg<K, DUAL>;
    constexpr int SB = K / 256, PITCH = C::PITCH;
    extern __shared__ __align__(128) uint8_t q3k_smem[];
    uint8_t * const raws = q3k_smem;                          // [2] raw rows of a unit
    uint8_t * const a_tiles = raws + 2 * C::RAW;              // [2] weights of one super-block as int8
    uint8_t * const b_tiles = a_tiles + 2 * C::TILE;          // [2] activations of the same super-block
    __shared__ uint2 s_prod[64];                              // six-bit scale v -> bytes (32 - v) * (c - 4), c = 0..7
    __shared__ float s_dw[2][C::ROWS], s_dx[2][C::TOK];
    __shared__ int s_pref[1025];                              // 64-row token tiles before expert e
    __shared__ uint64_t raw_full[2];
    __shared__ int s_abort;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&raw_full[0], 1);
        mbar_init(&raw_full[1], 1);
        mbar_fence_init();
        s_abort = 0;
    }
    if (tid < 64) {
        const int s = tid - 32;
        auto b = [&](int c) { return (uint32_t) ((s * (4 - c)) & 0xff); };
        s_prod[tid] = make_uint2(b(0) | b(1) << 8 | b(2) << 16 | b(3) << 24, b(4) | b(5) << 8 | b(6) << 16 | b(7) << 24);
    }
    if (warp == 0) {
        int run = 0;
        for (int base = 0; base < p.n_as; base += 32) {
            const int e = base + lane;
            const int t = e < p.n_as ? (p.offsets[e + 1] - p.offsets[e] + C::TOK - 1) / C::TOK : 0;
            int incl = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            if (e < p.n_as) s_pref[e] = run + incl - t;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) s_pref[p.n_as] = run;
    }
    __syncthreads();

    const int f_tiles = (p.n_out + C::FEAT - 1) / C::FEAT;
    const int n_units = s_pref[p.n_as] * f_tiles;
    struct Unit { int e, f0, row0, nt; };
    auto unit_at = [&](int u) {
        Unit w;
        const int tile = u / f_tiles;
        w.f0 = (u - tile * f_tiles) * C::FEAT;
        int lo = 0, hi = p.n_as;                              // largest e with s_pref[e] <= tile
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_pref[mid] <= tile) lo = mid; else hi = mid;
        }
        w.e = lo;
        w.row0 = p.offsets[lo] + (tile - s_pref[lo]) * C::TOK;
        w.nt = min(C::TOK, p.offsets[lo + 1] - w.row0);
        return w;
    };
    auto load_raw = [&](int u, int buf) {                     // one thread
        const Unit w = unit_at(u);
        const uint32_t bytes = (uint32_t) min(C::FEAT, p.n_out - w.f0) * C::ROW_BYTES;
        const size_t off = ((size_t) w.e * p.w_stride + w.f0) * C::ROW_BYTES;
        uint8_t * dst = raws + (size_t) buf * C::RAW;
        mbar_arrive_expect_tx(&raw_full[buf], bytes * (DUAL ? 2 : 1));
        bulk_g2s(dst, p.w0 + off, bytes, &raw_full[buf]);
        if (DUAL) bulk_g2s(dst + C::FEAT * C::ROW_BYTES, p.w1 + off, bytes, &raw_full[buf]);
    };
    // activation row that this thread copies (token tid / 4, a quarter of its 256 bytes); rows beyond the tile repeat its first
    auto act_row = [&](const Unit & w) {
        const int t = tid >> 2;
        const int r = p.perm[w.row0 + (t < w.nt ? t : 0)];
        return (r / p.n_ids) * p.ne11 + (r % p.n_ids) % p.ne11;
    };
    auto load_act = [&](int arow, int sb, int buf) {
        const int8_t * src = p.act.q + (size_t) arow * K + sb * 256 + (tid & 3) * 64;
        uint8_t * dst = b_tiles + (size_t) buf * C::TILE + (tid >> 2) * PITCH + (tid & 3) * 64;
#pragma unroll
        for (int i = 0; i < 4; ++i) cp_async16(dst + 16 * i, src + 16 * i);
        if ((tid & 3) == 0) cp_async4(&s_dx[buf][tid >> 2], p.act.d + (size_t) arow * SB + sb);
    };
    // thread = weight row tid / 4, lanes L = 2h and 2h + 1 (h = tid % 4) of its super-block
    auto decode = [&](int raw_buf, int sb, int buf) {
        const int row = tid >> 2, h = tid & 3;
        const uint32_t at = (uint32_t) (row * C::ROW_BYTES + sb * Q3K_BLOCK_BYTES);
        const uint32_t * blk = reinterpret_cast<const uint32_t *>(raws + (size_t) raw_buf * C::RAW + (at & ~3u));
        const int sh = (int) (at & 2u) * 8;                   // a block starts on a 2-byte boundary
        uint32_t hm[2], q[2][2], sc[4];
        {
            const uint32_t * s = blk + 2 * h;
            hm[0] = __funnelshift_r(s[0], s[1], sh);  hm[1] = __funnelshift_r(s[1], s[2], sh);
            q[0][0] = __funnelshift_r(s[8], s[9], sh);  q[0][1] = __funnelshift_r(s[9], s[10], sh);
            q[1][0] = __funnelshift_r(s[16], s[17], sh);  q[1][1] = __funnelshift_r(s[17], s[18], sh);
            const uint32_t w0 = blk[24], w1 = blk[25], w2 = blk[26], w3 = blk[27];
            const uint32_t s0 = __funnelshift_r(w0, w1, sh), s1 = __funnelshift_r(w1, w2, sh), s2 = __funnelshift_r(w2, w3, sh);
            const uint32_t m2 = 0x03030303u, m4 = 0x0f0f0f0fu;
            const int hi = h >= 2 ? 8 : 0;                    // lanes 4..7 use the odd sub-blocks' scales
            sc[0] = ((s0 & m4) | ((s2 & m2) << 4)) >> hi;
            sc[1] = ((s1 & m4) | (((s2 >> 2) & m2) << 4)) >> hi;
            sc[2] = (((s0 >> 4) & m4) | (((s2 >> 4) & m2) << 4)) >> hi;
            sc[3] = (((s1 >> 4) & m4) | (((s2 >> 6) & m2) << 4)) >> hi;
            if (h == 0) s_dw[buf][row] = __half2float(__ushort_as_half((unsigned short) (w3 >> sh)));
        }
        uint8_t * dst = a_tiles + (size_t) buf * C::TILE + row * PITCH + 8 * h;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int bit = 4 * j + s;
                const uint2 prod = s_prod[(sc[2 * j + (s >> 1)] >> (16 * (s & 1))) & 0x3fu];
                uint32_t out[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint32_t hb = bit >= 2 ? (hm[e] >> (bit - 2)) : (hm[e] << (2 - bit));
                    const uint32_t t = ((q[j][e] >> (2 * s)) & 0x03030303u) | (hb & 0x04040404u);   // codes 0..7, one per byte
                    out[e] = __byte_perm(prod.x, prod.y, __byte_perm(t | (t >> 4), 0u, 0x4420));    // packed to nibbles, looked up
                }
                *reinterpret_cast<uint2 *>(dst + bit * 32) = make_uint2(out[0], out[1]);
            }
    };

    const int wm = warp & 1, wn = warp >> 1;                  // a warp's half of the weight rows; its token groups are wn and wn + 4
    const int gq = lane >> 2, tq = lane & 3;
    const int m_row[2] = { DUAL ? wm * 16 : wm * 32, DUAL ? 32 + wm * 16 : wm * 32 + 16 };
    constexpr int MAGIC = 0x4B400000;                         // bits of 1.5 * 2^23: see small_int_to_float

    int issued = 0, waited = 0;
    const int first = blockIdx.x, step_u = gridDim.x;
    Unit cur{}, nxt{};
    int arow = 0;
    if (first < n_units) {
        if (tid == 0) {
            load_raw(first, 0);
            ++issued;
            if (first + step_u < n_units) { load_raw(first + step_u, 1); ++issued; }
        }
        cur = unit_at(first);
        arow = act_row(cur);
        load_act(arow, 0, 0);
        cp_async_commit();
        if (!mbar_wait_bounded(&raw_full[0], 0)) { report_error(p.err, DEV_ERR_BARRIER_TIMEOUT); s_abort = 1; }
        ++waited;
        decode(0, 0, 0);
        cp_async_wait<0>();
    }
    bool failed = __syncthreads_or(s_abort) != 0;
    float acc[2][2][8][4];
    int buf = 0;
    for (int u = first, ui = 0; u < n_units && !failed; u += step_u, ++ui) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int L = 0; L < 8; ++L)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[m][i][L][c] = 0.0f;
        const bool more = u + step_u < n_units;
        if (more) nxt = unit_at(u + step_u);
#pragma unroll 1
        for (int sb = 0; sb < SB; ++sb, buf ^= 1) {
            // operands of the next step (the next super-block, or the first one of the next unit)
            if (sb + 1 < SB) {
                load_act(arow, sb + 1, buf ^ 1);
                cp_async_commit();
                decode(ui & 1, sb + 1, buf ^ 1);
            } else {
                // every thread has decoded the last super-block of this unit: its raw rows give way to those of the next but one
                if (tid == 0 && u + 2 * step_u < n_units) { load_raw(u + 2 * step_u, ui & 1); ++issued; }
                if (more) {
                    arow = act_row(nxt);
                    load_act(arow, 0, buf ^ 1);
                    cp_async_commit();
                    if (!mbar_wait_bounded(&raw_full[(ui + 1) & 1], (uint32_t) ((ui + 1) >> 1) & 1u)) { report_error(p.err, DEV_ERR_BARRIER_TIMEOUT); s_abort = 1; }
                    ++waited;
                    decode((ui + 1) & 1, 0, buf ^ 1);
                }
            }
            if (8 * wn < cur.nt) {
                const uint8_t * at = a_tiles + (size_t) buf * C::TILE;
                const uint8_t * bt = b_tiles + (size_t) buf * C::TILE;
                const bool two = 8 * (wn + 4) < cur.nt;       // warp-uniform: the second token group exists
                float dw[2][2], dx[2][2];
#pragma unroll
                for (int m = 0; m < 2; ++m) { dw[m][0] = s_dw[buf][m_row[m] + gq]; dw[m][1] = s_dw[buf][m_row[m] + gq + 8]; }
#pragma unroll
                for (int i = 0; i < 2; ++i) { dx[i][0] = s_dx[buf][8 * (wn + 4 * i) + 2 * tq]; dx[i][1] = s_dx[buf][8 * (wn + 4 * i) + 2 * tq + 1]; }
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {              // lanes 4 hf .. 4 hf + 3
                    uint4 b[2][2];
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int g = 0; g < 2; ++g)
                            if (i == 0 || two)
                                b[i][g] = *reinterpret_cast<const uint4 *>(bt + (8 * (wn + 4 * i) + gq) * PITCH + (tq + 4 * g) * 32 + 16 * hf);
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        uint4 a[2][2];                        // [row gq, gq + 8][group tq, tq + 4]
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int g = 0; g < 2; ++g)
                                a[r][g] = *reinterpret_cast<const uint4 *>(at + (m_row[m] + gq + 8 * r) * PITCH + (tq + 4 * g) * 32 + 16 * hf);
                        auto word = [](const uint4 & v, int l) { return l == 0 ? v.x : l == 1 ? v.y : l == 2 ? v.z : v.w; };
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            if (i == 0 || two) {
                                const float s[4] = { __fmul_rn(dx[i][0], dw[m][0]), __fmul_rn(dx[i][1], dw[m][0]), __fmul_rn(dx[i][0], dw[m][1]),
                                                     __fmul_rn(dx[i][1], dw[m][1]) };
#pragma unroll
                                for (int l = 0; l < 4; ++l) {
                                    const uint32_t af[4] = { word(a[0][0], l), word(a[1][0], l), word(a[0][1], l), word(a[1][1], l) };
                                    int d[4];
                                    mma_s8_16832(d, af, word(b[i][0], l), word(b[i][1], l), MAGIC);
#pragma unroll
                                    for (int c = 0; c < 4; ++c)
                                        acc[m][i][4 * hf + l][c] = __fmaf_rn(s[c], __fsub_rn(12582912.0f, __int_as_float(d[c])), acc[m][i][4 * hf + l][c]);
                                }
                            }
                    }
                }
            }
            cp_async_wait<0>();
            if (__syncthreads_or(s_abort)) { failed = true; break; }
        }
        if (failed) break;
        // hsum_float_8 of every value, scales, SwiGLU, scatter
        const int se = p.w_stride ? cur.e : 0;   // every group of a dense product has the one matrix and its scale
        const float sc0 = p.scale0 ? p.scale0[se] : 1.0f;
        const float sc1 = (DUAL && p.scale1) ? p.scale1[se] : 1.0f;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int t = 8 * (wn + 4 * i) + 2 * tq + c;
                if (t < cur.nt) {
                    float * orow = p.out + (size_t) p.perm[cur.row0 + t] * p.n_out;
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        float v[2];
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            float s4[4];
#pragma unroll
                            for (int l = 0; l < 4; ++l) s4[l] = __fadd_rn(acc[m][i][l][2 * r + c], acc[m][i][l + 4][2 * r + c]);
                            v[m] = __fadd_rn(__fadd_rn(s4[0], s4[2]), __fadd_rn(s4[1], s4[3]));
                        }
                        if (DUAL) {
                            const int f = cur.f0 + wm * 16 + gq + 8 * r;
                            if (f < p.n_out) orow[f] = __fmul_rn(ggml_silu(__fmul_rn(v[0], sc0)), __fmul_rn(v[1], sc1));
                        } else {
#pragma unroll
                            for (int m = 0; m < 2; ++m) {
                                const int f = cur.f0 + m_row[m] + gq + 8 * r;
                                if (f < p.n_out) orow[f] = __fmul_rn(v[m], sc0);
                            }
                        }
                    }
                }
            }
        cur = nxt;
    }
    if (failed && tid == 0) {
        // bounded drain of copies still in flight before the block (and its shared memory) goes away
        cp_async_wait<0>();
        for (int k = waited; k < issued; ++k) mbar_wait_bounded(&raw_full[k & 1], (uint32_t) (k >> 1) & 1u, 200000000ull);
    }
}

}  // namespace b200moe
