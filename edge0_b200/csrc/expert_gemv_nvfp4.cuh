// Grouped NVFP4 expert matmul on the integer chains, bit-identical to the reference (see expert_gemv.cuh for the order of its sums): the
// indexed matmul as an operator, `down` of latent prompts, dense products of a few tokens.
//
// Four threads play the eight SIMD lanes of a weight row (two_lane_chains), eight rows to a warp, up to four routed rows to a pass.  A CTA
// of eight consumer warps takes items of 64 weight rows and one pass; their bytes arrive in K = 256 pieces as tiled copies of [8 rows][144
// bytes], one per warp and tensor, through a ring that a producer warp keeps ahead of them.  Pieces of that shape because their rows lie 36
// words apart - the 8 x 4 words a warp reads together fall on 32 different banks, where whole rows (K = 2048: 288 words apart) met on four -
// and because a ring of them leaves room for two or three CTAs on an SM at every width.  A further pass over an expert's rows brings them
// from L2 again; cutting the passes, too, over the CTAs is what fills the GPU when an expert has few weight rows and many routed ones.
// What bounds it is the arithmetic unit of integers and permutes (half rate: 15 of them per eight codes and row) and the issue of the rest.
// A lane to a thread, whole rows in the ring, spans of weight rows with all passes, us: 320 routed rows over 128 experts, 2048 -> 768, 104,
// now 57 (two CTAs on an SM instead of three 61); whole calls: 1024 rows 264, now 143; 3200 over 8 experts, 256 -> 512, 604, now 53.
#pragma once
#include "expert_gemm.cuh"
#include "expert_gemv.cuh"

namespace b200moe {

template <int K, bool DUAL>
struct Nvfp4GemvCfg {
    static constexpr int NT = 4;                              // routed rows to a pass
    static constexpr int WARPS = 8, ROWS = 8 * WARPS;         // consumer warps; weight rows of a chunk
    static constexpr int NTENS = DUAL ? 2 : 1;
    static constexpr int KC = K / 256;
    static constexpr int BOX = 8 * GEMM_RAW_ROW;              // a warp's rows of a piece
    static constexpr int STAGE = WARPS * BOX * NTENS;
    static constexpr int CTAS = DUAL || K > 2048 ? 2 : 3;
    static constexpr int STAGES = DUAL ? 4 : CTAS == 3 ? 6 : 8;
    static constexpr int ACT_D = K / 32;
    static constexpr int ACTS = NT * (K + 4 * ACT_D);
    static constexpr size_t SMEM = (size_t) STAGES * STAGE + ACTS + 256 * 4;
    static constexpr int THREADS = WARPS * 32 + 32;
    static_assert(K % 256 == 0 && BOX % 128 == 0 && CTAS * (SMEM + 2048) <= 228 * 1024, "the CTAs fit an SM, boxes keep their alignment");
};

template <int K, bool DUAL>
__global__ void __launch_bounds__(Nvfp4GemvCfg<K, DUAL>::THREADS, Nvfp4GemvCfg<K, DUAL>::CTAS)
nvfp4_gemv_kernel(const GemvParams p, const __grid_constant__ CUtensorMap map_w0, const __grid_constant__ CUtensorMap map_w1) {
    using C = Nvfp4GemvCfg<K, DUAL>;
    constexpr int NT = C::NT, NTENS = C::NTENS, CONSUMERS = C::WARPS * 32;
    extern __shared__ __align__(128) uint8_t nv4_smem[];
    uint8_t * const ring = nv4_smem;
    uint32_t * const acts = reinterpret_cast<uint32_t *>(ring + (size_t) C::STAGES * C::STAGE);   // [unit][act_slot][NT]
    float * const dys = reinterpret_cast<float *>(acts) + K / 4 * NT;                             // [unit][NT]
    float * const ue_tab = dys + C::ACT_D * NT;
    __shared__ uint64_t full[C::STAGES], empty[C::STAGES];
    __shared__ volatile int s_abort;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], C::WARPS); }
        mbar_fence_init();
        s_abort = 0;
    }
    if (tid < 256) ue_tab[tid] = ue4m3_half_to_f32(tid);
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();

    const int n_active = p.meta[0];
    const int * const cw = p.cost + (p.n_as + 1);
    // Chunks of 64 weight rows; while there are items for less than every CTA, of as few rows as leaves one to a CTA.  (A pass is 10 to 16 of
    // the work; of one group, a dense product of a few tokens, the passes are known, and twice as many would leave half of the CTAs out:
    // 2048 -> 8192, 3 tokens 24.8 us, so 19.0.)
    const long long passes = n_active == 1 ? (p.meta[1] + NT - 1) / NT : (cw[n_active] + 9) / 10;
    int log_rows = 3;                                        // boxes of eight rows each
    while (8 * C::WARPS >> log_rows > 1 && passes * ((p.n_out + (1 << log_rows) - 1) >> log_rows) > gridDim.x) ++log_rows;
    const int chunk_rows = 1 << log_rows, boxes = chunk_rows / 8;
    auto span = pass_span<C::THREADS, NT, 16>(cw, n_active, (p.n_out + chunk_rows - 1) >> log_rows);

    if (warp == C::WARPS) {
        // ---------------------------------------------------------------- weight producer
        Ring st;
        int at = -1, e = 0, n_e = 0;
        for (; !s_abort && span.more(); span.next(n_e)) {
            if (span.a != at) {
                at = span.a;
                e = p.active[at];
                n_e = p.offsets[e + 1] - p.offsets[e];
            }
            const int r0 = span.ch * chunk_rows, row0 = e * p.w_stride + r0, live = min(boxes, (p.n_out - r0) / 8);
            for (int kc = 0; kc < C::KC; ++kc) {
                if (!__all_sync(0xffffffffu, wait_or_abort<40>(&empty[st.stage], st.phase ^ 1u, &s_abort, p.err))) break;
                uint8_t * dst = ring + (size_t) st.stage * C::STAGE;
                if (lane == 0) mbar_arrive_expect_tx(&full[st.stage], (uint32_t) (live * C::BOX * NTENS));
                __syncwarp();
                const int b = lane & 15;
                if (b < live && lane < 16) tma_load_2d(dst + b * C::BOX, &map_w0, kc * GEMM_RAW_ROW, row0 + 8 * b, &full[st.stage]);
                if (DUAL && b < live && lane >= 16) tma_load_2d(dst + (C::WARPS + b) * C::BOX, &map_w1, kc * GEMM_RAW_ROW, row0 + 8 * b, &full[st.stage]);
                st.template advance<C::STAGES>();
            }
        }
    } else {
        // ---------------------------------------------------------------- chains
        // Every consumer warp walks every item and meets the others at the same barriers; after an abort they walk on without work.
        auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(CONSUMERS) : "memory"); };
        const int m = lane & 3, g = lane >> 2;
        int at = -1, row_beg = 0, n_e = 0, loaded = -1, my_row = 0;      // of the expert; the pass whose activations are in place
        float sc0 = 1.0f, sc1 = 1.0f;
        Ring st;
        for (; span.more(); span.next(n_e)) {
            if (span.a != at) {
                at = span.a;
                const int e = p.active[at], se = p.w_stride ? e : 0;     // every group of a dense product has the one matrix and its scale
                row_beg = p.offsets[e];
                n_e = p.offsets[e + 1] - row_beg;
                if (p.scale0) sc0 = p.scale0[se];
                if (DUAL && p.scale1) sc1 = p.scale1[se];
                loaded = -1;
            }
            const int r0 = span.ch * chunk_rows, t0 = 4 * span.ps;
            const int n = min(NT, n_e - t0);                             // routed rows of the pass: one or two run narrower chains
            const bool mine = warp < min(boxes, (p.n_out - r0) / 8);
            if (loaded != span.ps) {
                // the activation rows of this pass into shared memory; the loads of all four are in flight together
                size_t arow[NT];
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const int r = p.perm[row_beg + t0 + (t < n ? t : 0)];
                    arow[t] = (size_t) ((r / p.n_ids) * p.ne11 + (r % p.n_ids) % p.ne11);
                    if (t == m) my_row = r;
                }
                meet();
                if (p.act_f32) {
                    // Q8_0 on the fly, the arithmetic of quantize_q8_0_block: 8 lanes hold one block of 32 (4 values each)
                    for (int i0 = 0; i0 < K / 4; i0 += CONSUMERS) {
                        const int i = i0 + tid;
                        const bool in = i < K / 4;
                        float4 v[NT];
#pragma unroll
                        for (int t = 0; t < NT; ++t)
                            v[t] = in && t < n ? reinterpret_cast<const float4 *>(p.act_f32 + arow[t] * K)[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        uint32_t q[NT];
                        float d[NT];
#pragma unroll
                        for (int t = 0; t < NT; ++t) {
                            float amax = fmaxf(fmaxf(fabsf(v[t].x), fabsf(v[t].y)), fmaxf(fabsf(v[t].z), fabsf(v[t].w)));
                            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
                            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
                            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
                            const float id = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
                            q[t] = ((uint32_t) __float2int_rn(__fmul_rn(v[t].x, id)) & 0xffu) | (((uint32_t) __float2int_rn(__fmul_rn(v[t].y, id)) & 0xffu) << 8) |
                                   (((uint32_t) __float2int_rn(__fmul_rn(v[t].z, id)) & 0xffu) << 16) | (((uint32_t) __float2int_rn(__fmul_rn(v[t].w, id)) & 0xffu) << 24);
                            d[t] = __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
                        }
                        if (in) {
                            *reinterpret_cast<uint4 *>(acts + (size_t) ((i & ~7) | act_slot(i & 7)) * NT) = make_uint4(q[0], q[1], q[2], q[3]);
                            if ((i & 7) == 0) *reinterpret_cast<float4 *>(dys + (i >> 3) * NT) = make_float4(d[0], d[1], d[2], d[3]);
                        }
                    }
                } else {
                    for (int i = tid; i < K / 4; i += CONSUMERS) {
                        uint32_t q[NT];
#pragma unroll
                        for (int t = 0; t < NT; ++t) q[t] = t < n ? reinterpret_cast<const uint32_t *>(p.act.q + arow[t] * K)[i] : 0u;
                        *reinterpret_cast<uint4 *>(acts + (size_t) ((i & ~7) | act_slot(i & 7)) * NT) = make_uint4(q[0], q[1], q[2], q[3]);
                    }
                    if (tid < C::ACT_D) {
                        float d[NT];
#pragma unroll
                        for (int t = 0; t < NT; ++t) d[t] = t < n ? p.act.d[arow[t] * C::ACT_D + tid] : 0.0f;
                        *reinterpret_cast<float4 *>(dys + tid * NT) = make_float4(d[0], d[1], d[2], d[3]);
                    }
                }
                meet();
                loaded = span.ps;
            }
            float val[NTENS] = {};                       // thread m of a row ends up with the sums of routed row t0 + m
            auto run = [&](auto ntag) {
                constexpr int NTC = decltype(ntag)::value;
                TwoLaneAcc<NTENS, NTC> acc;
                acc.clear();
#pragma unroll 1
                for (int kc = 0; kc < C::KC; ++kc) {
                    const bool ok = __all_sync(0xffffffffu, wait_or_abort(&full[st.stage], st.phase, &s_abort, p.err));
                    if (ok && mine) {
                        const uint8_t * blk[NTENS];
#pragma unroll
                        for (int r = 0; r < NTENS; ++r) blk[r] = ring + (size_t) st.stage * C::STAGE + (r * C::WARPS + warp) * C::BOX + g * GEMM_RAW_ROW;
                        two_lane_chains<NTENS, NTC, NT>(blk, m, acts + kc * 64 * NT, dys + kc * 8 * NT, ue_tab, acc);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[st.stage]);
                    st.template advance<C::STAGES>();
                }
#pragma unroll
                for (int r = 0; r < NTENS; ++r)
#pragma unroll
                    for (int t = 0; t < NTC; ++t) {
                        float lo, hi;
                        acc.lanes(r, t, lo, hi);
                        const float v = hsum_two_lanes(lo, hi);
                        if (m == t) val[r] = v;
                    }
            };
            if (n >= 3) run(std::integral_constant<int, 4>{});
            else if (n == 2) run(std::integral_constant<int, 2>{});
            else run(std::integral_constant<int, 1>{});
            if (mine && m < n) {
                float v = __fmul_rn(val[0], sc0);
                if (DUAL) v = __fmul_rn(ggml_silu(v), __fmul_rn(val[NTENS - 1], sc1));
                p.out[(size_t) my_row * p.n_out + r0 + 8 * warp + g] = v;
            }
        }
    }
    if (s_abort) {   // copies still in flight land before the block (and its shared memory) goes away
        const uint64_t t = global_timer_ns();
        while (global_timer_ns() - t < 1000000ull) { }
    }
    __syncthreads();
}

}  // namespace b200moe
