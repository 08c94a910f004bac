// Routing kernels: fp32 router GEMV in the reference's summation order, activation quantisers,
// softmax + top-k + renormalise, and grouping of routed rows by expert.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace b200moe {

// Activation rows quantised the way the reference CPU backend feeds its dot products
// (vec_dot_type of the weight type): Q8_0 for NVFP4 weights, Q8_K for Q3_K weights.
// Stored as separate planes so the GEMV kernels read them with aligned vector loads:
//   q      int8  [rows][K]
//   d      float [rows][K/32]   (Q8_0: float(half(amax/127)))   or  [rows][K/256] (Q8_K: 1/iscale)
//   bsum   int16 [rows][K/16]   (Q8_K only: sums of 16 quants, used for the -4 offset of Q3_K codes)
struct ActQuant {
    int8_t *  q;
    float *   d;
    int16_t * bsum;
};

// eight neighbouring values; src 16-byte aligned
__device__ __forceinline__ void load8(const float * src, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4 *>(src), b = *reinterpret_cast<const float4 *>(src + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16 * src, float (&v)[8]) {
    const uint4 a = *reinterpret_cast<const uint4 *>(src);
    const uint32_t w[4] = { a.x, a.y, a.z, a.w };
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}

// ---- K0: router logits (+ optional bias) --------------------------------------------------------
// One warp per (expert, tile of TT tokens).  Lane l owns the reference's SIMD chain l: AVX2
// ggml_vec_dot_f32 keeps 4 accumulators x 8 lanes, element i feeding accumulator (i/8)%4 lane i%8,
// i.e. chain i%32, with FMAs in increasing i.  The cross-chain reduction follows GGML_F32x8_REDUCE:
// (a0+a2),(a1+a3) -> sum -> lanes j+(j+4) -> two horizontal adds.
// Single-token tiles of bf16 activations: the eight warps of a block work for one token when E is a multiple of 8, so its row goes through
// shared memory as fp32 - 32 two-byte loads per lane cost more than the weights (one token over 128 experts 7.0 -> 6.2 us, three tokens
// over 512 experts 13 -> 11 us).  fp32 rows are read directly (3.9 us; staged, four layers of one token took 6 us more).
constexpr int ROUTER_ROW = 4096;
// CH: steps of a lane's chain whose loads are in flight together
template <int TT, typename XT, int CH = TT == 1 ? 32 : 8>
__device__ __forceinline__ void router_warp(const float * W, const float * bias, const XT * x,
                                            float * __restrict__ logits, int H, int E, int T, int warp, int lane) {
    constexpr bool STAGE = TT == 1 && sizeof(XT) == 2;
    __shared__ __align__(16) float s_x[STAGE ? ROUTER_ROW : 4];
    const int n_tt = (T + TT - 1) / TT;
    const bool row_staged = STAGE && E % 8 == 0 && H <= ROUTER_ROW;
    const int e = warp % E;
    const float * w = W + (size_t) e * H;
    float wv[CH];                              // the first steps' weights are on their way while the row is staged
#pragma unroll
    for (int c = 0; c < CH; ++c) wv[c] = STAGE && lane + 32 * c < H ? w[lane + 32 * c] : 0.0f;
    if (row_staged) {
        const XT * xr = x + (size_t) min((warp & ~7) / E, T - 1) * H;
        if (H % 8 == 0 && ((uintptr_t) xr & 15) == 0) {
            for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
                float v[8];
                load8(xr + i, v);
                *reinterpret_cast<float4 *>(s_x + i) = make_float4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<float4 *>(s_x + i + 4) = make_float4(v[4], v[5], v[6], v[7]);
            }
        } else {
            for (int i = threadIdx.x; i < H; i += blockDim.x) s_x[i] = (float) xr[i];
        }
        __syncthreads();
    }
    if (warp >= E * n_tt) return;
    const int t0 = (warp / E) * TT;
    float acc[TT];
#pragma unroll
    for (int i = 0; i < TT; ++i) acc[i] = 0.0f;
    // The FMA chain of a lane is sequential by definition of the reference's order, but its loads are not:
    // fetch CH steps of weights and activations at once, then run the chain over them.
    for (int j0 = lane; j0 < H; j0 += 32 * CH) {
        float xv[TT][CH];
        if (!STAGE || j0 != lane) {
#pragma unroll
            for (int c = 0; c < CH; ++c) wv[c] = j0 + 32 * c < H ? w[j0 + 32 * c] : 0.0f;
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const int j = j0 + 32 * c;
#pragma unroll
            for (int i = 0; i < TT; ++i) {
                const int t = min(t0 + i, T - 1);
                xv[i][c] = j >= H ? 0.0f : row_staged ? s_x[j] : (float) x[(size_t) t * H + j];
            }
        }
#pragma unroll
        for (int c = 0; c < CH; ++c)
            if (j0 + 32 * c < H) {
#pragma unroll
                for (int i = 0; i < TT; ++i) acc[i] = __fmaf_rn(wv[c], xv[i][c], acc[i]);
            }
    }
#pragma unroll
    for (int i = 0; i < TT; ++i) {
        float v = acc[i];
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));  // a0+a2 (lanes 0-7), a1+a3 (lanes 8-15)
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));   // (a0+a2)+(a1+a3)
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));   // lane j + lane j+4
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));   // hadd
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));   // hadd
        if (lane == 0 && t0 + i < T) {
            if (bias) v = __fadd_rn(v, bias[e]);
            logits[(size_t) (t0 + i) * E + e] = v;
        }
    }
}

template <int TT, typename XT, int CH = TT == 1 ? 32 : 8>
__global__ void __launch_bounds__(256) router_logits_kernel(const float * W, const float * bias,
                                                           const XT * x, float * __restrict__ logits, int H,
                                                           int E, int T, int * __restrict__ zero_buf, int zero_n) {
    pdl_wait();
    pdl_launch_dependents();

    // block 0 also clears the per-expert counters the selection kernel accumulates into
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < zero_n; i += blockDim.x) zero_buf[i] = 0;
    router_warp<TT, XT, CH>(W, bias, x, logits, H, E, T, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, threadIdx.x & 31);
}

// Register-tiled form for batches: one warp per (TE experts x TT tokens).  Every (expert, token) pair still runs the reference's
// chains - lane l owns elements l, l + 32, ... in increasing order - but a weight value now meets TT tokens and an activation value
// TE experts per load, so the kernel is bound by FMAs instead of by re-reading x once per expert from L2.
template <int TE, int TT, typename XT>
__global__ void __launch_bounds__(256) router_logits_tiled_kernel(const float * W, const float * bias,
                                                                 const XT * x, float * __restrict__ logits, int H, int E, int T,
                                                                 int * __restrict__ zero_buf, int zero_n) {
    pdl_wait();
    pdl_launch_dependents();
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < zero_n; i += blockDim.x) zero_buf[i] = 0;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int n_te = (E + TE - 1) / TE, n_tt = (T + TT - 1) / TT;
    if (warp >= n_te * n_tt) return;
    const int e0 = (warp % n_te) * TE, t0 = (warp / n_te) * TT;
    float acc[TE][TT];
#pragma unroll
    for (int a = 0; a < TE; ++a)
#pragma unroll
        for (int b = 0; b < TT; ++b) acc[a][b] = 0.0f;
    const float * wrow[TE];
    const XT * xrow[TT];
#pragma unroll
    for (int a = 0; a < TE; ++a) wrow[a] = W + (size_t) min(e0 + a, E - 1) * H;
#pragma unroll
    for (int b = 0; b < TT; ++b) xrow[b] = x + (size_t) min(t0 + b, T - 1) * H;
#pragma unroll 2
    for (int j = lane; j < H; j += 32) {
        float wv[TE], xv[TT];
#pragma unroll
        for (int a = 0; a < TE; ++a) wv[a] = wrow[a][j];
#pragma unroll
        for (int b = 0; b < TT; ++b) xv[b] = (float) xrow[b][j];
#pragma unroll
        for (int a = 0; a < TE; ++a)
#pragma unroll
            for (int b = 0; b < TT; ++b) acc[a][b] = __fmaf_rn(wv[a], xv[b], acc[a][b]);
    }
#pragma unroll
    for (int a = 0; a < TE; ++a)
#pragma unroll
        for (int b = 0; b < TT; ++b) {
            float v = acc[a][b];
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
            if (lane == 0 && e0 + a < E && t0 + b < T) {
                if (bias) v = __fadd_rn(v, bias[e0 + a]);
                logits[(size_t) (t0 + b) * E + e0 + a] = v;
            }
        }
}

// ---- activation quantisers -------------------------------------------------------------------------
// Q8_0 as the reference's AVX2 quantize_row_q8_0 (ggml-cpu/arch/x86/quants.c:302-367): d = amax/127 kept
// as half, multiplier 127/amax in fp32, round to nearest even.  One warp per 32-element block... here one
// thread per element, a warp per block.
template <typename XT>
__device__ __forceinline__ void quantize_q8_0_block(const XT * src, int8_t * __restrict__ q, float * __restrict__ d,
                                                   int lane) {
    const float v = (float) src[lane];
    float amax = fabsf(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float dd = __fdiv_rn(amax, 127.0f);
    const float id = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    q[lane] = (int8_t) __float2int_rn(__fmul_rn(v, id));
    if (lane == 0) *d = __half2float(__float2half_rn(dd));
}

// Q8_0 for eight blocks at a time: a lane holds eight neighbouring values, four lanes one block.  src 16-byte aligned.  (A lane per value
// moved 16 MB of a 4096-token prompt in 39 us.)
template <typename XT>
__device__ __forceinline__ void quantize_q8_0_span(const XT * src, int8_t * __restrict__ q, float * __restrict__ d, int lane) {
    float v[8];
    load8(src + lane * 8, v);
    float amax = fabsf(v[0]);    // not zero: a block of nothing but NaN must come out with a NaN scale, as it does a value a lane
#pragma unroll
    for (int i = 1; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float dd = __fdiv_rn(amax, 127.0f);
    const float id = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
    uint32_t w[2] = { 0u, 0u };
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i >> 2] |= ((uint32_t) __float2int_rn(__fmul_rn(v[i], id)) & 0xffu) << (8 * (i & 3));
    *reinterpret_cast<uint2 *>(q + lane * 8) = make_uint2(w[0], w[1]);
    if ((lane & 3) == 0) d[lane >> 2] = __half2float(__float2half_rn(dd));
}

// Q8_K as quantize_row_q8_K_ref (ggml-quants.c:2768-2805): the FIRST element with the largest |x| sets
// iscale = -127/x; q = min(127, nearest_int(iscale*x)); d = 1/iscale; bsums over 16.
// One warp per 256-element block, 8 elements per lane (lane owns elements 8*lane .. 8*lane+7).
// src: the lane's eight values; q: its eight bytes; d: the block's scale, the same in every lane
template <typename XT>
__device__ __forceinline__ void q8_K_words(const XT * src, int lane, uint32_t (&q)[2], float & d) {
    float v[8];
    float amax = 0.0f, mx = 0.0f;
    int arg = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = (float) src[i];
        const float a = fabsf(v[i]);
        if (a > amax) { amax = a; mx = v[i]; arg = lane * 8 + i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, amax, o);
        const float om = __shfl_xor_sync(0xffffffffu, mx, o);
        const int oi = __shfl_xor_sync(0xffffffffu, arg, o);
        if (oa > amax || (oa == amax && oi < arg)) { amax = oa; mx = om; arg = oi; }
    }
    q[0] = q[1] = 0u;
    d = 0.0f;
    if (amax == 0.0f) return;
    const float iscale = __fdiv_rn(-127.0f, mx);
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i >> 2] |= ((uint32_t) min(127, __float2int_rn(__fmul_rn(iscale, v[i]))) & 0xffu) << (8 * (i & 3));
    d = __fdiv_rn(1.0f, iscale);
}
template <typename XT>
__device__ __forceinline__ void quantize_q8_K_block(const XT * src, int8_t * __restrict__ q, float * __restrict__ d,
                                                   int16_t * __restrict__ bsum, int lane) {
    uint32_t w[2];
    float dd;
    q8_K_words(src + lane * 8, lane, w, dd);
    *reinterpret_cast<uint2 *>(q + lane * 8) = make_uint2(w[0], w[1]);
    int s = dot4((int) w[0], 0x01010101, dot4((int) w[1], 0x01010101, 0));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    if ((lane & 1) == 0) bsum[lane >> 1] = (int16_t) s;
    if (lane == 0) *d = dd;
}

// rows x K activations -> ActQuant planes.  kind: 0 = Q8_0 (32-blocks), 1 = Q8_K (256-blocks).
// src row r starts at src + r*src_stride.
// spans: K is a multiple of 256 and the rows are 16-byte aligned, so a warp takes 256 values of either kind at a time
template <typename XT>
__device__ __forceinline__ void quantize_warp(const XT * src, int64_t src_stride, const ActQuant & dst, int rows, int K, int kind, bool spans,
                                              int warp, int n_warps, int lane) {
    const int nb = K / (kind == 0 && !spans ? 32 : 256);
    for (int i = warp; i < rows * nb; i += n_warps) {
        const int r = i / nb, b = i % nb;
        const XT * row = src + (size_t) r * src_stride;
        int8_t * q = dst.q + (size_t) r * K;
        if (kind) quantize_q8_K_block(row + b * 256, q + b * 256, dst.d + (size_t) r * nb + b, dst.bsum + (size_t) r * (K / 16) + b * 16, lane);
        else if (spans) quantize_q8_0_span(row + b * 256, q + b * 256, dst.d + (size_t) r * (K / 32) + b * 8, lane);
        else quantize_q8_0_block(row + b * 32, q + b * 32, dst.d + (size_t) r * nb + b, lane);
    }
}

template <typename XT>
__global__ void __launch_bounds__(256) quantize_act_kernel(const XT * src, int64_t src_stride, ActQuant dst, int rows,
                                                          int K, int kind, int spans) {
    pdl_wait();
    pdl_launch_dependents();
    quantize_warp<XT>(src, src_stride, dst, rows, K, kind, spans != 0, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5,
                      threadIdx.x & 31);
}

// Router logits and activation quantisation in one launch (few tokens): blocks [0, n_logit_blocks) compute logits,
// the rest quantise x for the expert matmuls.  Both only read x.
template <int TT, typename XT>
__global__ void __launch_bounds__(256) route_front_kernel(const float * W, const float * bias,
                                                         const XT * x, float * __restrict__ logits, int H, int E, int T,
                                                         int * __restrict__ zero_buf, int zero_n, int n_logit_blocks, ActQuant dst,
                                                         int kind, int spans) {
    pdl_wait();
    pdl_launch_dependents();

    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if ((int) blockIdx.x < n_logit_blocks) {
        if (blockIdx.x == 0)
            for (int i = threadIdx.x; i < zero_n; i += blockDim.x) zero_buf[i] = 0;
        router_warp<TT, XT>(W, bias, x, logits, H, E, T, (int) blockIdx.x * 8 + wib, lane);
        return;
    }
    quantize_warp<XT>(x, H, dst, T, H, kind, spans != 0, ((int) blockIdx.x - n_logit_blocks) * 8 + wib, ((int) gridDim.x - n_logit_blocks) * 8, lane);
}

// Shared-memory form for larger batches: a block owns (8 WE experts) x (RT WT tokens); weight and activation rows arrive in
// 128-element pieces through a three-deep cp.async ring, and every warp runs an 8 x RT register tile out of shared memory.  Blocks from
// n_logit_blocks on quantise x for the expert matmuls instead (dst.q null: there are none).  The
// chains are the reference's (lane l owns elements l, l + 32, ... in increasing order), so the logits keep its bits; what changes is
// that global loads are 16 bytes wide, issued two pieces ahead, and shared by the whole tile.
// Needs H to be a multiple of 128 and 16-byte aligned rows.
constexpr int ROUTER_KC = 128, ROUTER_ST = 3;
template <int WE, int WT, int RT, typename XT>
constexpr size_t router_smem_bytes() { return (size_t) ROUTER_ST * ROUTER_KC * (8 * WE * sizeof(float) + RT * WT * sizeof(XT)); }

__device__ __forceinline__ void cp_async16(void * smem, const void * gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t) __cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int WE, int WT, int RT, typename XT>
__global__ void __launch_bounds__(WE * WT * 32) router_logits_smem_kernel(const float * W, const float * bias,
                                                                         const XT * x, float * __restrict__ logits, int H, int E, int T,
                                                                         int * __restrict__ zero_buf, int zero_n, int n_logit_blocks, ActQuant dst,
                                                                         int kind, int spans) {
    constexpr int EB = 8 * WE, TB = RT * WT, KC = ROUTER_KC, ST = ROUTER_ST, NTHR = WE * WT * 32;
    constexpr int XP = 16 / sizeof(XT);   // activation elements per 16-byte piece
    extern __shared__ __align__(16) uint8_t router_smem[];
    float (*ws)[EB][KC] = reinterpret_cast<float (*)[EB][KC]>(router_smem);
    XT (*xs)[TB][KC] = reinterpret_cast<XT (*)[TB][KC]>(router_smem + (size_t) ST * EB * KC * sizeof(float));
    pdl_wait();
    pdl_launch_dependents();
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < zero_n; i += NTHR) zero_buf[i] = 0;
    if ((int) blockIdx.x >= n_logit_blocks) {
        quantize_warp<XT>(x, H, dst, T, H, kind, spans != 0, ((int) blockIdx.x - n_logit_blocks) * (NTHR / 32) + (int) (threadIdx.x >> 5),
                          ((int) gridDim.x - n_logit_blocks) * (NTHR / 32), threadIdx.x & 31);
        return;
    }
    const int n_eb = (E + EB - 1) / EB;
    const int e0 = (blockIdx.x % n_eb) * EB, t0 = (blockIdx.x / n_eb) * TB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int we = (warp % WE) * 8, wt = (warp / WE) * RT;
    const int n_chunks = H / KC;

    auto load_chunk = [&](int c) {
        const int s = c % ST;
        for (int i = threadIdx.x; i < EB * (KC / 4); i += NTHR) {
            const int r = i / (KC / 4), q = i % (KC / 4);
            cp_async16(&ws[s][r][q * 4], W + (size_t) min(e0 + r, E - 1) * H + (size_t) c * KC + q * 4);
        }
        for (int i = threadIdx.x; i < TB * (KC / XP); i += NTHR) {
            const int r = i / (KC / XP), q = i % (KC / XP);
            cp_async16(&xs[s][r][q * XP], x + (size_t) min(t0 + r, T - 1) * H + (size_t) c * KC + q * XP);
        }
    };
    float acc[8][RT];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < RT; ++b) acc[a][b] = 0.0f;
#pragma unroll
    for (int c = 0; c < ST - 1; ++c) {
        if (c < n_chunks) load_chunk(c);
        cp_async_commit();
    }
    for (int c = 0; c < n_chunks; ++c) {
        cp_async_wait<ST - 2>();   // piece c has landed (one younger group may still be in flight)
        __syncthreads();           // ... for every thread, and everybody is done with the stage the next load overwrites
        if (c + ST - 1 < n_chunks) load_chunk(c + ST - 1);
        cp_async_commit();
        const int s = c % ST;
#pragma unroll
        for (int kk = 0; kk < KC / 32; ++kk) {
            float wv[8], xv[RT];
#pragma unroll
            for (int a = 0; a < 8; ++a) wv[a] = ws[s][we + a][kk * 32 + lane];
#pragma unroll
            for (int b = 0; b < RT; ++b) xv[b] = (float) xs[s][wt + b][kk * 32 + lane];
#pragma unroll
            for (int a = 0; a < 8; ++a)
#pragma unroll
                for (int b = 0; b < RT; ++b) acc[a][b] = __fmaf_rn(wv[a], xv[b], acc[a][b]);
        }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < RT; ++b) {
            float v = acc[a][b];
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
            v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
            const int e = e0 + we + a, t = t0 + wt + b;
            if (lane == 0 && e < E && t < T) {
                if (bias) v = __fadd_rn(v, bias[e]);
                logits[(size_t) t * E + e] = v;
            }
        }
}

// ---- K1: softmax + top-k + renormalise, one warp per token ---------------------------------------------
// soft_max (ggml-cpu/ops.cpp:5584-5694, vec.cpp:531-551): exp via ggml_v_expf, groups of 8 summed in fp32 as
// ((v0+v4)+(v2+v6))+((v1+v5)+(v3+v7)), groups accumulated in double, p = exp * (float)(1/sum).
// top-k = argsort descending, first k (ggml.c:5441-5455); equal values: lower index first.
// weights = p[ids] / max((float)sum_double(p[ids]), 2^-14) (forward.cpp:268-269).
// Also counts rows per expert and remembers each row's arrival position for the grouping kernel.
template <int EPL>  // experts per lane; E <= 32*EPL, E % 8 == 0
__device__ __forceinline__ void route_select_token(const float * logits, int E, int K, int t, int lane,
                                                   int32_t * __restrict__ ids, float * __restrict__ weights,
                                                   float * __restrict__ probs_out, int * __restrict__ counts,
                                                   int * __restrict__ pos) {
    const float * l = logits + (size_t) t * E;

    // lane owns experts e = lane*EPL + i  (contiguous, so a group of 8 experts sits in 8/EPL lanes or one lane)
    float p[EPL];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
        const int e = lane * EPL + i;
        p[i] = e < E ? l[e] : -INFINITY;
        mx = fmaxf(mx, p[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
        const int e = lane * EPL + i;
        p[i] = e < E ? ggml_expf(__fsub_rn(p[i], mx)) : 0.0f;
    }
    // group-of-8 sums in the reference's order, then the double accumulation over groups in index order.  A group's values v0..v7 sit in
    // one lane (EPL >= 8) or in 8 / EPL neighbouring lanes, so each step of ((v0+v4)+(v2+v6))+((v1+v5)+(v3+v7)) is an addition inside the lane
    // or one exchange with the lane that holds the partner (addition commutes: both ends get the same bits).
    constexpr int GPL = EPL >= 8 ? EPL / 8 : 1;   // groups a lane holds
    float gs[GPL];
#pragma unroll
    for (int q = 0; q < GPL; ++q) {
        constexpr int N = EPL < 8 ? EPL : 8;
        float v[N];
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = p[8 * q + i];
#pragma unroll
        for (int step = 4; step > 0; step >>= 1) {
            if (step >= N) {
#pragma unroll
                for (int i = 0; i < N; ++i) v[i] = __fadd_rn(v[i], __shfl_xor_sync(0xffffffffu, v[i], step / N));
            } else {
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (i < step) v[i] = __fadd_rn(v[i], v[i + step]);
            }
        }
        gs[q] = v[0];
    }
    double sum = 0.0;
    if (EPL >= 8) {
        for (int o = 0; o * EPL < E; ++o) {
#pragma unroll
            for (int q = 0; q < GPL; ++q) {
                const float g = __shfl_sync(0xffffffffu, gs[q], o);
                if (o * EPL + 8 * q < E) sum += (double) g;
            }
        }
    } else {
        for (int g = 0; g < E / 8; ++g) sum += (double) __shfl_sync(0xffffffffu, gs[0], g * (8 / (EPL < 8 ? EPL : 8)));
    }
    const float inv = (float) (1.0 / sum);
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
        p[i] = __fmul_rn(p[i], inv);
        const int e = lane * EPL + i;
        if (probs_out && e < E) probs_out[(size_t) t * E + e] = p[i];
    }

    // iterative arg-max, K rounds; ties -> lower expert index
    float sel_p = 0.0f;
    int sel_e = -1;
    double wsum = 0.0;
    uint32_t taken = 0;  // bit i: p[i] already selected
    for (int k = 0; k < K; ++k) {
        float best = -1.0f;
        int best_e = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < EPL; ++i) {
            const int e = lane * EPL + i;
            if (e < E && !((taken >> i) & 1u) && p[i] > best) { best = p[i]; best_e = e; }
        }
        // candidates are not negative, so their bits order as they do; 0 marks a lane without one (all taken, or NaN)
        const uint32_t key = best >= 0.0f ? __float_as_uint(fabsf(best)) + 1u : 0u;
        const uint32_t top = __reduce_max_sync(0xffffffffu, key);
        best_e = (int) __reduce_min_sync(0xffffffffu, key == top ? (uint32_t) best_e : 0x7fffffffu);
        best = top ? __uint_as_float(top - 1u) : -1.0f;
        if (best_e / EPL == lane) taken |= 1u << (best_e % EPL);
        if (lane == k) { sel_p = best; sel_e = best_e; }
        wsum += (double) best;  // sum_rows accumulates in double in slot order (ggml-cpu/vec.h:1495-1505)
    }
    float den = (float) wsum;
    den = fmaxf(den, 6.103515625e-5f);
    if (lane < K) {
        // NaN logits leave no candidate; keep the index in range so nothing downstream is addressed with it
        sel_e = sel_e < 0 ? 0 : (sel_e >= E ? E - 1 : sel_e);
        ids[(size_t) t * K + lane] = sel_e;
        weights[(size_t) t * K + lane] = __fdiv_rn(sel_p, den);
        if (counts) pos[(size_t) t * K + lane] = atomicAdd(&counts[sel_e], 1);
    }
}

template <int EPL>
__global__ void __launch_bounds__(256) route_select_kernel(const float * logits, int E, int K, int T,
                                                          int32_t * __restrict__ ids, float * __restrict__ weights,
                                                          float * __restrict__ probs_out, int * __restrict__ counts,
                                                          int * __restrict__ pos) {
    pdl_wait();
    pdl_launch_dependents();

    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= T) return;
    route_select_token<EPL>(logits, E, K, t, threadIdx.x & 31, ids, weights, probs_out, counts, pos);
}

// ---- K2: grouping ----------------------------------------------------------------------------------------
// Group descriptor produced for the expert kernels (reference: matrix_rows / matrix_row_counts in
// ggml_compute_forward_mul_mat_id, ggml-cpu/ggml-cpu.c:1648-1663):
//   offsets[e]   first slot of expert e in perm, offsets[E] = total rows
//   perm[i]      routed row index (token*K + slot) placed i-th
//   active[a]    a-th expert that has at least one row; n_active in meta[0], total rows in meta[1]
// routed rows per token tile of the FP4 tensor-core kernels (6 digit planes each): few and many rows per expert
constexpr int TOKEN_TILE_SMALL = 14, TOKEN_TILE_LARGE = 27;

// Work per weight row of the NVFP4 integer kernel for n routed rows: passes of four, or of two or one for what is left.  A pass of one
// or two costs nearly what one of four does, the decode being most of it.
__host__ __device__ __forceinline__ constexpr int nvfp4_work(int n) { return n / 4 * 16 + (n % 4 == 0 ? 0 : n % 4 == 1 ? 10 : n % 4 == 2 ? 12 : 16); }

// The same for Q3_K in passes of TOK (16 or 32) routed rows, eight at a time: the decode is worth four times eight rows.
template <int TOK>
__host__ __device__ __forceinline__ constexpr int q3k_work(int n) { return n / TOK * (4 + TOK / 8) + (n % TOK ? 4 + (n % TOK + 7) / 8 : 0); }

struct Groups {
    int * counts;   // [E]
    int * offsets;  // [E+1]
    int * pos;      // [rows]
    int * perm;     // [rows]
    int * active;   // [E]
    int * meta;     // [4]: number of active experts, rows in a group, two counters of the re-quantisation fix-up (cleared by the grouping)
    int * cost;     // [4][E+1]: rows 0-2: prefix over active experts of the work per weight row for the integer kernels: Q3_K with 16
                    // routed rows to a pass (q3k_work), NVFP4 (nvfp4_work), Q3_K with 32;
                    // row 3, indexed by EXPERT id: index of the expert's first token tile (prefix of ceil(rows / tile_rows))
    int tile_rows;  // TOKEN_TILE_SMALL or TOKEN_TILE_LARGE
    int * done;     // [n_done] arrival counters of the one-or-two-token down kernel (GemvParams::comb_cnt), cleared by the grouping
    int n_done;
};

// Block-wide: counts must be final and visible to this block.  With several blocks every one scans the counts for itself (a
// microsecond) and fills its share of perm, which is what takes long with thousands of rows; block 0 writes the tables.
// allow_empty: ids equal to -1 mark routed rows that do not exist (empty slots of an expert-parallel exchange): they are in no group.
__device__ __forceinline__ void group_scan_body(Groups g, const int32_t * ids, int E, int rows, int * err, int * sh, bool allow_empty = false,
                                                int block = 0, int n_blocks = 1) {
    if (block == 0)
        for (int i = threadIdx.x; i < g.n_done; i += blockDim.x) g.done[i] = 0;
    // thread = expert (the launchers use 1024 threads, the largest expert count): a scan per warp, then one over the warps' totals
    int * off = sh;                      // [E]
    __shared__ int s_tot[7][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = tid < E ? g.counts[tid] : 0;
    // rows; active experts; work per weight row of the Q3_K kernel of few rows, of NVFP4's and of the Q3_K kernel of many; token tiles
    constexpr int N = 6;
    const int own[N] = { n, n > 0 ? 1 : 0, q3k_work<16>(n), nvfp4_work(n), q3k_work<32>(n), (n + g.tile_rows - 1) / g.tile_rows };
    int v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = own[i];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int up = __shfl_up_sync(0xffffffffu, v[i], o);
            if (lane >= o) v[i] += up;
        }
    if (lane == 31)
#pragma unroll
        for (int i = 0; i < N; ++i) s_tot[i][warp] = v[i];
    __syncthreads();
    if (warp < N) {
        const int own_t = lane < (int) (blockDim.x >> 5) ? s_tot[warp][lane] : 0;
        int t = own_t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += up;
        }
        s_tot[warp][lane] = t - own_t;
        if (lane == 31) s_tot[N][warp] = t;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += s_tot[i][warp] - own[i];     // exclusive prefixes
    if (tid < E) {
        off[tid] = v[0];
        if (block == 0) {
            g.offsets[tid] = v[0];
            g.cost[3 * (E + 1) + tid] = v[5];
            if (n > 0) {
                g.active[v[1]] = tid;
#pragma unroll
                for (int i = 0; i < 3; ++i) g.cost[i * (E + 1) + v[1]] = v[2 + i];
            }
        }
    }
    if (tid == 0 && block == 0) {
        const int run = s_tot[N][0], na = s_tot[N][1];
        g.offsets[E] = run;
#pragma unroll
        for (int i = 0; i < 3; ++i) g.cost[i * (E + 1) + na] = s_tot[N][2 + i];
        g.cost[3 * (E + 1) + E] = s_tot[N][5];
        g.meta[0] = na;
        g.meta[1] = run;
        g.meta[2] = g.meta[3] = 0;       // the counters of the re-quantisation fix-up
        if (allow_empty ? run > rows : run != rows) report_error(err, DEV_ERR_BAD_SHAPE);
    }
    __syncthreads();
    for (int r = block * blockDim.x + tid; r < rows; r += n_blocks * blockDim.x) {
        const int e = ids[r];
        if (allow_empty && e == -1) continue;
        if (e < 0 || e >= E) { report_error(err, DEV_ERR_BAD_EXPERT_ID); continue; }
        g.perm[off[e] + g.pos[r]] = r;
    }
}

// The grouping of a dense product: rows in order, gsize of them to a group (one launch instead of fill, count and scan; the same tables
// as group_scan_body leaves).
__global__ void __launch_bounds__(256) dense_groups_kernel(Groups g, int32_t * __restrict__ ids, int T, int gsize) {
    pdl_wait();
    pdl_launch_dependents();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < T) { ids[t] = t / gsize; g.perm[t] = t; g.pos[t] = t % gsize; }
    const int G = (T + gsize - 1) / gsize;
    if (t <= G) {
        // prefixes over t groups: all of gsize rows but for the last group
        const int last = T - (G - 1) * gsize, full = min(t, G - 1), tail = t == G ? 1 : 0;
        g.offsets[t] = full * gsize + tail * last;
        g.cost[t] = full * q3k_work<16>(gsize) + tail * q3k_work<16>(last);
        g.cost[(G + 1) + t] = full * nvfp4_work(gsize) + tail * nvfp4_work(last);
        g.cost[2 * (G + 1) + t] = full * q3k_work<32>(gsize) + tail * q3k_work<32>(last);
        g.cost[3 * (G + 1) + t] = full * ((gsize + g.tile_rows - 1) / g.tile_rows) + tail * ((last + g.tile_rows - 1) / g.tile_rows);
        if (t < G) g.active[t] = t;
    }
    if (t == 0) { g.meta[0] = G; g.meta[1] = T; g.meta[2] = g.meta[3] = 0; }
}

// counts must be final (selection kernel finished).
__global__ void __launch_bounds__(1024) group_scan_kernel(Groups g, const int32_t * ids, int E, int rows, int * err, int allow_empty) {
    pdl_wait();
    pdl_launch_dependents();

    extern __shared__ int sh[];  // [E] offsets
    group_scan_body(g, ids, E, rows, err, sh, allow_empty != 0, blockIdx.x, gridDim.x);
}

// Small batches: selection for every token and the grouping in ONE single-block launch (one warp per token, looping).
// grouped = 0: one or two tokens, whose kernels read the ids; only their arrival counters are cleared.
template <int EPL>
__global__ void __launch_bounds__(1024) route_select_group_kernel(const float * logits, int E, int K, int T,
                                                                 int32_t * __restrict__ ids, float * __restrict__ weights,
                                                                 float * __restrict__ probs_out, Groups g, int * err, int grouped) {
    pdl_wait();
    pdl_launch_dependents();

    extern __shared__ int sh[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int t = warp; t < T; t += nw) route_select_token<EPL>(logits, E, K, t, lane, ids, weights, probs_out, grouped ? g.counts : nullptr, g.pos);
    if (!grouped) {
        for (int i = threadIdx.x; i < g.n_done; i += blockDim.x) g.done[i] = 0;
        return;
    }
    __syncthreads();  // global writes of this block (counts, pos, ids) are visible to the whole block afterwards
    group_scan_body(g, ids, E, T * K, err, sh);
}

// Counting pass for routing that was not produced by route_select_kernel (ids given by the caller,
// possibly as a strided view: row t starts at ids + t*ids_stride).  Writes compact ids as well.
__global__ void __launch_bounds__(256) count_ids_kernel(const int32_t * ids, int64_t ids_stride, int n_ids, int T, int E,
                                                       int32_t * __restrict__ ids_compact, int * __restrict__ counts,
                                                       int * __restrict__ pos, int * err, int allow_empty = 0) {
    pdl_wait();
    pdl_launch_dependents();

    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_ids * T) return;
    const int t = r / n_ids, s = r % n_ids;
    const int e = ids[(size_t) t * ids_stride + s];
    ids_compact[r] = e;
    if (allow_empty && e == -1) { pos[r] = 0; return; }
    if (e < 0 || e >= E) { report_error(err, DEV_ERR_BAD_EXPERT_ID); pos[r] = 0; return; }
    pos[r] = atomicAdd(&counts[e], 1);
}

}  // namespace b200moe
