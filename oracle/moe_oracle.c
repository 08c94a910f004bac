/* TEST INFRASTRUCTURE — not product code.
 *
 * Plain-C, scalar restatement of the reference's quantised MoE-FFN path as the vendored ggml CPU
 * backend computes it when built for AVX2+FMA+F16C (the ISA the checker build of the reference is
 * pinned to).  Every SIMD lane of the reference is emulated as a scalar so that fp32 summation
 * order, FMA placement and rounding modes are the same; the restatement is meant to agree with the
 * compiled reference bit for bit, which tests/test_oracle_vs_ref.py checks, and the golden fixtures
 * under tests/golden/ (generated by the compiled reference) pin it where the reference sources are
 * not available.
 *
 * Paths are relative to edge0-infer/third_party/ggml/src/ unless they start with edge0-infer/.
 *
 * quantize_row_q3_K_ref (ggml-quants.c:1229-1303 with make_q3_quants, :697-754) is restated too, although it is not on the
 * measured path: it creates the Q3_K inputs of the tests where the compiled reference is not at hand.
 */
#define _GNU_SOURCE
#include "moe_oracle.h"

#include <math.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>
#include <time.h>
#include <unistd.h>

#define QK_K 256
#define QK8_0 32
#define QK_NVFP4 64
#define QK_NVFP4_SUB 16

/* block layouts: ggml-common.h:221-227 (nvfp4), :252-255 (q8_0), :315-321 (q3_K), :371-376 (q8_K) */
#pragma pack(push, 1)
typedef struct { uint8_t d[4]; uint8_t qs[32]; } blk_nvfp4;                                 /* 36 B / 64  */
typedef struct { uint16_t d; int8_t qs[32]; } blk_q8_0;                                     /* 34 B / 32  */
typedef struct { uint8_t hmask[32]; uint8_t qs[64]; uint8_t scales[12]; uint16_t d; } blk_q3_K; /* 110 B / 256 */
typedef struct { float d; int8_t qs[256]; int16_t bsums[16]; } blk_q8_K;                     /* 292 B / 256 */
#pragma pack(pop)

/* ggml-common.h:1126-1128: E2M1 values doubled */
static const int8_t kvalues_fp4[16] = { 0, 1, 2, 3, 4, 6, 8, 12, 0, -1, -2, -3, -4, -6, -8, -12 };

static inline uint32_t f2u(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static inline float u2f(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }

int64_t orc_row_size(int type, int64_t n) {
    switch (type) {
        case ORC_TYPE_F32:   return n * 4;
        case ORC_TYPE_Q3_K:  return n / QK_K * (int64_t) sizeof(blk_q3_K);
        case ORC_TYPE_NVFP4: return n / QK_NVFP4 * (int64_t) sizeof(blk_nvfp4);
        case 8:              return n / QK8_0 * (int64_t) sizeof(blk_q8_0);
        case 15:             return n / QK_K * (int64_t) sizeof(blk_q8_K);
        default:             return -1;
    }
}

/* ---- IEEE half <-> float, round to nearest even (what F16C's vcvtps2ph / vcvtph2ps do;
 *      ggml-cpu/simd-mappings.h maps GGML_CPU_FP32_TO_FP16 to them on x86 with F16C) */
float orc_fp16_to_fp32(uint16_t h) {
    const uint32_t sign = (uint32_t)(h & 0x8000u) << 16;
    const uint32_t exp = (h >> 10) & 0x1f;
    const uint32_t man = h & 0x3ffu;
    if (exp == 0) {
        if (man == 0) return u2f(sign);
        float v = ldexpf((float) man, -24);
        return (sign ? -v : v);
    }
    if (exp == 31) return u2f(sign | 0x7f800000u | (man << 13));
    return u2f(sign | ((exp + 112) << 23) | (man << 13));
}

uint16_t orc_fp32_to_fp16(float f) {
    const uint32_t u = f2u(f);
    const uint16_t sign = (uint16_t)((u >> 16) & 0x8000u);
    const uint32_t a = u & 0x7fffffffu;
    if (a >= 0x7f800000u) return (uint16_t)(sign | 0x7c00u | ((a > 0x7f800000u) ? 0x200u : 0));
    if (a >= 0x477ff000u) return (uint16_t)(sign | 0x7c00u);           /* rounds to inf (>= 65520) */
    if (a < 0x33000001u) return sign;                                   /* <= 2^-25 rounds to zero */
    int exp = (int)(a >> 23) - 127;
    uint32_t man = (a & 0x7fffffu) | 0x800000u;
    int shift;
    uint32_t base;
    if (exp < -14) { shift = 13 + (-14 - exp); base = 0; }              /* subnormal half */
    else { shift = 13; base = (uint32_t)(exp + 15) << 10; man &= 0x7fffffu; }
    uint32_t q = man >> shift;
    const uint32_t rem = man & ((1u << shift) - 1);
    const uint32_t half = 1u << (shift - 1);
    if (rem > half || (rem == half && (q & 1))) q++;
    return (uint16_t)(sign | (base + q));                               /* carry into exponent is correct */
}

/* ---- UE4M3 codec: ggml-impl.h:514-565 (decode returns value*0.5 to pair with the doubled E2M1 table) */
float orc_ue4m3_to_fp32(uint8_t x) {
    if (x == 0 || x == 0x7F) return 0.0f;
    const int exp = (x >> 3) & 0xF, man = x & 0x7;
    float raw = exp == 0 ? ldexpf((float) man, -9) : ldexpf(1.0f + (float) man / 8.0f, exp - 7);
    return raw * 0.5f;
}

uint8_t orc_fp32_to_ue4m3(float x) {
    if (!(x > 0.0f)) return 0;
    if (x > 448.0f) x = 448.0f;
    const uint32_t bits = f2u(x);
    const int fp32_exp = (int)((bits >> 23) & 0xFF) - 127;
    const int fp32_man = (bits >> 20) & 0x7;
    int ue_exp = fp32_exp + 7;
    if (ue_exp <= 0) {
        int man = (int)(x * 512.0f + 0.5f);
        if (man > 7) man = 7;
        if (man < 1) return 0;
        return (uint8_t) man;
    }
    if (ue_exp >= 15) return 0x7E;
    const int round_bit = (bits >> 19) & 1;
    int ue_man = fp32_man + round_bit;
    if (ue_man > 7) { ue_man = 0; ue_exp++; if (ue_exp >= 15) return 0x7E; }
    return (uint8_t)((ue_exp << 3) | ue_man);
}

/* ---- NVFP4 weight quantiser / dequantiser: ggml-quants.c:337-348, 384-417, 589-612 */
static int best_index_fp4(float x, float e) {
    int best = 0;
    float best_err = fabsf(kvalues_fp4[0] * e - x);
    for (int i = 1; i < 16; i++) {
        float err = fabsf(kvalues_fp4[i] * e - x);
        if (err < best_err) { best = i; best_err = err; }
    }
    return best;
}

void orc_quantize_row_nvfp4(const float * x, void * vy, int64_t k) {
    blk_nvfp4 * y = (blk_nvfp4 *) vy;
    const int64_t nb = k / QK_NVFP4;
    for (int64_t i = 0; i < nb; i++) {
        for (int s = 0; s < 4; s++) {
            const float * xb = x + i * QK_NVFP4 + s * QK_NVFP4_SUB;
            float amax = 0.0f;
            for (int j = 0; j < QK_NVFP4_SUB; j++) if (amax < fabsf(xb[j])) amax = fabsf(xb[j]);
            const uint8_t ue = orc_fp32_to_ue4m3(amax / 6.0f);
            y[i].d[s] = ue;
            const float d = orc_ue4m3_to_fp32(ue);
            for (int j = 0; j < 8; ++j) {
                const uint8_t x0 = (uint8_t) best_index_fp4(xb[j], d);
                const uint8_t x1 = (uint8_t) best_index_fp4(xb[8 + j], d);
                y[i].qs[s * 8 + j] = (uint8_t)(x0 | (x1 << 4));
            }
        }
    }
}

void orc_dequantize_row_nvfp4(const void * vx, float * y, int64_t k) {
    const blk_nvfp4 * x = (const blk_nvfp4 *) vx;
    const int64_t nb = k / QK_NVFP4;
    for (int64_t i = 0; i < nb; i++) {
        for (int s = 0; s < 4; s++) {
            const float d = orc_ue4m3_to_fp32(x[i].d[s]);
            float * yb = y + i * QK_NVFP4 + s * QK_NVFP4_SUB;
            for (int j = 0; j < 8; ++j) {
                yb[j]     = kvalues_fp4[x[i].qs[s * 8 + j] & 0x0F] * d;
                yb[j + 8] = kvalues_fp4[x[i].qs[s * 8 + j] >> 4] * d;
            }
        }
    }
}

/* 6-bit sub-block scales of a Q3_K super-block, as signed values (scale - 32):
 * unpacking of ggml-quants.c:1322-1327 */
static void q3k_scales(const uint8_t * sc12, int8_t out[16]) {
    uint32_t aux[4];
    memcpy(aux, sc12, 12);
    const uint32_t kmask1 = 0x03030303, kmask2 = 0x0f0f0f0f;
    const uint32_t tmp = aux[2];
    aux[2] = ((aux[0] >> 4) & kmask2) | (((tmp >> 4) & kmask1) << 4);
    aux[3] = ((aux[1] >> 4) & kmask2) | (((tmp >> 6) & kmask1) << 4);
    aux[0] = (aux[0] & kmask2) | (((tmp >> 0) & kmask1) << 4);
    aux[1] = (aux[1] & kmask2) | (((tmp >> 2) & kmask1) << 4);
    const uint8_t * s = (const uint8_t *) aux;
    for (int i = 0; i < 16; ++i) out[i] = (int8_t)((int) s[i] - 32);
}

/* element idx (0..255) of a Q3_K super-block as its signed 3-bit code in [-4,3]
 * (ggml-quants.c:1331-1348): idx = 128*half + 32*shift + l */
static inline int q3k_code(const blk_q3_K * b, int idx) {
    const int half = idx >> 7, shift = (idx >> 5) & 3, l = idx & 31;
    const int lo = (b->qs[32 * half + l] >> (2 * shift)) & 3;
    const int hb = (b->hmask[l] >> (4 * half + shift)) & 1;
    return lo - (hb ? 0 : 4);
}

void orc_dequantize_row_q3_K(const void * vx, float * y, int64_t k) {
    const blk_q3_K * x = (const blk_q3_K *) vx;
    const int64_t nb = k / QK_K;
    for (int64_t i = 0; i < nb; i++) {
        const float d_all = orc_fp16_to_fp32(x[i].d);
        int8_t sc[16];
        q3k_scales(x[i].scales, sc);
        for (int idx = 0; idx < QK_K; ++idx) {
            const float dl = d_all * sc[idx >> 4];
            y[i * QK_K + idx] = dl * (float) q3k_code(&x[i], idx);
        }
    }
}


/* ---- Q3_K weight quantiser (creates test inputs; ggml-quants.c:1229-1303 and its helper make_q3_quants, :697-754) */

/* nearest integer by the magic-number addition of ggml-quants.c:621-626 */
static inline int orc_nearest_int(float fval) {
    float val = fval + 12582912.f;
    int i;
    memcpy(&i, &val, sizeof(int));
    return (i & 0x007fffff) - 0x00400000;
}

/* scale of 16 values for codes in [-4, 3]: start from -4 / (value of largest magnitude), then up to five rounds of
 * coordinate descent on the weighted (w = x^2) least-squares objective; codes are returned shifted to [0, 7] */
static float orc_make_q3_quants(const float * x, int8_t * L) {
    const int n = 16, nmax = 4;
    float max = 0, amax = 0;
    for (int i = 0; i < n; ++i) { const float ax = fabsf(x[i]); if (ax > amax) { amax = ax; max = x[i]; } }
    if (amax < 1e-15f) { for (int i = 0; i < n; ++i) L[i] = 0; return 0.f; }
    const float iscale = -nmax / max;
    float sumlx = 0, suml2 = 0;
    for (int i = 0; i < n; ++i) {
        int l = orc_nearest_int(iscale * x[i]);
        l = l < -nmax ? -nmax : (l > nmax - 1 ? nmax - 1 : l);
        L[i] = (int8_t) l;
        const float w = x[i] * x[i];
        sumlx += w * x[i] * l;
        suml2 += w * l * l;
    }
    for (int itry = 0; itry < 5; ++itry) {
        int n_changed = 0;
        for (int i = 0; i < n; ++i) {
            const float w = x[i] * x[i];
            float slx = sumlx - w * x[i] * L[i];
            if (slx > 0) {
                float sl2 = suml2 - w * L[i] * L[i];
                int new_l = orc_nearest_int(x[i] * sl2 / slx);
                new_l = new_l < -nmax ? -nmax : (new_l > nmax - 1 ? nmax - 1 : new_l);
                if (new_l != L[i]) {
                    slx += w * x[i] * new_l;
                    sl2 += w * new_l * new_l;
                    if (sl2 > 0 && slx * slx * suml2 > sumlx * sumlx * sl2) {
                        L[i] = (int8_t) new_l; sumlx = slx; suml2 = sl2;
                        ++n_changed;
                    }
                }
            }
        }
        if (!n_changed) break;
    }
    for (int i = 0; i < n; ++i) L[i] += nmax;
    return suml2 > 0.0f ? sumlx / suml2 : 0.0f;
}

void orc_quantize_row_q3_K(const float * x, void * vy, int64_t k) {
    blk_q3_K * y = (blk_q3_K *) vy;
    const int64_t nb = k / QK_K;
    int8_t L[QK_K];
    float scales[QK_K / 16];
    for (int64_t i = 0; i < nb; i++, x += QK_K) {
        float max_scale = 0, amax = 0;
        for (int j = 0; j < QK_K / 16; ++j) {
            scales[j] = orc_make_q3_quants(x + 16 * j, L + 16 * j);
            const float scale = fabsf(scales[j]);
            if (scale > amax) { amax = scale; max_scale = scales[j]; }
        }
        memset(y[i].scales, 0, 12);
        if (max_scale) {
            const float iscale = -32.f / max_scale;
            for (int j = 0; j < QK_K / 16; ++j) {
                int8_t l = (int8_t) orc_nearest_int(iscale * scales[j]);
                l = (int8_t) ((l < -32 ? -32 : (l > 31 ? 31 : l)) + 32);
                if (j < 8) y[i].scales[j] = l & 0xF;
                else       y[i].scales[j - 8] |= ((l & 0xF) << 4);
                l >>= 4;
                y[i].scales[j % 4 + 8] |= (l << (2 * (j / 4)));
            }
            y[i].d = orc_fp32_to_fp16(1 / iscale);
        } else {
            y[i].d = orc_fp32_to_fp16(0.f);
        }
        const float dd = orc_fp16_to_fp32(y[i].d);
        for (int j = 0; j < QK_K / 16; ++j) {
            int sc = j < 8 ? y[i].scales[j] & 0xF : y[i].scales[j - 8] >> 4;
            sc = (sc | (((y[i].scales[8 + j % 4] >> (2 * (j / 4))) & 3) << 4)) - 32;
            const float d = dd * sc;
            if (!d) continue;
            for (int ii = 0; ii < 16; ++ii) {
                int l = orc_nearest_int(x[16 * j + ii] / d);
                l = l < -4 ? -4 : (l > 3 ? 3 : l);
                L[16 * j + ii] = (int8_t) (l + 4);
            }
        }
        memset(y[i].hmask, 0, QK_K / 8);
        int m = 0;
        uint8_t hm = 1;
        for (int j = 0; j < QK_K; ++j) {
            if (L[j] > 3) { y[i].hmask[m] |= hm; L[j] -= 4; }
            if (++m == QK_K / 8) { m = 0; hm <<= 1; }
        }
        for (int j = 0; j < QK_K; j += 128)
            for (int l = 0; l < 32; ++l)
                y[i].qs[j / 4 + l] = (uint8_t) (L[j + l] | (L[j + l + 32] << 2) | (L[j + l + 64] << 4) | (L[j + l + 96] << 6));
    }
}

/* rows are independent: spread them over the host's cores (input generation for whole layers takes 1e9 values) */
typedef struct { const float * src; char * dst; int64_t r0, r1, n, rs; } q3k_job;
static void * q3k_worker(void * arg) {
    const q3k_job * j = (const q3k_job *) arg;
    for (int64_t r = j->r0; r < j->r1; ++r) orc_quantize_row_q3_K(j->src + r * j->n, j->dst + r * j->rs, j->n);
    return NULL;
}
static void quantize_q3_K_rows(const float * src, void * dst, int64_t nrows, int64_t n_per_row) {
    long ncpu = sysconf(_SC_NPROCESSORS_ONLN);
    int nt = (int) (ncpu < 1 ? 1 : (ncpu > 64 ? 64 : ncpu));
    if (nrows < 64) nt = 1;
    pthread_t th[64];
    q3k_job jobs[64];
    for (int t = 0; t < nt; ++t) {
        jobs[t] = (q3k_job){ src, (char *) dst, nrows * t / nt, nrows * (t + 1) / nt, n_per_row, orc_row_size(ORC_TYPE_Q3_K, n_per_row) };
        if (nt == 1) q3k_worker(&jobs[t]);
        else pthread_create(&th[t], NULL, q3k_worker, &jobs[t]);
    }
    if (nt > 1) for (int t = 0; t < nt; ++t) pthread_join(th[t], NULL);
}

int orc_dequantize(int type, const void * src, float * dst, int64_t n) {
    if (type == ORC_TYPE_NVFP4) { orc_dequantize_row_nvfp4(src, dst, n); return 0; }
    if (type == ORC_TYPE_Q3_K)  { orc_dequantize_row_q3_K(src, dst, n); return 0; }
    if (type == ORC_TYPE_F32)   { memcpy(dst, src, (size_t) n * 4); return 0; }
    return 1;
}

int orc_quantize(int type, const float * src, void * dst, int64_t nrows, int64_t n_per_row) {
    if (type == ORC_TYPE_NVFP4) {
        const int64_t rs = orc_row_size(type, n_per_row);
        for (int64_t r = 0; r < nrows; ++r) orc_quantize_row_nvfp4(src + r * n_per_row, (char *) dst + r * rs, n_per_row);
        return 0;
    }
    if (type == ORC_TYPE_Q3_K) { quantize_q3_K_rows(src, dst, nrows, n_per_row); return 0; }
    if (type == ORC_TYPE_F32) { memcpy(dst, src, (size_t)(nrows * n_per_row) * 4); return 0; }
    return 1;
}

/* ---- activation quantisers */

/* Q8_0, AVX2 flavour: ggml-cpu/arch/x86/quants.c:302-367.  d = amax/127 stored as half;
 * the multiplier is 127/amax in fp32 and rounding is to nearest even (_mm256_round_ps NEAREST). */
void orc_quantize_row_q8_0(const float * x, void * vy, int64_t k) {
    blk_q8_0 * y = (blk_q8_0 *) vy;
    const int64_t nb = k / QK8_0;
    for (int64_t i = 0; i < nb; i++) {
        float amax = 0.0f;
        for (int j = 0; j < QK8_0; j++) { const float v = fabsf(x[i * QK8_0 + j]); if (v > amax) amax = v; }
        const float d = amax / 127.f;
        y[i].d = orc_fp32_to_fp16(d);
        const float id = (amax != 0.0f) ? 127.f / amax : 0.0f;
        for (int j = 0; j < QK8_0; j++) {
            const float v = x[i * QK8_0 + j] * id;
            y[i].qs[j] = (int8_t) (int) nearbyintf(v);
        }
    }
}

/* ggml-quants.c:621-626 */
static inline int nearest_int(float fval) {
    float val = fval + 12582912.f;
    int i; memcpy(&i, &val, sizeof(int));
    return (i & 0x007fffff) - 0x00400000;
}

/* Q8_K: ggml-quants.c:2768-2805 (arch/x86/quants.c:505-507 forwards to it) */
void orc_quantize_row_q8_K(const float * x, void * vy, int64_t k) {
    blk_q8_K * y = (blk_q8_K *) vy;
    const int64_t nb = k / QK_K;
    for (int64_t i = 0; i < nb; i++) {
        float max = 0, amax = 0;
        for (int j = 0; j < QK_K; ++j) {
            float ax = fabsf(x[j]);
            if (ax > amax) { amax = ax; max = x[j]; }
        }
        if (!amax) {
            y[i].d = 0;
            memset(y[i].qs, 0, QK_K);
            memset(y[i].bsums, 0, sizeof y[i].bsums);   /* reference leaves bsums untouched here; the dots never read them */
            x += QK_K;
            continue;
        }
        const float iscale = -127.f / max;
        for (int j = 0; j < QK_K; ++j) {
            int v = nearest_int(iscale * x[j]);
            y[i].qs[j] = (int8_t)(v < 127 ? v : 127);
        }
        for (int j = 0; j < QK_K / 16; ++j) {
            int sum = 0;
            for (int ii = 0; ii < 16; ++ii) sum += y[i].qs[j * 16 + ii];
            y[i].bsums[j] = (int16_t) sum;
        }
        y[i].d = 1 / iscale;
        x += QK_K;
    }
}

int64_t orc_quantize_activation(int wtype, const float * src, void * dst, int64_t n) {
    if (wtype == ORC_TYPE_NVFP4) { orc_quantize_row_q8_0(src, dst, n); return orc_row_size(8, n); }
    if (wtype == ORC_TYPE_Q3_K)  { orc_quantize_row_q8_K(src, dst, n); return orc_row_size(15, n); }
    return -1;
}

/* ---- dot products */

/* hsum_float_8 (ggml-cpu/arch/x86/quants.c:43-49): ((a0+a4)+(a2+a6)) + ((a1+a5)+(a3+a7)) */
static inline float hsum8(const float a[8]) {
    const float r0 = a[4] + a[0], r1 = a[5] + a[1], r2 = a[6] + a[2], r3 = a[7] + a[3];
    const float s0 = r0 + r2, s1 = r1 + r3;
    return s0 + s1;
}

/* ggml_vec_dot_f32 on AVX2: ggml-cpu/vec.cpp:104-126 with GGML_F32_STEP 32 / EPR 8 and
 * GGML_F32x8_REDUCE (ggml-cpu/simd-mappings.h:587-616): four 8-lane FMA accumulators, element i goes
 * to accumulator (i/8)%4 lane i%8; accumulators are added (0+2),(1+3),(0+1); lanes fold j + (j+4),
 * then two horizontal adds; leftovers are added after the reduction. */
float orc_vec_dot_f32(int n, const float * x, const float * y) {
    float acc[4][8];
    memset(acc, 0, sizeof acc);
    const int np = n & ~31;
    for (int i = 0; i < np; i += 32)
        for (int j = 0; j < 4; ++j)
            for (int l = 0; l < 8; ++l)
                acc[j][l] = fmaf(x[i + j * 8 + l], y[i + j * 8 + l], acc[j][l]);
    float v[8];
    for (int l = 0; l < 8; ++l) {
        const float a02 = acc[0][l] + acc[2][l];
        const float a13 = acc[1][l] + acc[3][l];
        v[l] = a02 + a13;
    }
    float t0[4];
    for (int l = 0; l < 4; ++l) t0[l] = v[l] + v[l + 4];
    const float t1a = t0[0] + t0[1], t1b = t0[2] + t0[3];
    float sumf = t1a + t1b;
    for (int i = np; i < n; ++i) sumf += x[i] * y[i];
    return sumf;
}

/* ggml_vec_dot_q3_K_q8_K, AVX2 branch: ggml-cpu/arch/x86/quants.c:1766-1880.  Integer part: each
 * group of 32 elements gives 8 int32 lanes (lane m = elements 4m..4m+3 of the group), multiplied by
 * the signed 6-bit scale of the 16-element sub-block the lane falls in, summed over the 8 groups of
 * the super-block; then acc[lane] = fma(d_x*d_w, (float)sumi[lane], acc[lane]); final hsum_float_8. */
float orc_vec_dot_q3_K_q8_K(int n, const void * vw, const void * va) {
    const blk_q3_K * w = (const blk_q3_K *) vw;
    const blk_q8_K * a = (const blk_q8_K *) va;
    const int nb = n / QK_K;
    float acc[8] = { 0 };
    for (int i = 0; i < nb; ++i) {
        const float d = a[i].d * orc_fp16_to_fp32(w[i].d);
        int8_t sc[16];
        q3k_scales(w[i].scales, sc);
        int32_t sumi[8] = { 0 };
        for (int idx = 0; idx < QK_K; ++idx) {
            const int lane = (idx & 31) >> 2;
            sumi[lane] += (int32_t) sc[idx >> 4] * (q3k_code(&w[i], idx) * (int32_t) a[i].qs[idx]);
        }
        for (int l = 0; l < 8; ++l) acc[l] = fmaf(d, (float) sumi[l], acc[l]);
    }
    return hsum8(acc);
}

/* ggml_vec_dot_nvfp4_q8_0, AVX2 branch: ggml-cpu/arch/x86/quants.c:1004-1062.  Per 64-element block:
 * lanes 0-3 of p_1 hold sub-block 0 (4 elements each), lanes 4-7 sub-block 1, scaled by
 * ue4m3(d[s])*dy; p_2 likewise for sub-blocks 2,3; two FMAs per lane per block; hsum_float_8.
 * GGML_CPU_UE4M3_TO_FP32 is a table of ggml_ue4m3_to_fp32 (ggml-cpu/simd-mappings.h:137-141). */
float orc_vec_dot_nvfp4_q8_0(int n, const void * vw, const void * va) {
    const blk_nvfp4 * w = (const blk_nvfp4 *) vw;
    const blk_q8_0 * a = (const blk_q8_0 *) va;
    const int nb = n / QK_NVFP4;
    float acc[8] = { 0 };
    for (int ib = 0; ib < nb; ++ib) {
        const float dy[2] = { orc_fp16_to_fp32(a[2 * ib].d), orc_fp16_to_fp32(a[2 * ib + 1].d) };
        for (int pair = 0; pair < 2; ++pair) {           /* p_1: sub-blocks 0,1 ; p_2: sub-blocks 2,3 */
            const blk_q8_0 * q8 = &a[2 * ib + pair];
            for (int half = 0; half < 2; ++half) {
                const int s = 2 * pair + half;
                const float scale = orc_ue4m3_to_fp32(w[ib].d[s]) * dy[pair];
                int8_t v[16];
                for (int j = 0; j < 8; ++j) {
                    v[j]     = kvalues_fp4[w[ib].qs[s * 8 + j] & 0xf];
                    v[j + 8] = kvalues_fp4[w[ib].qs[s * 8 + j] >> 4];
                }
                for (int m = 0; m < 4; ++m) {
                    int32_t p = 0;
                    for (int e = 0; e < 4; ++e) p += (int32_t) v[4 * m + e] * (int32_t) q8->qs[16 * half + 4 * m + e];
                    acc[4 * half + m] = fmaf(scale, (float) p, acc[4 * half + m]);
                }
            }
        }
    }
    return hsum8(acc);
}

int orc_vec_dot(int wtype, int64_t n, const void * wrow, const void * act, float * out) {
    if (wtype == ORC_TYPE_NVFP4) { *out = orc_vec_dot_nvfp4_q8_0((int) n, wrow, act); return 0; }
    if (wtype == ORC_TYPE_Q3_K)  { *out = orc_vec_dot_q3_K_q8_K((int) n, wrow, act); return 0; }
    if (wtype == ORC_TYPE_F32)   { *out = orc_vec_dot_f32((int) n, (const float *) wrow, (const float *) act); return 0; }
    return 1;
}

/* ---- ggml_v_expf, AVX2+FMA flavour, one lane: ggml-cpu/vec.h:1215-1252 */
float orc_expf(float x) {
    const float r = 0x1.8p23f;
    const float z = fmaf(x, 0x1.715476p+0f, r);
    const float n = z - r;
    const float b = fmaf(-n, 0x1.7f7d1cp-20f, fmaf(-n, 0x1.62e4p-1f, x));
    const uint32_t e = f2u(z) << 23;
    const float k = u2f(e + f2u(1.0f));
    const int c = fabsf(n) > 126.0f;
    const float u = b * b;
    const float j = fmaf(fmaf(fmaf(0x1.0e4020p-7f, b, 0x1.573e2ep-5f), u, fmaf(0x1.555e66p-3f, b, 0x1.fffdb6p-2f)), u,
                         0x1.ffffecp-1f * b);
    if (!c) return fmaf(j, k, k);
    const uint32_t g = (n <= 0.0f) ? 0x82000000u : 0u;
    const float s1 = u2f(g + 0x7f000000u);
    const float s2 = u2f(e - g);
    if (fabsf(n) > 192.0f) return s1 * s1;
    return fmaf(s2, j, s2) * s1;
}

/* ggml_v_silu: ggml-cpu/vec.h:1255-1262 (I is a multiple of 8 in every configuration, so the
 * vector branch of ggml_vec_silu_f32, ggml-cpu/vec.cpp:380-392, covers every element) */
float orc_silu(float x) {
    const float neg_x = 0.0f - x;
    return x / (1.0f + orc_expf(neg_x));
}

/* soft_max: ggml-cpu/ops.cpp:5584-5694 with scale 1, no mask; ggml_vec_soft_max_f32
 * (ggml-cpu/vec.cpp:531-551): each group of 8 exponentials is folded in fp32 as
 * ((v0+v4)+(v2+v6)) + ((v1+v5)+(v3+v7)) and added to a double; tail elements use expf. */
void orc_soft_max_row(int n, float * y, const float * x) {
    float max = -INFINITY;
    for (int i = 0; i < n; ++i) max = max > x[i] ? max : x[i];
    double sum = 0;
    int i = 0;
    for (; i + 7 < n; i += 8) {
        float v[8];
        for (int l = 0; l < 8; ++l) { v[l] = orc_expf(x[i + l] - max); y[i + l] = v[l]; }
        sum += (double) hsum8(v);
    }
    for (; i < n; ++i) { float v = expf(x[i] - max); y[i] = v; sum += (double) v; }
    sum = 1.0 / sum;
    const float inv = (float) sum;
    for (i = 0; i < n; ++i) y[i] *= inv;
}

/* argsort DESC + first k (ggml.c:5441-5455, ggml-cpu/ops.cpp:8477-8528). */
int orc_top_k_row(int n, int k, const float * p, int32_t * ids) {
    int tie = 0;
    unsigned char * used = (unsigned char *) calloc((size_t) n, 1);
    for (int s = 0; s < k; ++s) {
        int best = -1;
        for (int i = 0; i < n; ++i) {
            if (used[i]) continue;
            if (best < 0 || p[i] > p[best]) best = i;
        }
        used[best] = 1;
        ids[s] = best;
    }
    /* a value equal to a selected one, at another index, makes the reference order unspecified */
    for (int s = 0; s < k && !tie; ++s)
        for (int i = 0; i < n; ++i)
            if (i != ids[s] && p[i] == p[ids[s]]) { tie = 1; break; }
    free(used);
    return tie;
}

/* ---- the layer */

static void mul_mat_q(int wtype, int n_in, int n_out, const void * w, const float * x, float * y, void * act_buf) {
    /* ggml_compute_forward_mul_mat: src1 row -> vec_dot_type, then one vec_dot per weight row */
    orc_quantize_activation(wtype, x, act_buf, n_in);
    const int64_t rs = orc_row_size(wtype, n_in);
    for (int r = 0; r < n_out; ++r) orc_vec_dot(wtype, n_in, (const char *) w + r * rs, act_buf, &y[r]);
}

static double now_ms(void) {
    struct timespec ts; clock_gettime(CLOCK_MONOTONIC, &ts);
    return ts.tv_sec * 1e3 + ts.tv_nsec * 1e-6;
}

static int layer_once(const orc_moe_args * a) {
    const int H = a->H, L = a->latent ? a->L : a->H, E = a->E, K = a->K, I = a->I, T = a->T;
    const int wt = a->wtype;
    if (wt != ORC_TYPE_NVFP4 && wt != ORC_TYPE_Q3_K) return 1;
    const int64_t rs_L = orc_row_size(wt, L), rs_I = orc_row_size(wt, I);
    const int big = H > L ? H : L;
    float * logits = (float *) malloc(sizeof(float) * E);
    float * probs  = (float *) malloc(sizeof(float) * E);
    float * xl     = (float *) malloc(sizeof(float) * L);
    float * g      = (float *) malloc(sizeof(float) * I);
    float * u      = (float *) malloc(sizeof(float) * I);
    float * hid    = (float *) malloc(sizeof(float) * I);
    float * dn     = (float *) malloc(sizeof(float) * (size_t) L * K);
    float * moe    = (float *) malloc(sizeof(float) * L);
    void  * actx   = malloc((size_t) big * 2 + 1024);
    void  * acth   = malloc((size_t) I * 2 + 1024);
    int32_t * ids  = (int32_t *) malloc(sizeof(int32_t) * K);
    float * wts    = (float *) malloc(sizeof(float) * K);

    for (int t = 0; t < T; ++t) {
        const float * x = a->x + (size_t) t * H;
        /* route: edge0-infer/src/models/edge0_35b/forward.cpp:262-271 */
        for (int e = 0; e < E; ++e) {
            logits[e] = orc_vec_dot_f32(H, a->router_w + (size_t) e * H, x);
            if (a->router_bias) logits[e] = logits[e] + a->router_bias[e];
        }
        orc_soft_max_row(E, probs, logits);
        orc_top_k_row(E, K, probs, ids);
        double wsum = 0;                                /* sum_rows: ggml-cpu/vec.h:1495-1505, double accumulate */
        for (int s = 0; s < K; ++s) { wts[s] = probs[ids[s]]; wsum += (double) wts[s]; }
        float den = (float) wsum;
        if (den < 6.103515625e-5f) den = 6.103515625e-5f;   /* clamp(2^-14, inf) */
        for (int s = 0; s < K; ++s) wts[s] = wts[s] / den;

        /* latent down-projection (edge0-strata src/latent/latent_moe.cpp:38-92, one label group) */
        const float * xe = x;
        if (a->latent) {
            mul_mat_q(wt, H, L, a->lat_d, x, xl, actx);
            if (a->s_lat_d) for (int i = 0; i < L; ++i) xl[i] = xl[i] * a->s_lat_d[0];
            xe = xl;
        }

        /* ffn: forward.cpp:300-311; mul_mat_id: ggml-cpu/ggml-cpu.c:1550-1740 */
        orc_quantize_activation(wt, xe, actx, L);       /* gate/up share one activation row (ne11 == 1) */
        for (int s = 0; s < K; ++s) {
            const int e = ids[s];
            const char * wg = (const char *) a->gate + (size_t) e * I * rs_L;
            const char * wu = (const char *) a->up   + (size_t) e * I * rs_L;
            const char * wd = (const char *) a->down + (size_t) e * L * rs_I;
            for (int r = 0; r < I; ++r) {
                orc_vec_dot(wt, L, wg + r * rs_L, actx, &g[r]);
                orc_vec_dot(wt, L, wu + r * rs_L, actx, &u[r]);
                if (a->s_gate) g[r] = g[r] * a->s_gate[e];
                if (a->s_up)   u[r] = u[r] * a->s_up[e];
                hid[r] = orc_silu(g[r]) * u[r];
            }
            orc_quantize_activation(wt, hid, acth, I);
            float * d = dn + (size_t) s * L;
            for (int r = 0; r < L; ++r) {
                orc_vec_dot(wt, I, wd + r * rs_I, acth, &d[r]);
                if (a->s_down) d[r] = d[r] * a->s_down[e];
            }
            if (a->hidden)   memcpy(a->hidden + ((size_t) t * K + s) * I, hid, sizeof(float) * I);
            if (a->down_out) memcpy(a->down_out + ((size_t) t * K + s) * L, d, sizeof(float) * L);
        }
        /* weighted sum in slot order: forward.cpp:308-310 */
        for (int i = 0; i < L; ++i) {
            float acc = dn[i] * wts[0];
            for (int s = 1; s < K; ++s) acc = acc + dn[(size_t) s * L + i] * wts[s];
            moe[i] = acc;
        }
        if (a->logits)  memcpy(a->logits + (size_t) t * E, logits, sizeof(float) * E);
        if (a->probs)   memcpy(a->probs + (size_t) t * E, probs, sizeof(float) * E);
        if (a->ids)     memcpy(a->ids + (size_t) t * K, ids, sizeof(int32_t) * K);
        if (a->weights) memcpy(a->weights + (size_t) t * K, wts, sizeof(float) * K);
        if (a->moe_out) memcpy(a->moe_out + (size_t) t * L, moe, sizeof(float) * L);
        if (a->sh_gate && !a->latent) {
            /* shared expert: forward.cpp:312-314.  Dense quantised mul_mats (activation quantised to the type's vec_dot_type,
             * ggml-cpu/ggml-cpu.c:1255-1468), silu * up (vec.cpp:380-392), sigmoid of an F32 dot through libm's expf (vec.h:936) */
            const int Is = a->I_sh;
            float * sg = (float *) malloc(sizeof(float) * Is), * su = (float *) malloc(sizeof(float) * Is), * sh = (float *) malloc(sizeof(float) * H);
            void * acts = malloc((size_t) (Is > H ? Is : H) * 2 + 1024);
            mul_mat_q(wt, H, Is, a->sh_gate, x, sg, acts);
            mul_mat_q(wt, H, Is, a->sh_up, x, su, acts);
            for (int r = 0; r < Is; ++r) sg[r] = orc_silu(sg[r]) * su[r];
            mul_mat_q(wt, Is, H, a->sh_down, sg, sh, acts);
            const float gl = orc_vec_dot_f32(H, a->sh_gate_inp, x);
            const float sig = 1.f / (1.f + expf(-gl));
            for (int i = 0; i < H; ++i) {
                sh[i] = sh[i] * sig;
                moe[i] = moe[i] + sh[i];
            }
            if (a->shexp_gated) memcpy(a->shexp_gated + (size_t) t * H, sh, sizeof(float) * H);
            free(sg); free(su); free(sh); free(acts);
        }
        if (a->latent) {
            float * o = (float *) malloc(sizeof(float) * H);
            mul_mat_q(wt, L, H, a->lat_u, moe, o, actx);
            if (a->s_lat_u) for (int i = 0; i < H; ++i) o[i] = o[i] * a->s_lat_u[0];
            if (a->out) memcpy(a->out + (size_t) t * H, o, sizeof(float) * H);
            free(o);
        } else if (a->out) {
            memcpy(a->out + (size_t) t * L, moe, sizeof(float) * L);
        }
    }
    free(logits); free(probs); free(xl); free(g); free(u); free(hid); free(dn); free(moe);
    free(actx); free(acth); free(ids); free(wts);
    return 0;
}

int orc_moe_layer(const orc_moe_args * a) {
    int rc = layer_once(a);
    if (rc || a->repeats <= 0) return rc;
    double best = 1e300, * all = (double *) malloc(sizeof(double) * a->repeats);
    for (int r = 0; r < a->repeats; ++r) {
        const double t0 = now_ms();
        layer_once(a);
        all[r] = now_ms() - t0;
        if (all[r] < best) best = all[r];
    }
    for (int i = 1; i < a->repeats; ++i) for (int j = i; j > 0 && all[j] < all[j - 1]; --j) { double t = all[j]; all[j] = all[j - 1]; all[j - 1] = t; }
    if (a->ms_best) *a->ms_best = best;
    if (a->ms_median) *a->ms_median = all[a->repeats / 2];
    free(all);
    return 0;
}
