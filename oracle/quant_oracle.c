/*
 * quant_oracle.c -- CPU restatement of the reference's weight-only int8 quantized-linear arithmetic.
 *
 * TEST INFRASTRUCTURE ONLY.  This file is the checker the CUDA kernels are compared with, and the
 * CPU baseline that is timed next to them.  Nothing in the product (hidet_b200/) calls it.
 *
 * What it restates (paths are relative to the reference repository):
 *   - SymmetricQuantizationTask / SymmetricDeQuantizationTask, python/hidet/graph/ops/quant/symmetric.py:23-61,
 *     in the two arithmetics the reference really executes:
 *       f32 : the code its CPU (x86) backend generates -- fmaxf, '/', roundf
 *             (python/hidet/ir/primitives/cpu/math/float32.py:40), loops as generated by the
 *             auto-scheduler (one output per iteration, serial reduction);
 *       f16 : the code its CUDA backend generates -- __hmax, __half operator/, hrint, (int8_t)(short)
 *             cast (python/hidet/ir/primitives/cuda/math/float16.py:62-76,
 *             python/hidet/backend/codegen.py:452-453).  The division is taken as what it is documented to
 *             be, the quotient rounded to the nearest half, ties to even.
 *   - SymmetricQuantizedMatmulTask, python/hidet/graph/ops/quant/matmul.py:24-74, and the
 *     dequantize-then-matmul composition the quantization pass builds first
 *     (python/hidet/graph/transforms/graph_patterns/quant/linear.py:37-49).
 *
 * Parity status: the f32 functions are pinned against outputs of the reference's own compiled CPU
 * tasks (tests/golden/reference_cpu_*.npz).  The reference's own tests hold no bit-level vectors for
 * f16; the f16 functions are pinned against the reference's own CUDA kernels instead: its generated
 * quantize / dequantize sources, compiled for sm_100a with its flags (oracle/build_ref.py), run on the
 * GPU beside this oracle in tests/test_reference_kernels_gpu.py (codes, scales and dequantized values
 * bit for bit, on seeded and adversarial inputs).  That check needs a GPU; on a host without one the
 * f16 functions stand on the restatement alone.
 */
#include <math.h>
#include <float.h>
#include <stdint.h>
#include <stddef.h>
#include <string.h>
#include <stdlib.h>

#ifdef _OPENMP
#include <omp.h>
#endif

#define ORACLE_API __attribute__((visibility("default")))

/* ------------------------------------------------------------------------------------------- */
/* binary16 <-> binary32, written out so that the result does not depend on compiler support      */
/* ------------------------------------------------------------------------------------------- */
static inline float bits_to_float(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}
static inline uint32_t float_to_bits(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}

static inline float half_to_float(uint16_t h) {
    const uint32_t sign = (uint32_t)(h & 0x8000u) << 16;
    const uint32_t exp = (h >> 10) & 0x1fu;
    uint32_t man = h & 0x3ffu;
    if (exp == 0) {
        if (man == 0) return bits_to_float(sign);
        /* subnormal: man * 2^-24 */
        float f = (float)man * 5.9604644775390625e-08f;
        return (sign != 0) ? -f : f;
    }
    if (exp == 31) return bits_to_float(sign | 0x7f800000u | (man << 13));
    return bits_to_float(sign | ((exp + 112u) << 23) | (man << 13));
}

/* round to nearest, ties to even (cvt.rn.f16.f32) */
static inline uint16_t float_to_half(float f) {
    const uint32_t x = float_to_bits(f);
    const uint16_t sign = (uint16_t)((x >> 16) & 0x8000u);
    const uint32_t ax = x & 0x7fffffffu;
    if (ax > 0x7f800000u) return 0x7fffu;                  /* NaN: CUDA's canonical half NaN */
    if (ax >= 0x477ff000u) return (uint16_t)(sign | 0x7c00u); /* >= 65520 rounds to infinity (and inf) */
    if (ax < 0x33000001u) return sign;                      /* <= 2^-25 rounds to zero */
    int32_t e = (int32_t)(ax >> 23) - 127;
    uint32_t m = (ax & 0x7fffffu) | 0x800000u; /* 24-bit significand */
    uint32_t shift;
    uint32_t half_exp;
    if (e < -14) { /* subnormal half */
        shift = (uint32_t)(13 + (-14 - e));
        half_exp = 0;
    } else {
        shift = 13;
        half_exp = (uint32_t)(e + 15);
    }
    uint32_t q = m >> shift;
    const uint32_t rem = m & ((1u << shift) - 1u);
    const uint32_t halfway = 1u << (shift - 1);
    if (rem > halfway || (rem == halfway && (q & 1u))) q += 1;
    /* q includes the hidden bit for normals: adding it into the exponent field handles carries */
    uint32_t out;
    if (half_exp == 0) out = q;                      /* may carry into exponent 1: correct */
    else out = ((half_exp - 1u) << 10) + q;          /* q has bit 10 set */
    return (uint16_t)(sign | out);
}

static inline int half_is_nan(uint16_t h) { return (h & 0x7fffu) > 0x7c00u; }

/* ------------------------------------------------------------------------------------------- */
/* CUDA half operations used by the reference's generated kernels                                 */
/* ------------------------------------------------------------------------------------------- */

/* __hmax: the non-NaN operand if one is NaN, canonical NaN if both; -0 < +0 */
static inline uint16_t h_max(uint16_t a, uint16_t b) {
    if (half_is_nan(a)) return half_is_nan(b) ? 0x7fffu : b;
    if (half_is_nan(b)) return a;
    const float fa = half_to_float(a), fb = half_to_float(b);
    if (fa > fb) return a;
    if (fb > fa) return b;
    /* equal (possibly +0 / -0): prefer the one without sign bit */
    return (a & 0x8000u) ? b : a;
}

/* ((half)0.0f <= w) ? w : -w */
static inline uint16_t h_abs_ref(uint16_t w) {
    const int le = !half_is_nan(w) && (0.0f <= half_to_float(w));
    return le ? w : (uint16_t)(w ^ 0x8000u);
}

/* a / b, rounded to the nearest half.  The IEEE f32 quotient in between changes nothing: a quotient of two 11-bit
 * significands is either exactly half-way between two halves, and then f32 holds it exactly, or at least 2^-23 of its
 * value away from there, and one f32 rounding moves it by at most 2^-24. */
static inline uint16_t h_div(uint16_t a, uint16_t b) { return float_to_half(half_to_float(a) / half_to_float(b)); }

/* hrint: cvt.rni.f16.f16 */
static inline uint16_t h_rint(uint16_t h) {
    if (half_is_nan(h)) return 0x7fffu;
    return float_to_half(nearbyintf(half_to_float(h))); /* default rounding mode: ties to even */
}

/* __half2short_rz: cvt.rzi.s16.f16 -- NaN gives 0, out-of-range saturates */
static inline int16_t h_to_short_rz(uint16_t h) {
    if (half_is_nan(h)) return 0;
    const float f = truncf(half_to_float(h));
    if (f >= 32767.0f) return 32767;
    if (f <= -32768.0f) return -32768;
    return (int16_t)f;
}

/* __short2half_rn */
static inline uint16_t short_to_half(int16_t s) { return float_to_half((float)s); }

/* __hmul */
static inline uint16_t h_mul(uint16_t a, uint16_t b) { return float_to_half(half_to_float(a) * half_to_float(b)); }

/* ------------------------------------------------------------------------------------------- */
/* f16 path (the reference's CUDA arithmetic)                                                     */
/* ------------------------------------------------------------------------------------------- */

/*
 * w[rows, cols] half bits -> wq (int8 if q_bits == 8, int16 if 16), scale half bits.
 * reduce_dim 0: scale[cols] (Hidet dims=0); reduce_dim 1: scale[rows] (Hidet dims=-1).
 * Follows the three generated kernels: y (absmax), quantize, scaling.
 */
ORACLE_API void oracle_quantize_f16(const uint16_t *w, void *wq, uint16_t *scale, int64_t rows, int64_t cols,
                                    int reduce_dim, int q_bits) {
    const uint16_t qmax = float_to_half(q_bits == 8 ? 127.0f : 32767.0f);
    const int64_t n_out = reduce_dim == 0 ? cols : rows;
    const int64_t n_red = reduce_dim == 0 ? rows : cols;
    const int64_t out_stride = reduce_dim == 0 ? 1 : cols;
    const int64_t red_stride = reduce_dim == 0 ? cols : 1;
#pragma omp parallel for schedule(static)
    for (int64_t o = 0; o < n_out; ++o) {
        uint16_t acc = 0xfbffu; /* (half)-65504.0f */
        for (int64_t v = 0; v < n_red; ++v) acc = h_max(acc, h_abs_ref(w[o * out_stride + v * red_stride]));
        const uint16_t s = h_div(acc, qmax);
        scale[o] = s;
        for (int64_t v = 0; v < n_red; ++v) {
            const int64_t idx = o * out_stride + v * red_stride;
            const int16_t q = h_to_short_rz(h_rint(h_div(w[idx], s)));
            if (q_bits == 8) ((int8_t *)wq)[idx] = (int8_t)q; /* (int8_t)(short): keeps the low byte */
            else ((int16_t *)wq)[idx] = q;
        }
    }
}

/* w = (half) wq * scale */
ORACLE_API void oracle_dequantize_f16(const void *wq, const uint16_t *scale, uint16_t *w, int64_t rows, int64_t cols,
                                      int reduce_dim, int q_bits) {
#pragma omp parallel for schedule(static)
    for (int64_t r = 0; r < rows; ++r) {
        for (int64_t c = 0; c < cols; ++c) {
            const int64_t idx = r * cols + c;
            const int16_t q = q_bits == 8 ? (int16_t)((const int8_t *)wq)[idx] : ((const int16_t *)wq)[idx];
            w[idx] = h_mul(short_to_half(q), scale[reduce_dim == 0 ? c : r]);
        }
    }
}

/*
 * The reference's "dequantize, then fp16 matmul with fp32 accumulation" result, the yardstick the
 * quantized matmul is held to: b = half(wq) * scale rounded to half, c = half(sum_k a[m,k] * b[k,n]).
 * The sum is taken in double so the yardstick itself carries no accumulation-order noise.
 * layout 0: wq is [K, N]; layout 1: wq is [N, K].  Only k in [k_begin, k_end) is summed.
 */
ORACLE_API void oracle_qmatmul_f16(const uint16_t *a, const int8_t *wq, const uint16_t *scale, uint16_t *c, int64_t M,
                                   int64_t N, int64_t K, int layout, int64_t k_begin, int64_t k_end) {
#pragma omp parallel
    {
        float *b = (float *)malloc(sizeof(float) * (size_t)(K > 0 ? K : 1));
        float *arow = (float *)malloc(sizeof(float) * (size_t)(K > 0 ? K : 1));
#pragma omp for schedule(static)
        for (int64_t n = 0; n < N; ++n) {
            for (int64_t k = k_begin; k < k_end; ++k) {
                const int8_t q = layout == 0 ? wq[k * N + n] : wq[n * K + k];
                b[k] = half_to_float(h_mul(short_to_half(q), scale[n]));
            }
            for (int64_t m = 0; m < M; ++m) {
                double acc = 0.0;
                for (int64_t k = k_begin; k < k_end; ++k) acc += (double)half_to_float(a[m * K + k]) * (double)b[k];
                c[m * N + n] = float_to_half((float)acc);
            }
        }
        free(b);
        free(arow);
    }
}

/*
 * The arithmetic the new kernels use, for a tight comparison: exact integer-valued products summed
 * without rounding (double holds them exactly for any K here), one multiply by the scale in fp32 and
 * one rounding to half.
 */
ORACLE_API void oracle_qmatmul_f16_fused(const uint16_t *a, const int8_t *wq, const uint16_t *scale, uint16_t *c,
                                         int64_t M, int64_t N, int64_t K, int layout, int64_t k_begin, int64_t k_end) {
#pragma omp parallel for schedule(static)
    for (int64_t n = 0; n < N; ++n) {
        for (int64_t m = 0; m < M; ++m) {
            double acc = 0.0;
            for (int64_t k = k_begin; k < k_end; ++k) {
                const int8_t q = layout == 0 ? wq[k * N + n] : wq[n * K + k];
                acc += (double)half_to_float(a[m * K + k]) * (double)q;
            }
            c[m * N + n] = float_to_half((float)acc * half_to_float(scale[n]));
        }
    }
}

/* ------------------------------------------------------------------------------------------- */
/* f32 path (the reference's generated x86 code; the loops below are that code's loops)           */
/* ------------------------------------------------------------------------------------------- */

/*
 * x86_fast_math != 0 restates what g++ -O3 -ffast-math (the reference's CPU build flags,
 * python/hidet/backend/build.py:326-338) makes of `y / 127.0f`: a multiplication by the rounded
 * constant 1/127.  With it the scales equal the reference's CPU output bit for bit; the quotient
 * w / scale is then an IEEE division here, while the reference's build may use a reciprocal estimate
 * with a refinement step for it, which is not a portable function (int8 results agree on every
 * vector checked; int16 results differ by one step in about one element per thousand).
 */
ORACLE_API void oracle_quantize_f32(const float *w, void *wq, float *scale, int64_t rows, int64_t cols, int reduce_dim,
                                    int q_bits, int x86_fast_math) {
    const float qmax = q_bits == 8 ? 127.0f : 32767.0f;
    const float inv_qmax = 1.0f / qmax;
    const int64_t n_out = reduce_dim == 0 ? cols : rows;
    const int64_t n_red = reduce_dim == 0 ? rows : cols;
    const int64_t out_stride = reduce_dim == 0 ? 1 : cols;
    const int64_t red_stride = reduce_dim == 0 ? cols : 1;
#pragma omp parallel for schedule(static)
    for (int64_t o = 0; o < n_out; ++o) {
        float acc = -3.4028234663852886e+38f;
        for (int64_t v = 0; v < n_red; ++v) {
            const float x = w[o * out_stride + v * red_stride];
            acc = fmaxf(acc, (0.0f <= x) ? x : (-x));
        }
        scale[o] = x86_fast_math ? acc * inv_qmax : acc / qmax;
    }
    const int64_t total = rows * cols;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < total; ++i) {
        const int64_t o = reduce_dim == 0 ? (i % cols) : (i / cols);
        const float r = roundf(w[i] / scale[o]); /* scale[o] is y / qmax, the value the generated code recomputes */
        if (q_bits == 8) ((int8_t *)wq)[i] = (int8_t)r;
        else ((int16_t *)wq)[i] = (int16_t)r;
    }
}

ORACLE_API void oracle_dequantize_f32(const void *wq, const float *scale, float *w, int64_t rows, int64_t cols,
                                      int reduce_dim, int q_bits) {
    const int64_t total = rows * cols;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < total; ++i) {
        const int64_t o = reduce_dim == 0 ? (i % cols) : (i / cols);
        const float q = q_bits == 8 ? (float)((const int8_t *)wq)[i] : (float)((const int16_t *)wq)[i];
        w[i] = q * scale[o];
    }
}

/* auto-scheduled CPU matmul: one output per iteration, serial fp32 sum over k, b read with stride N */
ORACLE_API void oracle_matmul_f32(const float *a, const float *b, float *c, int64_t M, int64_t N, int64_t K) {
    const int64_t total = M * N;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < total; ++i) {
        const int64_t m = i / N, n = i % N;
        float acc = 0.0f;
        for (int64_t k = 0; k < K; ++k) acc = a[m * K + k] * b[n + k * N] + acc;
        c[i] = acc;
    }
}

/*
 * symmetric_quant_matmul as the reference's CPU backend runs it for f32 activations after its
 * quantization pass: c[m,n] = sum_k a[m,k] * ((float)wq[k,n] * scale[n]) (dequantize fused as a
 * prologue of the matmul; python/hidet/graph/transforms/graph_patterns/quant/linear.py:37-49).
 */
ORACLE_API void oracle_qmatmul_f32(const float *a, const int8_t *wq, const float *scale, float *c, int64_t M, int64_t N,
                                   int64_t K) {
    const int64_t total = M * N;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < total; ++i) {
        const int64_t m = i / N, n = i % N;
        float acc = 0.0f;
        for (int64_t k = 0; k < K; ++k) acc = a[m * K + k] * ((float)wq[n + k * N] * scale[n]) + acc;
        c[i] = acc;
    }
}

ORACLE_API int oracle_num_threads(void) {
#ifdef _OPENMP
    return omp_get_max_threads();
#else
    return 1;
#endif
}

/* conversions exported for the tests of this file */
ORACLE_API float oracle_half_to_float(uint16_t h) { return half_to_float(h); }
ORACLE_API uint16_t oracle_float_to_half(float f) { return float_to_half(f); }
ORACLE_API uint16_t oracle_hdiv(uint16_t a, uint16_t b) { return h_div(a, b); }
