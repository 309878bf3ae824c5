// Symmetric quantize / dequantize kernels.
//
// The arithmetic repeats, operation for operation, what the reference's generated kernels do for
// SymmetricQuantizationTask / SymmetricDeQuantizationTask (python/hidet/graph/ops/quant/symmetric.py:23-61):
//
//     x     = (0 <= w) ? w : -w
//     amax  = max over the reduced dimension of x, starting from the lowest finite value
//     scale = amax / (T)qmax
//     wq    = (Q) round(w / scale)          round = hrint for f16 / bf16, roundf for f32
//     w'    = (T) wq * scale
//
// in w's own type T, with CUDA's own operators for __half / __nv_bfloat16 or with operations shown to give
// the same values.  This file
// is compiled with -ftz=true -prec-div=false, the flags the reference compiles its kernels with
// (python/hidet/backend/build.py:142-177), because they decide the f32 division.
//
// What differs from the reference is the schedule: the reference reads the weight twice from HBM
// with one thread per column walking K serially; here a thread-block cluster owns a panel of
// columns, each CTA keeps its slice of the panel in shared memory, partial maxima are written into
// the other CTAs' shared memory, and the slice is quantized from shared memory, so the weight
// crosses HBM once.  max is exact and order-independent, so the result does not depend on the
// schedule.
//
// No kernel of this file lets the launch behind it start early: the small-M quantized linear asks for the codes of its weight
// before it waits for the kernel in front, and is safe behind these only because it starts when they have ended.  They are themselves
// launched as programmatic dependents, and every CTA waits for the kernel in front before it touches memory: what remains between two launches
// is shorter so (300 x 512 per column 4.2 -> 2.8 us, 285 x 2992 per row 5.3 -> 3.4, 300 x 400 restored 4.2 -> 1.6).
#include <cooperative_groups.h>
#include <cfloat>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace b200q {
namespace {

// ---------------------------------------------------------------------------------------------
// per-type arithmetic, spelled the way the reference's generated code spells it
// ---------------------------------------------------------------------------------------------
template <typename T>
struct Arith;

template <>
struct Arith<__half> {
    static __device__ __forceinline__ __half lowest() { return (__half)-65504.0f; }
    static __device__ __forceinline__ __half abs_(__half w) { return ((__half)0.0f <= w) ? w : (-w); }
    static __device__ __forceinline__ __half max_(__half a, __half b) { return __hmax(a, b); }
    static __device__ __forceinline__ __half div_(__half a, __half b) { return a / b; }
    static __device__ __forceinline__ __half qmax(int q) { return (__half)(float)q; }
    // w / scale for many w and one scale, as the correctly rounded reciprocal of the scale times w in f32, rounded to
    // half: that is the correctly rounded quotient, the value of `w / scale`, wherever the quotient is a normal half.
    // Let w and scale have the significands a, b < 2^11.  A midpoint between two halves has an odd 12-bit significand m,
    // so a / b - m / 2^j (j <= 12) is a non-zero multiple of 1 / (b 2^j), at least 1 / (a 2^12) of the quotient (j = 12
    // needs a < b <= 2047, so a <= 2046), which exceeds 2^-23 (1 + 2^-11); the two f32 roundings move it by less than
    // 2^-23 (1 + 2^-24).  A quotient below the normal halves rounds to the integer 0 either way, and zero, infinite
    // and NaN operands give the zeros, infinities and NaN of a division.
    typedef float Divisor;
    static __device__ __forceinline__ Divisor prepare(__half scale) { return __frcp_rn(__half2float(scale)); }
    template <typename Q>
    static __device__ __forceinline__ Q quant(__half w, Divisor rcp) {
        return (Q)(short)(hrint(__float2half(rcp * __half2float(w))));
    }
    template <typename Q>
    static __device__ __forceinline__ __half dequant(Q q, __half scale) {
        return __short2half_rn((short)q) * scale;
    }
};

template <>
struct Arith<__nv_bfloat16> {
    static __device__ __forceinline__ __nv_bfloat16 lowest() { return (__nv_bfloat16)-3.4e+38f; }
    static __device__ __forceinline__ __nv_bfloat16 abs_(__nv_bfloat16 w) { return ((__nv_bfloat16)0.0f <= w) ? w : (-w); }
    static __device__ __forceinline__ __nv_bfloat16 max_(__nv_bfloat16 a, __nv_bfloat16 b) { return __hmax(a, b); }
    static __device__ __forceinline__ __nv_bfloat16 div_(__nv_bfloat16 a, __nv_bfloat16 b) { return a / b; }
    static __device__ __forceinline__ __nv_bfloat16 qmax(int q) { return (__nv_bfloat16)(float)q; }
    // As for f16: the quotient of two significands below 2^8 is at least 2^-17 of itself away from a midpoint between two
    // bfloat16 numbers, and the reciprocal times w is within 2^-23 of it.  That holds where neither the scale nor its
    // reciprocal is near the ends of the exponent range (and a w that is flushed makes a quotient that rounds to zero).  Any
    // other scale, zero, infinity and NaN among them, is handed on in the low bits of a NaN, for `quant` to divide by: its
    // products are NaN, so the packed form below leaves it to `quant` too.
    typedef float Divisor;
    static __device__ __forceinline__ Divisor prepare(__nv_bfloat16 scale) {
        const float s = __bfloat162float(scale);
        return fabsf(s) >= 7.888609e-31f && fabsf(s) < 8.507059e37f ? __frcp_rn(s) : __uint_as_float(0x7fc00000u | __bfloat16_as_ushort(scale));  // 2^-100, 2^126
    }
    template <typename Q>
    static __device__ __forceinline__ Q quant(__nv_bfloat16 w, Divisor rcp) {
        const unsigned int bits = __float_as_uint(rcp);
        if ((bits & 0x7fc00000u) == 0x7fc00000u) return (Q)(hrint(w / __ushort_as_bfloat16((unsigned short)bits)));
        return (Q)(hrint(__float2bfloat16(rcp * __bfloat162float(w))));
    }
    template <typename Q>
    static __device__ __forceinline__ __nv_bfloat16 dequant(Q q, __nv_bfloat16 scale) {
        return __short2bfloat16_rn((short)q) * scale;
    }
};

template <>
struct Arith<float> {
    static __device__ __forceinline__ float lowest() { return -3.4028234663852886e+38f; }
    static __device__ __forceinline__ float abs_(float w) { return (0.0f <= w) ? w : (-w); }
    static __device__ __forceinline__ float max_(float a, float b) { return fmaxf(a, b); }
    static __device__ __forceinline__ float div_(float a, float b) { return a / b; }
    static __device__ __forceinline__ float qmax(int q) { return (float)q; }
    typedef float Divisor;
    static __device__ __forceinline__ Divisor prepare(float scale) { return scale; }
    template <typename Q>
    static __device__ __forceinline__ Q quant(float w, float scale) {
        return (Q)(roundf(w / scale));
    }
    template <typename Q>
    static __device__ __forceinline__ float dequant(Q q, float scale) {
        return ((float)q) * scale;
    }
};

template <typename Q>
struct QMax;
template <>
struct QMax<int8_t> {
    static constexpr int value = 127;
};
template <>
struct QMax<int16_t> {
    static constexpr int value = 32767;
};

// N elements of T moved as one naturally aligned vector.  Operands are read with ordinary loads, behind the wait that makes the results of
// the kernel in front visible, and not through pointers that promise no aliasing: those would let the compiler take the path for data that is
// constant while a kernel runs, which under programmatic launches it is not.  So the compiler cannot move a load over a store either,
// and where a thread handles several vectors their loads stand together in front of the stores.
template <typename T, int N>
struct alignas(sizeof(T) * N) Vec {
    T v[N];
};

template <typename T, int N>
__device__ __forceinline__ Vec<T, N> load_vec(const T *p) {
    return *reinterpret_cast<const Vec<T, N> *>(p);
}
// The same past the first-level cache, for what is read once by threads that have little else to do (codes of a narrow matrix restored per row:
// 100000 x 8 f16 9.1 us through it, 5.8 past it).  Volatile: where several are to be in flight they stand together.
template <int BYTES>
struct RawVec;
template <> struct RawVec<1> { typedef unsigned char Type; };
template <> struct RawVec<2> { typedef unsigned short Type; };
template <> struct RawVec<4> { typedef unsigned int Type; };
template <> struct RawVec<8> { typedef uint2 Type; };
template <> struct RawVec<16> { typedef uint4 Type; };
template <typename T, int N>
__device__ __forceinline__ Vec<T, N> load_l2(const T *p) {
    typedef typename RawVec<sizeof(T) * N>::Type Raw;
    const Raw raw = __ldcg(reinterpret_cast<const Raw *>(p));
    return *reinterpret_cast<const Vec<T, N> *>(&raw);
}
template <typename T, int N>
__device__ __forceinline__ void store_vec(T *p, const Vec<T, N> &x) {
    *reinterpret_cast<Vec<T, N> *>(p) = x;
}

// VEC quotients -> codes.  The general form applies Arith<T>::quant element by element.
template <typename T, typename Q, int VEC, typename D>
struct QuantVec {
    // scales: one divisor per element (PER_ELEMENT) or one for all
    template <bool PER_ELEMENT>
    static __device__ __forceinline__ void run(const Vec<T, VEC> &x, const D *s, Vec<Q, VEC> &q) {
        run_n<PER_ELEMENT, VEC>(x.v, s, q.v);
    }
    template <bool PER_ELEMENT, int N>
    static __device__ __forceinline__ void run_n(const T *x, const D *s, Q *q) {
#pragma unroll
        for (int i = 0; i < N; ++i) q[i] = Arith<T>::template quant<Q>(x[i], s[PER_ELEMENT ? i : 0]);
    }
};

// f16 -> int8, eight at a time, two per instruction where the arithmetic allows it, with the same bits as the
// general form:
//   * the quotient v is f16(rcp * f32(w)) as in Arith<__half>::quant;
//   * b = v + 1536 in f16 (1536 = 0x6600, where one ulp is 1) is v rounded to an integer, ties to even, plus 1536
//     for |v| < 512: the same integer hrint gives, and 1536 being even the same ties.  For |hrint(v)| <= 127 the
//     low mantissa byte of b is that integer's two's-complement byte, which replaces hrint and the two conversions
//     (short)(r), (int8_t)(short);
//   * b - 1536 is exact; where its magnitude is not a number <= 127 for one of the eight (|v| >= 512 lands there too,
//     and so do the NaN and infinities a zero scale produces) all eight take the general form, whose conversions
//     define the result.
template <>
struct QuantVec<__half, int8_t, 8, Arith<__half>::Divisor> {
    template <bool PER_ELEMENT>
    static __device__ __forceinline__ void run(const Vec<__half, 8> &x, const Arith<__half>::Divisor *s, Vec<int8_t, 8> &q) {
        const __half2 *x2 = reinterpret_cast<const __half2 *>(x.v);
        const __half2 magic = __floats2half2_rn(1536.0f, 1536.0f);
        __half2 b[4], far[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float d0 = s[PER_ELEMENT ? 2 * j : 0], d1 = s[PER_ELEMENT ? 2 * j + 1 : 0];
            const float2 f = __half22float2(x2[j]);
            b[j] = __hadd2(__floats2half2_rn(d0 * f.x, d1 * f.y), magic);
            far[j] = __habs2(__hsub2(b[j], magic));
        }
        // one test for the eight: the largest magnitude, a NaN if there is any
        const __half2 worst = __hmax2_nan(__hmax2_nan(far[0], far[1]), __hmax2_nan(far[2], far[3]));
        const __half2 in_range = __hle2(worst, __floats2half2_rn(127.0f, 127.0f));  // 1.0 where true; false for NaN
        if (*reinterpret_cast<const uint32_t *>(&in_range) != 0x3C003C00u) {
            QuantVec<__half, int8_t, 1, Arith<__half>::Divisor>::template run_n<PER_ELEMENT, 8>(x.v, s, q.v);
            return;
        }
        const uint32_t *bits = reinterpret_cast<const uint32_t *>(b);
        uint32_t *out = reinterpret_cast<uint32_t *>(q.v);
        out[0] = __byte_perm(bits[0], bits[1], 0x6420);  // the low byte of each half, in order
        out[1] = __byte_perm(bits[2], bits[3], 0x6420);
    }
};

// bf16 -> int8, the same way with what bfloat16 arithmetic has: the quotients are rounded to bfloat16 two per
// instruction; 8 bits of significand cannot hold v + 1.5 * 2^n for all |v| <= 127, so the rounding to an integer is the f32
// addition of 1.5 * 2^23, whose low mantissa byte is the code.  Against one exact division per element, which filled the
// issue slots: 11008 x 4096 per row 32.8 -> 26.6 us, 4096 x 4096 per column 24.0 -> 16.6.
template <>
struct QuantVec<__nv_bfloat16, int8_t, 8, Arith<__nv_bfloat16>::Divisor> {
    template <bool PER_ELEMENT>
    static __device__ __forceinline__ void run(const Vec<__nv_bfloat16, 8> &x, const Arith<__nv_bfloat16>::Divisor *s, Vec<int8_t, 8> &q) {
        const uint32_t *xw = reinterpret_cast<const uint32_t *>(x.v);
        __nv_bfloat162 v[4], far[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float d0 = s[PER_ELEMENT ? 2 * j : 0], d1 = s[PER_ELEMENT ? 2 * j + 1 : 0];
            v[j] = __floats2bfloat162_rn(d0 * __uint_as_float(xw[j] << 16), d1 * __uint_as_float(xw[j] & 0xffff0000u));
            far[j] = __habs2(v[j]);
        }
        const __nv_bfloat162 worst = __hmax2_nan(__hmax2_nan(far[0], far[1]), __hmax2_nan(far[2], far[3]));
        const __nv_bfloat162 in_range = __hle2(worst, __floats2bfloat162_rn(127.0f, 127.0f));  // 1.0 where true; false for NaN
        if (*reinterpret_cast<const uint32_t *>(&in_range) != 0x3F803F80u) {
            QuantVec<__nv_bfloat16, int8_t, 1, Arith<__nv_bfloat16>::Divisor>::template run_n<PER_ELEMENT, 8>(x.v, s, q.v);
            return;
        }
        const uint32_t *vw = reinterpret_cast<const uint32_t *>(v);
        uint32_t *out = reinterpret_cast<uint32_t *>(q.v);
        uint32_t pair[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float lo = __uint_as_float(vw[j] << 16) + 12582912.0f, hi = __uint_as_float(vw[j] & 0xffff0000u) + 12582912.0f;
            pair[j] = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x0040);
        }
        out[0] = __byte_perm(pair[0], pair[1], 0x5410);
        out[1] = __byte_perm(pair[2], pair[3], 0x5410);
    }
};

// The running absmax of VEC columns, in the reference's sense: max over abs_(w), starting from lowest().
template <typename T, int VEC>
struct AbsMaxVec {
    T m[VEC];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < VEC; ++i) m[i] = Arith<T>::lowest();
    }
    __device__ __forceinline__ void add(const Vec<T, VEC> &x) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) m[i] = Arith<T>::max_(m[i], Arith<T>::abs_(x.v[i]));
    }
    // The maxima over this thread's values and those of the lanes `TX`, `2 TX`, ... away in its warp (TX = 32: its own).
    template <int TX>
    __device__ __forceinline__ void finish(T *out) {
#pragma unroll
        for (int off = TX; off < 32; off <<= 1) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) m[i] = Arith<T>::max_(m[i], __shfl_xor_sync(0xffffffffu, m[i], off));
        }
#pragma unroll
        for (int i = 0; i < VEC; ++i) out[i] = m[i];
    }
};

// f16 and bf16, two columns per instruction: the running maximum `hi` and minimum `lo` of the values themselves (__hmax2 /
// __hmin2 skip a NaN operand and order -0 below +0, exactly as the __hmax of the element-wise form does), folded
// at the end.  abs_ leaves w >= 0 (both zeros and +inf included) as it is, negates w < 0, and turns a NaN into a
// NaN, which max_ skips; so the element-wise result over a set of values is
//     max(lowest, the largest non-NaN value, -(the smallest value) if that one is below zero)
// and hi starts at lowest (minus infinity for bf16, what -3.4e38 rounds to).  The zero cases: only -0 (and NaN) seen gives hi = lo = -0 and the result -0, as the
// element-wise form gives; one +0 makes hi = +0.  Nothing seen, or only NaN, leaves lowest.
template <typename T>
struct Packed;  // the two-element type of a 16-bit T
template <>
struct Packed<__half> {
    typedef __half2 Type;
    static __device__ __forceinline__ __half2 all(__half v) { return __half2half2(v); }
};
template <>
struct Packed<__nv_bfloat16> {
    typedef __nv_bfloat162 Type;
    static __device__ __forceinline__ __nv_bfloat162 all(__nv_bfloat16 v) { return __bfloat162bfloat162(v); }
};
template <typename T>
struct AbsMaxPacked {
    typedef typename Packed<T>::Type T2;
    T2 hi[4], lo[4];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            hi[j] = Packed<T>::all(Arith<T>::lowest());
            lo[j] = Packed<T>::all(-Arith<T>::lowest());
        }
    }
    __device__ __forceinline__ void add(const Vec<T, 8> &x) {
        const T2 *x2 = reinterpret_cast<const T2 *>(x.v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            hi[j] = __hmax2(hi[j], x2[j]);
            lo[j] = __hmin2(lo[j], x2[j]);
        }
    }
    template <int TX>
    __device__ __forceinline__ void finish(T *out) {
        const T2 zero = Packed<T>::all((T)0.0f), lowest = Packed<T>::all(Arith<T>::lowest());
        const uint32_t lowest2 = *reinterpret_cast<const uint32_t *>(&lowest);
        T2 m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // per half: lo < 0 ? max(hi, -lo) : hi, written as max(hi, lo < 0 ? -lo : lowest); hi >= lowest always
            const uint32_t below = __hlt2_mask(lo[j], zero);
            const T2 neg = __hneg2(lo[j]);
            const uint32_t cand = (*reinterpret_cast<const uint32_t *>(&neg) & below) | (lowest2 & ~below);
            m[j] = __hmax2(hi[j], *reinterpret_cast<const T2 *>(&cand));
        }
#pragma unroll
        for (int off = TX; off < 32; off <<= 1) {
#pragma unroll
            for (int j = 0; j < 4; ++j) m[j] = __hmax2(m[j], __shfl_xor_sync(0xffffffffu, m[j], off));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            out[2 * j] = m[j].x;
            out[2 * j + 1] = m[j].y;
        }
    }
};
template <>
struct AbsMaxVec<__half, 8> : AbsMaxPacked<__half> {};
template <>
struct AbsMaxVec<__nv_bfloat16, 8> : AbsMaxPacked<__nv_bfloat16> {};

constexpr int kThreads = 256;
constexpr int kMaxCluster = 8;   // the largest portable cluster

// ---------------------------------------------------------------------------------------------
// reduce over rows (Hidet dims=0): scale[cols]
// ---------------------------------------------------------------------------------------------
// 16 bytes global -> shared without passing through registers.
__device__ __forceinline__ void copy_async_16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// All of this thread's earlier asynchronous copies have landed.
__device__ __forceinline__ void copy_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// The two halves of a cluster barrier that publishes nothing: it only tells that every CTA of the cluster runs.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

// grid = (cluster_size, panels); the CTAs of one cluster share blockIdx.y (a panel of PW = TX*VEC
// columns) and split the rows.  TX threads lie across a panel row, kThreads / TX rows make a sweep.
// CACHE: the CTA's rows of the panel are kept in dynamic shared memory between the two phases
// (with VEC > 1 they are brought there by asynchronous 16-byte copies, all in flight at once, and the
// absmax is taken from shared memory); without, phase 2 reads them again from global memory.
// Each thread reads back only what it copied itself, so the copies need no barrier.
// Two kernels, since the one without holds a batch of vectors in registers: with both in one, four CTAs shared an SM for five and
// 1353 x 2432 f16 took 7.3 us for 5.6.  The one without gains from registers (one CTA asked for an SM, 100000 x 512 f32 129 us -> 106); element by
// element it is CTAs that count (eight an SM, 1000 x 40001 f32 per row 96 -> 73).
template <typename T, typename Q, int VEC, int TX, bool CACHE>
__global__ void __launch_bounds__(kThreads, VEC == 1 ? 8 : (CACHE ? 0 : 1)) quantize_cols_kernel(const T *w, Q *wq,
                                                                 T *scale, int64_t rows, int64_t cols,
                                                                 int64_t rows_per_cta) {
    constexpr int TY = kThreads / TX;          // rows per sweep
    constexpr int PW = TX * VEC;               // panel width in elements
    constexpr int WARPS = kThreads / 32;
    constexpr bool ASYNC = VEC > 1;            // a vector is 16 bytes whenever VEC > 1
    using A = Arith<T>;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) T red[WARPS][PW];
    __shared__ T recv[kMaxCluster][PW];        // recv[r]: the partial maxima of the cluster's CTA r
    __shared__ __align__(16) typename A::Divisor div_s[PW];

    T *tile = reinterpret_cast<T *>(smem_raw);

    cg::cluster_group cluster = cg::this_cluster();
    cluster_arrive_relaxed();                  // waited for before the first store into a peer's shared memory
    pdl_wait();
    const int tx = threadIdx.x % TX;
    const int ty = threadIdx.x / TX;
    const int64_t col = (int64_t)blockIdx.y * PW + (int64_t)tx * VEC;
    const bool col_ok = col < cols;            // cols % VEC == 0 whenever VEC > 1
    const int64_t row0 = (int64_t)blockIdx.x * rows_per_cta;
    int64_t nrows64 = rows - row0;
    if (nrows64 > rows_per_cta) nrows64 = rows_per_cta;
    if (nrows64 < 0) nrows64 = 0;
    const int nrows = (int)nrows64;            // at most rows_per_cta, which the launcher keeps below 2^31
    const int64_t sweep = (int64_t)TY * cols;  // elements between two rows of this thread

    // ---- phase 1: partial absmax of this CTA's rows ----
    AbsMaxVec<T, VEC> acc;
    acc.init();
    if (col_ok) {
        const T *src = w + (row0 + ty) * cols + col;
        if (ASYNC && CACHE) {
            uint32_t dst = smem_u32(tile) + (uint32_t)((ty * PW + tx * VEC) * sizeof(T));
            for (int r = ty; r < nrows; r += TY, src += sweep, dst += (uint32_t)(TY * PW * sizeof(T))) copy_async_16(dst, src);
            copy_async_wait_all();
            const T *t = tile + ty * PW + tx * VEC;
#pragma unroll 4
            for (int r = ty; r < nrows; r += TY, t += TY * PW) acc.add(load_vec<T, VEC>(t));
        } else {
            T *t = tile + ty * PW + tx * VEC;
#pragma unroll 4
            for (int r = ty; r < nrows; r += TY, src += sweep, t += TY * PW) {
                Vec<T, VEC> x = load_vec<T, VEC>(src);
                if (CACHE) store_vec<T, VEC>(t, x);
                acc.add(x);
            }
        }
    }
    T m[VEC];
    acc.template finish<TX>(m);                // over the rows of a sweep that this warp holds: lanes tx, tx + TX, ...
    if ((threadIdx.x & 31) < TX) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) red[threadIdx.x >> 5][tx * VEC + i] = m[i];
    }
    __syncthreads();
    // ---- exchange inside the cluster: every CTA writes its partial maxima into all the others' shared memory ----
    cluster_wait();                            // every CTA of the cluster has started
    const unsigned int n_cta = cluster.num_blocks();
    if (threadIdx.x < PW) {
        T a = A::lowest();
#pragma unroll
        for (int j = 0; j < WARPS; ++j) a = A::max_(a, red[j][threadIdx.x]);
        const unsigned int me = cluster.block_rank();
        for (unsigned int r = 0; r < n_cta; ++r) cluster.map_shared_rank(&recv[0][0], r)[me * PW + threadIdx.x] = a;
    }
    cluster.sync();  // the stores above are visible after it; nobody reads or writes a peer's memory from here on
    // one thread per column makes its scale and divisor
    if (threadIdx.x < PW) {
        T v[kMaxCluster];
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) v[r] = ((unsigned)r < n_cta) ? recv[r][threadIdx.x] : A::lowest();
        T a = A::lowest();
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) a = A::max_(a, v[r]);
        const T s = A::div_(a, A::qmax(QMax<Q>::value));
        div_s[threadIdx.x] = A::prepare(s);
        const int64_t c = (int64_t)blockIdx.y * PW + threadIdx.x;
        if (blockIdx.x == 0 && c < cols) scale[c] = s;
    }
    __syncthreads();

    // ---- phase 2: quantize ----
    if (col_ok) {
        typename A::Divisor s[VEC];
#pragma unroll
        for (int i = 0; i < VEC; ++i) s[i] = div_s[tx * VEC + i];
        const T *src = w + (row0 + ty) * cols + col;
        Q *dst = wq + (row0 + ty) * cols + col;
        if (CACHE) {
            const T *t = tile + ty * PW + tx * VEC;
#pragma unroll 4
            for (int r = ty; r < nrows; r += TY, dst += sweep, t += TY * PW) {
                Vec<Q, VEC> q;
                QuantVec<T, Q, VEC, typename A::Divisor>::template run<true>(load_vec<T, VEC>(t), s, q);
                store_vec<Q, VEC>(dst, q);
            }
        } else {
            constexpr int BATCH = 4;
            int left = nrows - ty;
            for (; left > (BATCH - 1) * TY; left -= BATCH * TY, src += BATCH * sweep, dst += BATCH * sweep) {
                Vec<T, VEC> x[BATCH];
#pragma unroll
                for (int i = 0; i < BATCH; ++i) x[i] = load_vec<T, VEC>(src + i * sweep);
#pragma unroll
                for (int i = 0; i < BATCH; ++i) {
                    Vec<Q, VEC> q;
                    QuantVec<T, Q, VEC, typename A::Divisor>::template run<true>(x[i], s, q);
                    store_vec<Q, VEC>(dst + i * sweep, q);
                }
            }
            for (; left > 0; left -= TY, src += sweep, dst += sweep) {
                Vec<Q, VEC> q;
                QuantVec<T, Q, VEC, typename A::Divisor>::template run<true>(load_vec<T, VEC>(src), s, q);
                store_vec<Q, VEC>(dst, q);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// reduce over columns (Hidet dims=-1): scale[rows]; one CTA per row, warp-shuffle reduction
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T warp_max(T a) {
    using A = Arith<T>;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) a = A::max_(a, __shfl_xor_sync(0xffffffffu, a, off));
    return a;
}

// REG_CHUNKS: vectors of the row each thread keeps in registers between the two phases; rows longer
// than blockDim * VEC * REG_CHUNKS read the remainder again (it is in L1/L2 by then).
// Four or five CTAs an SM (600 x 24576 f32 24 us with four, 19 with five), eight of the element-wise form.
template <typename T, typename Q, int VEC, int REG_CHUNKS>
__global__ void __launch_bounds__(kThreads, VEC == 1 ? 8 : (sizeof(T) == 4 ? 5 : 4)) quantize_rows_kernel(const T *w, Q *wq,
                                                                 T *scale, int64_t rows, int64_t cols) {
    using A = Arith<T>;
    __shared__ T warp_part[kThreads / 32];
    __shared__ T amax_s;

    pdl_wait();
    const int64_t row = blockIdx.x;
    const T *src = w + row * cols;
    Q *dst = wq + row * cols;
    const int64_t nvec = cols / VEC;  // cols % VEC == 0 whenever VEC > 1
    const int64_t stride = blockDim.x;

    Vec<T, VEC> keep[REG_CHUNKS];
    AbsMaxVec<T, VEC> acc;
    acc.init();
#pragma unroll
    for (int j = 0; j < REG_CHUNKS; ++j) {
        const int64_t i = threadIdx.x + j * stride;
        if (i < nvec) {
            keep[j] = load_vec<T, VEC>(src + i * VEC);
            acc.add(keep[j]);
        }
    }
    for (int64_t i = threadIdx.x + REG_CHUNKS * stride; i < nvec; i += stride) acc.add(load_vec<T, VEC>(src + i * VEC));
    T each[VEC];
    acc.template finish<32>(each);
    T m = A::lowest();
#pragma unroll
    for (int e = 0; e < VEC; ++e) m = A::max_(m, each[e]);
    m = warp_max<T>(m);
    if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int nwarps = (blockDim.x + 31) >> 5;
        T a = (threadIdx.x < nwarps) ? warp_part[threadIdx.x] : A::lowest();
        a = warp_max<T>(a);
        if (threadIdx.x == 0) amax_s = a;
    }
    __syncthreads();
    const T s_val = A::div_(amax_s, A::qmax(QMax<Q>::value));
    if (threadIdx.x == 0) scale[row] = s_val;
    const typename A::Divisor s = A::prepare(s_val);

#pragma unroll
    for (int j = 0; j < REG_CHUNKS; ++j) {
        const int64_t i = threadIdx.x + j * stride;
        if (i < nvec) {
            Vec<Q, VEC> q;
            QuantVec<T, Q, VEC, typename A::Divisor>::template run<false>(keep[j], &s, q);
            store_vec<Q, VEC>(dst + i * VEC, q);
        }
    }
    constexpr int BATCH = 4;
    int64_t i = threadIdx.x + REG_CHUNKS * stride;
    for (; i + (BATCH - 1) * stride < nvec; i += BATCH * stride) {
        Vec<T, VEC> x[BATCH];
#pragma unroll
        for (int j = 0; j < BATCH; ++j) x[j] = load_vec<T, VEC>(src + (i + j * stride) * VEC);
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            Vec<Q, VEC> q;
            QuantVec<T, Q, VEC, typename A::Divisor>::template run<false>(x[j], &s, q);
            store_vec<Q, VEC>(dst + (i + j * stride) * VEC, q);
        }
    }
    for (; i < nvec; i += stride) {
        Vec<Q, VEC> q;
        QuantVec<T, Q, VEC, typename A::Divisor>::template run<false>(load_vec<T, VEC>(src + i * VEC), &s, q);
        store_vec<Q, VEC>(dst + i * VEC, q);
    }
}

// A warp per row, for rows of at most half of kRowCtaBytes: the row is brought into the warp's part of shared memory by
// asynchronous 16-byte copies, all in flight at once, and both phases read it from there.  A lane reads back only
// what it copied itself and the warps of a CTA share nothing, so there is no barrier; the reduction is one round
// of warp shuffles instead of a CTA's.  grid = ceil(rows / W) CTAs of W <= kRowWarps warps (fewer for long rows, so
// that a CTA's rows stay near kRowCtaBytes and several CTAs fit an SM).
constexpr int kRowWarps = 4;
constexpr size_t kRowCtaBytes = 48 * 1024 - 64;  // the kernels keep a few bytes statically
constexpr size_t kLongRowBytes = 96 * 1024;       // two CTAs an SM

template <typename T, typename Q, int VEC>
__global__ void __launch_bounds__(kRowWarps * 32) quantize_rows_warp_kernel(const T *w, Q *wq,
                                                                            T *scale, int64_t rows, int64_t cols) {
    using A = Arith<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (row >= rows) return;
    const int nvec = (int)(cols / VEC);       // cols % VEC == 0, and a row is at most kRowCtaBytes
    T *mine = reinterpret_cast<T *>(smem_raw) + (size_t)warp * cols;
    const T *src = w + row * cols;
    Q *dst = wq + row * cols;

    {
        const uint32_t base = smem_u32(mine);
        for (int i = lane; i < nvec; i += 32) copy_async_16(base + (uint32_t)(i * VEC * sizeof(T)), src + (size_t)i * VEC);
        copy_async_wait_all();
    }
    AbsMaxVec<T, VEC> acc;
    acc.init();
#pragma unroll 4
    for (int i = lane; i < nvec; i += 32) acc.add(load_vec<T, VEC>(mine + (size_t)i * VEC));
    T each[VEC];
    acc.template finish<32>(each);
    T m = A::lowest();
#pragma unroll
    for (int e = 0; e < VEC; ++e) m = A::max_(m, each[e]);
    m = warp_max<T>(m);
    const T s_val = A::div_(m, A::qmax(QMax<Q>::value));
    if (lane == 0) scale[row] = s_val;
    const typename A::Divisor s = A::prepare(s_val);
#pragma unroll 4
    for (int i = lane; i < nvec; i += 32) {
        Vec<Q, VEC> q;
        QuantVec<T, Q, VEC, typename A::Divisor>::template run<false>(load_vec<T, VEC>(mine + (size_t)i * VEC), &s, q);
        store_vec<Q, VEC>(dst + (size_t)i * VEC, q);
    }
}

// ---------------------------------------------------------------------------------------------
// widths that are not multiples of a vector
// ---------------------------------------------------------------------------------------------
// A matrix without gaps between its rows is one run of elements, and runs are read and written in aligned vectors wherever the rows
// begin.  A vector at the end of a row holds elements of the next one, which each kernel leaves out in its own way.  Element by element,
// two bytes a load: 4147 x 8242 f16 per row 55.4 us, 31.8 so; 2024 x 3302 19.1 and 7.3; 2945 x 4447 restored with a scale per row 31.6 and
// 11.7.  (Per column such a form, panels of seven vectors read as eight, gains nothing: 2024 x 3302 16.3 us for 14.5, 4147 x 8242 61.9 for 65.8.)

// The bytes of a 16-byte piece that lie inside an array of `total` elements.
template <typename T, int VEC>
__device__ __forceinline__ int bytes_inside(int64_t first, int64_t total) {
    const int64_t left = total - first;
    return left >= VEC ? 16 : (left > 0 ? (int)(left * (int64_t)sizeof(T)) : 0);
}
__device__ __forceinline__ void copy_async_part(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
template <typename T>
__device__ __forceinline__ T nan_of();
template <>
__device__ __forceinline__ __half nan_of<__half>() { return __ushort_as_half(0x7fff); }
template <>
__device__ __forceinline__ __nv_bfloat16 nan_of<__nv_bfloat16>() { return __ushort_as_bfloat16(0x7fff); }
template <>
__device__ __forceinline__ float nan_of<float>() { return __uint_as_float(0x7fffffffu); }

// quantize_rows_warp_kernel for any row length: a warp, or for long rows a CTA (LONG), copies the vectors that its row touches.  In the
// first and the last one the neighbours' elements are NaN for the maximum, which skips it, and are not written.
template <typename T, typename Q, int VEC, bool LONG>
__global__ void __launch_bounds__(kRowWarps * 32) quantize_rows_flat_kernel(const T *w, Q *wq, T *scale, int64_t rows, int64_t cols, int row_bytes) {
    using A = Arith<T>;
    constexpr int STEP = LONG ? kRowWarps * 32 : 32;  // threads per row
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ T part[kRowWarps];
    pdl_wait();
    const int of_cta = threadIdx.x / STEP, lane = threadIdx.x % STEP;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x / STEP) + of_cta;
    if (row >= rows) return;
    const int64_t begin = row * cols, first = begin / VEC * VEC;
    const int head = (int)(begin - first), stop = head + (int)cols;  // the row's elements, counted from `first`
    const int nvec = (stop + VEC - 1) / VEC;
    T *mine = reinterpret_cast<T *>(smem_raw + (size_t)of_cta * row_bytes);
    const uint32_t base = smem_u32(mine);
    for (int i = lane; i < nvec; i += STEP) copy_async_part(base + i * 16, w + first + i * VEC, bytes_inside<T, VEC>(first + i * VEC, rows * cols));
    copy_async_wait_all();
    AbsMaxVec<T, VEC> acc;
    acc.init();
#pragma unroll 4
    for (int i = lane; i < nvec; i += STEP) {
        Vec<T, VEC> x = load_vec<T, VEC>(mine + i * VEC);
        if (i == 0 || i == nvec - 1) {
#pragma unroll
            for (int e = 0; e < VEC; ++e)
                if (i * VEC + e < head || i * VEC + e >= stop) x.v[e] = nan_of<T>();
        }
        acc.add(x);
    }
    T each[VEC];
    acc.template finish<32>(each);
    T m = A::lowest();
#pragma unroll
    for (int e = 0; e < VEC; ++e) m = A::max_(m, each[e]);
    m = warp_max<T>(m);
    if (LONG) {
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
        __syncthreads();
        m = A::lowest();
#pragma unroll
        for (int i = 0; i < kRowWarps; ++i) m = A::max_(m, part[i]);
    }
    const T s_val = A::div_(m, A::qmax(QMax<Q>::value));
    if (lane == 0) scale[row] = s_val;
    const typename A::Divisor s = A::prepare(s_val);
    Q *dst = wq + first;
#pragma unroll 4
    for (int i = lane; i < nvec; i += STEP) {
        const Vec<T, VEC> x = load_vec<T, VEC>(mine + i * VEC);
        Vec<Q, VEC> q;
        QuantVec<T, Q, VEC, typename A::Divisor>::template run<false>(x, &s, q);
        if (i * VEC >= head && (i + 1) * VEC <= stop) {
            store_vec<Q, VEC>(dst + i * VEC, q);
        } else {
#pragma unroll
            for (int e = 0; e < VEC; ++e)
                if (i * VEC + e >= head && i * VEC + e < stop) dst[i * VEC + e] = q.v[e];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// dequantize: a CTA covers kDqRows rows of kDqVecs vectors; a thread keeps its column and walks the rows
// ---------------------------------------------------------------------------------------------
// VEC codes -> values.  The general form applies Arith<T>::dequant element by element.
template <typename T, typename Q, int VEC>
struct DequantVec {
    template <bool PER_ELEMENT>
    static __device__ __forceinline__ void run(const Vec<Q, VEC> &q, const T *s, Vec<T, VEC> &out) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) out.v[e] = Arith<T>::template dequant<Q>(q.v[e], s[PER_ELEMENT ? e : 0]);
    }
};

// int8 -> f16, two per instruction with the same bits: 0x6400 | (b ^ 0x80) is the f16 number 1024 + (b + 128), and
// subtracting 1152 leaves b exactly, the value __short2half_rn gives; the product with the scale is then the same
// single f16 multiplication.
template <>
struct DequantVec<__half, int8_t, 8> {
    template <bool PER_ELEMENT>
    static __device__ __forceinline__ void run(const Vec<int8_t, 8> &q, const __half *s, Vec<__half, 8> &out) {
        const uint32_t *qw = reinterpret_cast<const uint32_t *>(q.v);
        const __half2 *s2 = reinterpret_cast<const __half2 *>(s);
        const __half2 s_all = PER_ELEMENT ? __half2() : __half2half2(s[0]);
        __half2 *o2 = reinterpret_cast<__half2 *>(out.v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // bytes (2j, 2j+1) of the vector into the low bytes of the two halves, 0x64 above each, sign bit flipped
            const uint32_t placed = __byte_perm(qw[j >> 1], 0x64646464u, (j & 1) ? 0x4342 : 0x4140) ^ 0x00800080u;
            uint32_t exact;
            asm("sub.f16x2 %0, %1, %2;" : "=r"(exact) : "r"(placed), "r"(0x64806480u));
            o2[j] = __hmul2(*reinterpret_cast<const __half2 *>(&exact), PER_ELEMENT ? s2[j] : s_all);
        }
    }
};

constexpr int kDqVecs = 32;                       // vectors across a CTA (one warp wide)
constexpr int kDqSweep = kThreads / kDqVecs;      // rows per sweep
constexpr int kDqRows = 2 * kDqSweep;             // rows per CTA

// grid = (column blocks, row blocks % kDqGridY, row blocks / kDqGridY): the CTAs that run together write whole rows, the pages of
// memory in order.  Row blocks first, four rows a thread: 4096 x 11008 28.8 us against 26.8, 1000 x 3000 6.3 against 4.2;
// eight rows a thread 33; streaming stores make no difference.
constexpr int64_t kDqGridY = 65535;
template <typename T, typename Q, int VEC>
__global__ void __launch_bounds__(kThreads) dequantize_kernel(const Q *wq, const T *scale,
                                                              T *w, int64_t rows, int64_t cols,
                                                              int reduce_dim) {
    pdl_wait();
    const int64_t c = ((int64_t)blockIdx.x * kDqVecs + (threadIdx.x % kDqVecs)) * VEC;
    if (c >= cols) return;                        // cols % VEC == 0 whenever VEC > 1
    const int64_t r0 = ((int64_t)blockIdx.z * kDqGridY + blockIdx.y) * kDqRows + threadIdx.x / kDqVecs;
    const Q *src = wq + r0 * cols + c;
    T *dst = w + r0 * cols + c;
    const int64_t sweep = (int64_t)kDqSweep * cols;
    static_assert(kDqRows == 2 * kDqSweep, "two rows a thread");
    if (r0 >= rows) return;
    if (r0 + kDqSweep >= rows) {                  // one row: a way of its own is shorter for the smallest matrices (5 x 256 1.0 -> 0.8 us)
        Vec<T, VEC> o;
        if (reduce_dim == 0) {
            DequantVec<T, Q, VEC>::template run<true>(load_l2<Q, VEC>(src), load_vec<T, VEC>(scale + c).v, o);
        } else {
            const T s = scale[r0];
            DequantVec<T, Q, VEC>::template run<false>(load_l2<Q, VEC>(src), &s, o);
        }
        store_vec<T, VEC>(dst, o);
        return;
    }
    const Vec<Q, VEC> q0 = load_l2<Q, VEC>(src), q1 = load_l2<Q, VEC>(src + sweep);
    Vec<T, VEC> o0, o1;
    if (reduce_dim == 0) {
        const Vec<T, VEC> s = load_vec<T, VEC>(scale + c);
        DequantVec<T, Q, VEC>::template run<true>(q0, s.v, o0);
        DequantVec<T, Q, VEC>::template run<true>(q1, s.v, o1);
    } else {
        const T s0 = scale[r0], s1 = scale[r0 + kDqSweep];
        DequantVec<T, Q, VEC>::template run<false>(q0, &s0, o0);
        DequantVec<T, Q, VEC>::template run<false>(q1, &s1, o1);
    }
    store_vec<T, VEC>(dst, o0);
    store_vec<T, VEC>(dst + sweep, o1);
}

// The same for any width of at least VEC: VEC rows together are whole vectors, so a thread takes the same vector of every group of
// VEC rows; it holds elements of one row or of two, at the same columns in each group.  grid = (vectors of a group, groups / kDqGroups)
// One vector at a time: all four in front of the stores take registers, and CTAs hide more (4000 x 20001 f16 70 us so, 54 one by one, bf16 102 and 55).
// The scales of the columns go through shared memory: fetched by each thread for itself, two bytes at a time, they ask the same few lines of L2
// too often (895 x 327 6.7 us, 4.1 element by element).
constexpr int kDqGroups = 4;                      // per thread and trip
template <typename T, typename Q, int VEC>
__global__ void __launch_bounds__(kThreads) dequantize_flat_kernel(const Q *wq, const T *scale, T *w, int64_t rows, int64_t cols, int reduce_dim) {
    __shared__ __align__(16) T col_scale[kThreads * VEC];
    pdl_wait();
    const int64_t v0 = (int64_t)blockIdx.x * kThreads, v = v0 + threadIdx.x;
    if (reduce_dim == 0) {
        const unsigned int width = (unsigned int)cols, c0 = (unsigned int)(v0 * VEC % cols);  // the launcher keeps cols below 2^22
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            const unsigned int at = threadIdx.x + i * kThreads;
            col_scale[at] = scale[(c0 + at) % width];
        }
        __syncthreads();
    }
    if (v >= cols) return;                        // a group is VEC * cols elements
    const int64_t row = v * VEC / cols, col = v * VEC - row * cols;
    const int here = cols - col < VEC ? (int)(cols - col) : VEC;  // elements in the first of the two rows
    const int64_t total = rows * cols, groups = (rows + VEC - 1) / VEC;
    Vec<T, VEC> s;
    if (reduce_dim == 0) s = load_vec<T, VEC>(col_scale + threadIdx.x * VEC);
    for (int64_t g0 = (int64_t)blockIdx.y * kDqGroups; g0 < groups; g0 += (int64_t)gridDim.y * kDqGroups) {
#pragma unroll
        for (int i = 0; i < kDqGroups; ++i) {
            const int64_t r = (g0 + i) * VEC + row, at = ((g0 + i) * cols + v) * VEC;
            if (r >= rows) break;
            if (reduce_dim != 0) {
                const T s0 = scale[r], s1 = here < VEC && r + 1 < rows ? scale[r + 1] : s0;
#pragma unroll
                for (int e = 0; e < VEC; ++e) s.v[e] = e < here ? s0 : s1;
            }
            Vec<T, VEC> out;
            if (at + VEC <= total) {
                DequantVec<T, Q, VEC>::template run<true>(load_vec<Q, VEC>(wq + at), s.v, out);
                store_vec<T, VEC>(w + at, out);
            } else {                              // the end of the matrix
                for (int e = 0; at + e < total; ++e) w[at + e] = Arith<T>::template dequant<Q>(wq[at + e], s.v[e]);
            }
        }
    }
}

bool aligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// ---------------------------------------------------------------------------------------------
// embedding lookup in a row-quantized table: out[i, :] = T(table[idx[i], :]) * scale[idx[i]]
// ---------------------------------------------------------------------------------------------
constexpr int kEmbRows = 4 * kDqSweep;            // indices per CTA
// dequantize_kernel over the looked-up rows: a thread keeps its column and walks kEmbRows / kDqSweep
// indices.  The arithmetic is that of dequantize_kernel with reduce_dim = 1, so a lookup equals the row of the
// dequantized table bit for bit.  An index outside [0, vocab) (after adding vocab to a negative one) yields a row of
// zeros and sets bit 30 of the device status word.  grid = (index blocks, column blocks)
template <typename T, typename Q, typename I, int VEC>
__global__ void __launch_bounds__(kThreads) embedding_dequant_kernel(const Q *table, const T *scale,
                                                                     const I *idx, T *out, int64_t vocab,
                                                                     int64_t dim, int64_t n_idx, unsigned int *status) {
    pdl_wait();
    const int64_t c = ((int64_t)blockIdx.y * kDqVecs + (threadIdx.x % kDqVecs)) * VEC;
    if (c >= dim) return;                         // dim % VEC == 0 whenever VEC > 1
    const int64_t r0 = (int64_t)blockIdx.x * kEmbRows + threadIdx.x / kDqVecs;
    constexpr int EACH = kEmbRows / kDqSweep;
    int64_t row[EACH];                            // -1: outside the table
    T s[EACH];
    Vec<Q, VEC> q[EACH];
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        const int64_t r = r0 + i * kDqSweep;
        row[i] = r < n_idx ? (int64_t)idx[r] : -1;
    }
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        if (r0 + i * kDqSweep >= n_idx) break;
        if (row[i] < 0) row[i] += vocab;
        if (row[i] < 0 || row[i] >= vocab) {
            row[i] = -1;
        } else {
            s[i] = scale[row[i]];
            q[i] = load_vec<Q, VEC>(table + row[i] * dim + c);
        }
    }
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
        const int64_t r = r0 + i * kDqSweep;
        if (r >= n_idx) break;
        Vec<T, VEC> o;
        if (row[i] < 0) {
#pragma unroll
            for (int e = 0; e < VEC; ++e) o.v[e] = (T)0.0f;
            if (c == 0 && status != nullptr) atomicOr(status, 0x40000000u);
        } else {
            DequantVec<T, Q, VEC>::template run<false>(q[i], &s[i], o);
        }
        store_vec<T, VEC>(out + r * dim + c, o);
    }
}

// A launch as a programmatic dependent of the kernel in front, in clusters of `cluster` CTAs along x.
template <typename... Params, typename... Args>
int launch_dependent(const char *name, void (*kernel)(Params...), dim3 grid, int threads, size_t smem, int cluster, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = (unsigned)cluster;
    attrs[1].val.clusterDim.y = 1;
    attrs[1].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    if (err != cudaSuccess) return set_error(B200Q_CUDA_ERROR, "launch of %s failed: %s", name, cudaGetErrorString(err));
    return B200Q_OK;
}

// Largest dynamic shared memory a quantize_cols CTA may ask for (the static arrays need a little).
constexpr size_t kMaxTileBytes = 200 * 1024;
// What it may ask for by default: 48 KB with the static arrays, a few KB of them.
constexpr size_t kDefaultTileBytes = 40 * 1024;

// Threads across a panel row when a thread moves a 16-byte vector: 4 make a panel of 64 bytes per row (32 f16
// columns), so that a [4096, 4096] weight gives 1024 CTAs of 32 KB, several to an SM and more than one wave.
constexpr int kPanelThreads = 4;

template <typename T, typename Q, int VEC, int TX>
int launch_quantize_cols(const T *w, Q *wq, T *scale, int64_t rows, int64_t cols, cudaStream_t stream) {
    constexpr int TY = kThreads / TX;
    constexpr int PW = TX * VEC;
    const int64_t panels = ceil_div(cols, PW);
    if (panels > 65535) return set_error(B200Q_UNSUPPORTED, "symmetric_quantize: %lld columns exceed the grid limit", (long long)cols);

    // Split the rows over the largest portable cluster that still leaves every CTA a full sweep,
    // and keep the slice in shared memory when it fits.
    int cluster = kMaxCluster;
    while (cluster > 1 && ceil_div(rows, cluster) < TY) cluster >>= 1;
    const int64_t rows_per_cta = ceil_div(rows, cluster);
    const size_t tile_bytes = (size_t)rows_per_cta * PW * sizeof(T);
    const dim3 grid((unsigned)cluster, (unsigned)panels, 1);
    if (tile_bytes > kMaxTileBytes) return launch_dependent("quantize_cols_kernel", quantize_cols_kernel<T, Q, VEC, TX, false>, grid, kThreads, 0, cluster, stream, w, wq, scale, rows, cols, rows_per_cta);
    auto kernel = quantize_cols_kernel<T, Q, VEC, TX, true>;
    if (tile_bytes > kDefaultTileBytes) {
        B200Q_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxTileBytes));
    }
    // Slices of about 32 KB leave six CTAs an SM.  Five are better where the sixth would empty the second wave but for a sliver (4096 x 4096 f16
    // 15.0 us with six, 14.3 with five), not where it is well filled or there are more (3800 x 5000 18.0 and 18.9, 4096 x 4096 f32 23.8 and 25.4,
    // 4096 x 14336 f16 39.1 and 39.5).
    size_t ask = tile_bytes;
    if (VEC > 1 && tile_bytes > 28 * 1024 && tile_bytes < 37 * 1024) {
        const int64_t wave = 6 * (int64_t)sm_count(), ctas = cluster * panels;
        if (wave > 0 && ctas > wave && ctas < 2 * wave && ctas % wave * 3 < wave) ask = 37 * 1024;
    }
    return launch_dependent("quantize_cols_kernel", kernel, grid, kThreads, ask, cluster, stream, w, wq, scale, rows, cols, rows_per_cta);
}

// VEC: elements per vector where bases are aligned (16 bytes of w), else 1.
template <typename T, typename Q, int VEC>
int launch_quantize_rows(const T *w, Q *wq, T *scale, int64_t rows, int64_t cols, cudaStream_t stream) {
    if (rows > 2147483647LL) return set_error(B200Q_UNSUPPORTED, "symmetric_quantize: %lld rows exceed the grid limit", (long long)rows);
    if constexpr (VEC > 1) {
        const bool whole = cols % VEC == 0;   // rows are whole vectors
        const size_t row_bytes = whole ? (size_t)cols * sizeof(T) : (size_t)(ceil_div(cols, VEC) + 1) * 16;
        int warps = (int)(kRowCtaBytes / row_bytes);
        warps = warps < 1 ? 1 : (warps > kRowWarps ? kRowWarps : warps);
        const size_t smem = warps * row_bytes;  // at most kRowCtaBytes, with a few static bytes the default limit for shared memory
        const dim3 grid((unsigned)ceil_div(rows, warps));
        // A row of more than half of a CTA's share has the whole CTA (a warp has few loads in flight for it, and few warps fit an SM): 4147 x 8242
        // f32 53 -> 34 us, 4096 x 12288 f16 39 -> 28, 674 x 6912 f32 12.2 -> 7.6.  Whole rows beyond that share are faster in the kernel below,
        // which keeps the SMs full (2000 x 20480 f32 61 us so, 45 there; 300 x 40960 f16 21 and 15), odd ones only beyond kLongRowBytes.
        // f32 rows that leave no SM more than one of them or two stay (120 x 24576 9.0 us so, 10.7 there; 64 x 12296 4.8 and 3.8).
        const int sms = sm_count() > 0 ? sm_count() : 148;
        const bool few = sizeof(T) == 4 && rows * 2 > sms && rows * 2 <= 3 * (int64_t)sms;
        if (row_bytes > kRowCtaBytes / 2 && row_bytes <= (whole && !few ? kRowCtaBytes : kLongRowBytes)) {
            auto kernel = quantize_rows_flat_kernel<T, Q, VEC, true>;
            if (row_bytes > kRowCtaBytes) B200Q_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLongRowBytes));
            return launch_dependent("quantize_rows_flat_kernel", kernel, dim3((unsigned)rows), kRowWarps * 32, row_bytes, 1, stream, w, wq, scale, rows, cols, (int)row_bytes);
        }
        if (whole && row_bytes <= kRowCtaBytes) return launch_dependent("quantize_rows_warp_kernel", quantize_rows_warp_kernel<T, Q, VEC>, grid, warps * 32, smem, 1, stream, w, wq, scale, rows, cols);
        // A warp a row needs rows to fill the SMs with, short ones more of them; with fewer, a CTA a row element by element is faster (256 x 513 f16
        // 1.7 us, 1.9 a warp a row, 256 x 4097 f32 3.7 and 5.2, 7 x 8466 bf16 6.0 and 7.9; but 1000 x 257 f16 2.4 and 1.9, 4000 x 33 2.6 and 2.2).
        if (!whole && row_bytes <= kRowCtaBytes && (rows >= 8 * (int64_t)sms || (rows >= 4 * (int64_t)sms && row_bytes >= 512)))
            return launch_dependent("quantize_rows_flat_kernel", quantize_rows_flat_kernel<T, Q, VEC, false>, grid, warps * 32, smem, 1, stream, w, wq, scale, rows, cols, (int)row_bytes);
        if (!whole) return launch_quantize_rows<T, Q, 1>(w, wq, scale, rows, cols, stream);
    }
    const int64_t nvec = cols / VEC;
    int threads = (int)round_up(nvec < 32 ? 32 : nvec, 32);
    if (threads > kThreads) threads = kThreads;
    return launch_dependent("quantize_rows_kernel", quantize_rows_kernel<T, Q, VEC, 4>, dim3((unsigned)rows), threads, 0, 1, stream, w, wq, scale, rows, cols);
}

template <typename T, typename Q>
int quantize_typed(const void *w_, void *wq_, void *scale_, int64_t rows, int64_t cols, int reduce_dim, cudaStream_t stream) {
    const T *w = static_cast<const T *>(w_);
    Q *wq = static_cast<Q *>(wq_);
    T *scale = static_cast<T *>(scale_);
    constexpr int VEC = 16 / sizeof(T);
    const bool bases_ok = aligned(w, 16) && aligned(wq, VEC * sizeof(Q));
    if (reduce_dim == 0) {
        return bases_ok && cols % VEC == 0 ? launch_quantize_cols<T, Q, VEC, kPanelThreads>(w, wq, scale, rows, cols, stream)
                                           : launch_quantize_cols<T, Q, 1, 32>(w, wq, scale, rows, cols, stream);
    }
    return bases_ok && cols >= VEC ? launch_quantize_rows<T, Q, VEC>(w, wq, scale, rows, cols, stream) : launch_quantize_rows<T, Q, 1>(w, wq, scale, rows, cols, stream);
}

template <typename T, typename Q>
int dequantize_typed(const void *wq_, const void *scale_, void *w_, int64_t rows, int64_t cols, int reduce_dim,
                     cudaStream_t stream) {
    const Q *wq = static_cast<const Q *>(wq_);
    const T *scale = static_cast<const T *>(scale_);
    T *w = static_cast<T *>(w_);
    constexpr int VEC = 16 / sizeof(T);  // 16-byte scale / output vectors; input vector is VEC * sizeof(Q)
    const bool vec_ok = (cols % VEC == 0) && aligned(w, 16) && aligned(wq, VEC * sizeof(Q)) && aligned(scale, 16);
    if (rows == 0 || cols == 0) return B200Q_OK;
    const int64_t row_blocks = ceil_div(rows, kDqRows);
    const int64_t col_blocks = ceil_div(vec_ok ? cols / VEC : cols, kDqVecs);
    if (row_blocks > kDqGridY * kDqGridY || col_blocks > 65535) {
        return set_error(B200Q_UNSUPPORTED, "symmetric_dequantize: [%lld, %lld] exceeds the grid limit", (long long)rows, (long long)cols);
    }
    // Vectors for widths that are not whole ones from 3 Mi elements and 96 columns on (48 with 16 Mi elements).  Below, element by element is faster: in
    // vectors a thread finds its rows by divisions and walks thirty-two of them, and a CTA covers 256 vectors of a row group that has `cols` (256 x 257
    // f16 1.0 us, 2.6 in vectors; 60000 x 9 2.9 and 6.2; 1000 x 2049 4.2 and 5.0; 1000 x 4097 8.4 and 6.3; 60000 x 129 16 and 11; 400000 x 63 42 and 29).
    const int64_t enough = (cols >= 96 ? 3 : 16) * (int64_t)1024 * 1024;
    if (cols % VEC != 0 && cols >= 48 && rows >= enough / cols && aligned(w, 16) && aligned(wq, VEC * sizeof(Q))) {
        const int64_t groups = ceil_div(ceil_div(rows, VEC), kDqGroups);
        return launch_dependent("dequantize_flat_kernel", dequantize_flat_kernel<T, Q, VEC>, dim3((unsigned)ceil_div(cols, kThreads), (unsigned)(groups < kDqGridY ? groups : kDqGridY)), kThreads, 0, 1,
                                stream, wq, scale, w, rows, cols, reduce_dim);
    }
    const dim3 grid((unsigned)col_blocks, (unsigned)(row_blocks < kDqGridY ? row_blocks : kDqGridY), (unsigned)ceil_div(row_blocks, kDqGridY));
    auto kernel = vec_ok ? dequantize_kernel<T, Q, VEC> : dequantize_kernel<T, Q, 1>;
    return launch_dependent("dequantize_kernel", kernel, grid, kThreads, 0, 1, stream, wq, scale, w, rows, cols, reduce_dim);
}

template <typename T, typename Q, typename I>
int embedding_typed(const void *table_, const void *scale_, const void *idx_, void *out_, int64_t vocab, int64_t dim, int64_t n_idx,
                    cudaStream_t stream) {
    const Q *table = static_cast<const Q *>(table_);
    const T *scale = static_cast<const T *>(scale_);
    const I *idx = static_cast<const I *>(idx_);
    T *out = static_cast<T *>(out_);
    constexpr int VEC = 16 / sizeof(T);
    const bool vec_ok = (dim % VEC == 0) && aligned(out, 16) && aligned(table, VEC * sizeof(Q));
    if (n_idx == 0 || dim == 0) return B200Q_OK;
    const int64_t row_blocks = ceil_div(n_idx, kEmbRows);
    const int64_t col_blocks = ceil_div(vec_ok ? dim / VEC : dim, kDqVecs);
    if (row_blocks > 2147483647LL || col_blocks > 65535) {
        return set_error(B200Q_UNSUPPORTED, "embedding_dequantize: %lld indices of %lld values exceed the grid limit", (long long)n_idx, (long long)dim);
    }
    const dim3 grid((unsigned)row_blocks, (unsigned)col_blocks, 1);
    unsigned int *status = device_status_word();
    auto kernel = vec_ok ? embedding_dequant_kernel<T, Q, I, VEC> : embedding_dequant_kernel<T, Q, I, 1>;
    return launch_dependent("embedding_dequant_kernel", kernel, grid, kThreads, 0, 1, stream, table, scale, idx, out, vocab, dim, n_idx, status);
}

int check_common(const char *op, const void *a, const void *b, const void *c, int64_t rows, int64_t cols, int f_type,
                 int q_type, int reduce_dim) {
    if (rows < 0 || cols < 0) return set_error(B200Q_INVALID_ARGUMENT, "%s: negative shape [%lld, %lld]", op, (long long)rows, (long long)cols);
    if (f_type < B200Q_F16 || f_type > B200Q_F32) return set_error(B200Q_INVALID_ARGUMENT, "%s: unknown float type %d", op, f_type);
    if (q_type < B200Q_I8 || q_type > B200Q_I16) return set_error(B200Q_INVALID_ARGUMENT, "%s: unknown quantized type %d", op, q_type);
    if (reduce_dim != 0 && reduce_dim != 1) return set_error(B200Q_INVALID_ARGUMENT, "%s: reduce_dim must be 0 or 1, got %d", op, reduce_dim);
    if (rows > 0 && cols > 0 && (a == nullptr || b == nullptr || c == nullptr)) return set_error(B200Q_INVALID_ARGUMENT, "%s: null pointer argument", op);
    return B200Q_OK;
}

}  // namespace
}  // namespace b200q

extern "C" {

B200Q_API int b200q_symmetric_quantize(const void *w, void *wq, void *scale, int64_t rows, int64_t cols, int w_type,
                                       int q_type, int reduce_dim, void *stream) {
    using namespace b200q;
    int rc = check_common("symmetric_quantize", w, wq, scale, rows, cols, w_type, q_type, reduce_dim);
    if (rc != B200Q_OK) return rc;
    // An empty reduced dimension has no maximum; the reference cannot build that task either.
    if (rows == 0 || cols == 0) {
        if ((reduce_dim == 0 ? cols : rows) == 0) return B200Q_OK;  // no outputs at all
        return set_error(B200Q_INVALID_ARGUMENT, "symmetric_quantize: empty reduction over shape [%lld, %lld]", (long long)rows, (long long)cols);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define B200Q_DISPATCH_Q(T)                                                                                    \
    (q_type == B200Q_I8 ? quantize_typed<T, int8_t>(w, wq, scale, rows, cols, reduce_dim, s)                   \
                        : quantize_typed<T, int16_t>(w, wq, scale, rows, cols, reduce_dim, s))
    switch (w_type) {
        case B200Q_F16: return B200Q_DISPATCH_Q(__half);
        case B200Q_BF16: return B200Q_DISPATCH_Q(__nv_bfloat16);
        default: return B200Q_DISPATCH_Q(float);
    }
#undef B200Q_DISPATCH_Q
}

B200Q_API int b200q_symmetric_dequantize(const void *wq, const void *scale, void *w, int64_t rows, int64_t cols,
                                         int scale_type, int q_type, int reduce_dim, void *stream) {
    using namespace b200q;
    int rc = check_common("symmetric_dequantize", wq, scale, w, rows, cols, scale_type, q_type, reduce_dim);
    if (rc != B200Q_OK) return rc;
    if (rows == 0 || cols == 0) return B200Q_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define B200Q_DISPATCH_DQ(T)                                                                                   \
    (q_type == B200Q_I8 ? dequantize_typed<T, int8_t>(wq, scale, w, rows, cols, reduce_dim, s)                 \
                        : dequantize_typed<T, int16_t>(wq, scale, w, rows, cols, reduce_dim, s))
    switch (scale_type) {
        case B200Q_F16: return B200Q_DISPATCH_DQ(__half);
        case B200Q_BF16: return B200Q_DISPATCH_DQ(__nv_bfloat16);
        default: return B200Q_DISPATCH_DQ(float);
    }
#undef B200Q_DISPATCH_DQ
}

B200Q_API int b200q_embedding_dequantize(const void *table, const void *scale, const void *indices, void *out, int64_t vocab,
                                         int64_t dim, int64_t n_indices, int scale_type, int q_type, int index_bytes, void *stream) {
    using namespace b200q;
    int rc = check_common("embedding_dequantize", table, scale, table, vocab, dim, scale_type, q_type, 1);
    if (rc != B200Q_OK) return rc;
    if (n_indices < 0) return set_error(B200Q_INVALID_ARGUMENT, "embedding_dequantize: negative index count %lld", (long long)n_indices);
    if (index_bytes != 4 && index_bytes != 8) return set_error(B200Q_INVALID_ARGUMENT, "embedding_dequantize: indices must be int32 or int64 (4 or 8 bytes), got %d", index_bytes);
    if (n_indices == 0 || dim == 0) return B200Q_OK;
    if (indices == nullptr || out == nullptr || table == nullptr || scale == nullptr) return set_error(B200Q_INVALID_ARGUMENT, "embedding_dequantize: null pointer argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define B200Q_DISPATCH_E2(T, Q)                                                                                    \
    (index_bytes == 8 ? embedding_typed<T, Q, int64_t>(table, scale, indices, out, vocab, dim, n_indices, s)      \
                      : embedding_typed<T, Q, int32_t>(table, scale, indices, out, vocab, dim, n_indices, s))
#define B200Q_DISPATCH_E(T) (q_type == B200Q_I8 ? B200Q_DISPATCH_E2(T, int8_t) : B200Q_DISPATCH_E2(T, int16_t))
    switch (scale_type) {
        case B200Q_F16: return B200Q_DISPATCH_E(__half);
        case B200Q_BF16: return B200Q_DISPATCH_E(__nv_bfloat16);
        default: return B200Q_DISPATCH_E(float);
    }
#undef B200Q_DISPATCH_E
#undef B200Q_DISPATCH_E2
}

}  // extern "C"
