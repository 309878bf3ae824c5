// Shared host/device helpers of libhidet_b200q.so: error state, launch checks and the sm_100a PTX
// wrappers (mbarrier, TMA, tcgen05) the kernels are written with.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/hidet_b200q.h"

namespace b200q {

// ---------------------------------------------------------------------------------------------
// host side: error state
// ---------------------------------------------------------------------------------------------

// Stores a printf-formatted message in the calling thread's error slot and returns `code`.
int set_error(int code, const char *fmt, ...);

#define B200Q_CUDA_TRY(expr)                                                                        \
    do {                                                                                            \
        cudaError_t err__ = (expr);                                                                 \
        if (err__ != cudaSuccess) {                                                                 \
            return ::b200q::set_error(B200Q_CUDA_ERROR, "%s failed: %s (%s:%d)", #expr,             \
                                      cudaGetErrorString(err__), __FILE__, __LINE__);               \
        }                                                                                           \
    } while (0)

// After a kernel launch: reports launch-configuration errors without synchronising.
#define B200Q_CHECK_LAUNCH(name)                                                                    \
    do {                                                                                            \
        cudaError_t err__ = cudaGetLastError();                                                     \
        if (err__ != cudaSuccess) {                                                                 \
            return ::b200q::set_error(B200Q_CUDA_ERROR, "launch of %s failed: %s", name,            \
                                      cudaGetErrorString(err__));                                   \
        }                                                                                           \
    } while (0)

// Device-global status word: a kernel whose bounded wait runs out ORs a code into it and returns.
// Code layout: bits 0..7 kernel id, bits 8..15 wait site, bit 31 set.
unsigned int *device_status_word();  // device address for the current device (nullptr on failure)

constexpr unsigned int kKernelDecode = 1;
constexpr unsigned int kKernelPrefill = 2;
constexpr unsigned int kKernelU4 = 3;
constexpr unsigned int kKernelUnaligned = 4;
constexpr unsigned int kKernelPair = 5;
constexpr unsigned int kKernelMid = 6;

// Number of SMs of the current device (cached per device).
int sm_count();

// Clusters of `cluster` CTAs (along y) of a kernel that run at once on the current device, asked of the runtime: clusters stay
// within a group of SMs, so it is less than what the slots add up to.  0 if it cannot be told.
int resident_clusters(const void *kernel, int threads, int smem, int cluster);
// True where the stream has only some of the device's SMs (a green context's): launches there may not hold what the device holds.
bool part_of_device(cudaStream_t stream);

// Encodes a 2-D tiled tensor map.  `inner`/`outer` are the tensor extents in elements, `row_bytes`
// the stride between consecutive outer indices, box_* the tile extents.  swizzle is a
// CUtensorMapSwizzle value.  Returns a b200q_status.
int make_tensor_map_2d(CUtensorMap *map, CUtensorMapDataType dtype, const void *base, uint64_t inner, uint64_t outer,
                       uint64_t row_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle,
                       CUtensorMapL2promotion promo);

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline int64_t round_up(int64_t a, int64_t b) { return ceil_div(a, b) * b; }

// ---------------------------------------------------------------------------------------------
// device side: PTX wrappers
// ---------------------------------------------------------------------------------------------
#ifdef __CUDACC__

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// One lane of the (fully converged) warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(pred));
    return pred != 0;
}

// ---- mbarrier ----
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One poll: returns true once the phase with the given parity has completed.  The thread may be
// suspended inside the instruction for up to about `kWaitHintNs` while the phase is pending, so a
// polling loop spends few issue slots.
constexpr uint32_t kWaitHintNs = 2000;
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(kWaitHintNs)
        : "memory");
    return ok != 0;
}

// The same without blocking.  An answer takes about 200 clocks even where the phase is long over, so a pipeline's loop asks for
// its next stage while it works on this one.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait on an mbarrier phase.  Returns false if `limit` polls passed without the phase
// completing; the caller then records the failure and leaves.  Each poll of try_wait already
// blocks for a hardware-defined interval, so the limit is a time bound of the order of a second.
constexpr uint32_t kSpinLimit = 1u << 20;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit = kSpinLimit) {
    for (uint32_t i = 0; i < limit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
    }
    return false;
}

// One answer for the 128 threads that meet at named barrier `id`: true where all of them bring true.  A wait that may give up is
// decided so in front of that barrier: with an answer per warp, one could leave and the others stay at the barrier for good.
__device__ __forceinline__ bool all_of_128(int id, bool ok) {
    uint32_t all;
    __syncwarp();
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.u32 p, %2, 0;\n\t"
        "bar.red.and.pred q, %1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}\n"
        : "=r"(all)
        : "r"(id), "r"((uint32_t)ok)
        : "memory");
    return all != 0;
}

// status[0] collects every wait that ran out (codes or-ed together: one failure starves the other
// roles, whose waits then run out too); status[1] keeps the first one.
__device__ __forceinline__ void report_timeout(unsigned int *status, unsigned int kernel, unsigned int site) {
    if (status != nullptr) {
        const unsigned int code = 0x80000000u | (site << 8) | kernel;
        atomicOr(status, code);
        atomicCAS(status + 1, 0u, code);
    }
}

// ---- TMA ----
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// 2-D tiled load global -> shared, completion counted in bytes on `bar`.  x is the inner
// (contiguous) coordinate in elements and must make x * element_size a multiple of 16.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int32_t x, int32_t y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap *map, int32_t x, int32_t y,
                                                 uint32_t bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%3, %4}], [%2], %5;"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "l"(policy)
        : "memory");
}
// Asks for a tile into L2 only.  L2 is where all writes meet, so this may run ahead of the kernel that writes the tile.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap *map, int32_t x, int32_t y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// Makes generic-proxy writes to shared memory visible to the async proxy (TMA, tcgen05.mma).
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- programmatic dependent launch ----
// launch_dependents: the next kernel in the stream may start its prologue once every CTA of this grid
// has said so.  wait: blocks until the previous kernel in the stream has completed and its writes are
// visible; a no-op when the kernel was not launched as a programmatic dependent.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// silu(g) = g / (1 + exp(-g)) for an epilogue: a quotient from an approximate reciprocal, corrected once by its remainder in fused multiply-adds
// (P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  Before its
// last rounding the corrected quotient is off by about 2^-44 of its value, so that it differs from the division's only where that lies on a rounding
// boundary, by one ulp: 2 of 350 million gates of 1e-38 to 88; largest and mean error against 64 bits are the division's (tests/test_silu_gpu.py).
// For gates of at most 2^125 in magnitude (sums of f16 times int8 end near 2^70); beyond, g * r may overflow.
// It has no branch: with the division a 32-row block of the kernel on SM pairs took 1.3 us, 3.6 where columns that only fill up the
// tile make its gates zeros, and 0.9 with this.
// d is a quarter of the divisor, which keeps its reciprocal a normal number for every finite exp(-g).  Where the remainder is zero (g may be
// -0) or, for an infinity, a NaN, the first quotient is the answer.
__device__ __forceinline__ float silu(float g) {
    const float d = fmaf(0.25f, __expf(-g), 0.25f);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    const float q = g * r, rest = fmaf(-d, q, g);
    return 0.25f * (fabsf(rest) > 0.0f ? fmaf(rest, r, q) : q);
}

// ---- warp-level tensor-core MMA ----
// D[16 x 8] += A[16 x 16] * B[16 x 8]: A row-major (the kernels here: 16 weight columns x 16 k), B column-major
// (16 k x 8 activation rows).
__device__ __forceinline__ void mma_m16n8k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                             uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- cluster primitives (a kernel launched without a cluster is a cluster of one) ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_acquire() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
    return r;
}
// Asynchronous stores into the shared memory of a CTA of the cluster; each adds its size to the transaction
// count of an mbarrier of that CTA once the data is there.
__device__ __forceinline__ void st_async_f32(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_v4f32(uint32_t addr, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar)
                 : "memory");
}
// One arrival on an mbarrier of a CTA of the cluster (address from map_to_rank).  The default release is at CTA scope: it publishes
// nothing that this thread stored in shared or global memory to the other CTA.  It is for a signal that carries no such stores,
// only that something is over: a phase of a barrier of this CTA whose copies have landed in its shared memory, accesses to tensor
// memory that tcgen05.wait and tcgen05.fence::before_thread_sync stand behind.  (With .release.cluster an arrival takes 350 clocks
// for 141, and the kernel on SM pairs, whose converters arrive once a stage, 1.6 to 2 times as long.)
__device__ __forceinline__ void mbar_arrive_remote(uint32_t remote_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
// Bounded wait on an mbarrier phase that remote CTAs complete (acquire at cluster scope).
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(kWaitHintNs)
            : "memory");
        if (ok) return true;
    }
    return false;
}
#endif  // __CUDACC__

}  // namespace b200q
