// What the streaming kernels on warp-level MMAs share (qlinear_u4.cu, qlinear_unaligned.cu): the warps of a CTA each hold an
// fp32 partial sum of the CTA's output tile, the CTAs of a cluster hold further ones (K is split over them), and all of
// them meet without a workspace and without a second launch.
#pragma once

#include <atomic>

#include "common.cuh"

namespace b200q {
namespace stream_mma {

constexpr int MAX_CLUSTER = 8;

#ifdef __CUDACC__

// Bytes of the receive buffer for a tile of `items` float4 partial sums.
__host__ __device__ constexpr int recv_bytes(int items) { return (items + MAX_CLUSTER) * 16; }

// Sums a tile over the CTAs of the cluster.  Item i (four fp32 sums) belongs to rank i % ranks: every CTA sends
// partial(i), its own sum over its warps, into the owner's shared memory with an asynchronous store counted in bytes on
// the owner's barrier; the owner adds what it got in rank order (the same result on every run) and calls
// finish(i, sum).  cluster_begin() sets up the barrier at the start of the kernel; its first half of a cluster
// barrier pairs with the wait in cluster_sum(), in front of the first remote store.
__device__ __forceinline__ void cluster_begin(uint32_t bar, int items) {
    if (threadIdx.x == 0) {
        const int ranks = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
        const int own = (items - rank + ranks - 1) / ranks;
        mbar_init(bar, 1);
        mbar_fence_init();
        mbar_expect_tx(bar, (uint32_t)(own * ranks) * 16u);
    }
    __syncthreads();
    cluster_arrive_release();
}

template <typename Partial, typename Finish>
__device__ __forceinline__ void cluster_sum(uint32_t bar, uint32_t recv, int items, unsigned int *status, unsigned int kernel, Partial partial, Finish finish) {
    const int ranks = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
    const int slots = (items + ranks - 1) / ranks;
    cluster_wait_acquire();  // every CTA of the cluster is running and has its barrier set up
    for (int i = threadIdx.x; i < items; i += blockDim.x) {
        const int slot = i / ranks, owner = i - slot * ranks;
        st_async_v4f32(map_to_rank(recv, owner) + (uint32_t)(rank * slots + slot) * 16u, partial(i), map_to_rank(bar, owner));
    }
    const int own = (items - rank + ranks - 1) / ranks;
    if (!mbar_wait_cluster(bar, 0)) report_timeout(status, kernel, 1);
    for (int slot = threadIdx.x; slot < own; slot += blockDim.x) {
        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int r = 0; r < ranks; ++r) {
            float4 v;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(recv + (uint32_t)(r * slots + slot) * 16u));
            sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
        }
        finish(slot * ranks + rank, sum);
    }
}

#endif  // __CUDACC__

// What is known about a kernel, per device: entry c the clusters of c CTAs that run at once, entry 0 that its shared-memory
// limit is set.  A repeated look-up by a racing thread is harmless.
using KnownClusters = std::atomic<int>[64][MAX_CLUSTER + 1];
inline int allow_smem(const void *kernel, int smem, KnownClusters &known) {
    int dev = 0;
    B200Q_CUDA_TRY(cudaGetDevice(&dev));
    const bool table = dev >= 0 && dev < 64;
    if (table && known[dev][0].load(std::memory_order_acquire) != 0) return B200Q_OK;
    B200Q_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (table) known[dev][0].store(1, std::memory_order_release);
    return B200Q_OK;
}

// The largest cluster along K (at most `limit`) with which the whole grid of `tiles` output tiles still runs at once: a
// few clusters left for a second wave double the time of a launch.  How many fit is looked up once per device, kernel and
// size.
inline int choose_cluster(const void *kernel, int threads, int smem, int64_t tiles, int64_t limit, KnownClusters &known) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 1;
    }
    int best = 1;
    for (int c = 2; c <= MAX_CLUSTER && c <= limit; ++c) {
        int n = known[dev][c].load(std::memory_order_relaxed);
        if (n == 0) {
            n = resident_clusters(kernel, threads, smem, c);
            if (n == 0) break;
            known[dev][c].store(n, std::memory_order_relaxed);
        }
        if (tiles > n) break;
        best = c;
    }
    return best;
}

// Launches grid (tiles along N, cluster, tiles along M) as a programmatic dependent of the kernel before it.
inline int launch(const char *name, const void *kernel, int64_t n_tiles, int cluster, int64_t m_tiles, int threads, int smem, cudaStream_t stream, void **args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_tiles, (unsigned)cluster, (unsigned)m_tiles);
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = 1;
    attrs[0].val.clusterDim.y = (unsigned)cluster;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 2;
    const cudaError_t err = cudaLaunchKernelExC(&cfg, kernel, args);
    if (err != cudaSuccess) return set_error(B200Q_CUDA_ERROR, "launch of %s failed: %s", name, cudaGetErrorString(err));
    return B200Q_OK;
}

}  // namespace stream_mma
}  // namespace b200q
