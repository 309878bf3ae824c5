// A kernel that lets the launch behind it start at once and writes its result a while later: dst = src, `words` 32-bit
// words, `clocks` after the start.  What follows it in the stream must wait for its end, not for its trigger.
#include <cuda_runtime.h>
#include <cstdint>

__global__ void late_copy_kernel(uint32_t *dst, const uint32_t *src, int words, int clocks) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long start = clock64();
    while (clock64() - start < clocks) {
    }
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}

// The same on every SM: each CTA first reads all of dst, so that the first-level caches hold what was there before, and block 0 writes.
__global__ void late_copy_everywhere_kernel(uint32_t *dst, const uint32_t *src, int words, int clocks, uint32_t *sink) {
    uint32_t old = 0, v;
    for (int i = threadIdx.x; i < words; i += blockDim.x) {
        asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(dst + i) : "memory");
        old ^= v;
    }
    if (words < 0) *sink = old;  // never
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long start = clock64();
    while (clock64() - start < clocks) {
    }
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}

extern "C" __attribute__((visibility("default"))) int late_copy_everywhere(uint32_t *dst, const uint32_t *src, int words, int clocks, int blocks, cudaStream_t stream) {
    late_copy_everywhere_kernel<<<blocks, 256, 0, stream>>>(dst, src, words, clocks, dst);
    return (int)cudaGetLastError();
}

extern "C" __attribute__((visibility("default"))) int late_copy(uint32_t *dst, const uint32_t *src, int words, int clocks, cudaStream_t stream) {
    late_copy_kernel<<<1, 256, 0, stream>>>(dst, src, words, clocks);
    return (int)cudaGetLastError();
}
