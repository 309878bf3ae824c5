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

extern "C" __attribute__((visibility("default"))) int late_copy(uint32_t *dst, const uint32_t *src, int words, int clocks, cudaStream_t stream) {
    late_copy_kernel<<<1, 256, 0, stream>>>(dst, src, words, clocks);
    return (int)cudaGetLastError();
}
