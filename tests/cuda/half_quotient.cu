// Counts the pairs (a, b) of halves for which the quantize kernels' quotient, the correctly rounded reciprocal of b times a
// in f32, rounded to half, is not what CUDA's a / b gives: another half where either is a normal number or beyond, another
// integer after rounding where both are below.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

__global__ void half_quotient_kernel(unsigned long long *mismatches) {
    const unsigned int b = blockIdx.x;
    const __half hb = __ushort_as_half((unsigned short)b);
    const float rcp = __frcp_rn(__half2float(hb));
    const __half least_normal = __ushort_as_half((unsigned short)0x0400);
    unsigned int wrong = 0;
    for (unsigned int a = threadIdx.x; a < 65536u; a += blockDim.x) {
        const __half ha = __ushort_as_half((unsigned short)a);
        const __half want = ha / hb, got = __float2half(rcp * __half2float(ha));
        if (__hisnan(want) && __hisnan(got)) continue;
        if (__hlt(__habs(want), least_normal) && __hlt(__habs(got), least_normal)) wrong += (short)hrint(want) != (short)hrint(got);
        else wrong += __half_as_ushort(want) != __half_as_ushort(got);
    }
    if (wrong != 0) atomicAdd(mismatches, (unsigned long long)wrong);
}

extern "C" __attribute__((visibility("default"))) int half_quotient_mismatches(unsigned long long *mismatches, cudaStream_t stream) {
    half_quotient_kernel<<<65536, 256, 0, stream>>>(mismatches);
    return (int)cudaGetLastError();
}
