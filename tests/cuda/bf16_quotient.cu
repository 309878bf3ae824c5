// Counts the pairs (a, b) of bfloat16 numbers for which the quantize kernels' quotient, the correctly rounded reciprocal of b times
// a in f32, rounded to bfloat16, is not what CUDA's a / b gives: another number where either is at least a quarter, another
// integer after rounding where both are below.  b runs over the divisors that are taken that way, 2^-100 to 2^126.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

__global__ void bf16_quotient_kernel(unsigned long long *mismatches) {
    const unsigned int b = blockIdx.x, exponent = (b >> 7) & 0xffu;
    if (exponent < 127u - 100u || exponent >= 127u + 126u) return;
    const __nv_bfloat16 hb = __ushort_as_bfloat16((unsigned short)b);
    const float rcp = __frcp_rn(__bfloat162float(hb));
    const __nv_bfloat16 quarter = __float2bfloat16(0.25f);
    unsigned int wrong = 0;
    for (unsigned int a = threadIdx.x; a < 65536u; a += blockDim.x) {
        const __nv_bfloat16 ha = __ushort_as_bfloat16((unsigned short)a);
        const __nv_bfloat16 want = ha / hb, got = __float2bfloat16(rcp * __bfloat162float(ha));
        if (__hisnan(want) && __hisnan(got)) continue;
        if (__hlt(__habs(want), quarter) && __hlt(__habs(got), quarter)) wrong += (int)hrint(want) != (int)hrint(got);
        else wrong += __bfloat16_as_ushort(want) != __bfloat16_as_ushort(got);
    }
    if (wrong != 0) atomicAdd(mismatches, (unsigned long long)wrong);
}

extern "C" __attribute__((visibility("default"))) int bf16_quotient_mismatches(unsigned long long *mismatches, cudaStream_t stream) {
    bf16_quotient_kernel<<<65536, 256, 0, stream>>>(mismatches);
    return (int)cudaGetLastError();
}
