// The epilogues' SiLU against the plain division and against 64 bits, on gates of consecutive bit patterns.
#include "../../hidet_b200/csrc/common.cuh"

struct Found {
    unsigned long long differ;       // gates whose results are neither the same bits nor both NaN
    unsigned long long apart;        // the most ulps between the two
    unsigned long long worst[2];     // largest error against 64 bits in thousandths of an ulp, of the division and of silu
    unsigned long long sum[2];       // the errors' sums
};

__device__ unsigned long long thousandths(float got, double want) {
    const float w = fabsf((float)want);
    const double ulp = (double)__uint_as_float(__float_as_uint(w) + 1) - (double)w;
    return (unsigned long long)(fabs((double)got - want) / ulp * 1000.0);
}

__global__ void compare_kernel(uint32_t begin, uint32_t step, uint32_t count, int errors, Found *out) {
    Found f = {};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += (uint64_t)gridDim.x * blockDim.x) {
        const float g = __uint_as_float(begin + (uint32_t)i * step);
        const float both[2] = {g / (1.0f + __expf(-g)), b200q::silu(g)};
        const int apart = abs((int)__float_as_uint(both[0]) - (int)__float_as_uint(both[1]));
        if (apart != 0 && !(both[0] != both[0] && both[1] != both[1])) {
            ++f.differ;
            if (apart > f.apart) f.apart = apart;
        }
        if (errors) {
            const double want = (double)g / (1.0 + exp(-(double)g));
            for (int k = 0; k < 2; ++k) {
                const unsigned long long e = thousandths(both[k], want);
                f.sum[k] += e;
                if (e > f.worst[k]) f.worst[k] = e;
            }
        }
    }
    atomicAdd(&out->differ, f.differ);
    atomicMax(&out->apart, f.apart);
    for (int k = 0; k < 2; ++k) {
        atomicAdd(&out->sum[k], f.sum[k]);
        atomicMax(&out->worst[k], f.worst[k]);
    }
}

// out: six 64-bit words, zero on entry
extern "C" __attribute__((visibility("default"))) int compare(uint32_t begin, uint32_t step, uint32_t count, int errors, Found *out, cudaStream_t stream) {
    compare_kernel<<<592, 256, 0, stream>>>(begin, step, count, errors, out);
    return (int)cudaGetLastError();
}
