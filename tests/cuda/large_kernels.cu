// The kernels for more than a few rows behind entry points that name the kernel, its tiles and its split, and the plan that chooses
// between them: compiled together with the library's own sources, for tests that have to know which kernel they run.
#include "../../hidet_b200/csrc/common.cuh"
#include "../../hidet_b200/csrc/qlinear.h"

#define EXPORT extern "C" __attribute__((visibility("default")))

using namespace b200q;

static OutTargets targets(void *const *dst, int count, int64_t ldc, int64_t col0) {
    OutTargets t;
    for (int i = 0; i < count; ++i) t.ptr[i] = dst[i];
    t.count = count;
    t.ldc = ldc;
    t.col0 = col0;
    return t;
}

// out: kind (0: the small-M kernel stays, 1: mid M, 2: SM pairs), rows per tile, cluster
EXPORT void plan(int64_t M, int64_t N, int64_t K, int silu, int *out) {
    const LargePlan p = plan_large(M, N, K, silu != 0);
    out[0] = p.kind, out[1] = p.tm, out[2] = p.cluster;
}

// out: rows per pass of the small-M kernel's plan, CTAs per cluster, clusters per tile
EXPORT void small_plan(int64_t M, int64_t N, int64_t K, int *out) {
    const DecodePlan p = plan_decode(M, N, K);
    out[0] = (int)((M + p.m_tiles - 1) / p.m_tiles), out[1] = p.cluster, out[2] = p.groups;
}

// The same for a launch on a stream.
EXPORT void small_plan_on(cudaStream_t stream, int64_t M, int64_t N, int64_t K, int *out) {
    const DecodePlan p = plan_decode_on(stream, M, N, K);
    out[0] = (int)((M + p.m_tiles - 1) / p.m_tiles), out[1] = p.cluster, out[2] = p.groups;
}

// The small-M kernel in its form for up to 4, 8, 16 or 24 rows a pass (0 to 3) with one cluster of that many CTAs a tile.
EXPORT int launch_small(int form, int cluster, const void *a, const void *wq, const void *scale, void *c, int64_t M, int64_t N, int64_t K, int nk, const void *bias,
                        const void *residual, int silu, cudaStream_t stream) {
    static const int rows[] = {4, 8, 16, 24};
    DecodePlan p;
    p.variant = form;
    p.n_tiles = (int)((N + 127) / 128);
    p.m_tiles = (int)((M + rows[form] - 1) / rows[form]);
    p.cluster = p.splits = cluster;
    p.iters_per_split = (int)(((K + 63) / 64 + cluster - 1) / cluster);
    Epilogue ep;
    ep.bias = bias;
    ep.residual = residual;
    ep.ldr = silu ? N / 2 : N;
    ep.act = silu ? kActSiluMul : kActNone;
    return launch_decode_kn(a, wq, scale, c, M, N, K, 0, K, true, nullptr, 0, stream, nullptr, &ep, nk != 0, &p);
}

EXPORT int launch(int kind, int tm, int cluster, const void *a, const void *wq, const void *scale, void *const *dst, int count, int64_t ldc, int64_t col0, int64_t M, int64_t N,
                  int64_t K, int64_t lda, int nk, const void *bias, const void *residual, int64_t ldr, int silu, cudaStream_t stream) {
    LargePlan p;
    p.kind = static_cast<LargePlan::Kind>(kind);
    p.tm = tm;
    p.cluster = cluster;
    Epilogue ep;
    ep.bias = bias;
    ep.residual = residual;
    ep.ldr = ldr;
    ep.act = silu ? kActSiluMul : kActNone;
    return launch_large(p, a, wq, scale, targets(dst, count, ldc, col0), M, N, K, stream, &ep, nk != 0, lda);
}

// The one-SM kernel on ordinary destinations (through the library it serves a multicast address, which one GPU does not have).
// Returns how many parts K was split into, or the negative status.
EXPORT int launch_one_sm(const void *a, const void *wq, const void *scale, void *const *dst, int count, int64_t ldc, int64_t col0, int64_t M, int64_t N, int64_t K,
                         void *workspace, size_t workspace_bytes, cudaStream_t stream) {
    const int rc = launch_prefill_kn(a, wq, scale, targets(dst, count, ldc, col0), M, N, K, stream, workspace, workspace_bytes);
    if (rc != B200Q_OK) return -rc;
    const PrefillSplit split = plan_prefill_split(M, N, K);
    return split.workspace_bytes <= workspace_bytes ? split.k_splits : 1;
}
