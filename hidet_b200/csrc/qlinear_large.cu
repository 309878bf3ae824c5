// Which kernel serves a quantized linear of more than a few rows, and with what tiles.
//
// The choice is by estimated time, in microseconds; the constants are measured (B200, graph replay of weights that exceed L2) and
// stand beside what they describe.  The small-M kernel stays for what it does better: up to 24 rows always (24 rows, small-M against the
// better of the others: (4096, 12288) 14.5 and 17.5 us, (4096, 22016) 24.8 and 29.8, (11008, 4096) 15.0 and 17.5, (1024, 1024) 3.1 and 5.2).
#include "common.cuh"
#include "qlinear.h"

namespace b200q {
namespace {

// The small-M kernel walks its 16-row blocks over the weight, from L2 after the first: (32, 4096, 4096) 8.8 us, (32, 4096, 12288) 25,
// (32, 11008, 4096) 17.9, (64, 4096, 4096) 13.5, (64, 2048, 2048) 5.9, (64, 1024, 1024) 3.4.
double small_m_us(int64_t M, int64_t N, int64_t K) { return 2.6 + (double)K * N / 3.9e6 * (1.0 + 0.55 * (double)(ceil_div(M, 16) - 1)); }

// A 64-k stage of the mid-M kernel takes 0.30 us with one CTA an SM and 0.46 with two, a fifth more at 128 rows than at 64; the launch
// and its tail 4.2, and each CTA of a cluster makes the exchange longer.  (64, 4096, 4096): 24.7 / 15.2 / 10.9 / 11.5 us in
// clusters of 1 / 2 / 4 / 8; (64, 4096, 11008) 20.2 in clusters of 2, 16.6 of 3; (64, 11008, 4096) 18.2 of 4, 15.1 of 8.
double mid_us(int64_t M, int64_t N, int64_t K, int *tm, int *cluster) {
    const int64_t m_tiles = ceil_div(M, 128), n_tiles = ceil_div(N, 128), k_blocks = ceil_div(K, 64);
    const int64_t tiles = m_tiles * n_tiles;
    *tm = (int)round_up(ceil_div(M, m_tiles), 16);
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    double best = 1e30;
    for (int c = 1; c <= 8 && (c == 1 || k_blocks >= 2 * c); ++c) {
        const int64_t resident = mid_resident_ctas(*tm, c), ctas = tiles * c;
        if (c > 1 && ctas > resident) break;  // a few clusters left for a second wave double the time
        const double stage = (ctas <= sms ? 0.30 : 0.46) * (*tm > 64 ? 1.0 + 0.2 * (*tm - 64) / 64.0 : 1.0);
        const double us = 4.2 + 0.3 * c + (double)ceil_div(ctas, resident) * (double)ceil_div(k_blocks, c) * stage;
        if (us < best) {
            best = us;
            *cluster = c;
        }
    }
    return best;
}

// A 64-k stage of the kernel on SM pairs by tile height, and what a tile costs on top: next to nothing where two accumulators
// fit in tensor memory (up to 192 rows), the epilogue where only one does.  (512, 4096, 22016) with SiLU: 124 / 96 / 88 / 87 us
// at 96 / 128 / 192 / 256 rows; (2048, 8192, 28672): 889 / 728 / 690 / 638 at 128 / 192 / 224 / 256; (256, 4096, 11008): 38 at
// 96 to 192 rows, 42 at 224, 26 at 256.
double pair_us(int64_t M, int64_t N, int64_t K, bool silu, int *tm) {
    static const struct {
        int tm;
        double stage;
    } forms[] = {{64, 0.262}, {96, 0.262}, {128, 0.265}, {160, 0.28}, {192, 0.315}, {224, 0.32}, {256, 0.335}};
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    double best = 1e30;
    for (const auto &f : forms) {
        const int64_t tiles = ceil_div(N, 256) * ceil_div(M, f.tm);
        const double tile = f.tm <= 192 ? 0.3 : (silu ? 6.0 : 2.5);
        const double us = 4.5 + (double)ceil_div(tiles, sms / 2) * ((double)ceil_div(K, 64) * f.stage + tile);
        if (us < best) {
            best = us;
            *tm = f.tm;
        }
    }
    return best;
}

}  // namespace

LargePlan plan_large(int64_t M, int64_t N, int64_t K, bool silu) {
    LargePlan p;
    if (M <= 24) return p;
    int mid_tm = 0, mid_cluster = 1, pair_tm = 0;
    const double mid = M <= 65535 * 128 ? mid_us(M, N, K, &mid_tm, &mid_cluster) : 1e30;  // the grid's limit
    const double pair = M > 32 ? pair_us(M, N, K, silu, &pair_tm) : 1e30;
    const double best = mid < pair ? mid : pair;
    // The estimates are within a tenth of each other's error, so nearly as good is good enough (a sixth was asked for before, and
    // (32, 4096, 12288) took 23.4 us for 17.7, (32, 4096, 22016) 36.0 for 29.8, (48, 4096, 4096) 13.6 for 9.9).
    if (!use_prefill_kernel(M, N, K) && best > 0.95 * small_m_us(M, N, K)) return p;
    p.kind = mid < pair ? LargePlan::kMid : LargePlan::kPair;
    p.tm = mid < pair ? mid_tm : pair_tm;
    p.cluster = mid_cluster;
    return p;
}

int check_large_outputs(const OutTargets &out) {
    for (int d = 0; d < out.count; ++d)
        if ((reinterpret_cast<uintptr_t>(out.ptr[d]) & 15u) != 0) return set_error(B200Q_INVALID_ARGUMENT, "qlinear: output %d is not 16-byte aligned", d);
    if (out.ldc % 8 != 0 || out.col0 % 8 != 0) return set_error(B200Q_INVALID_ARGUMENT, "qlinear: output row length and column offset must be multiples of 8 elements");
    return B200Q_OK;
}

bool try_large(const void *a, const void *wq, const void *scale, const OutTargets &c, int64_t M, int64_t N, int64_t K, cudaStream_t stream, const Epilogue *epilogue,
               bool weight_nk, int64_t lda, size_t scratch_bytes, int *rc) {
    if (M <= 24 || !(weight_nk ? prefill_nk_supported(a, wq, N, K) : prefill_kn_supported(a, wq, N, K))) return false;
    const bool only = use_prefill_kernel(M, N, K);  // the small-M kernel is out of the question
    if (!only) {
        const DecodePlan dp = plan_decode(M, N, K);
        if (dp.partial_bytes > 0 && scratch_bytes < dp.counter_bytes + dp.partial_bytes) return false;
    }
    const LargePlan plan = plan_large(M, N, K, epilogue != nullptr && epilogue->act == kActSiluMul);
    if (plan.kind == LargePlan::kNone) return false;
    *rc = check_large_outputs(c);
    if (*rc != B200Q_OK) return only;  // the small-M kernel stores at any element
    *rc = launch_large(plan, a, wq, scale, c, M, N, K, stream, epilogue, weight_nk, lda);
    return true;
}

int launch_large(const LargePlan &plan, const void *a, const void *wq, const void *scale, const OutTargets &out, int64_t M, int64_t N, int64_t K, cudaStream_t stream,
                 const Epilogue *epilogue, bool weight_nk, int64_t lda) {
    if (lda <= 0) lda = K;
    if (plan.kind == LargePlan::kMid) return launch_mid(a, wq, scale, out, M, N, K, stream, epilogue, weight_nk, lda, plan.tm, plan.cluster);
    return launch_pair(a, wq, scale, out, M, N, K, stream, epilogue, weight_nk, lda, plan.tm);
}

}  // namespace b200q
