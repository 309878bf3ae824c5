// Which kernel serves a quantized linear of more than a few rows, and with what tiles.
//
// The choice is by estimated time, in microseconds; the constants are measured (B200, graph replay of weights that exceed L2) and
// stand beside what they describe.  Over 580 drawn sizes of 25 to 2048 rows it is 1.1 % behind the best kernel, tile and cluster that were
// timed for each (10 % with estimates that left the epilogue out and took the SMs for evenly filled).  The small-M kernel stays for what it
// does better: up to 16 rows always, and up to 24 where one pass fills the SMs (see one_pass_or_mid).
#include "common.cuh"
#include "qlinear.h"

namespace b200q {
namespace {

// The small-M kernel walks its 16-row blocks over the weight, from L2 after the first: (32, 4096, 4096) 8.8 us, (32, 4096, 12288) 25,
// (32, 11008, 4096) 17.9, (64, 4096, 4096) 13.5, (64, 2048, 2048) 5.9, (64, 1024, 1024) 3.4.
double small_m_us(int64_t M, int64_t N, int64_t K) { return 2.6 + (double)K * N / 3.9e6 * (1.0 + 0.55 * (double)(ceil_div(M, 16) - 1)); }

// The mid-M kernel: a launch 2.9, each CTA of a cluster 0.12, and per tile what grows with its rows (loads of the accumulator, the exchange, the
// way out) 0.021 each, a block of eight rows that a CTA finishes 0.07 (with SiLU 0.26), and a 64-k stage: 0.32 with one CTA an SM, with two
// 0.27 to 0.41 and more with the rows (what two CTAs take from shared memory), and 2 to fill two rings.  How many CTAs get an SM of their
// own depends on the cluster: of 1 and 2 all of them, of 3 to 6 nine tenths, of 7 and 8 fifteen clusters (the jump is there at every size that
// was tried).  Estimate and time: (128, 4096, 4096) in clusters of 4 11.5 and 12.0 us, (59, 3792, 2928) in 5 8.8 and 9.1, in 6 10.5 and 11.0,
// (43, 9536, 13264) in 2 35.0 and 35.2, (249, 3376, 1744) in 4 10.8 and 11.6, (96, 2048, 19200) in 1 20.3 and 19.9.
// Rows of the weight that are not whole 32-byte sectors cost a sector more a row of a tile: with two CTAs an SM a stage is then 1.25 times as
// long for [N, K], whose tile rows are two sectors ((121, 3728, 20272) 43.1 us, (121, 5680, 28432) 69.1; on SM pairs 37.1 and 53.7), and 1.1
// times for [K, N] where no other row of tiles reads them again (38.7 and 59.8; 36.2 and 52.2).
double mid_us(int64_t M, int64_t N, int64_t K, bool silu, bool weight_nk, int *tm, int *cluster) {
    const int64_t m_tiles = ceil_div(M, 128), tiles = m_tiles * ceil_div(N, 128), k_blocks = ceil_div(K, 64);
    *tm = (int)round_up(ceil_div(M, m_tiles), 16);
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    double best = 1e30;
    for (int c = 1; c <= 8 && (c == 1 || k_blocks >= 2 * c); ++c) {
        const int64_t ctas = tiles * c, alone = c <= 2 ? sms : (c <= 6 ? sms * 9 / 10 : c * (sms / 10 + 1));
        if (c > 1 && ctas > 2 * sms) break;
        const int64_t resident = c == 1 || ctas * 5 <= sms * 8 ? 2 * sms : mid_resident_ctas(*tm, c);  // asked only where it may be short
        if (c > 1 && ctas > resident) break;  // a few clusters left for a second wave double the time
        const double shared = ctas >= 2 * sms ? 1.0 : (double)(ctas - sms) / sms;  // of the SMs: how many have two
        const double slow = (weight_nk ? K : N) % 32 == 0 ? 1.0 : (weight_nk ? 1.25 : (m_tiles == 1 ? 1.1 : 1.0));
        const double stage = ctas <= alone ? 0.32 : slow * (0.27 + 0.0012 * *tm + 0.135 * shared);
        const double tile = (ctas <= alone ? 0.0 : 2.0) + 0.021 * *tm + (silu ? 0.26 : 0.07) * (double)ceil_div(*tm / 8, c) + (double)ceil_div(k_blocks, c) * stage;
        const double us = 2.9 + 0.12 * c + (double)ceil_div(ctas, resident) * tile;
        if (us < best) {
            best = us;
            *cluster = c;
        }
    }
    return best;
}

// The kernel on SM pairs: a 64-k stage by tile height, for the only wave and for one of several, and the epilogue by rows.  Where two accumulators
// fit in tensor memory (up to 192 rows) the epilogue runs beside the next tile, which for short K it outlasts; where one does it comes on top.
// Estimate and time: (512, 4096, 22016) with SiLU 82 and 77 us at 256 rows, (1900, 368, 19264) 33.5 and 36.0 at 192, 35.3 and 38.9 at 160,
// (2048, 256, 8192) 16.9 and 16.6 at 192, 18.4 and 18.3 at 128, (1024, 320, 16384) 18.7 and 19.3 at 128, (1337, 464, 3008) 7.9 and 9.0 at 224.
double pair_us(int64_t M, int64_t N, int64_t K, bool silu, int *tm) {
    static const struct {
        int tm;
        double one, more;
    } forms[] = {{64, 0.29, 0.267}, {96, 0.285, 0.27}, {128, 0.28, 0.267}, {160, 0.26, 0.27}, {192, 0.262, 0.285}, {224, 0.284, 0.305}, {256, 0.32, 0.33}};
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    double best = 1e30;
    for (const auto &f : forms) {
        const int64_t waves = ceil_div(ceil_div(N, 256) * ceil_div(M, f.tm), sms / 2);
        const double rows = waves == 1 && M < f.tm ? (double)M : f.tm, loop = (double)ceil_div(K, 64) * (waves == 1 ? f.one : f.more);
        double us;
        if (f.tm <= 192) {
            const double epilogue = (silu ? 0.023 : 0.0085) * rows, next = loop + 0.65 > epilogue + 1.05 ? loop + 0.65 : epilogue + 1.05;
            us = 3.55 + loop + 0.9 * epilogue + (double)(waves - 1) * next;
        } else {
            us = 3.5 + (double)waves * (loop + (silu ? 0.02 : 0.0095) * rows);
        }
        if (us < best) {
            best = us;
            *tm = f.tm;
        }
    }
    return best;
}

// The kernels for more rows wait for the kernel in front before they read anything; the small-M kernel asks for its codes earlier.  A call that once
// waited goes on waiting, since its codes may be the result of that kernel: true for all calls of more than 24 rows that the first estimates of
// this rule gave to the kernels for more rows (and, by the roundings below, for 630 of 84 000 drawn ones of 25 to 64 rows that they did not).
// It is no slower there either: (64, 1536, 6144) 8.4 us, 11.8 in the small-M kernel, (60, 256, 28672) with SiLU 8.3 and 13.4, (51, 1680, 5776) 9.0 and 9.8.
bool codes_may_be_late(int64_t M, int64_t N, int64_t K) {
    const double enough = 0.85 * small_m_us(M, N, K);
    if (enough < 4.8) return false;  // the least that any size takes below
    const int sms = sm_count() > 0 ? sm_count() : 148;
    const int64_t tiles = ceil_div(N, 128), k_blocks = ceil_div(K, 64);
    double best = M > 32 ? 4.5 + (double)ceil_div(ceil_div(N, 256), sms / 2) * ((double)k_blocks * 0.262 + 0.3) : 1e30;
    for (int c = 1; c <= 8 && (c == 1 || (k_blocks >= 2 * c && tiles * c <= 2 * sms)); ++c) {
        const double us = 4.2 + 0.3 * c + (double)ceil_div(tiles * c, 2 * sms) * (double)ceil_div(k_blocks, c) * (tiles * c <= sms ? 0.30 : 0.46);
        if (us < best) best = us;
    }
    return best <= enough;
}

// 17 to 24 rows, which the small-M kernel takes in one pass: the mid-M kernel where that pass leaves the SMs thinly filled.  Its CTAs need about 0.62 us
// a 64-k step whether two or three share an SM, so time is its steps, and the mid-M kernel with as many CTAs is faster.  24 rows, one pass and mid M:
//   at most two CTAs an SM although K has work for more splits: (4096, 32000) 42.4 and 29.4 us, (8192, 28672) 76.8 and 53.0, (2048, 18432) 14.0
//     and 11.3; otherwise one pass is ahead, (4096, 12288) 13.8 and 16.6, (4096, 26624) 24.5 and 28.8, (1024, 8192) 6.1 and 6.6;
//   a second wave that is not full, in two of the mid-M kernel: (4096, 57344) 63.5 and 57.1, (4096, 65536) 65.3 and 59.1; (4096, 50000) 45.3 and 54.7,
//     (1760, 76368) 37.9 and 43.2;
//   long K, over at least two thirds as many CTAs: (28672, 4096) 31.1 and 27.4, (14336, 16384) 50.4 and 46.8; (28672, 12288) 73.2 and 88.7 with half.
LargePlan one_pass_or_mid(int64_t M, int64_t N, int64_t K, bool silu, bool weight_nk) {
    LargePlan p;
    const DecodePlan one = plan_decode(M, N, K);
    const int64_t sms = sm_count() > 0 ? sm_count() : 148, ctas = (int64_t)one.n_tiles * one.splits;
    const bool thin = one.splits < 8 && one.splits < one.most_splits && ctas <= 2 * sms;
    const bool second_wave = one.n_tiles > 3 * sms && one.n_tiles <= 4 * sms && K >= 512;
    if (one.m_tiles != 1 || !(thin || second_wave || K >= 12288)) return p;
    int tm = 0, cluster = 1;
    mid_us(M, N, K, silu, weight_nk, &tm, &cluster);
    const int64_t mid_ctas = (int64_t)one.n_tiles * cluster;
    const bool deep = K >= 12288 && mid_ctas <= 2 * sms && 3 * mid_ctas >= 2 * ctas;
    if (thin || second_wave || deep) p.kind = LargePlan::kMid, p.tm = tm, p.cluster = cluster;
    return p;
}

}  // namespace

LargePlan plan_large(int64_t M, int64_t N, int64_t K, bool silu, bool weight_nk) {
    LargePlan p;
    if (M <= 16 || (M <= 24 && N * K < kOnePassCodes)) return p;
    if (M <= 24) return one_pass_or_mid(M, N, K, silu, weight_nk);
    int mid_tm = 0, mid_cluster = 1, pair_tm = 0;
    const bool mid_takes = M <= (int64_t)65535 * 128;  // the grid's limit
    const double mid = mid_takes ? mid_us(M, N, K, silu, weight_nk, &mid_tm, &mid_cluster) : 1e30;
    // What was measured of the kernel on SM pairs ends at K = 256 and at columns that fill one tile and a sliver of another: below, the mid-M
    // kernel stays as long as its tiles run at once.
    const int sms = sm_count() > 0 ? sm_count() : 148;
    const bool pair_too = !mid_takes || (K >= 256 && N >= 288) || ceil_div(M, 128) * ceil_div(N, 128) > sms;
    const double pair = M > 32 && pair_too ? pair_us(M, N, K, silu, &pair_tm) : 1e30;
    const double best = mid < pair ? mid : pair;
    // The estimates are within a tenth of each other's error, so nearly as good is good enough (a sixth was asked for before, and
    // (32, 4096, 12288) took 23.4 us for 17.7, (32, 4096, 22016) 36.0 for 29.8, (48, 4096, 4096) 13.6 for 9.9).
    if (!use_prefill_kernel(M, N, K) && best > 0.95 * small_m_us(M, N, K) && !codes_may_be_late(M, N, K)) return p;
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
    if (M <= 16 || (M <= 24 && N * K < kOnePassCodes) || !(weight_nk ? prefill_nk_supported(a, wq, N, K) : prefill_kn_supported(a, wq, N, K))) return false;
    const bool only = use_prefill_kernel(M, N, K);  // the small-M kernel is out of the question
    if (!only) {
        const DecodePlan dp = plan_decode_portable(M, N, K);
        if (dp.partial_bytes > 0 && scratch_bytes < dp.counter_bytes + dp.partial_bytes) return false;
    }
    const LargePlan plan = plan_large(M, N, K, epilogue != nullptr && epilogue->act == kActSiluMul, weight_nk);
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
