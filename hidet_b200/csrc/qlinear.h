// Internal interface between the quantized-linear entry points and the kernels behind them.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace b200q {

// Where a kernel writes its result.  Element (m, n) of the result goes to
// ptr[i][m * ldc + col0 + n] for every i < count: one entry is the ordinary output; several entries
// are the same column block of output buffers on several GPUs (peer-mapped pointers), which is how a
// column-parallel layer delivers its slice to every rank without a separate all-gather.
constexpr int kMaxOutTargets = 8;
struct OutTargets {
    void *ptr[kMaxOutTargets] = {};
    int count = 0;
    int64_t ldc = 0;   // elements between consecutive rows of the destination
    int64_t col0 = 0;  // first destination column
    // ptr[0] is an NVLink multicast address (one store reaches the same place of every GPU bound to it, this one
    // included); count is 1.  Served by the large-M kernel only, whose epilogue then stores with multimem.st.
    int multicast = 0;
};

inline OutTargets one_output(void *c, int64_t columns) {
    OutTargets t;
    t.ptr[0] = c;
    t.count = 1;
    t.ldc = columns;
    return t;
}

// What a kernel does to the scaled fp32 sums y[m, n] before the one rounding to f16:
//   y += bias[n];  activation (silu_mul: the weight's columns come in pairs (gate_j, up_j) = (2j, 2j + 1), and
//   z[m, j] = silu(y[m, 2j]) * y[m, 2j + 1] is the result, half as wide);  z += residual[m, j].
// Takes the place of the element-wise operators the reference fuses into its matmul by IR rewriting
// (python/hidet/graph/transforms/fuse_operator.py, python/hidet/graph/ops/quant/matmul_f16_i8.py:95-99).
constexpr int kActNone = 0;
constexpr int kActSiluMul = 1;
struct Epilogue {
    const void *bias = nullptr;      // f16 [N]
    const void *residual = nullptr;  // f16 [M, ldr]
    int64_t ldr = 0;                 // elements between rows of residual
    int act = kActNone;
};

// How the small-M kernel splits a problem over CTAs, and the scratch that split needs.
struct DecodePlan {
    int variant = 0;           // which form of the kernel: rows per pass
    int n_tiles = 0;
    int m_tiles = 0;
    int splits = 1;            // CTAs along K per output tile
    int cluster = 1;           // of them, this many form a thread-block cluster that needs no workspace
    int groups = 1;            // clusters per tile; > 1: the clusters meet in the workspace
    int iters_per_split = 0;   // 64-row k steps each of them takes
    int most_splits = 1;       // as many as K has work for
    size_t counter_bytes = 0;  // head of the workspace: one arrival counter per output tile
    size_t partial_bytes = 0;  // then [groups][M][N] fp32 partial sums.  Both are asked of the caller where clusters of the portable size
                               // would meet in the workspace, also where larger ones (groups == 1) do without
};

// Codes of a weight from which on 17 to 24 rows are one pass.
constexpr int64_t kOnePassCodes = 6 * 1024 * 1024;
DecodePlan plan_decode(int64_t M, int64_t N, int64_t K);
DecodePlan plan_decode_portable(int64_t M, int64_t N, int64_t K);  // the same scratch, for less
DecodePlan plan_decode_on(cudaStream_t stream, int64_t M, int64_t N, int64_t K);  // the one that is launched on a stream

// True when the TMA-based [K, N] kernel can take these operands (16-byte aligned bases and rows).
bool decode_kn_supported(const void *a, const void *wq, int64_t N, int64_t K);

// c[M, N] = scale * (a[:, k_begin:k_end] x wq[k_begin:k_end, :]).  K is the row length of `a`.
int launch_decode_kn(const void *a, const void *wq, const void *scale, void *c, int64_t M, int64_t N, int64_t K,
                     int64_t k_begin, int64_t k_end, bool allow_split, void *workspace, size_t workspace_bytes,
                     cudaStream_t stream, const OutTargets *targets = nullptr, const Epilogue *epilogue = nullptr, bool weight_nk = false,
                     const DecodePlan *plan = nullptr);  // plan: instead of the one that plan_decode_on makes
// The same kernel on a weight stored [N, K] (weight_nk = true): needs 16-byte aligned bases and K % 16 == 0.
bool decode_nk_supported(const void *a, const void *wq, int64_t N, int64_t K);

// The operands that all kernels for more than a few rows take: as the small-M kernel, and for a weight stored [N, K] N % 8 == 0 too.
bool prefill_kn_supported(const void *a, const void *wq, int64_t N, int64_t K);
bool prefill_nk_supported(const void *a, const void *wq, int64_t N, int64_t K);
// Their outputs are written with 16-byte stores: B200Q_INVALID_ARGUMENT where those cannot write them.
int check_large_outputs(const OutTargets &out);

// The one-SM tensor-memory kernel for large M ([K, N] weights), which serves the multicast delivery.
// How it splits K (narrow problems only) and the scratch that takes: fp32 partial sums
// [k_splits][M][N] behind an untouched head of kSplitWorkspaceHead bytes (the small-M kernel's counters live there).
constexpr size_t kSplitWorkspaceHead = (size_t)65536 * 4;
struct PrefillSplit {
    int k_splits = 1;
    int kb_per_split = 0;
    size_t workspace_bytes = 0;
};
PrefillSplit plan_prefill_split(int64_t M, int64_t N, int64_t K);
// workspace: where K may be split (see plan_prefill_split); without it the kernel runs one CTA per output tile.
int launch_prefill_kn(const void *a, const void *wq, const void *scale, const OutTargets &out, int64_t M, int64_t N, int64_t K, cudaStream_t stream, void *workspace,
                      size_t workspace_bytes);

// More than a few rows: the kernel on pairs of SMs (tm, a multiple of 32 up to 256, rows per tile) and the mid-M
// kernel (tm, a multiple of 16 up to 128, rows per tile; K split over a cluster).  Operands as for the kernel above;
// outputs at any number of addresses but not a multicast one; no workspace.
struct LargePlan {
    enum Kind { kNone, kMid, kPair };  // kNone: the small-M kernel is the better one
    Kind kind = kNone;
    int tm = 0;
    int cluster = 1;
};
LargePlan plan_large(int64_t M, int64_t N, int64_t K, bool silu, bool weight_nk = false);
// True where these kernels serve the call and are better at it than the small-M one, or alone would serve it but for its
// outputs; *rc is then the launch's status or the refusal.  What the small-M kernel refuses for want of scratch stays refused.
bool try_large(const void *a, const void *wq, const void *scale, const OutTargets &c, int64_t M, int64_t N, int64_t K, cudaStream_t stream, const Epilogue *epilogue,
               bool weight_nk, int64_t lda, size_t scratch_bytes, int *rc);
int launch_large(const LargePlan &plan, const void *a, const void *wq, const void *scale, const OutTargets &out, int64_t M, int64_t N, int64_t K, cudaStream_t stream,
                 const Epilogue *epilogue, bool weight_nk, int64_t lda = 0);
int launch_pair(const void *a, const void *wq, const void *scale, const OutTargets &out, int64_t M, int64_t N, int64_t K, cudaStream_t stream,
                const Epilogue *epilogue, bool weight_nk, int64_t lda, int tm);
int launch_mid(const void *a, const void *wq, const void *scale, const OutTargets &out, int64_t M, int64_t N, int64_t K, cudaStream_t stream,
               const Epilogue *epilogue, bool weight_nk, int64_t lda, int tm, int cluster);
int mid_resident_ctas(int tm, int cluster);  // of the mid-M kernel, in clusters of that size, that run at once

// [K, N] weights whose rows are not multiples of 16 bytes: N even, K a multiple of 8, 16-byte aligned bases.
bool unaligned_supported(const void *a, const void *wq, const void *c, int64_t M, int64_t N, int64_t K);
int launch_unaligned(const void *a, const void *wq, const void *scale, void *c, int64_t M, int64_t N, int64_t K, cudaStream_t stream);

// Where the small-M kernel, which re-streams the weight once per 16 rows (from L2 after the first pass), is out of the question: the
// kernels for more rows then refuse what they cannot take.  (The line was drawn against the one-SM kernel, up to 64 rows by the size of
// the weight; below it plan_large compares estimates.  By those the small-M kernel would still be ahead of it in
// corners, (128, 1024, 1024) and (100, 4096, 1024) among them, which are not timed.)
constexpr int64_t kPrefillMinM = 33;
inline bool use_prefill_kernel(int64_t M, int64_t N, int64_t K) {
    if (M < kPrefillMinM) return false;
    if (M <= 64) return K * N > (int64_t)24 * 1024 * 1024;
    return true;
}

}  // namespace b200q
