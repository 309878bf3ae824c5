// Small-M (decode) f16 x int8 quantized linear for weights in the reference's [K, N] layout.
//
// The op is bound by streaming the int8 weight from HBM once, so the kernel is built around that
// stream.  A producer warp keeps a ring of TMA tile loads in flight: 64 k-rows x 128 columns of int8,
// 128B-swizzled, and copies the matching 16 x 64 f16 slice of the activations beside each with
// cp.async.  Four consumer warps own 32 columns each, so no sum ever crosses a warp.  A consumer
// fetches its slice with transposing matrix loads (four consecutive k of one column per register),
// turns the bytes into exact f16 pairs in registers and feeds warp-level m16n8k16 tensor-core MMAs
// with fp32 accumulators; the weight is the MMA's 16-row operand and the activations its 8-column operand, so up to 8 activation rows
// cost one MMA per 16 x 16 weight block, up to 16 rows two and up to 24 three (rows beyond M are zero-filled).
//
// K is split across CTAs to fill the machine.  Up to 16 splits of one output tile form a thread-block
// cluster: every CTA sends its partial tile into the shared memory of the CTA that owns those columns
// with asynchronous remote stores that count bytes on an mbarrier of the owner (no cluster barrier
// round trip); the owner waits for the byte count, adds the partials in rank order, applies the
// per-column scale and rounds to f16 once.  More splits than a cluster holds go through a
// caller-provided fp32 workspace, where the last CTA of a tile to arrive does the same.  Either way
// the order of every sum is fixed, so results are the same on every run.
//
// The kernel is launched as a programmatic dependent of the kernel before it in the stream: weight
// tiles do not depend on that kernel, so they are requested before waiting for it (the scales may, as the
// activations do; with 17 to 24 rows the weight may too, see below), and the kernel after this one may start as soon as that wait is over.
//
// Replaces the generated mma.sync kernel of python/hidet/graph/ops/quant/matmul_f16_i8.py:136-485
// (f16 accumulation, 64x128 tiles, no split-K by default) for up to 24 rows, and serves more where the
// kernels for more rows are not faster, by tiling M over blockIdx.z.
#include <atomic>

#include "common.cuh"
#include "qlinear.h"
#include "umma.cuh"

namespace b200q {
namespace decode {

constexpr int BK = 64;                       // k rows per pipeline stage
constexpr int BN = 128;                      // columns per CTA
constexpr int STAGES = 4;
constexpr int CONSUMER_WARPS = 4;            // each owns BN / 4 = 32 columns
constexpr int THREADS = 32 * (CONSUMER_WARPS + 1);
constexpr int W_STAGE_BYTES = BK * BN;       // 8192
constexpr int RECV_COLS = 168;               // most columns the slices of a cluster cover together (7 ranks x 24 columns, 14 x 12; see slices_fit)
constexpr int STAGING_ROW = 36;              // floats per row of a warp's 32-column staging block (padded: conflict-free)

// Shared memory of a CTA with MT blocks of eight activation rows.
template <int MT>
struct Config {
    static constexpr int ROWS = 8 * MT;                  // activation rows per CTA
    static constexpr int CTAS = MT <= 2 ? 4 : 3;         // that share an SM
    static constexpr int A_STAGE_BYTES = ROWS * BK * 2;
    static constexpr int PIPE_BYTES = STAGES * (W_STAGE_BYTES + A_STAGE_BYTES);
    static constexpr int RECV_BYTES = ROWS * RECV_COLS * 4;  // partial tiles sent by the CTAs of the cluster: [rank][row][cols_per] fp32
    // + alignment slack; and at least what keeps a fifth CTA off an SM.  The CTAs of the next launch move in beside this
    // one's (see the kernel) and fill their rings ahead of it; more of them than the fourth slots hold take the
    // memory system away from the launch they wait for: (1, 4096, 12288) 10.3 -> 11.1 us, (1, 4096, 32000) 22.1 -> 24.0 us.
    static constexpr int NEED = PIPE_BYTES + RECV_BYTES + 1024;
    static constexpr int SMEM_BYTES = NEED < 46 * 1024 + 512 ? 46 * 1024 + 512 : NEED;
    static_assert(CONSUMER_WARPS * ROWS * STAGING_ROW * 4 <= STAGES * W_STAGE_BYTES, "the staging blocks reuse the weight ring");
};
constexpr int64_t kMaxCounters = 65536;      // arrival counters at the head of the workspace
constexpr int kPortableCluster = 8;          // what every device runs; beyond it the occupancy query has the last word
constexpr int kMaxCluster = 16;              // largest cluster of the plan
// Columns of a tile that each CTA of a cluster owns, and whether a rank's slices from all of them have their place in the receive buffer (not
// those of 15 CTAs, 12 columns each).
constexpr int slice_cols(int cluster) {
    const int step = cluster <= kPortableCluster ? 8 : 4;
    return ((BN + cluster - 1) / cluster + step - 1) / step * step;
}
constexpr bool slices_fit(int cluster) { return slice_cols(cluster) * cluster <= RECV_COLS; }
constexpr bool all_slices_fit(int cluster) { return cluster == 0 || (slices_fit(cluster) && all_slices_fit(cluster - 1)); }
static_assert(all_slices_fit(kPortableCluster), "clusters up to the portable size are launched unasked");
static_assert(slices_fit(kMaxCluster), "the largest cluster of the plan");

__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

__device__ __forceinline__ float4 lds128f(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts32f(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

// 16 bytes global -> shared without passing through registers; src_bytes = 0 writes zeros instead.
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
// The barrier gets one arrival from this thread once all its earlier cp.async copies have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

constexpr int kModeDirect = 0;  // one CTA per output tile
constexpr int kModeSplit = 1;   // `splits` CTAs per tile: clusters of `cluster` CTAs, `groups` clusters per tile

// One result element to every destination.
__device__ __forceinline__ void store_out(const OutTargets &o, int row, int col, __half v) {
    const size_t off = (size_t)row * o.ldc + o.col0 + col;
#pragma unroll 1
    for (int i = 0; i < o.count; ++i) static_cast<__half *>(o.ptr[i])[off] = v;
}

// The end of every path: y is the scaled fp32 sum of column nn (in range or not), row `row`.  Adds the bias,
// applies the activation (the value of the partner column nn ^ 1 sits in lane ^ partner_xor; every lane
// of the calling warp that is active takes part), adds the residual, rounds once and stores.
__device__ __forceinline__ void finish(const OutTargets &o, const Epilogue &ep, int row, int nn, int n_limit, bool valid, float y, int partner_xor) {
    // Bias and residual come through L2: this CTA may be older than the kernel that wrote them, and so may be what the
    // first-level cache holds.
    if (valid && ep.bias != nullptr) y += __half2float(__ldcg(static_cast<const __half *>(ep.bias) + nn));
    int col = nn;
    if (ep.act == kActSiluMul) {
        const float other = __shfl_xor_sync(__activemask(), y, partner_xor);
        if (nn & 1) valid = false;  // the even column of a pair finishes both
        y = silu(y) * other;
        col = nn >> 1;
    }
    if (!valid || nn >= n_limit) return;
    if (ep.residual != nullptr) y += __half2float(__ldcg(static_cast<const __half *>(ep.residual) + (size_t)row * ep.ldr + col));
    store_out(o, row, col, __float2half_rn(y));
}

// Four adjacent halves, as one load / store where the address allows it.
__device__ __forceinline__ void load4(const __half *p, float (&v)[4]) {
    __align__(8) __half h[4];
    if ((reinterpret_cast<uintptr_t>(p) & 7u) == 0) {
        *reinterpret_cast<uint2 *>(h) = __ldcg(reinterpret_cast<const uint2 *>(p));
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) h[j] = __ldcg(p + j);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __half2float(h[j]);
}
// `finish` for four adjacent columns nn .. nn + 3 (nn a multiple of 4, all of them in the matrix) in one thread.
__device__ __forceinline__ void finish4(const OutTargets &o, const Epilogue &ep, int row, int nn, float4 y4) {
    float y[4] = {y4.x, y4.y, y4.z, y4.w}, t[4];
    if (ep.bias != nullptr) {
        load4(static_cast<const __half *>(ep.bias) + nn, t);
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] += t[j];
    }
    if (ep.act == kActSiluMul) {
        y[0] = silu(y[0]) * y[1];
        y[1] = silu(y[2]) * y[3];
        const int col = nn >> 1;
        if (ep.residual != nullptr) {
            const __half *r = static_cast<const __half *>(ep.residual) + (size_t)row * ep.ldr + col;
            y[0] += __half2float(__ldcg(r));
            y[1] += __half2float(__ldcg(r + 1));
        }
        store_out(o, row, col, __float2half_rn(y[0]));
        store_out(o, row, col + 1, __float2half_rn(y[1]));
        return;
    }
    if (ep.residual != nullptr) {
        load4(static_cast<const __half *>(ep.residual) + (size_t)row * ep.ldr + nn, t);
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] += t[j];
    }
    __align__(8) __half h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __float2half_rn(y[j]);
    const size_t off = (size_t)row * o.ldc + o.col0 + nn;
#pragma unroll 1
    for (int i = 0; i < o.count; ++i) {
        __half *dst = static_cast<__half *>(o.ptr[i]) + off;
        if ((reinterpret_cast<uintptr_t>(dst) & 7u) == 0) {
            *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(h);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[j] = h[j];
        }
    }
}

struct Params {
    const __half *a;          // activations [M, lda]
    int64_t lda;
    const __half *scale;
    OutTargets out;
    Epilogue ep;
    float *partial;           // [groups][M][N] fp32 in the workspace, used when groups > 1
    unsigned int *counters;   // [m_tiles * n_tiles * cluster] in the workspace, zero on entry, zero on exit
    unsigned int *status;
    int M, N;
    int k_begin, k_end;       // the k range this launch sums over (k_end is also the tensor maps' K extent)
    int iters_per_split;      // BK-sized k steps per split
    int groups;               // clusters per output tile (splits = groups * cluster size)
    int cols_per;             // columns of a tile each CTA of the cluster owns in the reduction (a multiple of 4)
    int mode;                 // kModeDirect or kModeSplit
    bool late;                // the weight may be a result of the kernel in front (with two row blocks; three always take it so)
};

// MT: 8-row blocks of activations per CTA (1: up to 8 rows, 2: up to 16, 3: up to 24).
// NK: the weight is [N, K] with K contiguous (the layout torch.nn.Linear keeps) instead of the reference's
//     [K, N]: a stage is then 128 weight rows of 64 k-bytes (64-byte swizzle) and the fragments come from
//     plain matrix loads; everything else is shared.
// QUAD: the elements that a CTA finishes in the split-K reduction are taken four adjacent columns of a row per thread (more than
//     four rows; with fewer one element per thread is one round anyway: (4, 9648, 1568) 7.9 us, 8.05 so).
// WIDE: clusters beyond the portable size (the eight partials that a smaller one sums at once stay one piece of code without a loop:
//     (16, 4096, 12288) 12.0 us, 12.4 with it).
// With 17 to 24 rows on weights of kOnePassCodes and more, the weight is not asked for ahead of the kernel in front: these calls were mostly served
// by a kernel that waits, and their codes may be that kernel's results.  In one pass (EARLY false) it is fetched into L2 meanwhile ((24, 4096, 4096) 7.6 us
// with, 8.1 without), and three CTAs share an SM.  Otherwise shared memory lets four CTAs share an SM; told so, the compiler takes up to 72 registers where it stopped at 56 (and spilled four
// bytes in one form): a decode step at 7B widths for one sequence 216 -> 209 us, for sixteen 256 -> 252.
template <int MT, bool NK, bool QUAD, bool WIDE>
__global__ void __launch_bounds__(THREADS, Config<MT>::CTAS) qlinear_decode_kn_kernel(const __grid_constant__ CUtensorMap map_w, const Params p) {
    using Cfg = Config<MT>;
    constexpr int ROWS = Cfg::ROWS, A_STAGE_BYTES = Cfg::A_STAGE_BYTES, PIPE_BYTES = Cfg::PIPE_BYTES, MAX_RANKS = WIDE ? kMaxCluster : kPortableCluster;
    constexpr bool EARLY = MT <= 2;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t full_bar[STAGES];
    __shared__ __align__(8) uint64_t empty_bar[STAGES];
    __shared__ __align__(8) uint64_t recv_bar;  // the partial tiles of this CTA's columns have landed, and their scales
    __shared__ __align__(8) unsigned short own_scales[BN];  // f16 bits
    __shared__ unsigned int is_last;

    // 128B-swizzled TMA tiles need 1024-byte aligned bases.
    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char *smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
    const uint32_t w_base = smem_base;
    const uint32_t a_base = smem_base + STAGES * W_STAGE_BYTES;
    const uint32_t recv_base = smem_base + PIPE_BYTES;
    float *recv = reinterpret_cast<float *>(smem_gen + PIPE_BYTES);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2;  // MMA group id
    const int t = lane & 3;   // thread in group
    const int n0 = blockIdx.x * BN;
    const int split = blockIdx.y;
    const int m0 = blockIdx.z * ROWS;
    const int total_iters = (p.k_end - p.k_begin + BK - 1) / BK;
    const int it_begin = split * p.iters_per_split;
    int n_iters = total_iters - it_begin;
    if (n_iters > p.iters_per_split) n_iters = p.iters_per_split;
    if (n_iters < 0) n_iters = 0;
    int rows = p.M - m0;
    if (rows > ROWS) rows = ROWS;
    const uint32_t nranks = cluster_nctarank();
    const uint32_t rank = cluster_ctarank();
    const int cols_per = p.cols_per;
    // Columns of the tile this CTA sums in the reduction: [own_first, own_first + own_cols).
    const int own_first = (int)rank * cols_per;
    int own_cols = BN - own_first;
    if (own_cols > cols_per) own_cols = cols_per;
    if (own_cols < 0) own_cols = 0;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1 + 32);  // the weight tile (TMA bytes) and the producer warp's 32 lanes, each when its activation copies have landed
            mbar_init(smem_u32(&empty_bar[s]), CONSUMER_WARPS);
        }
        mbar_init(smem_u32(&recv_bar), 1 + 1);  // the expected bytes, and the producer warp with the scales
        mbar_fence_init();
        // Bytes the cluster will send here: every rank, `rows` rows of this CTA's columns.
        if (p.mode == kModeSplit && own_cols > 0) mbar_expect_tx(smem_u32(&recv_bar), nranks * (uint32_t)rows * (uint32_t)own_cols * 4u);
    }
    __syncthreads();
    // First half of a cluster barrier whose second half sits in front of the first remote store: by
    // then every CTA of the cluster has started and set up its barriers, which remote access requires.
    cluster_arrive_release();

    // The scales may be a result of the kernel in front: they are asked for when that one is done, through L2, far from where they are
    // used, by the producer warp for the columns that this CTA sums (in shared memory at the end of its loop; by every thread for itself a
    // decode step takes 209.0 us for 207.6), without a split by every consumer for its own four.  They stay as they come until
    // they are used: a conversion where they are loaded waits for them in front of the main loop ((4, 4096, 1024) 4.4 us
    // for 3.9 to 4.1).
    const unsigned short *scale_bits = reinterpret_cast<const unsigned short *>(p.scale) + n0;
    unsigned short sc_bits[4] = {0, 0, 0, 0};
    auto scale_of = [&](int cc) { return __half2float(__ushort_as_half(own_scales[cc])); };

    // acc[j][mt][.]: 16 x 8 tile j of this warp's 32 columns, activation rows 8 * mt ... 8 * mt + 7.
    // Element (column 16 j + 8 h + g, row 8 mt + 2t + e) is acc[j][mt][2h + e].
    float acc[2][MT][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) acc[j][mt][0] = acc[j][mt][1] = acc[j][mt][2] = acc[j][mt][3] = 0.0f;

    if (warp == CONSUMER_WARPS) {
        // ---------------- producer warp ----------------
        // Lane 0 drives the TMA loads of the weight tiles.  The activation slices (8 MT rows x 64 k of f16 per stage,
        // 128-byte rows, 16-byte chunk c of row r at chunk c ^ 2 (r & 3), so that a consumer's 8-byte loads of four rows touch
        // every bank once)
        // are copied by all 32 lanes with cp.async: they are a few hundred bytes that sit in L2, and on the load/store
        // path they do not wait in the TMA queue behind weight tiles that are still on their way from HBM.
        uint32_t dst_off[2 * MT];
        const __half *src_row[2 * MT];
        int kc[2 * MT];
#pragma unroll
        for (int q = 0; q < 2 * MT; ++q) {
            const int chunk = lane + 32 * q;  // 8 chunks per row
            const int r = chunk >> 3, c = chunk & 7;
            dst_off[q] = r * 128 + ((c ^ ((r & 3) << 1)) << 4);
            src_row[q] = m0 + r < p.M ? p.a + (size_t)(m0 + r) * p.lda : nullptr;  // rows beyond M are zero-filled
            kc[q] = 8 * c;
        }
        auto load_weights = [&](int s, int it, uint64_t policy) {
            const uint32_t bar = smem_u32(&full_bar[s]);
            const int k0 = p.k_begin + (it_begin + it) * BK;
            mbar_expect_tx(bar, W_STAGE_BYTES);
            tma_load_2d_hint(w_base + s * W_STAGE_BYTES, &map_w, NK ? k0 : n0, NK ? n0 : k0, bar, policy);
        };
        auto copy_activations = [&](int s, int k0) {
#pragma unroll
            for (int q = 0; q < 2 * MT; ++q) {
                const int k = k0 + kc[q];
                const bool in = src_row[q] != nullptr && k < p.k_end;  // k_end is a multiple of 8 or the row's end: a chunk is in or out as a whole
                cp_async_16(a_base + s * A_STAGE_BYTES + dst_off[q], in ? static_cast<const void *>(src_row[q] + k) : static_cast<const void *>(p.a), in ? 16u : 0u);
            }
            cp_async_arrive(smem_u32(&full_bar[s]));
        };
        const int prologue = n_iters < STAGES ? n_iters : STAGES;
        uint64_t stream_policy = 0;
        if (lane == 0) {
            tma_prefetch_desc(&map_w);
            stream_policy = l2_policy_evict_first();  // the weight is read once
            // The weight does not depend on the kernel before this one in the stream; the activations
            // may.  Ask for the first weight tiles, then wait for that kernel, then ask for activations.
            if (MT == 2 && p.late) pdl_wait();
            for (int it = 0; it < prologue; ++it) {
                if (EARLY) load_weights(it, it, stream_policy);
                else tma_prefetch_2d(&map_w, NK ? p.k_begin + (it_begin + it) * BK : n0, NK ? n0 : p.k_begin + (it_begin + it) * BK);
            }
        }
        __syncwarp();
        pdl_wait();
        if (!EARLY && lane == 0) {
            for (int it = 0; it < prologue; ++it) load_weights(it, it, stream_policy);
        }
        __syncwarp();
        // The kernel in front is done; the one behind may move in now: its CTAs fill their rings while this launch streams
        // the rest of its weight, so that it starts with its first stages in shared memory.  Two launches at a time is as
        // far ahead as pays: allowed at the very start, its successors pile up and all their rings compete with this one's
        // (1, 4096, 4096: 4.9 us here, 5.5 at the end of the main loop, 5.9 at the start).  With several row blocks the
        // launch lives from L2, which the next one's rings would only crowd (19 rows through a 7B-shaped step: 458 us, 451
        // at the end of the main loop).
        if (gridDim.z == 1) pdl_launch_dependents();
        for (int it = 0; it < prologue; ++it) copy_activations(it, p.k_begin + (it_begin + it) * BK);
        if (p.mode == kModeSplit) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int cc = 4 * lane + j;
                if (cc < own_cols && n0 + own_first + cc < p.N) sc_bits[j] = __ldcg(scale_bits + own_first + cc);
            }
        }
        for (int it = STAGES; it < n_iters; ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(smem_u32(&empty_bar[s]), ((it / STAGES) - 1) & 1)) {
                if (lane == 0) report_timeout(p.status, kKernelDecode, 1);
                break;
            }
            const int k0 = p.k_begin + (it_begin + it) * BK;
            if (lane == 0) load_weights(s, it, stream_policy);
            copy_activations(s, k0);
        }
        if (p.mode == kModeSplit) {
            *reinterpret_cast<uint2 *>(own_scales + 4 * lane) = make_uint2(sc_bits[0] | (uint32_t)sc_bits[1] << 16, sc_bits[2] | (uint32_t)sc_bits[3] << 16);
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&recv_bar));
        }
    } else {
        // ---------------- consumers ----------------
        pdl_wait();
        if (p.mode == kModeDirect) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // i = 2 j + h, see below
                const int cc = 32 * warp + 8 * i + g;
                if (n0 + cc < p.N) sc_bits[i] = __ldcg(scale_bits + cc);
            }
        }
        // Weights: one transposing matrix load per 16 k-rows brings this warp's 32 columns (16-byte
        // chunks 2 warp and 2 warp + 1 of each row).  Lane l addresses row (l & 15) of chunk
        // 2 warp + (l >> 4); under the 128B swizzle chunk c of row r sits at chunk c ^ (r & 7).
        const uint32_t off_w = (lane & 15) * 128 + (((2 * warp + (lane >> 4)) ^ (lane & 7)) << 4);
        // [N, K] weights: lane l addresses row 32 warp + 8 (l / 8 % 2) + l % 8 (+ 16 j) of the stage, 16-byte
        // chunk l / 16 (+ 2 per 32 k); rows are 64 bytes, chunk c of row r sits at chunk c ^ (r / 2 % 4).
        const uint32_t nk_row = 32 * warp + 8 * ((lane >> 3) & 1) + (lane & 7);
        const uint32_t nk_chunk = (uint32_t)lane >> 4;
        // Activations: row g (and g + 8, same swizzle phase), k = 16 ks + 4t .. 4t+3: bytes 8 (t & 1) of
        // chunk 2 ks + (t >> 1).
        const uint32_t off_a = g * 128 + 8 * (t & 1);
        const uint32_t a_chunk = (uint32_t)(t >> 1) ^ (uint32_t)((g & 3) << 1);  // chunk index is (2 ks) ^ a_chunk: bit 0 of 2 ks is free
        for (int it = 0; it < n_iters; ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(smem_u32(&full_bar[s]), (it / STAGES) & 1)) {
                report_timeout(p.status, kKernelDecode, 2);
                break;
            }
            const uint32_t wb = w_base + s * W_STAGE_BYTES + off_w;
            const uint32_t ab = a_base + s * A_STAGE_BYTES + off_a;
            uint32_t q[4][4];
            uint2 b[4][MT];
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                if (!NK) umma::ldmatrix_x2_trans_b8(q[ks], wb + ks * 2048);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) b[ks][mt] = lds64(ab + mt * 1024 + (((2 * ks) ^ a_chunk) << 4));
            }
            if (NK) {
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int kh = 0; kh < 2; ++kh) {
                        const uint32_t row = nk_row + 16 * j;
                        uint32_t r[4];
                        umma::ldmatrix_x4(r, w_base + s * W_STAGE_BYTES + row * 64 + (((2 * kh + nk_chunk) ^ ((row >> 1) & 3)) << 4));
                        q[2 * kh][2 * j] = r[0];
                        q[2 * kh][2 * j + 1] = r[1];
                        q[2 * kh + 1][2 * j] = r[2];
                        q[2 * kh + 1][2 * j + 1] = r[3];
                    }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&empty_bar[s]));  // the stage is in registers now
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    // tile j: MMA rows g / g + 8 are columns 32 warp + 16 j + g / + 8 + g;
                    // k slots (2t, 2t+1) and (2t+8, 2t+9) carry k = 4t, 4t+1 and 4t+2, 4t+3
                    uint32_t a0, a1, a2, a3;
                    umma::cvt_s8x4_to_f16_pairs(q[ks][2 * j], a0, a2);
                    umma::cvt_s8x4_to_f16_pairs(q[ks][2 * j + 1], a1, a3);
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) mma_m16n8k16(acc[j][mt], a0, a1, a2, a3, b[ks][mt].x, b[ks][mt].y);
                }
            }
        }
    }
    __syncwarp();  // the role branches above are lane-divergent; the cluster barrier below wants whole warps
    if (gridDim.z > 1) pdl_launch_dependents();

    const bool consumer = warp < CONSUMER_WARPS;
    // This thread's four columns inside the tile: 32 warp + 16 j + 8 h + g.
    const int col_base = 32 * warp + g;

    if (p.mode == kModeDirect) {
        cluster_wait_acquire();
        if (consumer) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int nn = n0 + col_base + 16 * j + 8 * h;
                    const float sc = __half2float(__ushort_as_half(sc_bits[2 * j + h]));
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int r = 8 * mt + 2 * t + e;  // columns nn and nn ^ 1 live in lanes that differ in g by one
                            finish(p.out, p.ep, m0 + r, nn, p.N, r < rows, acc[j][mt][2 * h + e] * sc, 4);
                        }
                }
        }
        return;
    }

    // ---------------- split-K ----------------
    // Level 1, inside a cluster: every CTA sends its partial tile into the shared memory of the CTA that
    // owns those columns, counted in bytes on the owner's barrier; the owner then holds the partials of all
    // ranks.  (Without a cluster the CTA is its own owner and the same code runs on local shared memory.)
    // recv layout: [rank][row][cols_per] fp32.
    cluster_wait_acquire();  // every CTA of the cluster is running
    if (consumer) {
        if (rows <= 2) {
            // One or two rows live in the lanes with t == 0: a few scalar remote stores, no staging.
            if (t == 0) {
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int col = col_base + 16 * j + 8 * h;
                        const uint32_t owner = (uint32_t)(col / cols_per);
                        const int col_in = col - (int)owner * cols_per;
                        const uint32_t remote = map_to_rank(recv_base, owner);
                        const uint32_t rbar = map_to_rank(smem_u32(&recv_bar), owner);
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            if (e < rows) st_async_f32(remote + (((int)rank * ROWS + e) * cols_per + col_in) * 4, acc[j][0][2 * h + e], rbar);
                    }
            }
        } else {
            // More rows: transpose through a staging block in the (now idle) weight ring, then 16-byte remote stores.
            asm volatile("bar.sync 1, %0;" ::"n"(32 * CONSUMER_WARPS) : "memory");  // every consumer warp is done with the ring
            const uint32_t stage_w = w_base + warp * (ROWS * STAGING_ROW * 4);
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                        for (int e = 0; e < 2; ++e) sts32f(stage_w + ((8 * mt + 2 * t + e) * STAGING_ROW + 16 * j + 8 * h + g) * 4, acc[j][mt][2 * h + e]);
            __syncwarp();
            // lane -> row lane / 8 of each pass of four rows, columns 4 (lane % 8) .. + 3
            const int rr = lane >> 3, v4 = lane & 7;
            const int col = 32 * warp + 4 * v4;
            const uint32_t owner = (uint32_t)(col / cols_per);
            const int col_in = col - (int)owner * cols_per;
            const uint32_t remote = map_to_rank(recv_base, owner) + (((int)rank * ROWS) * cols_per + col_in) * 4;
            const uint32_t rbar = map_to_rank(smem_u32(&recv_bar), owner);
#pragma unroll
            for (int pass = 0; pass < ROWS / 4; ++pass) {
                const int r = pass * 4 + rr;
                if (r < rows) st_async_v4f32(remote + r * cols_per * 4, lds128f(stage_w + (r * STAGING_ROW + 4 * v4) * 4), rbar);
            }
        }
    }
    if (own_cols > 0) {
        if (!mbar_wait_cluster(smem_u32(&recv_bar), 0)) report_timeout(p.status, kKernelDecode, 4);
    }
    // Owner: the partials of the ranks are read eight together and added in rank order.
    const int col_first = n0 + own_first;  // first column this CTA owns
    auto sum_ranks = [&](int r, int cc) {
        float sum = 0.0f;
#pragma unroll
        for (int first = 0; first < MAX_RANKS; first += 8) {
            float v[8];
#pragma unroll
            for (int jr = 0; jr < 8; ++jr) v[jr] = first + jr < (int)nranks ? recv[((first + jr) * ROWS + r) * cols_per + cc] : 0.0f;
            if (first == 0) sum = v[0];
#pragma unroll
            for (int jr = first == 0 ? 1 : 0; jr < 8; ++jr) sum += v[jr];
        }
        return sum;
    };
    if (p.groups == 1) {
        if constexpr (QUAD) {
            // Four adjacent columns of one row per thread and round, so that 16 rows of a slice are one round (one element per thread
            // made four of them, each with its trips to memory: (16, 1408, 1408) with a residual 5.5 -> 3.6 us, (16, 4096,
            // 12288) 13.3 -> 11.9, (7, 896, 12112) 5.8 -> 4.7).  Item i is row i / per_row, columns 4 (i % per_row) .. + 3.
            const int per_row = cols_per / 4;
            auto sum_ranks4 = [&](int r, int cc) {
                float4 sum;
#pragma unroll
                for (int first = 0; first < MAX_RANKS; first += 8) {
                    float4 v[8];
#pragma unroll
                    for (int jr = 0; jr < 8; ++jr)
                        v[jr] = first + jr < (int)nranks ? *reinterpret_cast<const float4 *>(recv + ((first + jr) * ROWS + r) * cols_per + cc) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (first == 0) sum = v[0];
#pragma unroll
                    for (int jr = first == 0 ? 1 : 0; jr < 8; ++jr) sum.x += v[jr].x, sum.y += v[jr].y, sum.z += v[jr].z, sum.w += v[jr].w;
                }
                return sum;
            };
            for (int item = threadIdx.x; item < rows * per_row; item += THREADS) {
                const int r = item / per_row;
                const int cc = (item - r * per_row) * 4;
                const int nn = col_first + cc;
                if (cc >= own_cols || nn >= p.N) continue;  // own_cols is a multiple of 4
                float4 y = sum_ranks4(r, cc);
                const uint2 sc4 = *reinterpret_cast<const uint2 *>(own_scales + cc);
                const float2 sc01 = __half22float2(*reinterpret_cast<const __half2 *>(&sc4.x)), sc23 = __half22float2(*reinterpret_cast<const __half2 *>(&sc4.y));
                y.x *= sc01.x, y.y *= sc01.y, y.z *= sc23.x, y.w *= sc23.y;
                if (nn + 3 < p.N) {
                    finish4(p.out, p.ep, m0 + r, nn, y);
                } else {  // the end of an [N, K] weight's odd column count: no epilogue there
                    const float e[3] = {y.x, y.y, y.z};
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        if (nn + j < p.N) store_out(p.out, m0 + r, nn + j, __float2half_rn(e[j]));
                }
            }
        } else {
            // One element per thread and round; element i is row i / cols_per, column i % cols_per of the slice.
            for (int idx = threadIdx.x; idx < rows * cols_per; idx += THREADS) {
                const int r = idx / cols_per;
                const int cc = idx - r * cols_per;
                const int nn = col_first + cc;
                const bool valid = nn < p.N && cc < own_cols;  // N and own_cols are even: the two columns of a pair agree
                finish(p.out, p.ep, m0 + r, nn, p.N, valid, valid ? sum_ranks(r, cc) * scale_of(cc) : 0.0f, 1);
            }
        }
        return;
    }

    // Level 2, across the `groups` clusters of a tile: each owner publishes its cluster's sum in the
    // caller's workspace; the last of the `groups` owners of a column slice to arrive adds them in
    // group order and finishes.
    const int group = (int)(blockIdx.y / nranks);
    for (int idx = threadIdx.x; idx < rows * cols_per; idx += THREADS) {
        const int r = idx / cols_per;
        const int cc = idx - r * cols_per;
        const int nn = col_first + cc;
        if (nn < p.N && cc < own_cols) __stcg(&p.partial[((size_t)group * p.M + (m0 + r)) * p.N + nn], sum_ranks(r, cc));
    }
    __threadfence();
    __syncthreads();
    const unsigned int slot = (blockIdx.z * gridDim.x + blockIdx.x) * nranks + rank;
    if (threadIdx.x == 0) {
        const unsigned int prev = atomicAdd(&p.counters[slot], 1u);
        is_last = (prev == (unsigned int)(p.groups - 1)) ? 1u : 0u;
    }
    __syncthreads();
    if (is_last == 0) return;
    __threadfence();
    for (int idx = threadIdx.x; idx < rows * cols_per; idx += THREADS) {
        const int r = idx / cols_per;
        const int cc = idx - r * cols_per;
        const int nn = col_first + cc;
        const bool valid = nn < p.N && cc < own_cols;
        float v = 0.0f;
        if (valid) {
#pragma unroll 4
            for (int gr = 0; gr < p.groups; ++gr) v += __ldcg(&p.partial[((size_t)gr * p.M + (m0 + r)) * p.N + nn]);
            v *= scale_of(cc);
        }
        finish(p.out, p.ep, m0 + r, nn, p.N, valid, v, 1);
    }
    if (threadIdx.x == 0) p.counters[slot] = 0;  // leave the workspace ready for the next call
}

}  // namespace decode

namespace decode {

// Instantiations by rows: up to four, eight, sixteen and twenty-four; of each, by layout and for clusters beyond the portable size.
struct Variant {
    const void *kernel[2][2];  // [weight_nk][cluster > kPortableCluster]
    int rows, smem, ctas;
};
template <int MT, bool QUAD>
static Variant make_variant() {
    return {{{reinterpret_cast<const void *>(qlinear_decode_kn_kernel<MT, false, QUAD, false>), reinterpret_cast<const void *>(qlinear_decode_kn_kernel<MT, false, QUAD, true>)},
             {reinterpret_cast<const void *>(qlinear_decode_kn_kernel<MT, true, QUAD, false>), reinterpret_cast<const void *>(qlinear_decode_kn_kernel<MT, true, QUAD, true>)}},
            Config<MT>::ROWS, Config<MT>::SMEM_BYTES, Config<MT>::CTAS};
}
constexpr int kVariantCount = 4;
static const Variant kVariants[kVariantCount] = {make_variant<1, false>(), make_variant<1, true>(), make_variant<2, true>(), make_variant<3, true>()};
static int set_attributes() {
    static std::atomic<bool> attr_set[64];  // per device, zero-initialised; a repeated set by a racing thread is harmless
    int dev = 0;
    B200Q_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        for (const Variant &v : kVariants)
            for (int i = 0; i < 4; ++i) {
                const void *f = v.kernel[i >> 1][i & 1];
                B200Q_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem));
                if (i & 1) B200Q_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            }
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    return B200Q_OK;
}

// The current device, asked once a plan: a plan looks at up to fifteen cluster sizes, and a call makes several plans.  -1: none.
static int current_device() {
    int dev = -1;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) return dev;
    cudaGetLastError();
    return -1;
}

// CTAs of a variant that run at once in clusters of `cluster`: four per SM less what the clusters cannot use.  Looked up once
// per device; without a device, an estimate (none of clusters that not every device runs: the plan does without them).
static int resident_ctas(int dev, const Variant &v, int cluster) {
    static std::atomic<int> known[64][kVariantCount][kMaxCluster + 1];
    const int estimate = cluster <= kPortableCluster ? (148 - 8) * v.ctas : 0;
    if (dev < 0) return estimate;
    std::atomic<int> &slot = known[dev][&v - kVariants][cluster];
    int n = slot.load(std::memory_order_relaxed);
    if (n != 0) return n;
    if (set_attributes() != B200Q_OK) {
        cudaGetLastError();
        return estimate;
    }
    n = resident_clusters(v.kernel[0][cluster > kPortableCluster], THREADS, v.smem, cluster);
    if (n == 0) return estimate;
    n *= cluster;
    slot.store(n, std::memory_order_relaxed);
    return n;
}

}  // namespace decode

// The plan that every device can run: blocks of up to 16 rows, clusters of up to eight CTAs.  The scratch that callers are asked for is this
// plan's, whether the one that is launched needs any or not.
DecodePlan plan_decode_portable(int64_t M, int64_t N, int64_t K) {
    using namespace decode;
    DecodePlan pl;
    pl.n_tiles = (int)ceil_div(N, BN);
    const int k_iters = (int)ceil_div(K, BK);
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    const int dev = current_device();
    const Variant &v = kVariants[M <= 4 ? 0 : (M <= 8 ? 1 : 2)];
    pl.variant = (int)(&v - kVariants);
    pl.m_tiles = (int)ceil_div(M, v.rows);
    const int64_t tiles = (int64_t)pl.n_tiles * pl.m_tiles;
    // Each split has at least four 64-row steps of work, a ring's fill: with eight a narrow problem leaves most of the SMs
    // idle (a step of a 1024-wide decoder 72 -> 57 us), with two the exchange costs what the shorter loop gives (64 us).  Only where
    // that leaves fewer than four splits are two steps enough, for the last phase's sake: one CTA alone finishes 16 rows of 128
    // columns in several rounds ((16, 256, 688) 4.2 -> 3.0 us, (1, 256, 688) 2.75 -> 2.15, (16, 640, 2048) 3.8 -> 2.8), and where the grid has
    // the room: four splits up to four ninths as many tiles as SMs ((1, 512, 8192) 2.7 -> 2.6, (1, 512, 9472) 2.8 -> 3.1, (16, 512, 16384) 4.5 -> 4.8), two
    // of fewer than eight steps up to as many ((1, 384, 18688) 3.5 -> 2.9, (1, 384, 28160) 3.7 -> 4.0; with more than eight rows half as many again).
    int max_splits = k_iters >= 4 ? k_iters / 4 : 1;
    if (k_iters >= 4 && k_iters < 8) max_splits = tiles * 4 <= 2 * sms ? k_iters / 2 : (M > 16 || tiles <= (M <= 8 ? sms : sms * 3 / 2) ? 2 : 1);
    else if (max_splits < 4 && k_iters >= 8 && (M > 16 ? tiles * 4 <= 2 * sms : tiles * 9 <= 4 * sms)) max_splits = 4;
    // The splits of a tile form a cluster of up to eight CTAs (partials meet in distributed shared memory), as large as lets
    // the whole grid run at once: a few clusters left for a second wave double the time of the launch (96 tiles
    // in clusters of six are 576 CTAs and fit 148 x 4 slots by number, but not the groups of SMs clusters are confined to:
    // (1, 4096, 12288) 15.1 us, and 10.3 us in clusters of five).
    int c = 1;
    // (With several row blocks the second pass over the weight comes from L2 and a second wave costs little.)
    while (c < kPortableCluster && c < max_splits && tiles * (c + 1) <= (pl.m_tiles > 1 ? (int64_t)sms * v.ctas : resident_ctas(dev, v, c + 1))) ++c;
    // More splits than a cluster holds become several full clusters per tile that meet in the workspace.  They pay three
    // dependent trips through L2 at the end of the launch (publish, count, read back), about 3 us more than partials
    // that meet in distributed shared memory.  That is worth it only when one cluster per tile would leave most of the
    // machine idle, and only for splits of eight steps or more: with four, (1, 4096, 1024) takes 5.7 us against 3.8 and
    // (1, 8192, 1024) 6.5 against 6.3, though (1, 8192, 256) gains, 4.8 against 5.7.  (It is also what the scratch is sized by: with
    // four the partial sums of (16, 11008, 1024) would not fit the array of b200q_qlinear_f16_i8_static any more.)
    int groups = 1;
    if (c == kPortableCluster && tiles * c * 2 < sms) {
        int64_t splits = tiles > 0 ? (int64_t)sms * 4 / tiles : 1;
        if (splits > k_iters / 8) splits = k_iters / 8;
        if (splits > 64) splits = 64;
        groups = (int)(splits / c);
        if (groups < 1 || tiles * c > kMaxCounters) groups = 1;
    }
    // The counter region has one fixed size, so that counters never land on bytes an earlier call of
    // another shape used for partial sums: the region stays all-zero between calls.
    pl.counter_bytes = groups > 1 ? (size_t)kMaxCounters * 4 : 0;
    pl.partial_bytes = groups > 1 ? (size_t)groups * M * N * 4 : 0;
    pl.cluster = c;
    pl.groups = groups;
    pl.most_splits = max_splits;
    pl.splits = c * groups;  // the grid holds whole clusters; a split may get fewer steps than others, or none
    pl.iters_per_split = (int)ceil_div(k_iters, pl.splits);
    return pl;
}

// The plan where all SMs are at hand.
DecodePlan plan_decode(int64_t M, int64_t N, int64_t K) {
    using namespace decode;
    DecodePlan pl = plan_decode_portable(M, N, K);
    const int k_iters = (int)ceil_div(K, BK), c = pl.cluster, groups = pl.groups;
    const bool one_pass = M > 16 && M <= 24 && N * K >= kOnePassCodes;
    if (!one_pass && (pl.m_tiles > 1 || c < kPortableCluster || k_iters < 48)) return pl;
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    const int dev = current_device();
    // Up to 24 rows in one pass where the weight is more than what L2 delivers again for nothing: (24, 4096, 4096) 8.5 -> 8.2 us, (24, 4096, 12288)
    // 23.0 -> 14.5, (17, 2304, 6912) 8.3 -> 7.3 against two passes of 16 rows; below the line the passes run side by side ((24, 2048, 2048)
    // 4.0 us, 4.4 in one).  A form for 32 rows was no better than two passes or the mid-M kernel ((32, 4096, 4096) 8.8 and 8.5 us, (32, 4096,
    // 12288) 16.1 and 17.7): the warp-level MMAs of four row blocks take longer than the stream.
    int variant = pl.variant, m_tiles = pl.m_tiles, one = c;  // of the plan with one cluster a tile, of `one` CTAs
    // With three CTAs an SM, of clusters that are not of one, two or a multiple of four the last few that the query allows wait for CTAs of the launch
    // behind that have moved in ((24, 4096, 17408), 408 CTAs, 17.4 us; 414 19.6, 420 23.3, 426 24.9; (24, 8192, 8704), 408, 17.1 and with 426 22.1).
    auto full = [&](int cluster) {
        const int n = resident_ctas(dev, kVariants[variant], cluster), most = sms * 69 / 25;
        return variant == 3 && cluster > 2 && cluster % 4 != 0 && n > most ? most : n;
    };
    if (one_pass) {
        variant = 3, m_tiles = 1, one = 1;
        while (one < kPortableCluster && one < pl.most_splits && pl.n_tiles * (one + 1) <= full(one + 1)) ++one;
    }
    // Beyond the portable size where that leaves SMs idle ((1, 4096, 1024) 4.0 -> 3.1 us, (8, 8192, 1024) 6.7 -> 4.7, (16, 8192, 1024) 8.3 -> 5.4,
    // (1, 11008, 512) 7.0 -> 4.8 instead of clusters that meet in the workspace), and where the runs are long: with few CTAs an SM a stage
    // takes as long as its chain of waits and loads, not as its bytes ((1, 11008, 4096), 256 CTAs of 22 steps, 11.4 us; 448 of 13, 10.1;
    // (16, 11008, 4096) 12.9 -> 12.0, (1, 16384, 5120) 19.1 -> 16.1; not with three CTAs an SM, (7, 10080, 7088) 14.5 -> 16.8).  Short runs in many parts lose more in the exchange, which grows with the rows: (1, 4096, 4096) 5.0 -> 5.8
    // in sixteen parts of four steps, (16, 5376, 2304) 6.1 -> 6.4, (24, 4608, 1536) 5.3 -> 6.1 ((24, 5120, 1280) 5.6 -> 5.1).
    if (m_tiles == 1 && one == kPortableCluster && k_iters >= 48) {
        const int portable = pl.n_tiles * one;
        const bool narrow = M <= 8 ? portable <= sms : (M <= 16 ? portable * 3 <= sms * 2 : portable * 11 <= sms * 6), deep = k_iters >= (M <= 8 ? 12 : 16) * one && portable * 4 <= sms * 9;
        for (int wide = kMaxCluster; wide > kPortableCluster && (narrow || deep); --wide) {
            if (!slices_fit(wide) || pl.n_tiles * wide > full(wide)) continue;
            one = wide;
            break;
        }
    }
    // Several clusters a tile stay where one would leave each CTA so many more steps (0.24 to 0.3 us each) that the three trips through L2 cost less;
    // what goes through L2 grows with the tiles and the rows.  Over 378 sizes of K 16384 to 65536 and N 16 to 1536 within 0.7 % of the better
    // one: (1, 65536, 128) 8.4 us in eight clusters a tile, 17.2 in one; (16, 32768, 256) 8.7 and 10.8, (24, 65536, 512) 17.6 and 22.3;
    // but (8, 16384, 512) 6.4 and 6.0, (16, 24576, 768) 11.7 and 9.2, (24, 24576, 512) 11.7 and 10.0.
    const double extra = 8.0 + 1.4 * (double)pl.n_tiles * pl.m_tiles + (M <= 8 ? 0.0 : (M <= 16 ? 0.8 * (double)(M - 9) : 2.0));
    const bool other = one > c || m_tiles != pl.m_tiles;
    if (other && (groups == 1 || (double)(ceil_div(k_iters, one) - ceil_div(k_iters, c * groups)) <= extra)) {
        pl.variant = variant, pl.m_tiles = m_tiles;
        pl.cluster = pl.splits = one, pl.groups = 1;
        pl.iters_per_split = (int)ceil_div(k_iters, one);
    }
    return pl;
}

// Clusters beyond the portable size are taken by what the device holds; a part of its SMs may hold none of them, and the launch would fail.
DecodePlan plan_decode_on(cudaStream_t stream, int64_t M, int64_t N, int64_t K) {
    const DecodePlan pl = plan_decode(M, N, K);
    return pl.cluster > decode::kPortableCluster && part_of_device(stream) ? plan_decode_portable(M, N, K) : pl;
}

bool decode_kn_supported(const void *a, const void *wq, int64_t N, int64_t K) {
    return (N % 16 == 0) && (K % 8 == 0) && ((reinterpret_cast<uintptr_t>(a) & 15u) == 0) &&
           ((reinterpret_cast<uintptr_t>(wq) & 15u) == 0);
}

bool decode_nk_supported(const void *a, const void *wq, int64_t N, int64_t K) {
    (void)N;
    return (K % 16 == 0) && ((reinterpret_cast<uintptr_t>(a) & 15u) == 0) && ((reinterpret_cast<uintptr_t>(wq) & 15u) == 0);
}

int launch_decode_kn(const void *a, const void *wq, const void *scale, void *c, int64_t M, int64_t N, int64_t K,
                     int64_t k_begin, int64_t k_end, bool allow_split, void *workspace, size_t workspace_bytes,
                     cudaStream_t stream, const OutTargets *targets, const Epilogue *epilogue, bool weight_nk, const DecodePlan *plan) {
    using namespace decode;
    DecodePlan pl = plan != nullptr ? *plan : plan_decode_on(stream, M, N, k_end - k_begin);
    if (pl.cluster > kMaxCluster || !slices_fit(pl.cluster)) return set_error(B200Q_INVALID_ARGUMENT, "qlinear: no clusters of %d CTAs", pl.cluster);
    if (!allow_split) {
        pl.iters_per_split = (int)ceil_div(k_end - k_begin, BK);
        pl.splits = 1;
        pl.cluster = 1;
        pl.groups = 1;
        pl.partial_bytes = 0;
        pl.counter_bytes = 0;
    }
    if (pl.partial_bytes > 0 && (workspace == nullptr || workspace_bytes < pl.counter_bytes + pl.partial_bytes)) {
        return set_error(B200Q_WORKSPACE_TOO_SMALL, "qlinear: workspace of %zu bytes given, %zu needed for M=%lld N=%lld K=%lld",
                         workspace_bytes, pl.counter_bytes + pl.partial_bytes, (long long)M, (long long)N, (long long)K);
    }
    if (pl.m_tiles > 65535 || pl.splits > 65535) return set_error(B200Q_UNSUPPORTED, "qlinear: M=%lld is too large for the small-M kernel", (long long)M);

    CUtensorMap map_w;
    int rc = weight_nk ? make_tensor_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, wq, (uint64_t)k_end, (uint64_t)N, (uint64_t)K, BK, BN,
                                            CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)
                       : make_tensor_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, wq, (uint64_t)N, (uint64_t)k_end, (uint64_t)N, BN, BK,
                                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200Q_OK) return rc;

    Params p;
    p.a = static_cast<const __half *>(a);
    p.lda = K;
    p.scale = static_cast<const __half *>(scale);
    if (targets != nullptr) {
        p.out = *targets;
    } else {
        p.out.ptr[0] = c;
        p.out.count = 1;
        p.out.ldc = (epilogue != nullptr && epilogue->act == kActSiluMul) ? N / 2 : N;
        p.out.col0 = 0;
    }
    if (epilogue != nullptr) p.ep = *epilogue;
    p.counters = static_cast<unsigned int *>(workspace);
    p.partial = pl.groups > 1 ? reinterpret_cast<float *>(static_cast<unsigned char *>(workspace) + pl.counter_bytes) : nullptr;
    p.status = device_status_word();
    p.M = (int)M;
    p.N = (int)N;
    p.k_begin = (int)k_begin;
    p.k_end = (int)k_end;
    p.iters_per_split = pl.iters_per_split;
    p.groups = pl.groups;
    p.cols_per = slice_cols(pl.cluster);
    p.mode = pl.splits == 1 ? kModeDirect : kModeSplit;
    p.late = M > 16 && M <= 24 && N * (k_end - k_begin) >= kOnePassCodes;

    const Variant &v = kVariants[pl.variant];
    const void *kernel = v.kernel[weight_nk][pl.cluster > kPortableCluster];
    const int rc_attr = set_attributes();
    if (rc_attr != B200Q_OK) return rc_attr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)pl.n_tiles, (unsigned)pl.splits, (unsigned)pl.m_tiles);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = v.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = 1;
    attrs[0].val.clusterDim.y = (unsigned)pl.cluster;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 2;
    void *args[2] = {&map_w, &p};
    B200Q_CUDA_TRY(cudaLaunchKernelExC(&cfg, kernel, args));
    return B200Q_OK;
}

}  // namespace b200q
