// Mid-M f16 x int8 quantized linear (a few dozen activation rows): bound by streaming the weight, computed on tcgen05.
//
// D[n, m] = sum_k W[k, n] * A[m, k], the weight converted to f16 in tensor memory (where the tensor core takes its first
// operand from), one CTA per 128 weight columns x TM activation rows (TM a multiple of 16, at most 128) and K split over the CTAs
// of a cluster, so that the weight is in flight on every SM: two CTAs per SM with 48 KB of int8 tiles on their way each.  (One CTA
// per SM with 96 KB and twice the converters: 25 us for 17 on (64, 4096, 11008).)  The partial tiles meet in distributed
// shared memory: no workspace, no second launch, the same result on every run.
//
// Warps: converters in two groups that take stages in turn, then do the reduction and the epilogue; a TMA producer of the int8
// tiles; a TMA producer of the activation tiles; the MMA issuer.
// Nothing is read before the kernel in front is done, the weight included; the first tiles are asked into L2 meanwhile.  Every wait is bounded (see qlinear_prefill.cu).
#include <atomic>

#include "common.cuh"
#include "qlinear.h"
#include "umma.cuh"

namespace b200q {
namespace mid {

constexpr int TN = 128, BK = 64;
constexpr int RAW_BYTES = BK * TN;
constexpr int CONV_GROUPS = 2, GROUP_WARPS = 4, CONV_WARPS = CONV_GROUPS * GROUP_WARPS;
constexpr int RAW_SLOTS = 6;
constexpr int W_SLOTS = 4;                    // converted weight tiles in tensor memory, 32 columns each
constexpr uint32_t TMEM_COLS = 256;           // two CTAs share an SM
constexpr uint32_t W_COL0 = TMEM_COLS - 32 * W_SLOTS;
constexpr int MAX_SLOTS = 8;
static_assert(RAW_SLOTS % CONV_GROUPS == 0 && W_SLOTS % CONV_GROUPS == 0, "a slot stays with one converter group");
constexpr int RAW_WARP = CONV_WARPS, ACT_WARP = RAW_WARP + 1, MMA_WARP = ACT_WARP + 1;
constexpr int THREADS = 32 * (MMA_WARP + 1);
constexpr int CONV_THREADS = 32 * CONV_WARPS;
constexpr int BLOCK_BYTES = TN * 8 * 4;       // fp32 sums of 8 rows: the unit of the reduction
constexpr int ROW_BYTES = TN * 2 + 16;        // one output row in the staging buffer, padded
constexpr int CTA_SMEM = 110 * 1024;          // with the static part and what the system takes, twice per SM

struct Params {
    const __half *scale;
    OutTargets out;              // [M, N], or [M, N / 2] with the gate / up pairing; not a multicast address
    Epilogue ep;
    unsigned int *status;
    int M, N;
    int tm;                      // activation rows per tile
    int k_blocks;
    int act_slots;               // length of the activation ring
};

// Shared memory: activation ring, int8 ring; after the main loop the partial sums (own 8-row blocks x ranks) and then
// the staging rows take the place of both.
static int act_slots_of(int tm) {
    const int n = (CTA_SMEM - 1024 - RAW_SLOTS * RAW_BYTES) / (tm * BK * 2);
    return n < MAX_SLOTS ? n : MAX_SLOTS;
}
static int smem_of(int tm, int cluster) {
    const int rings = act_slots_of(tm) * tm * BK * 2 + RAW_SLOTS * RAW_BYTES, own = (tm / 8 + cluster - 1) / cluster;
    const int exchange = own * cluster * BLOCK_BYTES + own * 8 * ROW_BYTES;
    return (rings > exchange ? rings : exchange) + 1024;
}

template <bool FUSED, bool NK>
__global__ void __launch_bounds__(THREADS, 2)
    qlinear_mid_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const Params p) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t raw_full[RAW_SLOTS];    // an int8 tile has landed
    __shared__ __align__(8) uint64_t raw_empty[RAW_SLOTS];   // its converter group has read it
    __shared__ __align__(8) uint64_t act_full[MAX_SLOTS];    // an activation tile has landed
    __shared__ __align__(8) uint64_t act_empty[MAX_SLOTS];   // the MMAs that read it have completed
    __shared__ __align__(8) uint64_t ready[W_SLOTS];         // a converted weight tile is in tensor memory
    __shared__ __align__(8) uint64_t done[W_SLOTS];          // the MMAs that read it have completed
    __shared__ __align__(8) uint64_t acc_full;               // all MMAs have completed
    __shared__ __align__(8) uint64_t recv_bar;               // the partial sums of this CTA's blocks have landed
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char *smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int ranks = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
    const int n0 = blockIdx.x * TN, m0 = blockIdx.z * p.tm;
    const int kb_begin = (int)((int64_t)p.k_blocks * rank / ranks), kb_end = (int)((int64_t)p.k_blocks * (rank + 1) / ranks);
    const uint32_t n_it = (uint32_t)(kb_end - kb_begin);     // at least one: clusters are no larger than k_blocks
    constexpr uint32_t raw_slots = RAW_SLOTS;
    const uint32_t act_slots = p.act_slots;
    const uint32_t act_bytes = (uint32_t)p.tm * BK * 2;
    const uint32_t raw_off = act_slots * act_bytes;
    // 8-row blocks of the tile in the reduction: block b belongs to rank b % ranks
    const int blocks = p.tm / 8, own_blocks = (blocks - rank + ranks - 1) / ranks;

    if (threadIdx.x == 0) {
        for (int s = 0; s < RAW_SLOTS; ++s) {
            mbar_init(smem_u32(&raw_full[s]), 1);
            mbar_init(smem_u32(&raw_empty[s]), GROUP_WARPS);
        }
        for (int s = 0; s < MAX_SLOTS; ++s) {
            mbar_init(smem_u32(&act_full[s]), 1);
            mbar_init(smem_u32(&act_empty[s]), 1);
        }
        for (int w = 0; w < W_SLOTS; ++w) {
            mbar_init(smem_u32(&ready[w]), GROUP_WARPS);
            mbar_init(smem_u32(&done[w]), 1);
        }
        mbar_init(smem_u32(&acc_full), 1);
        mbar_init(smem_u32(&recv_bar), 1);
        abort_flag = 0;
        mbar_fence_init();
        if (own_blocks > 0) mbar_expect_tx(smem_u32(&recv_bar), (uint32_t)(own_blocks * ranks) * BLOCK_BYTES);
    }
    if (warp == MMA_WARP) {
        umma::alloc(smem_u32(&tmem_base_slot), TMEM_COLS);
        umma::relinquish();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    // A ring's fill of the weight, into L2 only, while the kernel in front ends: (64, 4096, 11008) 16.2 -> 15.8 us, [N, K] 16.8 -> 16.1,
    // (64, 2304, 6912) 10.6 -> 10.3.
    if (warp == RAW_WARP && lane == 0) {
        for (uint32_t i = 0; i < n_it && i < raw_slots; ++i) {
            const int k0 = (kb_begin + (int)i) * BK;
            tma_prefetch_2d(&map_w, NK ? k0 : n0, NK ? n0 : k0);
        }
    }
    if (warp == ACT_WARP && lane == 0) tma_prefetch_desc(&map_a);
    pdl_wait();  // every role: none of the bounded waits below runs against the kernel in front

    auto wait = [&](uint32_t bar, uint32_t parity, unsigned int site) -> bool {
        bool ok = mbar_wait(bar, parity, umma::kFastPolls);
        if (__all_sync(0xffffffffu, ok)) return true;
        if (!ok) ok = umma::wait_or_abort<kKernelMid>(bar, parity, site, &abort_flag, p.status);
        return __all_sync(0xffffffffu, ok);
    };

    auto wait_one = [&](uint32_t bar, uint32_t parity, unsigned int site) -> bool {  // one thread's
        return mbar_wait(bar, parity, umma::kFastPolls) || umma::wait_or_abort<kKernelMid>(bar, parity, site, &abort_flag, p.status);
    };

    if (warp == RAW_WARP) {
        // ---------------- TMA producer: int8 weight tiles ----------------
        const uint64_t once = l2_policy_evict_first();
        pdl_launch_dependents();  // tensor memory is allocated: a kernel that moves in cannot take it away from this one
        uint32_t i = 0;
        umma::Ring r;
        for (; i < n_it; ++i, r.advance(1, raw_slots)) {
            if (i >= raw_slots && !wait(smem_u32(&raw_empty[r.slot]), r.phase ^ 1u, 1)) break;
            if (elect_one()) {
                const int k0 = (kb_begin + (int)i) * BK;
                const uint32_t bar = smem_u32(&raw_full[r.slot]);
                mbar_expect_tx(bar, RAW_BYTES);
                if (gridDim.z == 1) tma_load_2d_hint(smem_base + raw_off + r.slot * RAW_BYTES, &map_w, NK ? k0 : n0, NK ? n0 : k0, bar, once);
                else tma_load_2d(smem_base + raw_off + r.slot * RAW_BYTES, &map_w, NK ? k0 : n0, NK ? n0 : k0, bar);
            }
            __syncwarp();
        }
        // Teardown: every copy armed must have landed.  Slot s was last used for the largest j < i with j % raw_slots == s.
        for (uint32_t s = 0; s < raw_slots; ++s) {
            if (i <= s) continue;
            const uint32_t j = i - 1 - (i - 1 - s) % raw_slots;
            if (!mbar_wait(smem_u32(&raw_full[s]), (j / raw_slots) & 1)) report_timeout(p.status, kKernelMid, 7);
        }
    } else if (warp == ACT_WARP) {
        // ---------------- TMA producer: activation tiles ----------------
        const uint64_t keep = l2_policy_evict_last();
        uint32_t i = 0;
        umma::Ring r;
        for (; i < n_it; ++i, r.advance(1, act_slots)) {
            if (i >= act_slots && !wait(smem_u32(&act_empty[r.slot]), r.phase ^ 1u, 2)) break;
            if (elect_one()) {
                const uint32_t bar = smem_u32(&act_full[r.slot]);
                mbar_expect_tx(bar, act_bytes);
                tma_load_2d_hint(smem_base + r.slot * act_bytes, &map_a, (kb_begin + (int)i) * BK, m0, bar, keep);
            }
            __syncwarp();
        }
        for (uint32_t s = 0; s < act_slots; ++s) {
            if (i <= s) continue;
            const uint32_t j = i - 1 - (i - 1 - s) % act_slots;
            if (!mbar_wait(smem_u32(&act_full[s]), (j / act_slots) & 1)) report_timeout(p.status, kKernelMid, 7);
        }
    } else if (warp == MMA_WARP) {
        // ---------------- MMA issuer ----------------
        // One thread for the whole loop: with the election inside it the four MMAs of a stage take 260 clocks to issue, with it
        // outside 47.  The barriers of the next stage are asked while this one's MMAs are on their way.
        if (elect_one()) {
            const uint32_t idesc = umma::instr_desc_f16(TN, p.tm);
            umma::Ring a, w;
            bool act_ok = false, w_ok = false;
            for (uint32_t i = 0; i < n_it; ++i) {
                if (!act_ok && !wait_one(smem_u32(&act_full[a.slot]), a.phase, 3)) break;
                if (!w_ok && !wait_one(smem_u32(&ready[w.slot]), w.phase, 4)) break;
                umma::fence_after_sync();
                const uint32_t a_addr = tmem_base + W_COL0 + 32 * w.slot;
                const uint64_t b_desc = umma::smem_desc_sw128(smem_base + a.slot * act_bytes);
#pragma unroll
                for (int ks = 0; ks < BK / 16; ++ks) umma::mma_ts(tmem_base, a_addr + 8 * ks, b_desc + 2 * ks, idesc, (i > 0 || ks > 0) ? 1u : 0u);
                umma::commit(smem_u32(&done[w.slot]));
                umma::commit(smem_u32(&act_empty[a.slot]));
                a.advance(1, act_slots), w.advance(1, W_SLOTS);
                act_ok = i + 1 < n_it && mbar_test(smem_u32(&act_full[a.slot]), a.phase);
                w_ok = i + 1 < n_it && mbar_test(smem_u32(&ready[w.slot]), w.phase);
            }
            umma::commit(smem_u32(&acc_full));
        }
        __syncwarp();
    } else {
        // ---------------- converters ----------------
        const int group = warp / GROUP_WARPS, q = warp & 3;
        const uint32_t w_lane = tmem_base + ((uint32_t)(32 * q) << 16) + W_COL0;
        // where this lane's matrix-load rows lie in a tile
        //   [K, N]: rows of 128 columns, 128B swizzle; lanes 0-15 / 16-31 address the first / second 16-column block
        //   [N, K]: rows of 64 k, 64B swizzle; lane = row, 16-byte chunk = 16 k
        const uint32_t kn_off = (uint32_t)(lane & 15) * 128u + (((uint32_t)(2 * q + (lane >> 4)) ^ (uint32_t)(lane & 7)) << 4);
        const uint32_t nk_row = (uint32_t)(32 * q + lane);
        const uint32_t nk_off = nk_row * 64u, nk_sw = (nk_row >> 1) & 3u;
        umma::Ring r, w;
        r.slot = group, w.slot = group;
        bool raw_ok = false;
        for (uint32_t i = group; i < n_it; i += CONV_GROUPS, w.advance(CONV_GROUPS, W_SLOTS)) {
            if (!__all_sync(0xffffffffu, raw_ok) && !wait(smem_u32(&raw_full[r.slot]), r.phase, 5)) break;
            const uint32_t raw = smem_base + raw_off + r.slot * RAW_BYTES;
            uint32_t v[4][4];  // [k block of 16][column block of 8]: four consecutive k of one column
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                if (NK) umma::ldmatrix_x4(v[ks], raw + nk_off + (((uint32_t)ks ^ nk_sw) << 4));
                else umma::ldmatrix_x2_trans_b8(v[ks], raw + ks * 16 * 128 + kn_off);
            }
            const uint32_t raw_bar = smem_u32(&raw_empty[r.slot]);
            r.advance(CONV_GROUPS, raw_slots);
            raw_ok = i + CONV_GROUPS < n_it && mbar_test(smem_u32(&raw_full[r.slot]), r.phase);
            const bool done_ok = i < (uint32_t)W_SLOTS || mbar_test(smem_u32(&done[w.slot]), w.phase ^ 1u);
            uint32_t h[2][16];
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
#pragma unroll
                for (int b = 0; b < 4; ++b) umma::cvt_s8x4_to_f16_pairs(v[ks][b], h[b >> 1][4 * ks + 2 * (b & 1)], h[b >> 1][4 * ks + 2 * (b & 1) + 1]);
            __syncwarp();
            if (lane == 0) mbar_arrive(raw_bar);  // the int8 tile is in registers
            if (!__all_sync(0xffffffffu, done_ok) && !wait(smem_u32(&done[w.slot]), w.phase ^ 1u, 6)) break;
            umma::fence_after_sync();
            umma::st_16x256b_x4(w_lane + 32 * w.slot, h[0]);
            umma::st_16x256b_x4(w_lane + (16u << 16) + 32 * w.slot, h[1]);
            umma::st_wait();
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ready[w.slot]));
        }
    }

    // ---------------- the main loop is over in this CTA, then in all of them: the rings are free ----------------
    __syncwarp();
    // What the end needs from memory is asked for now, so that it is there when the sums are, and converted then: a conversion waits.
    const int cw = warp & 7;  // this warp: columns 16 cw + 8 e + g of the tile
    unsigned short sc_bits[2] = {0, 0}, bias_bits[2] = {0, 0};
    if (warp < CONV_WARPS) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int n = n0 + 16 * cw + 8 * e + g;
            if (n < p.N) sc_bits[e] = __ldcg(reinterpret_cast<const unsigned short *>(p.scale) + n);
            if (FUSED && n < p.N && p.ep.bias != nullptr) bias_bits[e] = __ldcg(static_cast<const unsigned short *>(p.ep.bias) + n);
        }
    }
    if (!mbar_wait(smem_u32(&acc_full), 0)) report_timeout(p.status, kKernelMid, 8);
    __syncthreads();  // the producers' copies have landed
    umma::fence_after_sync();
    cluster_arrive_release();
    cluster_wait_acquire();

    if (warp < CONV_WARPS) {
        // Every CTA sends each 8-row block of its partial tile to the block's owner, in the order in which the lanes hold it
        // (lane (g, t): rows 2t, 2t + 1 of column g, then of column g + 8, of 16 columns); the owner adds the ranks' blocks
        // in rank order and finishes.
        const int q = warp & 3;
        // Two blocks are loaded together: one at a time, each waits for its own way out of tensor memory ((128, 4096, 4096) 12.6 us, 12.0 with
        // this and two of the last phase's blocks side by side, (64, 4096, 12288) 20.6 and 20.0; four of either are more code and no faster).
        constexpr int TOGETHER = 2, STEP = CONV_WARPS / 4;
        for (int b0 = warp >> 2; b0 < blocks; b0 += TOGETHER * STEP) {
            uint32_t v[TOGETHER][2][4];
#pragma unroll
            for (int i = 0; i < TOGETHER; ++i) {
                if (b0 + i * STEP < blocks) {
                    umma::ld_16x256b_x1(tmem_base + ((uint32_t)(32 * q) << 16) + 8 * (b0 + i * STEP), v[i][0]);
                    umma::ld_16x256b_x1(tmem_base + ((uint32_t)(32 * q + 16) << 16) + 8 * (b0 + i * STEP), v[i][1]);
                }
            }
            umma::ld_wait();
#pragma unroll
            for (int i = 0; i < TOGETHER; ++i) {
                const int b = b0 + i * STEP;
                if (b >= blocks) break;
                const int owner = b % ranks, slot = b / ranks;
                const uint32_t dst = map_to_rank(smem_base, owner) + (uint32_t)((slot * ranks + rank) * BLOCK_BYTES) + (uint32_t)(2 * q * 32 + lane) * 16u;
                const uint32_t bar = map_to_rank(smem_u32(&recv_bar), owner);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    st_async_v4f32(dst + h * 512, make_float4(__uint_as_float(v[i][h][0]), __uint_as_float(v[i][h][1]), __uint_as_float(v[i][h][2]), __uint_as_float(v[i][h][3])), bar);
            }
        }
        umma::fence_before_sync();
        if (own_blocks > 0 && !mbar_wait_cluster(smem_u32(&recv_bar), 0)) report_timeout(p.status, kKernelMid, 10);
        const bool pairs = FUSED && p.ep.act == kActSiluMul;
        const __half *res = FUSED ? static_cast<const __half *>(p.ep.residual) : nullptr;
        const int out_n = pairs ? p.N >> 1 : p.N, out_n0 = pairs ? n0 >> 1 : n0;
        const float sc[2] = {__half2float(__ushort_as_half(sc_bits[0])), __half2float(__ushort_as_half(sc_bits[1]))};
        const float bias[2] = {__half2float(__ushort_as_half(bias_bits[0])), __half2float(__ushort_as_half(bias_bits[1]))};
        const uint32_t staging = smem_base + (uint32_t)(own_blocks * ranks) * BLOCK_BYTES;
        unsigned char *staging_gen = smem_gen + own_blocks * ranks * BLOCK_BYTES;
        // SLOTS blocks side by side: their residuals are on their way together, and the sums of one fill the waits of another.
        static_assert(CONV_WARPS == 8, "a warp finishes its columns of every block");
        constexpr int SLOTS = 2;
        const bool odd = g & 1;
        for (int slot0 = 0; slot0 < own_blocks; slot0 += SLOTS) {
            float r[SLOTS][2][2];  // [column half][row], or [row] in the first half with pairs
            if (FUSED && res != nullptr) {
#pragma unroll
                for (int i = 0; i < SLOTS; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int n = pairs ? out_n0 + 8 * cw + (odd ? 4 : 0) + (g >> 1) : n0 + 16 * cw + 8 * e + g, m = m0 + ((slot0 + i) * ranks + rank) * 8 + 2 * tq + k;
                            r[i][e][k] = 0.0f;
                            if (n < out_n && m < p.M && slot0 + i < own_blocks && !(pairs && e == 1)) r[i][e][k] = __half2float(__ldcg(res + (size_t)m * p.ep.ldr + n));
                        }
            }
            float4 sum[SLOTS];
#pragma unroll
            for (int i = 0; i < SLOTS; ++i)
                if (slot0 + i < own_blocks) sum[i] = reinterpret_cast<const float4 *>(smem_gen + (size_t)(slot0 + i) * ranks * BLOCK_BYTES)[cw * 32 + lane];
            for (int k = 1; k < ranks; ++k) {
#pragma unroll
                for (int i = 0; i < SLOTS; ++i)
                    if (slot0 + i < own_blocks) {
                        const float4 x = reinterpret_cast<const float4 *>(smem_gen + ((size_t)(slot0 + i) * ranks + k) * BLOCK_BYTES)[cw * 32 + lane];
                        sum[i].x += x.x, sum[i].y += x.y, sum[i].z += x.z, sum[i].w += x.w;
                    }
            }
#pragma unroll
            for (int i = 0; i < SLOTS; ++i) {
                if (slot0 + i >= own_blocks) break;
                float y[2][2] = {{sum[i].x * sc[0], sum[i].y * sc[0]}, {sum[i].z * sc[1], sum[i].w * sc[1]}};  // [column half][row]
                if (FUSED) {
#pragma unroll
                    for (int e = 0; e < 2; ++e) y[e][0] += bias[e], y[e][1] += bias[e];
                }
                const uint32_t row = staging + (uint32_t)((slot0 + i) * 8 + (lane & 7)) * ROW_BYTES;
                if (pairs) {
                    // Lanes with even g hold gates, the lanes with g + 1 what they multiply; of the two 8-column halves each lane of
                    // such a pair finishes one, for its two rows.
                    float z[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float other = __shfl_xor_sync(0xffffffffu, odd ? y[0][k] : y[1][k], 4);
                        z[k] = silu(odd ? other : y[0][k]) * (odd ? y[1][k] : other);
                        if (res != nullptr) z[k] += r[i][0][k];
                    }
                    const __half2 z2 = __floats2half2_rn(z[0], z[1]);
                    umma::stmatrix_x1_trans(row + 16 * cw, *reinterpret_cast<const uint32_t *>(&z2));
                } else {
                    uint32_t pk[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        if (FUSED && res != nullptr) y[e][0] += r[i][e][0], y[e][1] += r[i][e][1];
                        const __half2 y2 = __floats2half2_rn(y[e][0], y[e][1]);
                        pk[e] = *reinterpret_cast<const uint32_t *>(&y2);
                    }
                    umma::stmatrix_x2_trans(row + (16 * cw + 8 * ((lane >> 3) & 1)) * 2, pk);
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(CONV_THREADS) : "memory");
        // whole rows out: 16 (8 with pairs) pieces of 16 bytes each
        const int log2_chunks = pairs ? 3 : 4;
        for (int idx = threadIdx.x; idx < (own_blocks * 8) << log2_chunks; idx += CONV_THREADS) {
            const int r = idx >> log2_chunks, chunk = idx & ((1 << log2_chunks) - 1);
            const int m = m0 + ((r >> 3) * ranks + rank) * 8 + (r & 7), col = out_n0 + chunk * 8;
            if (m >= p.M || col >= out_n) continue;
            uint4 val = *reinterpret_cast<const uint4 *>(staging_gen + r * ROW_BYTES + chunk * 16);
            if (pairs) {  // columns stand in the order 0 4 1 5 2 6 3 7
                val = make_uint4(__byte_perm(val.x, val.y, 0x5410), __byte_perm(val.z, val.w, 0x5410), __byte_perm(val.x, val.y, 0x7632),
                                 __byte_perm(val.z, val.w, 0x7632));
            }
            const size_t off = (size_t)m * p.out.ldc + p.out.col0 + col;
#pragma unroll 1
            for (int d = 0; d < p.out.count; ++d) *reinterpret_cast<uint4 *>(static_cast<__half *>(p.out.ptr[d]) + off) = val;
        }
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        umma::fence_after_sync();
        umma::dealloc(tmem_base, TMEM_COLS);
    }
}

static int allow_smem(int dev) {
    static std::atomic<bool> attr_set[64];  // per device, zero-initialised; a repeated set by a racing thread is harmless
    if (dev >= 0 && dev < 64 && attr_set[dev].load(std::memory_order_acquire)) return B200Q_OK;
    B200Q_CUDA_TRY(cudaFuncSetAttribute(qlinear_mid_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, CTA_SMEM));
    B200Q_CUDA_TRY(cudaFuncSetAttribute(qlinear_mid_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, CTA_SMEM));
    B200Q_CUDA_TRY(cudaFuncSetAttribute(qlinear_mid_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, CTA_SMEM));
    if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    return B200Q_OK;
}

}  // namespace mid

// The runtime's occupancy query counts one CTA per SM for kernels that allocate tensor memory; two run (measured: the time of a
// launch steps up beyond these counts and not before).  Clusters of c CTAs with two on an SM are clusters of c / 2 SMs, so
// for an even c the query for c / 2 counts them; for an odd one twice what it counts for c is less than what fits.
int mid_resident_ctas(int tm, int cluster) {
    using namespace mid;
    static std::atomic<int> known[64][9][9];  // per device, tm / 16 and cluster; a repeated look-up by a racing thread is harmless
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 2 * 148 - 32;
    }
    std::atomic<int> &slot = known[dev][tm / 16][cluster];
    int n = slot.load(std::memory_order_relaxed);
    if (n != 0) return n;
    if (allow_smem(dev) != B200Q_OK) return 2 * 148 - 32;
    const int half = cluster % 2 == 0 ? cluster / 2 : cluster;
    n = resident_clusters(reinterpret_cast<const void *>(qlinear_mid_kernel<true, false>), THREADS, smem_of(tm, cluster), half) * (cluster % 2 == 0 ? cluster : 2 * cluster);
    if (n == 0) return 2 * 148 - 32;
    slot.store(n, std::memory_order_relaxed);
    return n;
}

int launch_mid(const void *a, const void *wq, const void *scale, const OutTargets &out, int64_t M, int64_t N, int64_t K, cudaStream_t stream,
               const Epilogue *epilogue, bool weight_nk, int64_t lda, int tm, int cluster) {
    using namespace mid;
    CUtensorMap map_w, map_a;
    int rc = weight_nk ? make_tensor_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, wq, (uint64_t)K, (uint64_t)N, (uint64_t)K, BK, TN,
                                            CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)
                       : make_tensor_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, wq, (uint64_t)N, (uint64_t)K, (uint64_t)N, TN, BK,
                                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200Q_OK) return rc;
    rc = make_tensor_map_2d(&map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, (uint32_t)tm,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200Q_OK) return rc;
    Params p = {};
    p.scale = static_cast<const __half *>(scale);
    p.out = out;
    if (epilogue != nullptr) p.ep = *epilogue;
    p.status = device_status_word();
    p.M = (int)M;
    p.N = (int)N;
    p.tm = tm;
    p.k_blocks = (int)ceil_div(K, BK);
    p.act_slots = act_slots_of(tm);
    const int64_t n_tiles = ceil_div(N, TN), m_tiles = ceil_div(M, tm);
    if (m_tiles > 65535) return set_error(B200Q_UNSUPPORTED, "qlinear: M=%lld is too large for the mid-M kernel", (long long)M);
    const bool fused = p.ep.bias != nullptr || p.ep.residual != nullptr || p.ep.act != kActNone;
    if (weight_nk && fused) return set_error(B200Q_UNSUPPORTED, "qlinear: the fused epilogue is served for [K, N] weights");
    const void *kernel = weight_nk ? reinterpret_cast<const void *>(qlinear_mid_kernel<false, true>)
                                   : (fused ? reinterpret_cast<const void *>(qlinear_mid_kernel<true, false>) : reinterpret_cast<const void *>(qlinear_mid_kernel<false, false>));
    int dev = 0;
    B200Q_CUDA_TRY(cudaGetDevice(&dev));
    rc = allow_smem(dev);
    if (rc != B200Q_OK) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_tiles, (unsigned)cluster, (unsigned)m_tiles);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem_of(tm, cluster);
    cfg.stream = stream;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = 1;
    attrs[0].val.clusterDim.y = (unsigned)cluster;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 2;
    void *args[3] = {&map_w, &map_a, &p};
    B200Q_CUDA_TRY(cudaLaunchKernelExC(&cfg, kernel, args));
    return B200Q_OK;
}

}  // namespace b200q
