// Large-M (prefill) f16 x int8 quantized linear on pairs of SMs: tcgen05.mma with cta_group::2, the converted weight in
// tensor memory.
//
// The product is computed transposed, D[n, m] = sum_k W[k, n] * A[m, k].  A cluster of two CTAs owns a tile of 256 weight
// columns x TM activation rows (TM a multiple of 32, at most 256): each CTA converts its own 128 columns and keeps the f16
// image in its tensor memory, where the tensor core takes its first operand from; of the activations each CTA fetches
// half of the rows and the pair's MMA reads both halves.  Shared memory then carries, per 64-k stage and CTA, 8 KB of
// int8 in and out and TM / 2 rows of activations in and out: 48 KB at TM = 256, for 512 clocks of MMA.  The single-SM form
// (qlinear_prefill.cu) writes and reads the f16 weight there too and fetches every activation row itself: 112 KB.
//
// One persistent CTA per SM, nineteen warps:
//   warps 0-3, 15-18 epilogue, two groups that take the 32-row blocks of a tile in turn: tensor memory -> scale, bias, gate / up pairing, residual -> f16, transposed through a staging
//               buffer (two per group, taken in turn) by matrix stores, 16-byte stores of whole output rows.  (One group:
//               (512, 4096, 22016) with SiLU 109 us for 87 in tiles of 256 rows, (1000, 4096, 4096) with a residual 37.6 for
//               31.7, (2048, 256, 28672) 58.7 for 45.7.)
//   warps 4-11  converters, two groups that take stages in turn: int8 tile -> registers by matrix loads (transposing ones for
//               [K, N] weights) that leave a lane four consecutive k of one column, int8 -> exact f16, tcgen05.st.  The
//               fragment of the loads is the fragment of the 16x256b store, so nothing is exchanged between lanes.
//   warp 12     TMA producer of the int8 tiles
//   warp 13     TMA producer of the activation tiles
//   warp 14     MMA issuer (first CTA of the pair only): one thread for the whole loop, one barrier a stage: each CTA's converters
//               tell it that their weight tile is in tensor memory and that their CTA's activations have landed (arrivals on
//               the first CTA's barriers that carry no stores with them: see mbar_arrive_remote)
//
// Every wait is bounded, as in qlinear_prefill.cu: a wait that runs out records where and raises a CTA-wide flag, all roles
// leave, the producers wait for the copies they armed, the MMA thread for what it issued, and the two CTAs meet at a cluster
// barrier before either gives back tensor memory or retires.
#include <atomic>

#include "common.cuh"
#include "qlinear.h"
#include "umma.cuh"

namespace b200q {
namespace pair {

constexpr int TN = 128;                      // weight columns per CTA; a pair's tile has twice as many
constexpr int BK = 64;                       // k per stage = four MMAs of K = 16
constexpr int RAW_BYTES = BK * TN;           // int8 tile of one CTA
constexpr int RAW_SLOTS = 10;                // 80 KB in flight
constexpr int ACT_RING_BYTES = 96 * 1024;    // halves of activation tiles: as many slots as fit, at most MAX_SLOTS
constexpr int MAX_SLOTS = 12;
constexpr int MAX_W_SLOTS = 8;               // converted weight tiles in tensor memory, 32 columns each, behind the accumulators
constexpr int TMEM_COLS = 512;
constexpr int CONV_WARPS = 8, CONV_GROUPS = 2, GROUP_WARPS = CONV_WARPS / CONV_GROUPS;
constexpr int CONV_WARP0 = 4, RAW_WARP = 12, ACT_WARP = 13, MMA_WARP = 14;
constexpr int EPI_GROUPS = 2, EPI_WARP1 = 15;
constexpr int THREADS = 32 * 19;
constexpr int ROW_BYTES = TN * 2 + 16;       // one output row in the staging buffer, padded: matrix stores touch every bank once
constexpr int STAGING_BYTES = 32 * ROW_BYTES;
constexpr int SMEM_BYTES = ACT_RING_BYTES + RAW_SLOTS * RAW_BYTES + EPI_GROUPS * 2 * STAGING_BYTES + 1024;  // + alignment slack

// A parity wait tells a phase only from its neighbours, so a waiter has to see every phase of its barriers: stage i belongs
// to converter group i % CONV_GROUPS, and every ring's length is a multiple of CONV_GROUPS, so that a slot stays with one group.
static_assert(RAW_SLOTS % CONV_GROUPS == 0, "slots must not change groups");

struct Params {
    const __half *scale;
    OutTargets out;            // [M, N], or [M, N / 2] with the gate / up pairing; not a multicast address
    Epilogue ep;
    unsigned int *status;
    int M, N;
    int tm;                    // activation rows per tile
    int n_tiles, m_tiles;
    int band;                  // row tiles that are walked together, column tile by column tile
    int k_blocks;
    int n_acc;                 // accumulators of tm columns in tensor memory: two where four weight slots still fit beside them
    int act_slots, w_slots;    // ring lengths, even
    int residual_vec;          // residual rows can be read as 16-byte vectors
};

// Tile u of the grid's work.  Within a band of row tiles the row tile runs fastest, so that the pairs that work at the same
// time share weight tiles, and a band's activations stay in L2.
__device__ __forceinline__ void tile_of(const Params &p, int u, int &n0, int &m0) {
    const int band_tiles = p.band * p.n_tiles;
    const int b = u / band_tiles, r = u - b * band_tiles;
    const int rows = min(p.band, p.m_tiles - b * p.band);
    const int n = r / rows;
    n0 = n * 2 * TN;
    m0 = (b * p.band + (r - n * rows)) * p.tm;
}

// NK: the weight is [N, K] with K contiguous.
template <bool FUSED, bool NK>
__global__ void __launch_bounds__(THREADS, 1) __cluster_dims__(2, 1, 1)
    qlinear_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const Params p) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t raw_full[RAW_SLOTS];    // an int8 tile has landed
    __shared__ __align__(8) uint64_t raw_empty[RAW_SLOTS];   // its converter group has read it
    __shared__ __align__(8) uint64_t act_full[MAX_SLOTS];    // this CTA's half of an activation tile has landed
    __shared__ __align__(8) uint64_t act_empty[MAX_SLOTS];   // the MMAs that read it have completed
    __shared__ __align__(8) uint64_t ready[MAX_W_SLOTS];     // (first CTA) both CTAs have the stage's operands in place
    __shared__ __align__(8) uint64_t done[MAX_W_SLOTS];      // the MMAs that read the weight slot have completed
    __shared__ __align__(8) uint64_t acc_full[2];            // an accumulator holds a finished tile
    __shared__ __align__(8) uint64_t acc_empty[2];           // (first CTA) both CTAs' epilogue warps have read it out
    __shared__ __align__(8) uint64_t drain_bar;              // every MMA issued has completed (teardown)
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const uint32_t smem_base = (smem_u32(smem_dyn) + 1023u) & ~1023u;  // swizzled operands; the same in both CTAs
    unsigned char *smem_gen = smem_dyn + (smem_base - smem_u32(smem_dyn));
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int units = p.n_tiles * p.m_tiles;
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
    const uint32_t n_acc = p.n_acc, act_slots = p.act_slots, w_slots = p.w_slots;
    const uint32_t act_bytes = (uint32_t)(p.tm / 2 * BK * 2), w_col0 = n_acc * p.tm;
    constexpr int RAW_OFF = ACT_RING_BYTES, STAGING_OFF = RAW_OFF + RAW_SLOTS * RAW_BYTES;

    if (threadIdx.x == 0) {
        for (int r = 0; r < RAW_SLOTS; ++r) {
            mbar_init(smem_u32(&raw_full[r]), 1);
            mbar_init(smem_u32(&raw_empty[r]), GROUP_WARPS);
        }
        for (int s = 0; s < MAX_SLOTS; ++s) {
            mbar_init(smem_u32(&act_full[s]), 1);
            mbar_init(smem_u32(&act_empty[s]), 1);
        }
        for (int w = 0; w < MAX_W_SLOTS; ++w) {
            mbar_init(smem_u32(&ready[w]), 2 * GROUP_WARPS);
            mbar_init(smem_u32(&done[w]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), 2 * 4 * EPI_GROUPS);
        }
        mbar_init(smem_u32(&drain_bar), 1);
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == MMA_WARP) {
        umma::alloc_pair(smem_u32(&tmem_base_slot), TMEM_COLS);
        umma::relinquish_pair();
    }
    umma::fence_before_sync();
    __syncthreads();
    cluster_arrive_release();
    cluster_wait_acquire();  // both CTAs' barriers are set up and both have their tensor memory
    umma::fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;
    if (lane == 0 && (warp == RAW_WARP || warp == ACT_WARP)) tma_prefetch_desc(warp == RAW_WARP ? &map_w : &map_a);
    pdl_wait();  // every role: none of the bounded waits below runs against the kernel in front

    // Bounded wait of a whole warp (true in all lanes or false in all lanes) / of one thread.
    auto wait = [&](uint32_t bar, uint32_t parity, unsigned int site) -> bool {
        bool ok = mbar_wait(bar, parity, umma::kFastPolls);
        if (__all_sync(0xffffffffu, ok)) return true;
        if (!ok) ok = umma::wait_or_abort<kKernelPair>(bar, parity, site, &abort_flag, p.status);
        return __all_sync(0xffffffffu, ok);
    };
    auto wait_one = [&](uint32_t bar, uint32_t parity, unsigned int site) -> bool {
        return mbar_wait(bar, parity, umma::kFastPolls) || umma::wait_or_abort<kKernelPair>(bar, parity, site, &abort_flag, p.status);
    };

    if (warp == RAW_WARP) {
        // ---------------- TMA producer: int8 weight tiles ----------------
        pdl_launch_dependents();  // tensor memory is allocated: a kernel that is placed as this one's CTAs leave cannot take it away
        if (lane == 0) {
            uint32_t i = 0;
            umma::Ring r;
            bool ok = true;
            for (int u = first; u < units && ok; u += step) {
                int n, m0;
                tile_of(p, u, n, m0);
                n += (int)rank * TN;
                for (int kb = 0; kb < p.k_blocks; ++kb, ++i, r.advance(1, RAW_SLOTS)) {
                    if (i >= (uint32_t)RAW_SLOTS && !wait_one(smem_u32(&raw_empty[r.slot]), r.phase ^ 1u, 1)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&raw_full[r.slot]);
                    mbar_expect_tx(bar, RAW_BYTES);
                    tma_load_2d(smem_base + RAW_OFF + r.slot * RAW_BYTES, &map_w, NK ? kb * BK : n, NK ? n : kb * BK, bar);
                }
            }
            // Teardown: every copy armed must have landed before the CTA may retire.  Slot s was last used for the largest
            // j < i with j % RAW_SLOTS == s.
            for (uint32_t s = 0; s < (uint32_t)RAW_SLOTS; ++s) {
                if (i <= s) continue;
                const uint32_t j = i - 1 - (i - 1 - s) % RAW_SLOTS;
                if (!mbar_wait(smem_u32(&raw_full[s]), (j / RAW_SLOTS) & 1)) report_timeout(p.status, kKernelPair, 7);
            }
        }
    } else if (warp == ACT_WARP) {
        // ---------------- TMA producer: this CTA's half of the activation tiles ----------------
        if (lane == 0) {
            const uint64_t keep = l2_policy_evict_last();  // every column tile reads them again
            uint32_t i = 0;
            umma::Ring r;
            bool ok = true;
            for (int u = first; u < units && ok; u += step) {
                int n0, m;
                tile_of(p, u, n0, m);
                m += (int)rank * (p.tm / 2);
                for (int kb = 0; kb < p.k_blocks; ++kb, ++i, r.advance(1, act_slots)) {
                    if (i >= act_slots && !wait_one(smem_u32(&act_empty[r.slot]), r.phase ^ 1u, 2)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&act_full[r.slot]);
                    mbar_expect_tx(bar, act_bytes);
                    tma_load_2d_hint(smem_base + r.slot * act_bytes, &map_a, kb * BK, m, bar, keep);
                }
            }
            for (uint32_t s = 0; s < act_slots; ++s) {
                if (i <= s) continue;
                const uint32_t j = i - 1 - (i - 1 - s) % act_slots;
                if (!mbar_wait(smem_u32(&act_full[s]), (j / act_slots) & 1)) report_timeout(p.status, kKernelPair, 7);
            }
        }
    } else if (warp == MMA_WARP) {
        // ---------------- MMA issuer ----------------
        // The election stands outside the loop: inside it the four MMAs and the commit of a stage take 260 clocks to issue, here
        // 47.  The next stage's barrier is asked while this one's MMAs are on their way.
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = umma::instr_desc_f16(2 * TN, p.tm);
            uint32_t t_iter = 0;
            umma::Ring ra, rw;
            bool ok = true, here = false;
            for (int u = first; u < units && ok; u += step, ++t_iter) {
                const uint32_t buf = n_acc == 2 ? (t_iter & 1) : 0, acc_use = n_acc == 2 ? (t_iter >> 1) : t_iter;
                if (acc_use >= 1 && !wait_one(smem_u32(&acc_empty[buf]), (acc_use - 1) & 1, 3)) break;
                umma::fence_after_sync();
                const uint32_t d_addr = tmem_base + buf * p.tm;
                for (int kb = 0; kb < p.k_blocks; ++kb) {
                    if (!here && !wait_one(smem_u32(&ready[rw.slot]), rw.phase, 4)) {
                        ok = false;
                        break;
                    }
                    umma::fence_after_sync();
                    const uint32_t a_addr = tmem_base + w_col0 + 32 * rw.slot;
                    // K-major activations, 8-row groups 1024 B apart; K = 16 is 32 bytes along the swizzled row
                    const uint64_t b_desc = umma::smem_desc_sw128(smem_base + ra.slot * act_bytes);
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks)
                        umma::mma_pair_ts(d_addr, a_addr + 8 * ks, b_desc + 2 * ks, idesc, (kb > 0 || ks > 0) ? 1u : 0u);
                    umma::commit_pair(smem_u32(&done[rw.slot]));
                    umma::commit_pair(smem_u32(&act_empty[ra.slot]));
                    ra.advance(1, act_slots), rw.advance(1, w_slots);
                    here = mbar_test(smem_u32(&ready[rw.slot]), rw.phase);
                }
                if (ok) umma::commit_pair(smem_u32(&acc_full[buf]));
            }
            // Teardown: no MMA may still be running when tensor memory is given back or the peer retires.
            umma::commit_pair_self(smem_u32(&drain_bar));
            if (!mbar_wait(smem_u32(&drain_bar), 0)) report_timeout(p.status, kKernelPair, 8);
        }
    } else if (warp >= CONV_WARP0 && warp < RAW_WARP) {
        // ---------------- converters ----------------
        const int cw = warp - CONV_WARP0;
        const int group = cw / GROUP_WARPS;   // converts stages group, group + CONV_GROUPS, ...
        const int q = warp & 3;               // 32 columns of the tile = the tensor-memory lanes this warp may write
        const uint32_t w_lane = tmem_base + ((uint32_t)(32 * q) << 16) + w_col0;
        const uint32_t ready0 = map_to_rank(smem_u32(&ready[0]), 0);
        // where this lane's matrix-load rows lie in a tile
        //   [K, N]: rows of 128 columns, 128B swizzle; lanes 0-15 / 16-31 address the first / second 16-column block
        //   [N, K]: rows of 64 k, 64B swizzle; lane = row, 16-byte chunk = 16 k
        const uint32_t kn_off = (uint32_t)(lane & 15) * 128u + (((uint32_t)(2 * q + (lane >> 4)) ^ (uint32_t)(lane & 7)) << 4);
        const uint32_t nk_row = (uint32_t)(32 * q + lane);
        const uint32_t nk_off = nk_row * 64u, nk_sw = (nk_row >> 1) & 3u;
        const int my_units = units > first ? (units - first + step - 1) / step : 0;
        const uint32_t stages = (uint32_t)my_units * (uint32_t)p.k_blocks;
        umma::Ring rr, ra, rw;
        rr.slot = ra.slot = rw.slot = (uint32_t)group;
        bool raw_ok = false;
        for (uint32_t i = group; i < stages; i += CONV_GROUPS, ra.advance(CONV_GROUPS, act_slots), rw.advance(CONV_GROUPS, w_slots)) {
            if (!raw_ok && !wait(smem_u32(&raw_full[rr.slot]), rr.phase, 5)) break;
            const uint32_t raw = smem_base + RAW_OFF + rr.slot * RAW_BYTES, read_bar = smem_u32(&raw_empty[rr.slot]);
            uint32_t v[4][4];  // [k block of 16][column block of 8]: four consecutive k of one column
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                if (NK) umma::ldmatrix_x4(v[ks], raw + nk_off + (((uint32_t)ks ^ nk_sw) << 4));
                else umma::ldmatrix_x2_trans_b8(v[ks], raw + ks * 16 * 128 + kn_off);
            }
            // Asked for here, looked at after the conversion: the next tile, the weight slot's last readers and, by one warp of the
            // group, which answers for them, the activations.
            rr.advance(CONV_GROUPS, RAW_SLOTS);
            const bool t_raw = i + CONV_GROUPS < stages && mbar_test(smem_u32(&raw_full[rr.slot]), rr.phase);
            const bool t_done = i < w_slots || mbar_test(smem_u32(&done[rw.slot]), rw.phase ^ 1u);
            const bool t_act = q != 0 || mbar_test(smem_u32(&act_full[ra.slot]), ra.phase);
            uint32_t h[2][16];
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
#pragma unroll
                for (int b = 0; b < 4; ++b) umma::cvt_s8x4_to_f16_pairs(v[ks][b], h[b >> 1][4 * ks + 2 * (b & 1)], h[b >> 1][4 * ks + 2 * (b & 1) + 1]);
            __syncwarp();
            if (lane == 0) mbar_arrive(read_bar);  // the int8 tile is in registers
            raw_ok = __all_sync(0xffffffffu, t_raw);
            if (!__all_sync(0xffffffffu, t_done) && !wait(smem_u32(&done[rw.slot]), rw.phase ^ 1u, 6)) break;
            umma::fence_after_sync();
            umma::st_16x256b_x4(w_lane + 32 * rw.slot, h[0]);
            umma::st_16x256b_x4(w_lane + (16u << 16) + 32 * rw.slot, h[1]);
            umma::st_wait();
            umma::fence_before_sync();
            if (!__all_sync(0xffffffffu, t_act) && !wait(smem_u32(&act_full[ra.slot]), ra.phase, 9)) break;
            __syncwarp();
            // What the MMA reads behind this arrival is the weight in this CTA's tensor memory, stored (st_wait) and fenced above, and the
            // activations that the copy engine put into this CTA's shared memory, complete before the phase that was waited for: no
            // store of this warp is among it, so the arrival needs no wider scope.
            if (lane == 0) mbar_arrive_remote(ready0 + 8 * rw.slot);
        }
    } else {
        // ---------------- epilogue ----------------
        const int eg = warp >= EPI_WARP1 ? 1 : 0;  // takes blocks eg, eg + EPI_GROUPS, ...
        const int q = warp & 3;                 // tensor-memory lanes 32 q .. 32 q + 31
        const int et = 32 * q + lane;           // 0 .. 127
        auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + eg) : "memory"); };
        const int g = lane >> 2, tq = lane & 3; // fragment coordinates: column g of an 8-column block, rows 2 tq, 2 tq + 1 of an 8-row block
        const bool pairs = FUSED && p.ep.act == kActSiluMul;  // columns (2j, 2j + 1) = (gate, up)
        const __half *res = FUSED ? static_cast<const __half *>(p.ep.residual) : nullptr;
        const bool res_vec = FUSED && !pairs && p.residual_vec;
        const int out_n = pairs ? p.N >> 1 : p.N;
        const int row_chunks_log2 = pairs ? 3 : 4;             // 16-byte pieces of a tile's output row
        const int chunk = et & ((1 << row_chunks_log2) - 1);
        const int row_in_pass = et >> row_chunks_log2;
        const int pass_rows = 128 >> row_chunks_log2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * q) << 16);
        uint32_t t_iter = 0, block = 0;         // block: the group's 32-row blocks so far, staging buffers in turn
        for (int u = first; u < units; u += step, ++t_iter) {
            int n0, m0;
            tile_of(p, u, n0, m0);
            n0 += (int)rank * TN;
            const uint32_t buf = n_acc == 2 ? (t_iter & 1) : 0, acc_use = n_acc == 2 ? (t_iter >> 1) : t_iter;
            const int m_left = min(p.M - m0, p.tm);
            const int blocks = (m_left + 31) / 32;
            const uint32_t acc = lane_addr + buf * p.tm;
            float sc[2][2], bias[2][2];  // [16-column block][8-column half]: column 16 h + 8 e + g of this warp's 32
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int n = n0 + 32 * q + 16 * h + 8 * e + g;
                    sc[h][e] = n < p.N ? __half2float(__ldcg(p.scale + n)) : 0.0f;
                    bias[h][e] = (FUSED && n < p.N && p.ep.bias != nullptr) ? __half2float(__ldcg(static_cast<const __half *>(p.ep.bias) + n)) : 0.0f;
                }
            if (!all_of_128(1 + eg, wait(smem_u32(&acc_full[buf]), acc_use & 1, 10))) break;  // the group stays or leaves as one
            umma::fence_after_sync();
            const int out_n0 = pairs ? n0 >> 1 : n0;
            const bool cols_ok = out_n0 + chunk * 8 < out_n;  // widths are multiples of 8: eight columns are in or out together
            const size_t out_off = (size_t)m0 * p.out.ldc + p.out.col0 + out_n0 + chunk * 8;
            if (eg >= blocks) {  // a tile of a single block: nothing for this group
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(map_to_rank(smem_u32(&acc_empty[buf]), 0));
            }
#pragma unroll 1
            for (int cb = eg; cb < blocks; cb += EPI_GROUPS, ++block) {
                unsigned char *staging = smem_gen + STAGING_OFF + (2 * eg + (block & 1)) * STAGING_BYTES;
                const uint32_t staging_a = smem_base + STAGING_OFF + (2 * eg + (block & 1)) * STAGING_BYTES;
                if (res_vec && res != nullptr) {
                    // the residual's block goes through the staging buffer into the fragments' layout
#pragma unroll
                    for (int pass = 0; pass < 4; ++pass) {
                        const int r = pass * 8 + row_in_pass, m = cb * 32 + r;
                        uint4 val = make_uint4(0, 0, 0, 0);
                        if (m < m_left && cols_ok) val = __ldcg(reinterpret_cast<const uint4 *>(res + (size_t)(m0 + m) * p.ep.ldr + out_n0 + chunk * 8));
                        *reinterpret_cast<uint4 *>(staging + r * ROW_BYTES + chunk * 16) = val;
                    }
                    group_sync();
                }
                uint32_t v[2][16];
                umma::ld_16x256b_x4(acc + cb * 32, v[0]);
                umma::ld_16x256b_x4(acc + (16u << 16) + cb * 32, v[1]);
                umma::ld_wait();
                if (cb + EPI_GROUPS >= blocks) {  // the group's part of the accumulator is in registers
                    umma::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(map_to_rank(smem_u32(&acc_empty[buf]), 0));
                }
                // v[h][4 j + 2 e + i]: column 16 h + 8 e + g, row 8 j + 2 tq + i
                if (pairs) {
                    // Lanes with even g hold gates, the lanes with g + 1 what they multiply; of the two 8-column halves each
                    // lane of such a pair finishes one, for its two rows.
                    const bool odd = g & 1;
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        // Eight results side by side, and no branch between them: one after the other, with the residual's test in each, a
                        // block of 32 rows took 1.45 us for 0.9.
                        float z[2][2][2];  // [row block j, j + 1][column block h][row]
#pragma unroll
                        for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                            for (int h = 0; h < 2; ++h)
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    float y0 = __uint_as_float(v[h][4 * (j + jj) + i]) * sc[h][0], y1 = __uint_as_float(v[h][4 * (j + jj) + 2 + i]) * sc[h][1];
                                    y0 += bias[h][0];
                                    y1 += bias[h][1];
                                    const float other = __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 4);
                                    z[jj][h][i] = silu(odd ? other : y0) * (odd ? y1 : other);
                                }
                        if (res != nullptr) {
#pragma unroll
                            for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                                for (int h = 0; h < 2; ++h)
#pragma unroll
                                    for (int i = 0; i < 2; ++i) {
                                        const int oc = out_n0 + 16 * q + 8 * h + (odd ? 4 : 0) + (g >> 1), m = cb * 32 + 8 * (j + jj) + 2 * tq + i;
                                        if (oc < out_n && m < m_left) z[jj][h][i] += __half2float(__ldcg(res + (size_t)(m0 + m) * p.ep.ldr + oc));
                                    }
                        }
                        uint32_t pk[4];
#pragma unroll
                        for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const __half2 z2 = __floats2half2_rn(z[jj][h][0], z[jj][h][1]);
                                pk[2 * jj + h] = *reinterpret_cast<const uint32_t *>(&z2);
                            }
                        // result column g / 2 (even g) or 4 + g / 2 (odd g) of each 8: stored in the order of g, put right on the way out
                        const int mi = lane >> 3;
                        umma::stmatrix_x4_trans(staging_a + (8 * (j + (mi >> 1)) + (lane & 7)) * ROW_BYTES + (16 * q + 8 * (mi & 1)) * 2, pk);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t place = staging_a + (8 * j + (lane & 7)) * ROW_BYTES + (32 * q + 8 * (lane >> 3)) * 2;
                        uint32_t rs[4] = {0u, 0u, 0u, 0u}, pk[4];
                        if (res_vec && res != nullptr) umma::ldmatrix_x4_trans(rs, place);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                float y[2];
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    y[i] = __uint_as_float(v[h][4 * j + 2 * e + i]) * sc[h][e];
                                    if (FUSED) y[i] += bias[h][e];
                                }
                                if (FUSED && res != nullptr) {
                                    if (res_vec) {
                                        const float2 r2 = __half22float2(*reinterpret_cast<const __half2 *>(&rs[2 * h + e]));
                                        y[0] += r2.x;
                                        y[1] += r2.y;
                                    } else {
                                        const int n = n0 + 32 * q + 16 * h + 8 * e + g;
#pragma unroll
                                        for (int i = 0; i < 2; ++i) {
                                            const int m = cb * 32 + 8 * j + 2 * tq + i;
                                            if (n < p.N && m < m_left) y[i] += __half2float(__ldcg(res + (size_t)(m0 + m) * p.ep.ldr + n));
                                        }
                                    }
                                }
                                const __half2 y2 = __floats2half2_rn(y[0], y[1]);
                                pk[2 * h + e] = *reinterpret_cast<const uint32_t *>(&y2);
                            }
                        umma::stmatrix_x4_trans(place, pk);
                    }
                }
                group_sync();  // the four warps: block complete; the other buffer is free
#pragma unroll 4
                for (int r = row_in_pass; r < 32; r += pass_rows) {
                    const int m = cb * 32 + r;
                    if (m < m_left && cols_ok) {
                        uint4 val = *reinterpret_cast<const uint4 *>(staging + r * ROW_BYTES + chunk * 16);
                        if (pairs) {  // columns stand in the order 0 4 1 5 2 6 3 7
                            val = make_uint4(__byte_perm(val.x, val.y, 0x5410), __byte_perm(val.z, val.w, 0x5410), __byte_perm(val.x, val.y, 0x7632),
                                             __byte_perm(val.z, val.w, 0x7632));
                        }
                        // this GPU's output and, for a column-parallel layer, the peer-mapped outputs of the other ranks
                        const size_t off = out_off + (size_t)m * p.out.ldc;
#pragma unroll 1
                        for (int d = 0; d < p.out.count; ++d) *reinterpret_cast<uint4 *>(static_cast<__half *>(p.out.ptr[d]) + off) = val;
                    }
                }
            }
        }
    }

    // ---------------- teardown: both CTAs are done with each other's shared and tensor memory ----------------
    __syncwarp();
    umma::fence_before_sync();
    cluster_arrive_release();
    cluster_wait_acquire();
    if (warp == MMA_WARP) {
        umma::fence_after_sync();
        umma::dealloc_pair(tmem_base, TMEM_COLS);
    }
}

}  // namespace pair

int launch_pair(const void *a, const void *wq, const void *scale, const OutTargets &out, int64_t M, int64_t N, int64_t K, cudaStream_t stream,
                const Epilogue *epilogue, bool weight_nk, int64_t lda, int tm) {
    using namespace pair;
    CUtensorMap map_w, map_a;
    int rc = weight_nk ? make_tensor_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, wq, (uint64_t)K, (uint64_t)N, (uint64_t)K, BK, TN,
                                            CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)
                       : make_tensor_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, wq, (uint64_t)N, (uint64_t)K, (uint64_t)N, TN, BK,
                                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200Q_OK) return rc;
    rc = make_tensor_map_2d(&map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, (uint32_t)(tm / 2),
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200Q_OK) return rc;

    Params p = {};
    p.scale = static_cast<const __half *>(scale);
    p.out = out;
    if (epilogue != nullptr) p.ep = *epilogue;
    p.residual_vec = p.ep.residual != nullptr && p.ep.ldr % 8 == 0 && (reinterpret_cast<uintptr_t>(p.ep.residual) & 15u) == 0;
    p.status = device_status_word();
    p.M = (int)M;
    p.N = (int)N;
    p.tm = tm;
    p.n_tiles = (int)ceil_div(N, 2 * TN);
    p.m_tiles = (int)ceil_div(M, tm);
    // as many row tiles in a band as leave the band's activations well inside L2
    int64_t band = ((int64_t)48 << 20) / ((int64_t)tm * K * 2);
    if (band < 1) band = 1;
    p.band = (int)(band < p.m_tiles ? band : p.m_tiles);
    p.k_blocks = (int)ceil_div(K, BK);
    p.n_acc = 2 * tm + 4 * 32 <= TMEM_COLS ? 2 : 1;
    const int w_slots = (TMEM_COLS - p.n_acc * tm) / 32, act_slots = ACT_RING_BYTES / (tm / 2 * BK * 2);
    p.w_slots = (w_slots < MAX_W_SLOTS ? w_slots : MAX_W_SLOTS) & ~1;
    p.act_slots = (act_slots < MAX_SLOTS ? act_slots : MAX_SLOTS) & ~1;
    const int64_t units = (int64_t)p.n_tiles * p.m_tiles;
    if (units * 2 > 2147483647LL) return set_error(B200Q_UNSUPPORTED, "qlinear: problem too large for the tile counter");
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    const int64_t pairs_at_once = sms / 2;
    const unsigned grid = 2u * (unsigned)(units < pairs_at_once ? units : pairs_at_once);

    const bool fused = p.ep.bias != nullptr || p.ep.residual != nullptr || p.ep.act != kActNone;
    if (weight_nk && fused) return set_error(B200Q_UNSUPPORTED, "qlinear: the fused epilogue is served for [K, N] weights");
    const void *kernel = weight_nk ? reinterpret_cast<const void *>(qlinear_pair_kernel<false, true>)
                                   : (fused ? reinterpret_cast<const void *>(qlinear_pair_kernel<true, false>) : reinterpret_cast<const void *>(qlinear_pair_kernel<false, false>));
    static std::atomic<bool> attr_set[64];  // per device, zero-initialised; a repeated set by a racing thread is harmless
    int dev = 0;
    B200Q_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        B200Q_CUDA_TRY(cudaFuncSetAttribute(qlinear_pair_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        B200Q_CUDA_TRY(cudaFuncSetAttribute(qlinear_pair_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        B200Q_CUDA_TRY(cudaFuncSetAttribute(qlinear_pair_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 1;
    void *args[3] = {&map_w, &map_a, &p};
    B200Q_CUDA_TRY(cudaLaunchKernelExC(&cfg, kernel, args));
    return B200Q_OK;
}

}  // namespace b200q
