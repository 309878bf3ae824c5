// PTX wrappers of the tensor-memory kernels: tcgen05 (allocation, MMA, commit, loads and stores of tensor memory), the matrix
// loads and stores around them, and the int8 -> f16 conversion in the order those loads deliver.
#pragma once

#include "common.cuh"

namespace b200q {
namespace umma {

// ---- tensor memory: of one CTA, and of the two CTAs of a pair ----
__device__ __forceinline__ void alloc(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
}
__device__ __forceinline__ void relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void alloc_pair(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
}
__device__ __forceinline__ void relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- MMA ----
// Instruction descriptor, kind::f16: D = f32, A = B = f16, both K-major; N / 8 in bits 17..22, M / 16 in bits 24..28.
__device__ __forceinline__ uint32_t instr_desc_f16(int m, int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }
// Shared-memory descriptor of a K-major operand in rows of 128 swizzled bytes, 8-row groups 1024 bytes apart (addresses and
// offsets in 16-byte units, descriptor version 1, 128-byte swizzle).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3fffu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// D[tmem] (+)= A[tmem] * B[smem]; accumulate == 0 overwrites D.  _pair: over the two CTAs of a pair.
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_pair_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// One arrival on the barrier when every MMA issued so far by this thread has completed.  _pair: on the barrier at this place
// of both CTAs; _pair_self: of pair MMAs, in this CTA alone.
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void commit_pair_self(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---- tensor memory <-> registers ----
// 16 lanes x 32 columns; per 8 columns thread (g = lane / 4, t = lane % 4) holds, in four registers, columns 2t, 2t + 1 of
// lane g and then of lane g + 8.
__device__ __forceinline__ void ld_16x256b_x4(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void ld_16x256b_x1(uint32_t taddr, uint32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void st_16x256b_x4(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- matrix loads and stores ----
// Two 16 x 16 byte tiles, transposed on the way to registers.  Lanes 0-15 give the addresses of the 16 rows (16 bytes
// each) of the first tile, lanes 16-31 those of the second.  With a tile stored as [k][column], lane (g = lane / 4,
// t = lane % 4) receives, for tile i, in r[2i] the bytes (k = 4t .. 4t+3, column g) and in r[2i+1] the bytes
// (k = 4t .. 4t+3, column g + 8).
__device__ __forceinline__ void ldmatrix_x2_trans_b8(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// Four 8 x 16 byte tiles; lane i gives the address of row i % 8 of tile i / 8; lane (g, t) receives bytes 4t .. 4t+3 of row g.
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// Four 8 x 8 tiles of 16-bit values, transposed: lane (g, t) receives elements (row 2t, column g) and (row 2t + 1, column g).
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// The inverse: lane (g, t) holds elements (row 2t, column g), (row 2t + 1, column g) of each tile.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void stmatrix_x2_trans(uint32_t addr, const uint32_t (&r)[2]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(addr), "r"(r[0]), "r"(r[1]) : "memory");
}
__device__ __forceinline__ void stmatrix_x1_trans(uint32_t addr, uint32_t r) {
    asm volatile("stmatrix.sync.aligned.m8n8.x1.trans.shared.b16 [%0], {%1};" ::"r"(addr), "r"(r) : "memory");
}

// Four signed bytes (b0 .. b3) -> f16 pairs (b0, b1) and (b2, b3), exactly (0x6400 | u is 1024 + u).
__device__ __forceinline__ void cvt_s8x4_to_f16_pairs(uint32_t v, uint32_t &p01, uint32_t &p23) {
    const uint32_t u = v ^ 0x80808080u;
    const uint32_t e01 = __byte_perm(u, 0x64646464u, 0x4140);
    const uint32_t e23 = __byte_perm(u, 0x64646464u, 0x4342);
    const uint32_t bias = 0x64806480u;
    asm("sub.f16x2 %0, %1, %2;" : "=r"(p01) : "r"(e01), "r"(bias));
    asm("sub.f16x2 %0, %1, %2;" : "=r"(p23) : "r"(e23), "r"(bias));
}

// ---- what the kernels' pipelines share ----
// A position in a ring of `n` slots, with the parity of the slot's phase.
struct Ring {
    uint32_t slot = 0, phase = 0;
    __device__ __forceinline__ void advance(uint32_t by, uint32_t n) {
        slot += by;
        if (slot >= n) slot -= n, phase ^= 1u;
    }
};

// A bounded wait is this many plain polls, inline, and then `wait_or_abort`: the code around the hot loops stays what it is without
// the flag (with the flag tested at every wait the one-SM kernel lost a tenth of its speed, although the test never ran).
constexpr uint32_t kFastPolls = 4096;
// Polls on, looking at the CTA's abort flag between runs of polls; when its own limit runs out it records the site and raises
// the flag for the other roles of the CTA.
template <unsigned int KERNEL>
__device__ __noinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, unsigned int site, int *abort_flag, unsigned int *status) {
    for (uint32_t round = 0; round < kSpinLimit / 1024u; ++round) {
        if (mbar_wait(bar, parity, 1024u)) return true;
        if (*reinterpret_cast<volatile int *>(abort_flag) != 0) return false;
    }
    report_timeout(status, KERNEL, site);
    atomicExch(abort_flag, 1);
    return false;
}

}  // namespace umma
}  // namespace b200q
