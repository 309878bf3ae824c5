// Sub-byte weights: 4-bit unsigned codes with per-group scales and zero points (w4a16), the format of the
// reference's CuTe test programs (tests/cute_kernel/quantized_linear.py:494-517, tests/cute_kernel/test_quant_linear.py:36-85):
//
//     c[M, N] = a[M, K] x w[K, N],   w[k, n] = scale[k / G, n] * (q[k, n] - zeros[k / G, n])     (zeros optional)
//
// with a, scale, zeros in f16 and q a u4 matrix [K, N] packed as the reference packs sub-byte types: element i of
// a row sits in bits 4 (i % 2) .. 4 (i % 2) + 3 of byte i / 2 (python/hidet/transforms/lower_integer_subbyte.py:103-113).
// The weight is taken in that plain row-major form; the reference's tests first permute it into a layout private to
// their kernel (preprocess_weight), which has no meaning outside that kernel.
//
// Two kernels: on tensor cores for group sizes that are multiples of 16 (further down), and this one for the others.  A thread owns eight adjacent columns (one 32-bit
// word per k row; a warp reads 128 contiguous bytes per row) and a slice of k.  Inside a group the scale and the zero
// point of a column are constant, so the inner loop multiplies activations with the bare codes and keeps the sum of
// the activations beside it; at the end of the group
//     out[m, n] += scale[n] * (sum_k a[m, k] q[k, n] - zeros[n] * sum_k a[m, k]),
// all in fp32 (the codes are exact in fp32; the reference multiplies every weight by its scale in f16 first and
// accumulates the products, tests/cute_kernel/quantized_linear.py:1044-1047: same value up to rounding).  The k slices
// of a CTA meet in shared memory; the CTAs that split K further write fp32 partial sums to the caller's workspace,
// and a second kernel adds them in slice order and rounds to f16 once: the same result on every run.  (Without room for
// partial sums K is not split.)
#include "stream_mma.cuh"

namespace b200q {
namespace u4 {

constexpr int COLS_PER_THREAD = 8;   // one 32-bit word of packed codes
constexpr int WORDS_X = 32;          // threads along N: a warp covers 256 columns
constexpr int K_SLICES = 8;          // warps of a CTA, each on its own k rows
constexpr int THREADS = WORDS_X * K_SLICES;
// The head of a workspace is where the int8 kernels keep their arrival counters (all-zero between calls); this op
// leaves it alone, so one workspace can serve both.
constexpr size_t kReservedHead = (size_t)65536 * 4;

struct Params {
    const __half *a;        // [M, K]
    const uint32_t *q;      // [K, N / 8] words
    const __half *scale;    // [K / G, N]
    const __half *zeros;    // [K / G, N] or null
    float *partial;         // [splits][M, N] fp32
    __half *direct;         // [M, N]: the result itself, in place of partial sums (one split), or null
    int M, N, K, G;
    int k_per_split;        // a multiple of G
};

// Codes of one word as exact floats: 0x4B000000 | code is 8388608 + code.
__device__ __forceinline__ void unpack8(uint32_t w, float (&v)[8]) {
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = __uint_as_float(((w >> (4 * c)) & 0xFu) | 0x4B000000u) - 8388608.0f;
}

// MT: activation rows per pass (1, 2 or 4: the smallest that covers M, so that a single row costs a single row's
// multiplications).  The k loop is taken 4 to 16 rows at a time with all loads issued first: a thread has only a few
// dozen rows, and one load per iteration would leave it waiting for memory most of the time.
template <int MT>
__global__ void __launch_bounds__(THREADS) qlinear_u4_partial_kernel(const Params p) {
    __shared__ float red[K_SLICES][MT][WORDS_X * COLS_PER_THREAD + 8];
    const int word = blockIdx.x * WORDS_X + threadIdx.x;  // which group of eight columns
    const int n0 = word * COLS_PER_THREAD;
    const int slice = threadIdx.y;
    const int split = blockIdx.y;
    const int k_begin = split * p.k_per_split;
    const int k_end = min(p.K, k_begin + p.k_per_split);
    const int words_per_row = p.N / COLS_PER_THREAD;
    const bool in = n0 < p.N;
    float *out = p.partial + (size_t)split * p.M * p.N;
    constexpr int UNROLL = MT == 1 ? 16 : (MT == 2 ? 8 : 4);  // rows whose loads are in flight together

    for (int m0 = 0; m0 < p.M; m0 += MT) {
        float acc[MT][8];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[m][c] = 0.0f;
        if (in) {
            const __half *arow[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) arow[m] = p.a + (size_t)min(m0 + m, p.M - 1) * p.K;  // rows beyond M repeat the last one and are not stored
            for (int g0 = k_begin; g0 < k_end; g0 += p.G) {
                float gs[MT][8], asum[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    asum[m] = 0.0f;
#pragma unroll
                    for (int c = 0; c < 8; ++c) gs[m][c] = 0.0f;
                }
                const int g_end = min(k_end, g0 + p.G);
                for (int kb = g0 + slice; kb < g_end; kb += UNROLL * K_SLICES) {
                    uint32_t w[UNROLL];
                    float av[UNROLL][MT];
#pragma unroll
                    for (int u = 0; u < UNROLL; ++u) {
                        const int k = kb + u * K_SLICES;
                        const bool ok = k < g_end;
                        w[u] = ok ? __ldg(p.q + (size_t)k * words_per_row + word) : 0u;
#pragma unroll
                        for (int m = 0; m < MT; ++m) av[u][m] = ok ? __half2float(__ldg(arow[m] + k)) : 0.0f;
                    }
#pragma unroll
                    for (int u = 0; u < UNROLL; ++u) {
                        float v[8];
                        unpack8(w[u], v);
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            asum[m] += av[u][m];
#pragma unroll
                            for (int c = 0; c < 8; ++c) gs[m][c] = fmaf(av[u][m], v[c], gs[m][c]);
                        }
                    }
                }
                const size_t grow = (size_t)(g0 / p.G) * p.N + n0;
                const uint4 sraw = __ldg(reinterpret_cast<const uint4 *>(p.scale + grow));
                const __half *sh = reinterpret_cast<const __half *>(&sraw);
                uint4 zraw = make_uint4(0, 0, 0, 0);
                if (p.zeros != nullptr) zraw = __ldg(reinterpret_cast<const uint4 *>(p.zeros + grow));
                const __half *zh = reinterpret_cast<const __half *>(&zraw);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float s = __half2float(sh[c]), z = __half2float(zh[c]);
#pragma unroll
                    for (int m = 0; m < MT; ++m) acc[m][c] = fmaf(s, gs[m][c] - z * asum[m], acc[m][c]);
                }
            }
        }
        // the k slices of the CTA meet in shared memory, slice order
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int c = 0; c < 8; ++c) red[slice][m][threadIdx.x * COLS_PER_THREAD + c] = acc[m][c];
        __syncthreads();
        for (int idx = threadIdx.y * WORDS_X + threadIdx.x; idx < MT * WORDS_X * COLS_PER_THREAD; idx += THREADS) {
            const int m = idx / (WORDS_X * COLS_PER_THREAD);
            const int col = idx - m * (WORDS_X * COLS_PER_THREAD);
            const int n = blockIdx.x * WORDS_X * COLS_PER_THREAD + col;
            if (m0 + m < p.M && n < p.N) {
                float s = 0.0f;
#pragma unroll
                for (int sl = 0; sl < K_SLICES; ++sl) s += red[sl][m][col];
                const size_t at = (size_t)(m0 + m) * p.N + n;
                if (p.direct != nullptr) p.direct[at] = __float2half_rn(s);
                else out[at] = s;
            }
        }
        __syncthreads();
    }
}

__global__ void qlinear_u4_reduce_kernel(const float *partial, __half *c, int64_t mn, int splits) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= mn) return;
    float s = 0.0f;
    for (int sp = 0; sp < splits; ++sp) s += partial[(size_t)sp * mn + i];
    c[i] = __float2half_rn(s);
}

// ---- group sizes that are multiples of 16: tensor cores, one launch ----
// Warp-level m16n8k16 MMAs with the bare codes as the 16-row operand (exact in f16) and the activations as the 8-column
// operand, so that the codes are unpacked once for up to 8 MT activation rows and nothing is multiplied per row outside
// the tensor core.  A CTA owns 64 W columns; its warps and the CTAs of its cluster each take a contiguous
// run of 16-row steps.  A lane (g, t) copies W words (8 W columns) of rows 4t .. 4t + 3 of a step, DEPTH steps
// ahead, into places of shared memory that only it reads, so the main loop has no barrier; the two columns
// 2j, 2j + 1 of a word are rows g and g + 8 of MMA j, and the activations of the same four k are one 8-byte load.  One more
// MMA per step with ones as the 16-row operand gives every lane the sums of its activations.  At the end of a group (or of
// the warp's run; a part of a group is a term like any other)
//     sum += scale * (group sum - zero * activation sum)
// goes to the lane's own place in shared memory, where the warps, and then the cluster, are summed in a fixed order.
// What is left is not bytes: at (1, 4096, 12288) a scheduler issues 8 900 times (mostly unpacking; 10 300 before the constants were kept in
// registers), in half of its active clocks, and four warps each, in chains of short dependent steps, do not hide the latency between; then the
// exchange at the end.  (Built like the small-M int8 kernel, with a TMA producer and transposing matrix loads of bytes, it takes
// 11.2 us there for 11.6, 6.4 for 6.0 at (1, 4096, 4096), and 16.3 for 11.7 where rows are not multiples of 16 bytes.)
// Per launch in a replayed graph, with the kernel below it before: (1, 4096, 12288) 25.8 -> 11.6 us, (8, 4096, 4096) 28.7 ->
// 6.1; (16, 12288, 4096) 127 (a call) -> 16.0, (64, 4096, 11008) 42.
struct MmaParams {
    const __half *a;        // [M, K]
    const uint32_t *q;      // [K, N / 8] words
    const __half *scale;    // [K / G, N]
    const __half *zeros;    // [K / G, N] or null
    __half *c;              // [M, N]
    unsigned int *status;
    int M, N, K;
    int steps_per_group;    // G / 16
};

constexpr int MMA_WARPS = 4;
constexpr int MMA_THREADS = 32 * MMA_WARPS;

template <int MT, int W>
struct MmaConfig {
    static constexpr int TILES = 4 * W;                                 // 16-row MMAs per step
    static constexpr int ITEMS = TILES * MT * 32;                       // float4 sums of a CTA
    static constexpr int RED_BYTES = MMA_WARPS * ITEMS * 16;
    static constexpr int RING_OFF = RED_BYTES + stream_mma::recv_bytes(ITEMS);
    static constexpr int CTAS = MT * MT * W > 4 ? 3 : 4;                // per SM
    // Steps in flight.  Short rings are enough, and let the clusters fit better (measured while codes were copied ahead of the
    // wait, 0.4 us less than now): (1, 4096, 12288) takes 12.7 us with four
    // CTAs of three steps, 15.5 with four of seven; (16, 12288, 4096) 15.9 with three and 19.3 with eight.
    static constexpr int DEPTH = 3;
    static constexpr int SLOT_BYTES = 32 * (16 * W + 8 * MT);           // of one warp and step: [row][lane] words, [row][32 bytes] activations
    static constexpr int SMEM_BYTES = RING_OFF + MMA_WARPS * DEPTH * SLOT_BYTES;
    static_assert(CTAS * (SMEM_BYTES + 1024 + 16) <= 228 * 1024, "room for CTAS per SM");
};

// Codes 0 .. 3 of two rows as f16 pairs (row 0, row 1): x holds the rows' 16-bit pieces.  0x6400 | c is 1024 + c, and with
// the code four bits up 1024 + 16 c, of which a sixteenth less 64 is c; both exact.  (The bare bits as subnormal numbers take
// half the instructions, but the tensor core aligns products by the operands' unnormalised exponents and the sums lose bits.)
// The constants are kept in registers, where the compiler cannot see them: a logical operation takes one immediate, so that
// with two constants in place (x & mask) | bias becomes two operations: 65 instructions for four words, 50 so; (1, 4096, 12288)
// 13.3 -> 12.3 us, (8, 4096, 4096) 6.6 -> 6.1.
struct UnpackConstants {
    uint32_t lower, upper, bias, sixteenth, minus64;
    __device__ __forceinline__ UnpackConstants() {
        asm volatile("mov.b32 %0, 0x000f000f;" : "=r"(lower));
        asm volatile("mov.b32 %0, 0x00f000f0;" : "=r"(upper));
        asm volatile("mov.b32 %0, 0x64006400;" : "=r"(bias));
        asm volatile("mov.b32 %0, 0x2c002c00;" : "=r"(sixteenth));
        asm volatile("mov.b32 %0, 0xd400d400;" : "=r"(minus64));
    }
};
__device__ __forceinline__ void unpack_pairs(uint32_t x, uint32_t (&h)[4], const UnpackConstants &k) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        uint32_t lo, hi;  // (x & mask) | bias
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(lo) : "r"(x >> (8 * i)), "r"(k.lower), "r"(k.bias));
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(hi) : "r"(x >> (8 * i)), "r"(k.upper), "r"(k.bias));
        asm("sub.f16x2 %0, %1, %2;" : "=r"(h[2 * i]) : "r"(lo), "r"(k.bias));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(h[2 * i + 1]) : "r"(hi), "r"(k.sixteenth), "r"(k.minus64));
    }
}

template <int N>
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(N) : "memory");
}

// WIDE: W words are loaded together (rows are multiples of 4 W bytes).
template <int MT, int W, bool WIDE>
__global__ void __launch_bounds__(MMA_THREADS, MmaConfig<MT, W>::CTAS) qlinear_u4_mma_kernel(const MmaParams p) {
    using Cfg = MmaConfig<MT, W>;
    constexpr int DEPTH = Cfg::DEPTH, TILES = Cfg::TILES;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t recv_bar;
    stream_mma::cluster_begin(smem_u32(&recv_bar), Cfg::ITEMS);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int m0 = blockIdx.z * 8 * MT;
    const int words_per_row = p.N / COLS_PER_THREAD;
    const int word0 = (blockIdx.x * 8 + g) * W;      // this lane's words
    const int n_lane = word0 * COLS_PER_THREAD;      // and their first column
    // this warp's run of 16-row steps
    const int steps = p.K / 16, workers = (int)cluster_nctarank() * MMA_WARPS, worker = (int)cluster_ctarank() * MMA_WARPS + warp;
    const int share = steps / workers, extra = steps % workers;
    const int s_begin = worker * share + min(worker, extra), s_end = s_begin + share + (worker < extra ? 1 : 0);

    // Words beyond the row repeat the last ones: their columns of the result are not stored.  Rows beyond M are zeros.
    bool in[W];
    const uint32_t *q_src[4][W];  // the words of the next step to fetch
#pragma unroll
    for (int i = 0; i < W; ++i) {
        in[i] = word0 + i < words_per_row;
#pragma unroll
        for (int r = 0; r < 4; ++r) q_src[r][i] = p.q + (size_t)(s_begin * 16 + 4 * t + r) * words_per_row + min(word0 + (WIDE ? 0 : i), words_per_row - (WIDE ? W : 1));
    }
    // The activations of a step are 32 bytes of each row; half a row per lane, lanes 2 (8 mt + row) and + 1, through L2 (this CTA
    // may be older than the kernel that wrote them, and so may be what the first-level cache holds).
    constexpr int A_COPIES = (MT + 1) / 2;
    const __half *a_src[A_COPIES];
    int a_size[A_COPIES];  // bytes to copy, the rest of the 16 is zeros (rows beyond M used to repeat the last one, whose lines every CTA then asked
                           // for many times over: (24, 4096, 12288) 33 -> 22 us, (9, 4096, 4096) 9.9 -> 7.5, (1, 4096, 12288) 12.3 -> 11.6)
#pragma unroll
    for (int i = 0; i < A_COPIES; ++i) {
        const int row = m0 + 16 * i + (lane >> 1);
        a_size[i] = row < p.M ? 16 : 0;
        a_src[i] = p.a + (size_t)min(row, p.M - 1) * p.K + s_begin * 16 + 8 * (lane & 1);
    }
    const uint32_t ring = smem_u32(smem) + Cfg::RING_OFF + (uint32_t)warp * DEPTH * Cfg::SLOT_BYTES + lane * 4 * W;
    const uint32_t ring_a = smem_u32(smem) + Cfg::RING_OFF + (uint32_t)warp * DEPTH * Cfg::SLOT_BYTES + 4 * W * 4 * 32;
    const size_t step_words = (size_t)16 * words_per_row;
    auto fetch_codes = [&](uint32_t slot) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int i = 0; i < (WIDE ? 1 : W); ++i) {
                cp_async<WIDE ? 4 * W : 4>(ring + slot + r * 32 * 4 * W + 4 * i, q_src[r][i]);
                q_src[r][i] += step_words;
            }
    };
    auto fetch_activations = [&](uint32_t slot) {
#pragma unroll
        for (int i = 0; i < A_COPIES; ++i) {
            if (MT > 1 || lane < 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ring_a + slot + (i * 32 + lane) * 16), "l"(a_src[i]), "r"(a_size[i]) : "memory");
            a_src[i] += 16;
        }
    };
    auto commit = [&]() { asm volatile("cp.async.commit_group;" ::: "memory"); };  // one group per step, empty ones past the end included
    // scales and zero points of this lane's columns in a group
    uint4 sc[W], zp[W];
    auto load_group = [&](int group) {
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const size_t off = (size_t)group * p.N + n_lane + 8 * i;
            sc[i] = zp[i] = make_uint4(0, 0, 0, 0);
            if (in[i]) sc[i] = __ldcg(reinterpret_cast<const uint4 *>(p.scale + off));
            if (in[i] && p.zeros != nullptr) zp[i] = __ldcg(reinterpret_cast<const uint4 *>(p.zeros + off));
        }
    };

    // acc[j][mt]: element (column n_lane + 2 j + h, row 8 mt + 2 t + e) is acc[j][mt][2 h + e]; asum[mt][e]: row 8 mt + 2 t + e
    float acc[TILES][MT][4], asum[MT][4];
    auto clear = [&]() {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
            for (int j = 0; j < TILES; ++j) acc[j][mt][0] = acc[j][mt][1] = acc[j][mt][2] = acc[j][mt][3] = 0.0f;
            asum[mt][0] = asum[mt][1] = asum[mt][2] = asum[mt][3] = 0.0f;
        }
    };
    float4 *red = reinterpret_cast<float4 *>(smem) + warp * Cfg::ITEMS + lane;
    bool first = true;
    auto flush = [&]() {
#pragma unroll
        for (int j = 0; j < TILES; ++j) {
            const __half2 s2 = reinterpret_cast<const __half2 *>(&sc[j / 4])[j % 4], z2 = reinterpret_cast<const __half2 *>(&zp[j / 4])[j % 4];
            const float s0 = __low2float(s2), s1 = __high2float(s2), z0 = __low2float(z2), z1 = __high2float(z2);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                float4 *dst = red + (j * MT + mt) * 32;
                float4 v = first ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : *dst;
                v.x = fmaf(s0, acc[j][mt][0] - z0 * asum[mt][0], v.x);
                v.y = fmaf(s0, acc[j][mt][1] - z0 * asum[mt][1], v.y);
                v.z = fmaf(s1, acc[j][mt][2] - z1 * asum[mt][0], v.z);
                v.w = fmaf(s1, acc[j][mt][3] - z1 * asum[mt][1], v.w);
                *dst = v;
            }
        }
        first = false;
    };

    const UnpackConstants constants;
    uint32_t ones[4];  // a register each, as above: otherwise the four are put in place again for every MMA
#pragma unroll
    for (int i = 0; i < 4; ++i) asm volatile("mov.b32 %0, 0x3c003c00;" : "=r"(ones[i]));
    clear();
    int group = s_begin / p.steps_per_group;
    int left = (group + 1) * p.steps_per_group - s_begin;  // steps to the end of the group
    // Nothing is read before the kernel in front is done, so codes and scales may be its results like the activations; the
    // first codes are only asked into L2, which is coherent: (1, 4096, 4096) 6.5 us, 7.2 without, and 6.3 with the codes copied
    // ahead of the wait.  The kernel after this one may move in once the wait is over.
#pragma unroll
    for (int d = 0; d < DEPTH; ++d)
        if (s_begin + d < s_end) {
#pragma unroll
            for (int r = 0; r < 4; ++r) asm volatile("prefetch.global.L2 [%0];" ::"l"(q_src[r][0] + d * step_words));
        }
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
        if (s_begin + d < s_end) {
            fetch_codes(d * Cfg::SLOT_BYTES);
            fetch_activations(d * Cfg::SLOT_BYTES);
        }
        commit();
    }
    if (s_begin < s_end) load_group(group);
    uint32_t slot = 0;
    for (int step = s_begin; step < s_end; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
        __syncwarp();  // the activations come from other lanes
        uint32_t w[4][W];
        uint2 b[MT];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t src = ring + slot + r * 32 * 4 * W;
            if (W == 2) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[r][0]), "=r"(w[r][W - 1]) : "r"(src) : "memory");
            else asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[r][0]) : "r"(src) : "memory");
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(b[mt].x), "=r"(b[mt].y) : "r"(ring_a + slot + (8 * mt + g) * 32 + t * 8) : "memory");
#pragma unroll
        for (int i = 0; i < W; ++i)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const uint32_t sel = half == 0 ? 0x5410u : 0x7632u;
                uint32_t h01[4], h23[4];
                unpack_pairs(__byte_perm(w[0][i], w[1][i], sel), h01, constants);
                unpack_pairs(__byte_perm(w[2][i], w[3][i], sel), h23, constants);
#pragma unroll
                for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt)
                        mma_m16n8k16(acc[4 * i + 2 * half + jj][mt], h01[2 * jj], h01[2 * jj + 1], h23[2 * jj], h23[2 * jj + 1], b[mt].x, b[mt].y);
            }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) mma_m16n8k16(asum[mt], ones[0], ones[1], ones[2], ones[3], b[mt].x, b[mt].y);
        __syncwarp();
        if (step + DEPTH < s_end) {  // into the place just read
            fetch_codes(slot);
            fetch_activations(slot);
        }
        commit();
        slot = slot == (DEPTH - 1) * Cfg::SLOT_BYTES ? 0 : slot + Cfg::SLOT_BYTES;
        if (--left == 0 || step + 1 == s_end) {
            flush();
            if (step + 1 < s_end) {
                clear();
                load_group(++group);
                left = p.steps_per_group;
            }
        }
    }
    if (first) {  // no steps: this warp's sum is zero
#pragma unroll
        for (int j = 0; j < TILES * MT; ++j) red[j * 32] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncthreads();
    auto partial = [&](int i) {
        const float4 *src = reinterpret_cast<const float4 *>(smem) + i;
        float4 s = src[0];
#pragma unroll
        for (int r = 1; r < MMA_WARPS; ++r) {
            const float4 v = src[r * Cfg::ITEMS];
            s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
        }
        return s;
    };
    auto finish = [&](int i, float4 s) {
        const int ln = i & 31, tile = i >> 5, mt = tile % MT, j = tile / MT;
        const int n = (blockIdx.x * 8 + (ln >> 2)) * W * COLS_PER_THREAD + 2 * j, m = m0 + 8 * mt + 2 * (ln & 3);
        if (n >= p.N) return;
        __half2 *dst = reinterpret_cast<__half2 *>(p.c + (size_t)m * p.N + n);
        if (m < p.M) *dst = __floats2half2_rn(s.x, s.z);
        if (m + 1 < p.M) dst[p.N / 2] = __floats2half2_rn(s.y, s.w);
    };
    stream_mma::cluster_sum(smem_u32(&recv_bar), smem_u32(smem) + Cfg::RED_BYTES, Cfg::ITEMS, p.status, kKernelU4, partial, finish);
}

template <int MT, int W, bool WIDE>
int launch_mma(const MmaParams &p, cudaStream_t stream) {
    using Cfg = MmaConfig<MT, W>;
    const void *kernel = reinterpret_cast<const void *>(qlinear_u4_mma_kernel<MT, W, WIDE>);
    static stream_mma::KnownClusters known;
    const int rc = stream_mma::allow_smem(kernel, Cfg::SMEM_BYTES, known);
    if (rc != B200Q_OK) return rc;
    const int64_t n_tiles = ceil_div(p.N, (int64_t)64 * W), m_tiles = ceil_div(p.M, (int64_t)8 * MT);
    // every warp should have two steps or more
    const int cluster = stream_mma::choose_cluster(kernel, MMA_THREADS, Cfg::SMEM_BYTES, n_tiles * m_tiles, p.K / (16 * 2 * MMA_WARPS), known);
    MmaParams copy = p;
    void *args[1] = {&copy};
    return stream_mma::launch("qlinear_u4_mma_kernel", kernel, n_tiles, cluster, m_tiles, MMA_THREADS, Cfg::SMEM_BYTES, stream, args);
}

// The tensor-core kernel's conditions: steps of 16 rows that never cross a group, and what its loads and stores need.
bool mma_supported(const void *a, const void *c, int64_t M, int64_t G) {
    return G % 16 == 0 && M <= (int64_t)65535 * 32 && (reinterpret_cast<uintptr_t>(a) & 15u) == 0 && (reinterpret_cast<uintptr_t>(c) & 3u) == 0;
}

// f16 (integral values) -> u4 codes, two per byte; C conversion to int, low four bits kept.  Like every kernel here that
// writes weights, this one never lets dependents start early (the small-M int8 kernel reads weights ahead of its wait).
__global__ void u4_pack_kernel(const __half *w, uint8_t *out, int64_t bytes) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= bytes) return;
    const __half2 v = reinterpret_cast<const __half2 *>(w)[i];
    const int lo = (int)__low2float(v), hi = (int)__high2float(v);
    out[i] = (uint8_t)((lo & 15) | ((hi & 15) << 4));
}

__global__ void u4_unpack_kernel(const uint8_t *packed, __half *out, int64_t bytes) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= bytes) return;
    const uint8_t b = packed[i];
    reinterpret_cast<__half2 *>(out)[i] = __floats2half2_rn((float)(b & 15), (float)(b >> 4));
}

struct Plan {
    int splits;
    int k_per_split;
};

Plan plan(int64_t M, int64_t N, int64_t K, int64_t G) {
    (void)M;
    int sms = sm_count();
    if (sms <= 0) sms = 148;
    const int64_t col_blocks = ceil_div(N, (int64_t)WORDS_X * COLS_PER_THREAD);
    const int64_t groups = ceil_div(K, G);
    int64_t splits = ceil_div((int64_t)4 * sms, col_blocks);  // four CTAs per SM: the loads of many rows in flight
    if (splits > groups) splits = groups;
    if (splits < 1) splits = 1;
    Plan pl;
    pl.k_per_split = (int)(ceil_div(groups, splits) * G);
    pl.splits = (int)ceil_div(K, pl.k_per_split);
    return pl;
}

// Scratch a call asks for.  The tensor-core kernel has no use for any: its group sizes are held to what the shared head
// takes, whatever the problem, and a call without a workspace is refused for every group size alike.
size_t workspace_bytes(int64_t M, int64_t N, int64_t K, int64_t G) {
    if (G % 16 == 0) return kReservedHead + 256;
    return kReservedHead + (size_t)plan(M, N, K, G).splits * M * N * sizeof(float);
}

}  // namespace u4
}  // namespace b200q

extern "C" {

B200Q_API size_t b200q_qlinear_f16_u4_workspace_bytes(int64_t M, int64_t N, int64_t K, int64_t group_size) {
    using namespace b200q;
    if (M <= 0 || N <= 0 || K <= 0 || group_size <= 0) return 0;
    return u4::workspace_bytes(M, N, K, group_size);
}

B200Q_API int b200q_qlinear_f16_u4(const void *a, const void *q, const void *scale, const void *zeros, void *c, int64_t M, int64_t N, int64_t K,
                                   int64_t group_size, void *workspace, size_t workspace_bytes, void *stream) {
    using namespace b200q;
    if (M < 0 || N < 0 || K < 0) return set_error(B200Q_INVALID_ARGUMENT, "qlinear_f16_u4: negative size M=%lld N=%lld K=%lld", (long long)M, (long long)N, (long long)K);
    if (group_size <= 0 || K % group_size != 0) {
        return set_error(B200Q_INVALID_ARGUMENT, "qlinear_f16_u4: K=%lld is not a multiple of the group size %lld", (long long)K, (long long)group_size);
    }
    if (N % 8 != 0) return set_error(B200Q_UNSUPPORTED, "qlinear_f16_u4: N=%lld is not a multiple of 8 (whole 32-bit words of codes per row)", (long long)N);
    if (M > 2147483647LL || N > 2147483647LL || K > 2147483647LL) return set_error(B200Q_UNSUPPORTED, "qlinear_f16_u4: sizes beyond 2^31-1 are not supported");
    if (M == 0 || N == 0) return B200Q_OK;
    if (c == nullptr) return set_error(B200Q_INVALID_ARGUMENT, "qlinear_f16_u4: null output pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (K == 0) {
        B200Q_CUDA_TRY(cudaMemsetAsync(c, 0, (size_t)M * N * sizeof(__half), s));
        return B200Q_OK;
    }
    if (a == nullptr || q == nullptr || scale == nullptr) return set_error(B200Q_INVALID_ARGUMENT, "qlinear_f16_u4: null input pointer");
    if ((reinterpret_cast<uintptr_t>(q) & 3u) != 0 || (reinterpret_cast<uintptr_t>(scale) & 15u) != 0 || (reinterpret_cast<uintptr_t>(zeros) & 15u) != 0) {
        return set_error(B200Q_UNSUPPORTED, "qlinear_f16_u4: codes need a 4-byte aligned base, scales and zero points 16-byte aligned bases");
    }
    const size_t need = u4::workspace_bytes(M, N, K, group_size);
    if (workspace == nullptr || workspace_bytes < need) {
        return set_error(B200Q_WORKSPACE_TOO_SMALL, "qlinear_f16_u4: workspace of %zu bytes given, %zu needed for M=%lld N=%lld K=%lld", workspace_bytes, need,
                         (long long)M, (long long)N, (long long)K);
    }
    if (u4::mma_supported(a, c, M, group_size)) {
        u4::MmaParams mp;
        mp.a = static_cast<const __half *>(a);
        mp.q = static_cast<const uint32_t *>(q);
        mp.scale = static_cast<const __half *>(scale);
        mp.zeros = static_cast<const __half *>(zeros);
        mp.c = static_cast<__half *>(c);
        mp.status = device_status_word();
        mp.M = (int)M;
        mp.N = (int)N;
        mp.K = (int)K;
        mp.steps_per_group = (int)(group_size / 16);
        // Wider column strips while one block of rows is enough (64 contiguous bytes of a row: (1, 4096, 12288) 13 us
        // against 20 with 32), except where they leave too few CTAs ((1, 12288, 256) 7.0 us wide, 5.7 narrow).  With two blocks they
        // take a CTA off the SM for the accumulators' registers: wide where columns abound and K is long enough ((16, 4096, 12288) 19.6 -> 13.3,
        // (9, 4096, 8192) 12.4 -> 10.6, (16, 2432, 7040) 8.7 -> 7.8; (16, 1024, 8192) 5.8 -> 6.2, (16, 4096, 4096) 8.1 -> 8.3,
        // (16, 12288, 4096) 16.1 -> 17.4); narrow with four, where two CTAs an SM are left ((24, 4096, 12288) 22.2 and 24.3).
        const bool whole = N % 16 == 0 && (reinterpret_cast<uintptr_t>(q) & 7u) == 0;  // rows of 8-byte pieces
        if (M > 16) return u4::launch_mma<4, 1, true>(mp, s);
        if (M > 8) return N >= 6144 && K >= 2048 && whole ? u4::launch_mma<2, 2, true>(mp, s) : u4::launch_mma<2, 1, true>(mp, s);
        if (N <= 1024) return u4::launch_mma<1, 1, true>(mp, s);
        return whole ? u4::launch_mma<1, 2, true>(mp, s) : u4::launch_mma<1, 2, false>(mp, s);
    }
    u4::Plan pl = u4::plan(M, N, K, group_size);
    // Operands the tensor-core kernel cannot take (an unaligned a or c) with its amount of scratch: one split.
    const bool direct = workspace_bytes < u4::kReservedHead + (size_t)pl.splits * M * N * sizeof(float);
    if (direct) pl = {1, (int)K};
    u4::Params p;
    p.direct = direct ? static_cast<__half *>(c) : nullptr;
    p.a = static_cast<const __half *>(a);
    p.q = static_cast<const uint32_t *>(q);
    p.scale = static_cast<const __half *>(scale);
    p.zeros = static_cast<const __half *>(zeros);
    p.partial = reinterpret_cast<float *>(static_cast<unsigned char *>(workspace) + u4::kReservedHead);
    p.M = (int)M;
    p.N = (int)N;
    p.K = (int)K;
    p.G = (int)group_size;
    p.k_per_split = pl.k_per_split;
    const dim3 grid((unsigned)ceil_div(N, (int64_t)u4::WORDS_X * u4::COLS_PER_THREAD), (unsigned)pl.splits, 1);
    const dim3 block(u4::WORDS_X, u4::K_SLICES, 1);
    if (M == 1) {
        u4::qlinear_u4_partial_kernel<1><<<grid, block, 0, s>>>(p);
    } else if (M == 2) {
        u4::qlinear_u4_partial_kernel<2><<<grid, block, 0, s>>>(p);
    } else {
        u4::qlinear_u4_partial_kernel<4><<<grid, block, 0, s>>>(p);
    }
    B200Q_CHECK_LAUNCH("qlinear_u4_partial_kernel");
    if (direct) return B200Q_OK;
    const int64_t mn = M * N;
    u4::qlinear_u4_reduce_kernel<<<(unsigned)ceil_div(mn, 256), 256, 0, s>>>(p.partial, static_cast<__half *>(c), mn, pl.splits);
    B200Q_CHECK_LAUNCH("qlinear_u4_reduce_kernel");
    return B200Q_OK;
}

B200Q_API int b200q_u4_pack(const void *w, void *packed, int64_t rows, int64_t cols, void *stream) {
    using namespace b200q;
    if (rows < 0 || cols < 0 || cols % 2 != 0) return set_error(B200Q_INVALID_ARGUMENT, "u4_pack: rows=%lld cols=%lld (cols must be even)", (long long)rows, (long long)cols);
    const int64_t bytes = rows * cols / 2;
    if (bytes == 0) return B200Q_OK;
    if (w == nullptr || packed == nullptr) return set_error(B200Q_INVALID_ARGUMENT, "u4_pack: null pointer");
    u4::u4_pack_kernel<<<(unsigned)ceil_div(bytes, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __half *>(w), static_cast<uint8_t *>(packed), bytes);
    B200Q_CHECK_LAUNCH("u4_pack_kernel");
    return B200Q_OK;
}

B200Q_API int b200q_u4_unpack(const void *packed, void *w, int64_t rows, int64_t cols, void *stream) {
    using namespace b200q;
    if (rows < 0 || cols < 0 || cols % 2 != 0) return set_error(B200Q_INVALID_ARGUMENT, "u4_unpack: rows=%lld cols=%lld (cols must be even)", (long long)rows, (long long)cols);
    const int64_t bytes = rows * cols / 2;
    if (bytes == 0) return B200Q_OK;
    if (w == nullptr || packed == nullptr) return set_error(B200Q_INVALID_ARGUMENT, "u4_unpack: null pointer");
    u4::u4_unpack_kernel<<<(unsigned)ceil_div(bytes, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint8_t *>(packed), static_cast<__half *>(w), bytes);
    B200Q_CHECK_LAUNCH("u4_unpack_kernel");
    return B200Q_OK;
}

}  // extern "C"
