// f16 x int8 quantized linear for [K, N] weights whose rows are not multiples of 16 bytes (N even: vocabularies with
// added tokens, odd feature counts), which neither TMA nor 16-byte loads can take row by row.
//
// Eight rows together are a multiple of 16 bytes, so rows with the same k % 8 all start at the same place between two
// 16-byte boundaries.  Each of a CTA's eight warps therefore takes one residue of k mod 8 and loads, from every row of
// its residue, the 128 bytes that start at the 16-byte boundary at or in front of the tile's first column: aligned 16-byte
// loads, no shifting anywhere in the main loop.  The warps' partial sums are merely offset against each other by up to 15
// columns, which the sum over the warps at the end takes into account; 112 of the 128 columns are common to all eight, and
// those are the tile.  (The 16 columns read twice come from L2: neighbouring tiles run side by side.)
//
// A lane (g, t) loads 16 bytes of four rows: for MMA j of a step its columns are 16 g + 2 j and + 2 j + 1 and its k slots
// the four rows, so byte permutations alone turn the loads into m16n8k16 operands (weights as the 16-row operand, fp32
// accumulators).  The activations of a chunk of k are spread by residue through shared memory, double-buffered.
//
// Bound by streaming the weight once, and by how much of it is in flight.  (7, 4096, 32002), 131 MB: 32 us, 4.1 TB/s; the
// one-thread-per-element kernel that served it before takes 420 us.  Copying the weights to shared memory asynchronously
// instead of into registers: 46 us (the extra trip through shared memory costs more than the deeper pipeline gives).
#include "qlinear.h"
#include "stream_mma.cuh"

namespace b200q {
namespace unaligned {

constexpr int WARPS = 8;              // one per residue of k mod 8
constexpr int THREADS = 32 * WARPS;
constexpr int COLS = 128;             // columns a warp computes
constexpr int TILE = COLS - 16;       // columns of them that every residue covers
constexpr int STEP = 16;              // rows of one residue per MMA step
constexpr int RED_PITCH = COLS + 4;

template <int MT>
struct Config {
    static constexpr int ROWS = 8 * MT;
    // Steps whose activations are in shared memory together, and whose weights are in flight.  Two, with two CTAs on an SM,
    // against four: (7, 4096, 32002) 32 and 40 us; with two blocks of rows one CTA with four fits: (16, 4096, 32002)
    // 48 us, and 64 us with two steps and spilled accumulators.
    static constexpr int CHUNK = MT == 1 ? 2 : 4;
    static constexpr int CHUNK_ROWS = STEP * CHUNK;
    static constexpr int A_PITCH = CHUNK_ROWS + 16;                    // halves between activation rows: 8-byte loads of four rows spread over the banks
    static constexpr int A_BYTES = 8 * ROWS * A_PITCH * 2;             // [residue][row][k / 8] of one chunk
    static constexpr int RED_BYTES = WARPS * ROWS * RED_PITCH * 4;      // the warps' sums, over the activation buffers
    static constexpr int ITEMS = ROWS * (TILE / 4);
    static constexpr int MAIN_BYTES = 2 * A_BYTES > RED_BYTES ? 2 * A_BYTES : RED_BYTES;
    static constexpr int SMEM_BYTES = MAIN_BYTES + stream_mma::recv_bytes(ITEMS);
};

struct Params {
    const __half *a;       // [M, K]
    const uint8_t *wq;     // [K, N]
    const __half *scale;   // [N]
    __half *c;             // [M, N]
    unsigned int *status;
    int M, N, K;
};

// pair: bytes (k0.c, k1.c, k0.c+1, k1.c+1) of rows k0 and k1, each biased by 128 -> the exact f16 pairs (k0, k1) of
// column c and of column c + 1 (0x6400 | u is 1024 + u).
__device__ __forceinline__ void to_f16(uint32_t pair, uint32_t &first, uint32_t &second) {
    const uint32_t bias = 0x64806480u;  // 1152 = 1024 + 128, twice
    const uint32_t e0 = __byte_perm(pair, 0x64646464u, 0x4140), e1 = __byte_perm(pair, 0x64646464u, 0x4342);
    asm("sub.f16x2 %0, %1, %2;" : "=r"(first) : "r"(e0), "r"(bias));
    asm("sub.f16x2 %0, %1, %2;" : "=r"(second) : "r"(e1), "r"(bias));
}

// Through L2: under programmatic launches this CTA may be older than the kernel that wrote the activations.  (The weight,
// too, is read after that kernel, with coherent loads.)
__device__ __forceinline__ uint4 load_l2(const void *p) { return __ldcg(static_cast<const uint4 *>(p)); }

template <int MT>
__global__ void __launch_bounds__(THREADS, MT == 1 ? 2 : 1) qlinear_unaligned_kernel(const Params p) {
    using Cfg = Config<MT>;
    constexpr int ROWS = Cfg::ROWS, CHUNK = Cfg::CHUNK, CHUNK_ROWS = Cfg::CHUNK_ROWS, A_PITCH = Cfg::A_PITCH;
    constexpr int A_LOADS = ROWS * CHUNK_ROWS / THREADS;  // 16-byte activation pieces per thread and chunk
    static_assert(A_LOADS * THREADS == ROWS * CHUNK_ROWS, "whole pieces per thread");
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) uint64_t recv_bar;
    stream_mma::cluster_begin(smem_u32(&recv_bar), Cfg::ITEMS);
    pdl_wait();
    pdl_launch_dependents();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * TILE, m0 = blockIdx.z * ROWS;
    const int ranks = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
    const int groups = p.K / 8;  // rows of each residue
    const int64_t group_bytes = (int64_t)p.N * 8;
    // this CTA's share of the chunks
    const int chunks = (groups + CHUNK_ROWS - 1) / CHUNK_ROWS;
    const int chunk_begin = (int)((int64_t)chunks * rank / ranks), chunk_end = (int)((int64_t)chunks * (rank + 1) / ranks);

    // this lane's 16 bytes of row 8 j + warp start at byte j * group_bytes + x
    const int64_t x = (((int64_t)warp * p.N + n0) & ~(int64_t)15) + 16 * g;
    const bool x_in = x < group_bytes;  // the last tile reaches past the last row; group_bytes is a multiple of 16
    auto load_weights = [&](uint4 (&w)[4], int step) {
        const int j = step * STEP + 4 * t;
        const uint8_t *src = p.wq + j * group_bytes + x;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[i] = make_uint4(0, 0, 0, 0);
            if (x_in && j + i < groups) asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[i].x), "=r"(w[i].y), "=r"(w[i].z), "=r"(w[i].w) : "l"(src + i * group_bytes));
        }
    };
    // piece q of a chunk: activation row q / CHUNK_ROWS, k = 8 j .. 8 j + 7 for the chunk's j = q % CHUNK_ROWS
    auto load_activations = [&](uint4 (&v)[A_LOADS], int chunk) {
#pragma unroll
        for (int l = 0; l < A_LOADS; ++l) {
            const int q = l * THREADS + threadIdx.x;
            const int row = q / CHUNK_ROWS, j = chunk * CHUNK_ROWS + q % CHUNK_ROWS;
            v[l] = make_uint4(0, 0, 0, 0);
            if (m0 + row < p.M && j < groups) v[l] = load_l2(p.a + (size_t)(m0 + row) * p.K + (size_t)j * 8);
        }
    };
    auto store_activations = [&](const uint4 (&v)[A_LOADS], int buffer) {
#pragma unroll
        for (int l = 0; l < A_LOADS; ++l) {
            const int q = l * THREADS + threadIdx.x;
            __half *dst = reinterpret_cast<__half *>(smem + buffer * Cfg::A_BYTES) + (q / CHUNK_ROWS) * A_PITCH + q % CHUNK_ROWS;
            const __half *h = reinterpret_cast<const __half *>(&v[l]);
#pragma unroll
            for (int r = 0; r < 8; ++r) dst[r * ROWS * A_PITCH] = h[r];
        }
    };

    // acc[j][mt]: element (column 16 g + 2 j + h, row 8 mt + 2 t + e) is acc[j][mt][2 h + e]
    float acc[8][MT][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) acc[j][mt][0] = acc[j][mt][1] = acc[j][mt][2] = acc[j][mt][3] = 0.0f;

    uint4 w[CHUNK][4];
    uint4 av[A_LOADS];
    if (chunk_begin < chunk_end) {
        load_activations(av, chunk_begin);
#pragma unroll
        for (int d = 0; d < CHUNK; ++d) load_weights(w[d], chunk_begin * CHUNK + d);
        store_activations(av, chunk_begin & 1);
    }
    for (int chunk = chunk_begin; chunk < chunk_end; ++chunk) {
        const bool more = chunk + 1 < chunk_end;
        if (more) load_activations(av, chunk + 1);
        __syncthreads();  // this chunk's activations are in shared memory; the other buffer is free
        const unsigned char *buf = smem + (chunk & 1) * Cfg::A_BYTES + ((warp * ROWS + g) * A_PITCH + 4 * t) * 2;
#pragma unroll
        for (int d = 0; d < CHUNK; ++d) {
            uint2 b[MT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) b[mt] = *reinterpret_cast<const uint2 *>(buf + (mt * 8 * A_PITCH + d * STEP) * 2);
            uint32_t r[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i][0] = w[d][i].x ^ 0x80808080u, r[i][1] = w[d][i].y ^ 0x80808080u, r[i][2] = w[d][i].z ^ 0x80808080u, r[i][3] = w[d][i].w ^ 0x80808080u;
            if (more) load_weights(w[d], (chunk + 1) * CHUNK + d);
#pragma unroll
            for (int word = 0; word < 4; ++word)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const uint32_t sel = half == 0 ? 0x5140u : 0x7362u;
                    uint32_t a0, a1, a2, a3;
                    to_f16(__byte_perm(r[0][word], r[1][word], sel), a0, a1);
                    to_f16(__byte_perm(r[2][word], r[3][word], sel), a2, a3);
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) mma_m16n8k16(acc[2 * word + half][mt], a0, a1, a2, a3, b[mt].x, b[mt].y);
                }
        }
        if (more) store_activations(av, (chunk + 1) & 1);
    }

    // the warps' sums meet in shared memory, each at its own column offset
    __syncthreads();
    float *red = reinterpret_cast<float *>(smem);
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                *reinterpret_cast<float2 *>(red + (warp * ROWS + 8 * mt + 2 * t + e) * RED_PITCH + 16 * g + 2 * j) = make_float2(acc[j][mt][e], acc[j][mt][2 + e]);
    __syncthreads();
    auto partial = [&](int i) {
        const int row = i / (TILE / 4), col = (i - row * (TILE / 4)) * 4;
        float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < WARPS; ++r) {
            const int off = (int)(((int64_t)r * p.N + n0) & 15);
            const float *v = red + (r * ROWS + row) * RED_PITCH + off + col;
            s.x += v[0], s.y += v[1], s.z += v[2], s.w += v[3];
        }
        return s;
    };
    auto finish = [&](int i, float4 s) {
        const int row = i / (TILE / 4), n = n0 + (i - row * (TILE / 4)) * 4;
        if (m0 + row >= p.M) return;
        __half *dst = p.c + (size_t)(m0 + row) * p.N + n;
        if (n < p.N) *reinterpret_cast<__half2 *>(dst) = __floats2half2_rn(s.x * __half2float(p.scale[n]), s.y * __half2float(p.scale[n + 1]));
        if (n + 2 < p.N) *reinterpret_cast<__half2 *>(dst + 2) = __floats2half2_rn(s.z * __half2float(p.scale[n + 2]), s.w * __half2float(p.scale[n + 3]));
    };
    stream_mma::cluster_sum(smem_u32(&recv_bar), smem_u32(smem) + Cfg::MAIN_BYTES, Cfg::ITEMS, p.status, kKernelUnaligned, partial, finish);
}

template <int MT>
static int launch(const Params &p, cudaStream_t stream) {
    using Cfg = Config<MT>;
    const void *kernel = reinterpret_cast<const void *>(qlinear_unaligned_kernel<MT>);
    static stream_mma::KnownClusters known;
    const int rc = stream_mma::allow_smem(kernel, Cfg::SMEM_BYTES, known);
    if (rc != B200Q_OK) return rc;
    const int64_t n_tiles = ceil_div(p.N, TILE), m_tiles = ceil_div(p.M, Cfg::ROWS);
    const int cluster = stream_mma::choose_cluster(kernel, THREADS, Cfg::SMEM_BYTES, n_tiles * m_tiles, ceil_div(p.K / 8, Cfg::CHUNK_ROWS), known);
    Params copy = p;
    void *args[1] = {&copy};
    return stream_mma::launch("qlinear_unaligned_kernel", kernel, n_tiles, cluster, m_tiles, THREADS, Cfg::SMEM_BYTES, stream, args);
}

}  // namespace unaligned

bool unaligned_supported(const void *a, const void *wq, const void *c, int64_t M, int64_t N, int64_t K) {
    return N % 2 == 0 && K % 8 == 0 && M <= 65535 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(wq)) & 15u) == 0 &&
           (reinterpret_cast<uintptr_t>(c) & 3u) == 0;
}

int launch_unaligned(const void *a, const void *wq, const void *scale, void *c, int64_t M, int64_t N, int64_t K, cudaStream_t stream) {
    unaligned::Params p;
    p.a = static_cast<const __half *>(a);
    p.wq = static_cast<const uint8_t *>(wq);
    p.scale = static_cast<const __half *>(scale);
    p.c = static_cast<__half *>(c);
    p.status = device_status_word();
    p.M = (int)M;
    p.N = (int)N;
    p.K = (int)K;
    return M <= 8 ? unaligned::launch<1>(p, stream) : unaligned::launch<2>(p, stream);
}

}  // namespace b200q
