// C[M, N] = A[M, K] * W[N, K]^T in true float on the FMA pipe (no tensor cores, no reduced-precision mode): the 32-bit path's
// products of up to 32 rows wherever these are 16-byte aligned (K % 4 == 0).  More rows are gemm_f32_tc.cu's, but for a result off a 16-byte boundary
// whose rows are multiples of 16 bytes.  gemm_simt.cu keeps the other alignments and bfloat16 operands.
//
// Both kernels multiply with fma.rn.f32x2 along K: a 16-byte piece of a row is two pairs of neighbouring k, which is how both
// operands lie in memory, so no value is duplicated or repacked; the even and the odd k of a sum are added at the end.
//
// gemm_f32_tile_kernel   tiles of 16 x 128 and 32 x 128 (64 x 128 for such results), 128 threads of 2 x 8 and 4 x 8 results (8 x 8), K slices of 32
//   through a three-stage cp.async ring, two blocks an SM.  Per 4 k a thread issues 128 packed FMAs and 16 16-byte reads, nearly free of bank
//   conflicts (rows are 36 floats apart).  549 rows, 6144 x 1024 (ncu): the FMA pipe busy 62 % of an SM's active cycles, shared memory 50 %; the rest are
//   fixed latencies of the two warps a scheduler that 255 registers leave.  8 x 4 results a thread (12 reads for 64
//   FMAs) ran at 35 TFLOP/s where 8 x 8 run at 41.  Up to eight blocks of a cluster share a tile's K and add their parts through
//   distributed shared memory in the order of the ranks: for tiles that do not fill the SMs, and because a running sum over a K of
//   thousands would lose low-order bits.  A slice's sums go into a second set of floats for the same reason.
// gemm_f32_rows_kernel   up to 8 rows: bound by the weight's bytes.  A warp takes 4 weight rows (and, where N gives too few blocks, a
//   share of K that the block's warps add through shared memory); its lanes walk K in 16-byte pieces, the first of which are
//   asked for ahead of the dependency wait, since no kernel of a step writes weights.
//
// Against gemm_simt_kernel (before), N x K 6144 x 1024: 2 rows 10 us (119), 64 rows 36 us (126), 549 rows 178 us (313), 1,024 rows 319 us (617);
// 151,936 x 1,024 at 2 rows 111 us (878), 5.6 TB/s; error against 64 bits 0.9e-7 to 1.18e-7 (1.13e-7 to 1.26e-7) of the result's norm.
#include "common.cuh"

using namespace qt;

namespace {

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float halves(uint64_t v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }

constexpr int GF_BN = 128, GF_BK = 32, GF_THREADS = 128, GF_STAGES = 3, GF_MOST_RANKS = 8;
constexpr int GF_ROW = GF_BK + 4;                                          // floats between rows in shared memory


__device__ __forceinline__ void copy16(float* to, const float* from, bool there) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(to);
    const int bytes = there ? 16 : 0;                                       // nothing read, zeros written
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(from), "r"(bytes) : "memory");
}

// TM x 8 results a thread, tiles of 8 TM x 128; grid (ranks x N tiles, M tiles); k_steps slices of 32 per rank
template <int TM>
__global__ void __launch_bounds__(GF_THREADS, 2) gemm_f32_tile_kernel(const float* a, const float* w, float* __restrict__ c,
                                                                     int M, int N, int K, int ranks, int k_steps) {
    constexpr int BM = 8 * TM, STAGE = (BM + GF_BN) * GF_ROW;
    static_assert(GF_STAGES * STAGE >= BM * GF_BN, "a block's part of the result is exchanged in the ring's memory");
    extern __shared__ __align__(16) float ring[];
    const int rank = ranks > 1 ? (int)cluster_rank() : 0;
    if (ranks > 1) cluster_arrive_started();
    const int n0 = blockIdx.x / ranks * GF_BN, m0 = blockIdx.y * BM;
    const int k_begin = rank * k_steps * GF_BK;
    const int k_end = min(K, k_begin + k_steps * GF_BK);
    const int steps = k_end > k_begin ? (k_end - k_begin + GF_BK - 1) / GF_BK : 0;
    const int row = threadIdx.x >> 3, piece = (threadIdx.x & 7) * 4;        // a warp copies four rows of 128 bytes

    auto fetch = [&](const float* from, float* to, int rows, int first, int limit, int step) {
        const int k = k_begin + step * GF_BK + piece;
#pragma unroll
        for (int r = 0; r < rows; r += GF_THREADS / 8) {
            const int at = first + r + row;
            const bool there = at < limit && k < k_end;
            copy16(to + (r + row) * GF_ROW + piece, there ? from + (size_t)at * K + k : from, there);
        }
    };
    auto fetch_w = [&](int step) { fetch(w, ring + step % GF_STAGES * STAGE + BM * GF_ROW, GF_BN, n0, N, step); };
    auto fetch_a = [&](int step) { fetch(a, ring + step % GF_STAGES * STAGE, BM, m0, M, step); };
    // weights do not depend on the kernels before this one
#pragma unroll
    for (int s = 0; s < GF_STAGES - 1; ++s)
        if (s < steps) fetch_w(s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < GF_STAGES - 1; ++s) {
        if (s < steps) fetch_a(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tm = (warp >> 1) * (4 * TM) + (lane >> 3), tn = (warp & 1) * 64 + (lane & 7);   // rows tm + 4 i, columns tn + 8 j
    float sum[TM][8] = {};
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GF_STAGES - 2) : "memory");
        __syncthreads();                                                    // the slice is there, and the one before it is read
        if (step + GF_STAGES - 1 < steps) { fetch_w(step + GF_STAGES - 1); fetch_a(step + GF_STAGES - 1); }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = ring + step % GF_STAGES * STAGE + tm * GF_ROW;
        const float* ws = ring + step % GF_STAGES * STAGE + (BM + tn) * GF_ROW;
        uint64_t part[TM][8];
#pragma unroll
        for (int k = 0; k < GF_BK; k += 4) {
            ulonglong2 av[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(as + i * 4 * GF_ROW + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(ws + j * 8 * GF_ROW + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) part[i][j] = fma2(av[i].x, wv.x, k == 0 ? 0ull : part[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) part[i][j] = fma2(av[i].y, wv.y, part[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) sum[i][j] += halves(part[i][j]);
    }
    pdl_launch_dependents();                                                // late: their blocks would take this kernel's places
    if (ranks == 1) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int m = m0 + tm + 4 * i, n = n0 + tn + 8 * j;
                if (m < M && n < N) c[(size_t)m * N + n] = sum[i][j];
            }
        return;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                                        // the ring is read out and nothing more arrives in it
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) ring[(tm + 4 * i) * GF_BN + tn + 8 * j] = sum[i][j];
    cluster_wait_started();
    cluster_barrier();
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(ring);
    for (int at = (rank * GF_THREADS + threadIdx.x) * 4; at < BM * GF_BN; at += ranks * GF_THREADS * 4) {
        const int m = m0 + at / GF_BN, n = n0 + at % GF_BN;
        float v[GF_MOST_RANKS][4];
#pragma unroll
        for (int r = 0; r < GF_MOST_RANKS; ++r) {                           // every peer is asked before the first answer is used
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mine + at * 4), "r"(r < ranks ? r : 0));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[r][0]), "=f"(v[r][1]), "=f"(v[r][2]), "=f"(v[r][3]) : "r"(remote) : "memory");
        }
        float total[4] = {};
#pragma unroll
        for (int r = 0; r < GF_MOST_RANKS; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j) total[j] += r < ranks ? v[r][j] : 0.f;
        if (m < M)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < N) c[(size_t)m * N + n + j] = total[j];
    }
    cluster_barrier();                                                      // a block leaves only when nobody reads its part any more
}

template <int TM>
int launch_tiles(const float* a, const float* w, float* c, int M, int N, int K, cudaStream_t s) {
    constexpr int SMEM = GF_STAGES * (8 * TM + GF_BN) * GF_ROW * 4;
    const cudaError_t raised = raise_shared<gemm_f32_tile_kernel<TM>>(SMEM);
    if (raised != cudaSuccess) QT_FAIL(QT_ERR_LAUNCH, "gemm_f32: %d bytes of shared memory: %s", SMEM, cudaGetErrorString(raised));
    const long long tiles_n = (N + GF_BN - 1) / GF_BN, tiles_m = (M + 8 * TM - 1) / (8 * TM), slices = (K + GF_BK - 1) / GF_BK;
    QT_REQUIRE(tiles_m <= 65535, "gemm_f32: M=%d is too large for one launch", M);
    const int slots = 2 * sm_count();
    // K ranges.  At least one per 16 slices: a chain of 16 products, 16 slices and the ranges rounds no more than the three levels of
    // gemm_simt.cu do (16 products, 16 tiles, K / 256 groups).  Beyond that the count with the shortest product of waves and slices a
    // block walks (plus about six slices' time for a block's start, exchange and end).
    int least = 1;
    while (least < GF_MOST_RANKS && slices > 16 * least) least *= 2;
    int ranks = least;
    double best = 1e30;
    for (int r = least; r <= GF_MOST_RANKS; r *= 2) {
        if (r > least && slices < 4 * r) break;
        const long long waves = (tiles_n * tiles_m * r + slots - 1) / slots;
        const double cost = (double)waves * ((double)((slices + r - 1) / r) + 6.0);
        if (cost < 0.97 * best) { best = cost; ranks = r; }
    }
    const int k_steps = (int)((slices + ranks - 1) / ranks);
    const dim3 grid((unsigned)(tiles_n * ranks), (unsigned)tiles_m);
    if (ranks == 1) launch_kernel(gemm_f32_tile_kernel<TM>, grid, dim3(GF_THREADS), SMEM, s, a, w, c, M, N, K, ranks, k_steps);
    else launch_kernel_cluster(gemm_f32_tile_kernel<TM>, grid, dim3(GF_THREADS), SMEM, s, (unsigned)ranks, a, w, c, M, N, K, ranks, k_steps);
    QT_CHECK_LAUNCH("gemm_f32");
    return QT_OK;
}

// MT rows of A at most (1, 2, 4 or 8), 4 weight rows a warp; shares: warps of a block that divide a weight row's K
constexpr int GR_WARPS = 8, GR_ROWS = 4;

template <int MT>
__global__ void __launch_bounds__(GR_WARPS * 32) gemm_f32_rows_kernel(const float* a, const float* w, float* __restrict__ c,
                                                                     int M, int N, int K, int shares) {
    constexpr int AHEAD = MT <= 2 ? 4 : 2;                                  // 16-byte pieces of each weight row in flight
    __shared__ float exchange[GR_WARPS][MT * GR_ROWS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int share = warp % shares, n0 = (blockIdx.x * (GR_WARPS / shares) + warp / shares) * GR_ROWS;
    const int pieces = K >> 2, stride = shares * 32;
    const ulonglong2* wr[GR_ROWS];
#pragma unroll
    for (int r = 0; r < GR_ROWS; ++r) wr[r] = reinterpret_cast<const ulonglong2*>(w + (size_t)min(n0 + r, N - 1) * K);   // rows beyond N: read, not stored
    uint64_t acc[MT][GR_ROWS];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < GR_ROWS; ++r) acc[m][r] = 0ull;
    ulonglong2 next[AHEAD][GR_ROWS];
    int at = share * 32 + lane;
    auto load = [&](int first) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
#pragma unroll
            for (int r = 0; r < GR_ROWS; ++r)
                if (first + u * stride < pieces) next[u][r] = __ldg(wr[r] + first + u * stride);
    };
    load(at);
    pdl_launch_dependents();
    pdl_wait();
    for (; at < pieces; at += AHEAD * stride) {
        ulonglong2 now[AHEAD][GR_ROWS];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
#pragma unroll
            for (int r = 0; r < GR_ROWS; ++r) now[u][r] = next[u][r];
        load(at + AHEAD * stride);
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            if (at + u * stride >= pieces) break;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const ulonglong2 x = m < M ? *(reinterpret_cast<const ulonglong2*>(a + (size_t)m * K) + at + u * stride) : make_ulonglong2(0ull, 0ull);
#pragma unroll
                for (int r = 0; r < GR_ROWS; ++r) acc[m][r] = fma2(x.y, now[u][r].y, fma2(x.x, now[u][r].x, acc[m][r]));
            }
        }
    }
    float mine = 0.f;                                                       // lane m * GR_ROWS + r keeps that sum
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < GR_ROWS; ++r) {
            const float total = warp_sum(halves(acc[m][r]));
            if (lane == m * GR_ROWS + r) mine = total;
        }
    const int m = lane / GR_ROWS, n = n0 + lane % GR_ROWS;
    if (shares > 1) {
        if (lane < MT * GR_ROWS) exchange[warp][lane] = mine;
        __syncthreads();
        if (share == 0 && lane < MT * GR_ROWS)
            for (int s = 1; s < shares; ++s) mine += exchange[warp + s][lane];
    }
    if (share == 0 && m < M && m < MT && n < N) c[(size_t)m * N + n] = mine;
}

}  // namespace

extern "C" int qt_gemm_f32(const float* a, const float* w, float* c, int M, int N, int K, void* stream) {
    QT_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    QT_REQUIRE(K % 4 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)w & 15) == 0, "gemm_f32: rows must be 16-byte aligned (K=%d)", K);
    if (M == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (M <= 8) {
        // as many warps to a weight row as it takes to give every SM two blocks, each with at least one piece of K
        int shares = 1;
        while (shares < GR_WARPS && (long long)N * shares < 2ll * sm_count() * GR_WARPS * GR_ROWS && shares * 2 * 128 <= K) shares *= 2;
        const int per_block = GR_WARPS / shares * GR_ROWS;
        const dim3 grid((N + per_block - 1) / per_block), block(GR_WARPS * 32);
        if (M == 1) launch_kernel(gemm_f32_rows_kernel<1>, grid, block, 0, s, a, w, c, M, N, K, shares);
        else if (M == 2) launch_kernel(gemm_f32_rows_kernel<2>, grid, block, 0, s, a, w, c, M, N, K, shares);
        else if (M <= 4) launch_kernel(gemm_f32_rows_kernel<4>, grid, block, 0, s, a, w, c, M, N, K, shares);
        else launch_kernel(gemm_f32_rows_kernel<8>, grid, block, 0, s, a, w, c, M, N, K, shares);
        QT_CHECK_LAUNCH("gemm_f32");
        return QT_OK;
    }
    if (M <= 16) return launch_tiles<2>(a, w, c, M, N, K, s);
    if (M <= 32) return launch_tiles<4>(a, w, c, M, N, K, s);
    return launch_tiles<8>(a, w, c, M, N, K, s);
}

QT_DEFINE_LAST_ERROR(gemm_f32)
