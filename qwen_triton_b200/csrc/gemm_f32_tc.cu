// C[M, N] = A[M, K] * W[N, K]^T of float operands on the fifth-generation tensor cores, exact in what it multiplies: the 32-bit path's
// products of more than a few rows.
//
// A float of 24 bits is the sum of three bfloat16 numbers (round to nearest, subtract, twice more: 8 + 8 + 8 bits, nothing is lost), and a product of
// two bfloat16 numbers is exact in the float that tcgen05.mma adds it to.  Of the nine products of pieces six are formed: 1.1, 1.2, 2.1, 2.2,
// 1.3, 3.1; the others are below 2^-25 of the operands' product and of either sign.  What could lose bits is the adding: the tensor pipe
// does not round to nearest, so an accumulator takes one K slice of 64 (small products first) and is then added, rounded to nearest, to sums in registers.
//
// A block forms 128 x 128 results.  Sixteen warps load the next slice's floats into registers, split them and store the pieces where the MMAs read
// them, two stages deep: A's in tensor memory, half a row a thread (from shared memory both operands of 128 x 128 x 16 would be 128 bytes a clock, all it
// gives), W's as swizzled tiles.  A's floats come by TMA: a row a thread read straight from memory is 32 lines an instruction, 2,048 cycles a slice.  One thread issues 24 MMAs a slice (1,536 cycles of the tensor pipe), and the sixteen
// warps add a finished slice's accumulator up while the next one is multiplied.  Up to eight blocks of a cluster share K where the tiles do not fill
// the SMs, and add up through distributed shared memory in the order of the ranks.
//
// What bounds it now is the splitting: a slice takes 1.9 us (3,300 cycles), and with one product in the place of six 0.9 of that.
//
// N x K, rows, us before (gemm_f32.cu) / here, L2 flushed ahead of each: 4096 x 1024 64 27 / 21, 549 129 / 64, 4,096 807 / 236; 6144 x 1024 549 184 / 74; 1024 x 3072 549 117 / 39; 4096 x 12288
// 549 1,458 / 512, 4,096 9,940 / 2,290 (180 TFLOP/s); up to 32 rows the FMA pipe's kernels are as fast or faster.
//
// What is exact in float stays so (one number a row, powers of two, whole numbers up to 2^24).  Error against 64 bits over the result's norm, before / here, 64 to 12,288 of K: random signs
// 0.84e-7 to 1.61e-7 / 0.78e-7 to 1.40e-7; operands of one sign 0.40e-7 to 0.63e-7 / 0.86e-7 to 0.98e-7, of which 0.79e-7 is the mean of the large instructions' cuts towards zero.  A factor for that
// mean would round off sums that nothing was cut from; accumulators read back every 32 or 16 of K (0.60e-7 to 0.83e-7, 0.56e-7 to 0.91e-7) cost 10 to 25 % and 35 to 140 % of the time.
//
// Infinities, NaN and numbers that round to an infinite bfloat16 have no such pieces: a block that meets one forms its results again with FMAs.
#include "tc_common.cuh"

using namespace qt;
using namespace qt_tc;

namespace {

constexpr int TILE = 128, BK = 64;                     // rows of either operand a block takes, K elements of a slice
constexpr int WORK_WARPS = 16, MMA_WARP = 16, COPY_WARP = 17, THREADS = 18 * 32;
constexpr int A_STAGES = 3;                            // slices of A as floats, ahead of their splitting
constexpr uint32_t A_HALF_BYTES = TILE * 128, A_STAGE_BYTES = 2 * A_HALF_BYTES;      // [128 rows][32 floats] twice, 128-byte swizzle
constexpr uint32_t PIECE_BYTES = TILE * BK * 2;        // one piece of W: [128 rows][64] bfloat16, 128-byte swizzle
constexpr uint32_t STAGE_BYTES = 3 * PIECE_BYTES;
constexpr int A_COLS = BK / 2;                         // one piece of A in tensor memory: row i in lane i, two elements a column
constexpr uint32_t TMEM_A = 2 * TILE, TMEM_COLS = 512; // two accumulators, two stages of A's pieces
constexpr int UNITS = 4;                               // runs of eight elements a thread splits per slice
constexpr int COLS = 32;                               // results a thread keeps the sums of
constexpr int MOST_RANKS = 8, PARK_ROW = TILE + 4;
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TILE >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
static_assert(TILE * PARK_ROW * 4 <= 2 * STAGE_BYTES, "a block's part of the result is parked in the stages' memory");


struct Params {
    const float* a; const float* w; float* c;
    int M, N, K, ranks, slices_per_rank;
    int* status;
};

__device__ __forceinline__ uint32_t pack_rn(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ float low_of(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float high_of(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ void store16(uint32_t at, const uint32_t (&v)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void store_columns(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                   "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ float4 load4(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float4 peer4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ Params p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t a_floats = base + 2 * STAGE_BYTES;
    // full[2], empty[2], summed[2] (an accumulator is complete), added[2] (and read), arrived[3] (floats of A), taken[3]
    constexpr uint32_t BARS = 2 * STAGE_BYTES + A_STAGES * A_STAGE_BYTES;
    const uint32_t bars = base + BARS, full = bars, empty = bars + 16, summed = bars + 32, added = bars + 48, arrived = bars + 64, taken = arrived + 8 * A_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + BARS + 64 + 16 * A_STAGES);
    int* odd = reinterpret_cast<int*>(tmem_slot + 1);                       // a number without pieces was met

    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = p.ranks > 1 ? (int)cluster_ctarank() : 0;
    const int n0 = (int)(blockIdx.x / (unsigned)p.ranks) * TILE, m0 = blockIdx.y * TILE;
    const int k_begin = rank * p.slices_per_rank * BK, k_end = min(p.K, k_begin + p.slices_per_rank * BK);
    const int slices = (k_end - k_begin + BK - 1) / BK;                     // >= 1: the host sizes the ranks so
    int* status = p.status;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(full + 8 * s, WORK_WARPS); mbar_init(empty + 8 * s, 1);
            mbar_init(summed + 8 * s, 1); mbar_init(added + 8 * s, WORK_WARPS);
        }
        for (int s = 0; s < A_STAGES; ++s) { mbar_init(arrived + 8 * s, 1); mbar_init(taken + 8 * s, WORK_WARPS / 2); }
        *odd = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == COPY_WARP) {
        if (lane == 0) {
            prefetch_tensor_map(&map_a);
            pdl_wait();
            for (int i = 0, s = 0, turn = 0; i < slices; ++i) {
                if (!mbar_wait(taken + 8 * s, (uint32_t)turn ^ 1u, status, 1)) break;
                mbar_expect_tx(arrived + 8 * s, A_STAGE_BYTES);
                for (int h = 0; h < 2; ++h)                                 // the map counts 16-bit elements, two a float
                    tma_load_2d(a_floats + s * A_STAGE_BYTES + h * A_HALF_BYTES, &map_a, arrived + 8 * s, 2 * (k_begin + i * BK + 32 * h), m0);
                if (++s == A_STAGES) { s = 0; turn ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == MMA_WARP) {
        if (lane == 0) {
            const uint64_t desc0 = operand_desc(base);
            for (int i = 0; i < slices; ++i) {
                const int s = i & 1;
                const uint32_t turn = (uint32_t)(i >> 1) & 1u;
                if (!mbar_wait(full + 8 * s, turn, status, 2)) break;
                if (!mbar_wait(added + 8 * s, turn ^ 1u, status, 4)) break;
                tc_fence_after();
                const uint64_t w0 = desc0 + (uint64_t)(s * (STAGE_BYTES >> 4));
                const uint32_t acc = tmem_base + s * TILE, a0 = tmem_base + TMEM_A + s * 3 * A_COLS;
                auto product = [&](int x, int y, bool first) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma_bf16_a_tmem(acc, a0 + x * A_COLS + 8 * k, w0 + y * (PIECE_BYTES >> 4) + 2 * k, IDESC, first && k == 0 ? 0u : 1u);
                };
                product(0, 2, true); product(2, 0, false); product(1, 1, false);
                product(0, 1, false); product(1, 0, false); product(0, 0, false);
                umma_commit(empty + 8 * s);
                umma_commit(summed + 8 * s);
            }
        }
        __syncwarp();
    } else {
        // Warps 0 to 7: a thread holds half a row of A's slice (warps 0 to 3 the first), unit u is its elements 8 u .. 8 u + 7.  Warps 8 to 15: unit u
        // of a thread is eight neighbouring elements of row 32 u + (thread / 8) of W's.
        const bool of_a = warp < 8;
        const int chunk = threadIdx.x & 7, w_row = (threadIdx.x & 255) >> 3, a_row = threadIdx.x & 127, a_half = (warp >> 2) & 1;
        float v[UNITS][8];
        auto put = [&](int u, const float4& x, const float4& y) {
            v[u][0] = x.x; v[u][1] = x.y; v[u][2] = x.z; v[u][3] = x.w; v[u][4] = y.x; v[u][5] = y.y; v[u][6] = y.z; v[u][7] = y.w;
        };
        auto ask = [&](int u, int slice) {                                  // of W
            const int at = n0 + 32 * u + w_row, k = k_begin + slice * BK + 8 * chunk;
            const float* from = p.w + (size_t)at * p.K + k;
            const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
            put(u, at < p.N && k < k_end ? load4(from) : none, at < p.N && k + 4 < k_end ? load4(from + 4) : none);              // K is a multiple of 4
        };
        float sums[COLS];                                                   // row 32 (warp % 4) + lane, columns 32 (warp / 4) ..
#pragma unroll
        for (int j = 0; j < COLS; ++j) sums[j] = 0.f;
        const uint32_t mine = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(warp >> 2) * COLS;
        auto add = [&](int i) {
            const int s = i & 1;
            if (!mbar_wait(summed + 8 * s, (uint32_t)(i >> 1) & 1u, status, 3)) return false;
            tc_fence_after();
#pragma unroll
            for (int part = 0; part < COLS / 16; ++part) {
                uint32_t x[16];
                tmem_load16(mine + s * TILE + 16 * part, x);
#pragma unroll
                for (int j = 0; j < 16; ++j) sums[16 * part + j] += __uint_as_float(x[j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(added + 8 * s);
            return true;
        };
        if (!of_a) {                                                        // weights depend on no earlier kernel
#pragma unroll
            for (int u = 0; u < UNITS; ++u) ask(u, 0);
        }
        pdl_wait();                                                         // the result may still be read by one
        int a_stage = 0;
        uint32_t a_turn = 0;
        float none = 0.f;                                                   // stays 0 while every number has its pieces
        // the next piece of a unit: its numbers rounded, and what is left of them
        auto piece_of = [&](int u, uint32_t* h, bool first, bool last) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float& lo = v[u][2 * j];
                float& hi = v[u][2 * j + 1];
                h[j] = pack_rn(lo, hi);
                if (last) continue;
                lo -= low_of(h[j]); hi -= high_of(h[j]);
                if (first) { none = fmaf(0.f, lo, none); none = fmaf(0.f, hi, none); }
            }
        };
        bool ok = true;
        for (int i = 0; i < slices && ok; ++i) {
            const int s = i & 1;
            ok = mbar_wait(empty + 8 * s, ((uint32_t)(i >> 1) & 1u) ^ 1u, status, 1);
            if (!ok) break;
            if (of_a) {
                ok = mbar_wait(arrived + 8 * a_stage, a_turn, status, 3);
                if (!ok) break;
                const uint8_t* floats = smem + 2 * STAGE_BYTES + a_stage * A_STAGE_BYTES + a_half * A_HALF_BYTES + a_row * 128;
#pragma unroll
                for (int u = 0; u < UNITS; ++u)                             // a row's 16-byte pieces lie in the swizzle's order
                    put(u, *reinterpret_cast<const float4*>(floats + (((2 * u) ^ (a_row & 7)) << 4)), *reinterpret_cast<const float4*>(floats + (((2 * u + 1) ^ (a_row & 7)) << 4)));
                __syncwarp();
                if (lane == 0) mbar_arrive(taken + 8 * a_stage);
                if (++a_stage == A_STAGES) { a_stage = 0; a_turn ^= 1u; }
                tc_fence_after();
#pragma unroll
                for (int piece = 0; piece < 3; ++piece) {
                    uint32_t h[16];
#pragma unroll
                    for (int u = 0; u < UNITS; ++u) {
                        piece_of(u, h + 4 * u, piece == 0, piece == 2);
                    }
                    store_columns(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + TMEM_A + (s * 3 + piece) * A_COLS + 16 * a_half, h);
                }
                tmem_wait_st();
                tc_fence_before();
            } else {
#pragma unroll
                for (int u = 0; u < UNITS; ++u) {
                    uint32_t h[3][4];
#pragma unroll
                    for (int piece = 0; piece < 3; ++piece) piece_of(u, h[piece], piece == 0, piece == 2);
                    if (i + 1 < slices) ask(u, i + 1);
                    const int row = 32 * u + w_row;
                    const uint32_t at = base + s * STAGE_BYTES + (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4));
#pragma unroll
                    for (int piece = 0; piece < 3; ++piece) store16(at + piece * PIECE_BYTES, h[piece]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(full + 8 * s);
            if (i > 0) ok = add(i - 1);
        }
        if (ok) ok = add(slices - 1);
        if (none != 0.f) atomicOr(odd, 1);                                  // NaN
        asm volatile("bar.sync 1, %0;" ::"n"(WORK_WARPS * 32) : "memory");
        const int row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * COLS, m = m0 + row;
        if (*(volatile int*)odd != 0) {
            const float* x = p.a + (size_t)min(m, p.M - 1) * p.K;
#pragma unroll 1
            for (int j0 = 0; j0 < COLS; ++j0) {
                const float* y = p.w + (size_t)min(n0 + col0 + j0, p.N - 1) * p.K;
                float sum = 0.f;
                for (int k = k_begin; k < k_end; ++k) sum = fmaf(x[k], y[k], sum);
#pragma unroll
                for (int j = 0; j < COLS; ++j) if (j == j0) sums[j] = sum;    // registers have no index
            }
        }
        if (p.ranks > 1) {                                                  // every MMA has read the stages: they are free
            float* park = reinterpret_cast<float*>(smem) + row * PARK_ROW + col0;
#pragma unroll
            for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4*>(park + j) = make_float4(sums[j], sums[j + 1], sums[j + 2], sums[j + 3]);
        } else if (m < p.M && ok) {
            float* to = p.c + (size_t)m * p.N + n0 + col0;
#pragma unroll
            for (int j = 0; j < COLS; j += 4) {
                if (n0 + col0 + j + 3 < p.N && (p.N & 3) == 0) *reinterpret_cast<float4*>(to + j) = make_float4(sums[j], sums[j + 1], sums[j + 2], sums[j + 3]);
                else
#pragma unroll
                    for (int e = 0; e < 4; ++e) if (n0 + col0 + j + e < p.N) to[j + e] = sums[j + e];
            }
        }
    }
    // The tensor memory goes back before a block waits for its peers: one that waits for tensor memory then waits for none that waits for it.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (*(volatile int*)status != 0) {                                      // a wait gave up: let MMAs in flight finish first
        const unsigned long long t0 = global_timer();
        while (global_timer() - t0 < 2000000ull) __nanosleep(1000);
    }
    if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    if (p.ranks > 1) {
        cluster_sync_all();
        // a block finishes every ranks-th row: a warp a row, four columns a lane
        if (*(volatile int*)status == 0 && warp < WORK_WARPS) {
            for (int row = rank + p.ranks * warp; row < TILE && m0 + row < p.M; row += p.ranks * WORK_WARPS) {
                const uint32_t off = (uint32_t)(row * PARK_ROW + 4 * lane) * 4u;
                float4 part[MOST_RANKS];
#pragma unroll
                for (int r = 0; r < MOST_RANKS; ++r) if (r < p.ranks) part[r] = peer4(map_to_cta(base, (uint32_t)r) + off);
                float4 sum = part[0];
#pragma unroll
                for (int r = 1; r < MOST_RANKS; ++r) if (r < p.ranks) { sum.x += part[r].x; sum.y += part[r].y; sum.z += part[r].z; sum.w += part[r].w; }
                const int n = n0 + 4 * lane;
                float* to = p.c + (size_t)(m0 + row) * p.N + n;
                if (n + 3 < p.N && (p.N & 3) == 0) *reinterpret_cast<float4*>(to) = sum;
                else {
                    const float e[4] = {sum.x, sum.y, sum.z, sum.w};
                    for (int j = 0; j < 4; ++j) if (n + j < p.N) to[j] = e[j];
                }
            }
        }
        cluster_sync_all();                                                 // nobody leaves while its sums are read
    }
}

}  // namespace

// a [M, K], w [N, K], c [M, N] float; K a multiple of 4, a and w 16-byte aligned, c too where N is a multiple of 4; `status` as in qt_gemm_tc.
extern "C" int qt_gemm_f32_tc(const float* a, const float* w, float* c, int M, int N, int K, int* status, void* stream) {
    QT_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32_tc: bad sizes M=%d N=%d K=%d", M, N, K);
    QT_REQUIRE(K % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0 && (N % 4 != 0 || ((uintptr_t)c & 15) == 0), "gemm_f32_tc: rows must be 16-byte aligned (K=%d)", K);
    QT_REQUIRE(status != nullptr, "gemm_f32_tc: a status word is required");
    const int n_tiles = (N + TILE - 1) / TILE, m_tiles = (M + TILE - 1) / TILE, slices = (K + BK - 1) / BK;
    QT_REQUIRE(m_tiles <= 65535, "gemm_f32_tc: M=%d is too many rows", M);
    if (M == 0) return QT_OK;
    // Waves of blocks, one to an SM, times a block's slices and what it does besides (about two slices' time, three with peers).
    const int sms = sm_count();
    int ranks = 1, per = slices;
    long long best = -1;
    for (int r = 1; r <= MOST_RANKS; ++r) {
        const int each = (slices + r - 1) / r;
        if ((r - 1) * each >= slices) continue;                             // a rank without slices
        const long long cost = (((long long)n_tiles * m_tiles * r + sms - 1) / sms) * (each + (r > 1 ? 3 : 2));
        if (best < 0 || cost < best) { best = cost; ranks = r; per = each; }
    }
    CUtensorMap map_a;
    const int rc = tensor_map(&map_a, a, (uint64_t)M, 2 * (uint64_t)K, TILE);     // floats as pairs of 16-bit elements: only copied
    if (rc) return rc;
    const Params p{a, w, c, M, N, K, ranks, per, status};
    const size_t smem = 2 * STAGE_BYTES + A_STAGES * A_STAGE_BYTES + 1024 + 64 + 16 * A_STAGES + 16;
    const cudaError_t raised = raise_shared<gemm_f32_tc_kernel>(227 * 1024);
    if (raised != cudaSuccess) QT_FAIL(QT_ERR_LAUNCH, "gemm_f32_tc: cannot raise shared memory: %s", cudaGetErrorString(raised));
    launch_kernel_cluster(gemm_f32_tc_kernel, dim3((unsigned)(n_tiles * ranks), (unsigned)m_tiles), dim3(THREADS), smem, (cudaStream_t)stream, (unsigned)ranks, map_a, p);
    QT_CHECK_LAUNCH("gemm_f32_tc");
    return QT_OK;
}

QT_DEFINE_LAST_ERROR(gemm_f32_tc)
