// bfloat16 matrix product for up to 16 tokens (a decode step of a few sequences) with what follows it done in the same launch.
//
// Y[M, N] = X[M, K] * W[N, K]^T with the epilogues of fused_epilogue.cuh.  Such a product is bound by reading the weight and, on a
// small model, by the chain of launches it stands in: each waits for the one before it, and what it does between that moment and its
// own end is the step's time.  So the chain is kept as short as it can be:
//
//   * A block holds 16 or 32 rows of W whole: its warps share K (64 elements a warp and turn, interleaved) and add up through shared
//     memory.  No cluster, no partial sums in memory, no TMEM, no tensor maps (gemm_fused.cu has all of these between the arrival of X
//     and its result); only q/k/v, whose heads span 128 rows, is a cluster of four blocks that hand each other finished sums.
//   * The weight goes from memory into the registers that mma.sync reads (few_tokens.cuh).  Every warp asks for its first turns ahead of
//     the wait for the kernel that produces X: at the small shapes that is all of W.
//   * X comes from L2 the same way.  With 8 tokens on the instruction's N nothing is padded up to 16 as tcgen05 would, and the tensor
//     pipe is idle either way: the weight arrives at 22 bytes a clock and SM.
//
// A step of the 0.6B shape (28 layers of q/k/v, o, gate/up and down), before (gemm_fused.cu) / with this kernel: one sequence 832 / 570-590 us, two 876 / 617, eight
// 1,005 / 718, sixteen 1,019 / 797.
//
// Counterparts in luozoupi/Qwen-Triton: kernels/matmul.py:52-97, kernels/rmsnorm.py:100-133, kernels/residual_add.py:50-60,
// kernels/swiglu.py:84-92, kernels/rope.py:99-120, kernels/cache.py:71-98 (one launch each, or two).
#include "few_tokens.cuh"
#include "fused_epilogue.cuh"

using namespace qt;
using namespace qt_epi;
using namespace qt_few;

namespace {

constexpr int QKV_BLOCKS = 4;              // blocks of 32 rows that hold a 128-row group of heads

// RT: tiles of 16 weight rows of a block; NT: tiles of 8 tokens; DEPTH: turns whose operands are in flight
template <int EPI, int RT, int NT, int WARPS, int DEPTH>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS) gemm_few_kernel(const __nv_bfloat16* w, const __nv_bfloat16* x, int K, const __grid_constant__ EpilogueParams ep) {
    constexpr int W = 16 * RT, LANES = W / 4, TOKENS = 8 * NT, STEP = 4 * PIECE;
    constexpr int FINISHERS = TOKENS * LANES / 32;                  // warps that add the others' sums up
    static_assert(EPI != EPI_QKV || W * QKV_BLOCKS == TILE, "a cluster holds the 128 rows that the heads' epilogue takes");
    static_assert(FINISHERS <= WARPS, "");
    __shared__ __align__(16) float sums[WARPS][TOKENS][W + 4];      // 4 more: a quad's tokens lie in different banks
    __shared__ __align__(16) float heads[EPI == EPI_QKV ? TOKENS / QKV_BLOCKS : 1][EPI == EPI_QKV ? TILE : 4];

    pdl_launch_dependents();
    if (EPI == EPI_QKV) cluster_arrive_started();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int w_tile = blockIdx.x, n0 = w_tile * W;
    const int turns = (K + STEP - 1) / STEP;
    const int mine = (turns - warp + WARPS - 1) / WARPS;            // this warp's: warp, warp + WARPS, ...

    const __nv_bfloat16* row[RT][2];                                // rows beyond N repeat the last one; their sums are not stored
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h) row[r][h] = w + (size_t)min(n0 + 16 * r + 8 * h + g, ep.N - 1) * K;
    Line a[DEPTH][RT][2], b[DEPTH][NT];
    auto ask_weight = [&](int slot, int i) {
        const int k = (warp + i * WARPS) * STEP + PIECE * t;
        const bool inside = k < K;                                  // K is a multiple of 16: a lane's elements are all in or out
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (inside) a[slot][r][h] = load_weight(row[r][h] + k);
                else a[slot][r][h] = Line{};
            }
    };
    auto ask_rows = [&](int slot, int i) {
        const int k = (warp + i * WARPS) * STEP + PIECE * t;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            if (k < K && 8 * n + g < ep.M) b[slot][n] = load_rows(x + (size_t)(8 * n + g) * K + k);
            else b[slot][n] = Line{};
        }
    };
#pragma unroll
    for (int u = 0; u < DEPTH; ++u)
        if (u < mine) ask_weight(u, u);
    pdl_wait();
#pragma unroll
    for (int u = 0; u < DEPTH; ++u)
        if (u < mine) ask_rows(u, u);

    // the epilogue's operands, under the product: of (token, lane) pairs of this block, or, for heads, of a whole token of the cluster's 128 rows
    Operands ops;
    const int rank = EPI == EPI_QKV ? w_tile % QKV_BLOCKS : 0, head_tile = w_tile / QKV_BLOCKS;
    const int token = (warp * 32 + lane) / LANES, l = lane % LANES, whole = rank + QKV_BLOCKS * warp;
    if (EPI == EPI_QKV) {
        if (whole < ep.M) ops = load_operands<EPI, TILE>(ep, whole, head_tile * TILE, lane);
    } else if (warp < FINISHERS) {
        ops = load_operands<EPI, W>(ep, min(token, ep.M - 1), n0, l);
    }

    constexpr int CHAINS = RT * NT == 1 ? 2 : 1;                    // sums that do not wait for one another
    float c[RT][NT][CHAINS][4] = {};
    for (int i0 = 0; i0 < mine; i0 += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
            if (i0 + u >= mine) break;
#pragma unroll
            for (int j = 0; j < PIECE / 4; ++j)
#pragma unroll
                for (int r = 0; r < RT; ++r)
#pragma unroll
                    for (int n = 0; n < NT; ++n)
                        mma_16x8x16(c[r][n][j % CHAINS], a[u][r][0].r[2 * j], a[u][r][1].r[2 * j], a[u][r][0].r[2 * j + 1], a[u][r][1].r[2 * j + 1],
                                    b[u][n].r[2 * j], b[u][n].r[2 * j + 1]);
            if (i0 + u + DEPTH < mine) { ask_weight(u, i0 + u + DEPTH); ask_rows(u, i0 + u + DEPTH); }
        }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float v = c[r][n][0][e];
                if (CHAINS == 2) v += c[r][n][CHAINS - 1][e];
                sums[warp][8 * n + 2 * t + (e & 1)][16 * r + g + 8 * (e >> 1)] = v;
            }
    __syncthreads();

    // every warp's sums in the order of the warps
    const bool live = token < ep.M;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (warp < FINISHERS) {
        if (EPI == EPI_SWIGLU) {
            const int at = swiglu_gate_row(l);
            float2 gate = make_float2(0.f, 0.f), up = make_float2(0.f, 0.f);
#pragma unroll
            for (int s = 0; s < WARPS; ++s) {
                const float2 gs = *reinterpret_cast<const float2*>(&sums[s][token][at]), us = *reinterpret_cast<const float2*>(&sums[s][token][at + 16]);
                gate.x += gs.x; gate.y += gs.y; up.x += us.x; up.y += us.y;
            }
            finish_swiglu<W>(ep, ops, gate, up, token, w_tile, l, live);
        } else {
#pragma unroll
            for (int s = 0; s < WARPS; ++s) {
                const float4 part = *reinterpret_cast<const float4*>(&sums[s][token][4 * l]);
                v.x += part.x; v.y += part.y; v.z += part.z; v.w += part.w;
            }
            if (EPI != EPI_QKV) finish<EPI, W>(ep, ops, v, token, w_tile, l, live);
        }
    }
    if (EPI == EPI_QKV) {
        cluster_wait_started();
        if (warp < FINISHERS && live) cluster_store4(&heads[token / QKV_BLOCKS][rank * W + 4 * l], (uint32_t)(token % QKV_BLOCKS), v);
        cluster_barrier();
        if (whole < ep.M) finish<EPI, TILE>(ep, ops, *reinterpret_cast<const float4*>(&heads[warp][4 * lane]), whole, head_tile, lane);
    }
}

template <int EPI, int RT, int NT, int WARPS, int DEPTH>
int launch(const void* w, const void* x, int K, const EpilogueParams& e, cudaStream_t stream) {
    const dim3 block(WARPS * 32);
    if (EPI == EPI_QKV)
        launch_kernel_cluster(gemm_few_kernel<EPI, RT, NT, WARPS, DEPTH>, dim3((unsigned)((e.N + TILE - 1) / TILE * QKV_BLOCKS)), block, 0, stream, (unsigned)QKV_BLOCKS,
                              (const __nv_bfloat16*)w, (const __nv_bfloat16*)x, K, e);
    else
        launch_kernel(gemm_few_kernel<EPI, RT, NT, WARPS, DEPTH>, dim3((unsigned)((e.N + 16 * RT - 1) / (16 * RT))), block, 0, stream,
                      (const __nv_bfloat16*)w, (const __nv_bfloat16*)x, K, e);
    QT_CHECK_LAUNCH("gemm_few");
    return QT_OK;
}

template <int EPI, int RT>
int dispatch(const void* w, const void* x, int K, int warps, const EpilogueParams& e, cudaStream_t stream) {
    constexpr int DEPTH = RT == 1 ? 4 : 2, DEPTH2 = RT == 1 ? 2 : 1;
    if (e.M <= 8) {
        if (warps == 16) return launch<EPI, RT, 1, 16, DEPTH>(w, x, K, e, stream);
        return launch<EPI, RT, 1, 8, DEPTH>(w, x, K, e, stream);
    }
    if (warps == 16) return launch<EPI, RT, 2, 16, DEPTH2>(w, x, K, e, stream);
    return launch<EPI, RT, 2, 8, DEPTH2>(w, x, K, e, stream);
}

}  // namespace

// x [M, K] bfloat16 (M up to 16), w [N, K] bfloat16, K a multiple of 16 and both 32-byte aligned.  `epilogue` picks what is done with
// the product and which of the pointers are read, as in qt_gemm_fused; `block_rows` (16, or 32 as q/k/v and the gate always take) is
// how many rows of w a block holds, and the width of the tiles whose sums of squares sq_out receives; `warps` (8 or 16) share K.  The engine takes 16 rows with 16
// warps, and 32 rows for heads and gates (Linear.few_plan); 16 rows with 8 warps, and 32 with the other epilogues, are for other callers.
extern "C" int qt_gemm_few(const void* x, const void* w, int M, int N, int K, int block_rows, int warps, int epilogue,
                           const float* sq_in, int sq_tiles, int norm_width, float eps, const float* bias,
                           void* out, int out_dtype, int act, float limit,
                           float* residual, const float* norm_w, void* xw, float* sq_out,
                           void* q_out, void* k_cache, void* v_cache, const int* token_seq, const int* token_pos,
                           const int* block_table, int max_blocks, const float* q_w, const float* k_w, float qk_eps,
                           const float* cos_sin, int rotary_dim, int max_pos, int nq, int nkv, int d, int page_tokens,
                           int ring_tokens, int write_kv, int interleaved, void* stream) {
    QT_REQUIRE(M > 0 && M <= 16 && N > 0 && K > 0, "gemm_few: bad sizes M=%d N=%d K=%d (up to 16 tokens)", M, N, K);
    QT_REQUIRE(K % 16 == 0 && (uintptr_t)x % 32 == 0 && (uintptr_t)w % 32 == 0, "gemm_few: rows must start on 32-byte boundaries (K=%d)", K);
    QT_REQUIRE(warps == 8 || warps == 16, "gemm_few: %d warps (8 or 16)", warps);
    QT_REQUIRE(block_rows == 32 || (block_rows == 16 && epilogue != EPI_SWIGLU && epilogue != EPI_QKV), "gemm_few: blocks of %d rows for epilogue %d", block_rows, epilogue);
    EpilogueParams e = {};
    e.M = M; e.N = N;
    e.sq_in = sq_in; e.sq_tiles = sq_tiles; e.inv_hidden = norm_width > 0 ? 1.f / (float)norm_width : 0.f; e.eps = eps;
    e.bias = bias;
    e.out = out; e.out_is_float = out_dtype == QT_F32; e.act = act; e.limit = limit;
    e.residual = residual; e.norm_w = norm_w; e.xw = (__nv_bfloat16*)xw; e.sq_out = sq_out;
    e.q_out = (__nv_bfloat16*)q_out; e.k_cache = (__nv_bfloat16*)k_cache; e.v_cache = (__nv_bfloat16*)v_cache;
    e.token_seq = token_seq; e.token_pos = token_pos; e.block_table = block_table; e.max_blocks = max_blocks;
    e.q_w = q_w; e.k_w = k_w; e.qk_eps = qk_eps; e.cos_sin = cos_sin; e.rotary_dim = rotary_dim; e.max_pos = max_pos;
    e.nq = nq; e.nkv = nkv; e.d = d; e.page_tokens = page_tokens; e.ring_tokens = ring_tokens; e.write_kv = write_kv; e.interleaved = interleaved;
    e.activated = epilogue == EPI_ACTIVATED;
    if (e.activated) epilogue = EPI_STORE;
    const int rc = check_epilogue("gemm_few", epilogue, e, out_dtype);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    switch (epilogue) {
        case EPI_STORE: return block_rows == 16 ? dispatch<EPI_STORE, 1>(w, x, K, warps, e, s) : dispatch<EPI_STORE, 2>(w, x, K, warps, e, s);
        case EPI_RESIDUAL: return block_rows == 16 ? dispatch<EPI_RESIDUAL, 1>(w, x, K, warps, e, s) : dispatch<EPI_RESIDUAL, 2>(w, x, K, warps, e, s);
        case EPI_SWIGLU: return dispatch<EPI_SWIGLU, 2>(w, x, K, warps, e, s);
        default: return dispatch<EPI_QKV, 2>(w, x, K, warps, e, s);
    }
}

QT_DEFINE_LAST_ERROR(gemm_few)
