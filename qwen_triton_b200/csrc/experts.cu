// Feed-forward experts chosen per token by a table: each token runs the `top` experts that the table's row of its
// token id names, out[t] = sum_k weight_k * W_down[e_k] act(W_up[e_k] x[t]).  The routing is read on the device
// (token ids and table are device arrays), so a step with these kernels has the same launches whatever the tokens
// are and can be captured in a CUDA graph.
//
// Two forms.  Few tokens (a decode step): one pass of matrix-vector products per (token, expert) pair, the expert's
// rows streamed once per pair.  Many tokens: the pairs are ordered by expert on the device (count, offsets, scatter;
// every expert's run padded to whole tiles of rows), and the two products run tile by tile, a tile's rows all of one
// expert, so that an expert's weights are read once per tile instead of once per pair.
//
// The same kernels serve experts chosen by a learned router: without token ids the "table" is read by token (row t
// holds the experts that a router kernel chose for token t), every pair has a weight of its own (`pair_weights`),
// an expert may be gated (its first matrix holds [gate; up] rows, mid = gate(g, u)), and a further term
// row_scale[t] * base[t] (a shared expert behind a gate of one number per token) may be added to the sum.
#include "common.cuh"
#include "few_tokens.cuh"

#include <math.h>

#include <type_traits>

using namespace qt;

// ----------------------------------------------------------------------------- few tokens: per pair
constexpr int EV_WARPS = 8;
constexpr int EV_FEATS = 4;        // output features per warp and pass

struct ExpertParams {
    const void* x;            // [T, width] normed rows
    const int* token_ids;     // [T]
    const int* table;         // [vocab, top]
    const void* up;           // [E, ff, width]
    const void* down;         // [E, width, ff]
    void* mid;                // [T * top, ff] activations
    float* out;               // [T, width] float
    int n_tokens, vocab, top, experts, width, ff, act;
    float pair_weight;        // weight of every chosen expert (1 / top for an unweighted mean)
    const float* pair_weights;  // [T, top] a weight per pair instead, or null
    int gated; float limit;     // up holds [E, 2 ff, width]: ff gate rows, then ff up rows; mid = gated_value(g, u, act, limit)
    const float* base; int base_splits; size_t base_stride;   // [splits, T, width] float added to out, times row_scale[t]; or null
    const float* row_scale;     // [T] or null (1)
    const float* in_weights;    // [T, top] or null: a pair's expert reads its token's row times this (a weight on the input, not the output)
};

__device__ __forceinline__ int expert_of(const ExpertParams& p, int t, int k) {
    int id = p.token_ids ? p.token_ids[t] : t;            // no ids: the table's row t is token t's
    id = id < 0 ? 0 : (id >= p.vocab ? p.vocab - 1 : id);
    int e = p.table[(size_t)id * p.top + k];
    return e < 0 ? 0 : (e >= p.experts ? p.experts - 1 : e);          // never read outside the weights
}

// EV_FEATS dot products of consecutive weight rows (`stride` apart, `n` elements each) with a vector in shared memory,
// summed over the warp, for rows that do not lie on 16-byte boundaries.
template <typename T>
__device__ __forceinline__ void warp_dots(const T* __restrict__ w, size_t stride, int rows, int n, const float* __restrict__ xs, int lane,
                                          float (&acc)[EV_FEATS]) {
#pragma unroll
    for (int j = 0; j < EV_FEATS; ++j) acc[j] = 0.f;
    for (int i = lane; i < n; i += 32) {
        const float xv = xs[i];
#pragma unroll
        for (int j = 0; j < EV_FEATS; ++j)
            if (j < rows) acc[j] += to_float(w[(size_t)j * stride + i]) * xv;
    }
#pragma unroll
    for (int j = 0; j < EV_FEATS; ++j) acc[j] = warp_sum(acc[j]);
}

// mid[pair, f] = act(W_up[e][f, :] . x[t, :]).  grid (pairs, feature blocks); x[t] in shared memory as float.
template <typename T>
__global__ void __launch_bounds__(EV_WARPS * 32) expert_up_kernel(const ExpertParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float xs[];
    const int pair = blockIdx.x, t = pair / p.top, k = pair % p.top;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* x = (const T*)p.x + (size_t)t * p.width;
    const float in_weight = p.in_weights ? p.in_weights[pair] : 1.f;
    for (int i = threadIdx.x; i < p.width; i += blockDim.x) xs[i] = to_float(x[i]) * in_weight;
    __syncthreads();
    const int e = expert_of(p, t, k);
    const T* w = (const T*)p.up + (size_t)e * (p.gated ? 2 : 1) * p.ff * p.width;
    T* mid = (T*)p.mid + (size_t)pair * p.ff;
    const int f0 = (blockIdx.y * EV_WARPS + warp) * EV_FEATS;
    if (f0 >= p.ff) return;
    float acc[EV_FEATS];
    warp_dots<T>(w + (size_t)f0 * p.width, (size_t)p.width, p.ff - f0, p.width, xs, lane, acc);
    if (p.gated) {
        float up[EV_FEATS];
        warp_dots<T>(w + (size_t)(p.ff + f0) * p.width, (size_t)p.width, p.ff - f0, p.width, xs, lane, up);
#pragma unroll
        for (int j = 0; j < EV_FEATS; ++j)
            if (lane == 0 && f0 + j < p.ff) mid[f0 + j] = from_float<T>(gated_value<false>(acc[j], up[j], p.act, p.limit));
        return;
    }
#pragma unroll
    for (int j = 0; j < EV_FEATS; ++j)
        if (lane == 0 && f0 + j < p.ff) mid[f0 + j] = from_float<T>(gate_activation<false>(acc[j], p.act));
}

// The result of token t, column c: the weighted sum over its experts, the further term, into out.
__device__ __forceinline__ void expert_put(const ExpertParams& p, int t, int c, float total) {
    const size_t at = (size_t)t * p.width + c;
    float y = p.pair_weights ? total : total * p.pair_weight;
    if (p.base) y += (p.row_scale ? p.row_scale[t] : 1.f) * load_sum(p.base, at, p.base_splits, p.base_stride);
    p.out[at] = y;
}

// out[t, c] = pair_weight * sum_k W_down[e_k][c, :] . mid[t * top + k, :].  grid (tokens, column blocks).
template <typename T>
__global__ void __launch_bounds__(EV_WARPS * 32) expert_down_kernel(const ExpertParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float ms[];                 // [top, ff]
    const int t = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* mid = (const T*)p.mid + (size_t)t * p.top * p.ff;
    for (int i = threadIdx.x; i < p.top * p.ff; i += blockDim.x) ms[i] = to_float(mid[i]);
    __syncthreads();
    const int c0 = (blockIdx.y * EV_WARPS + warp) * EV_FEATS;
    if (c0 >= p.width) return;
    float total[EV_FEATS];
#pragma unroll
    for (int j = 0; j < EV_FEATS; ++j) total[j] = 0.f;
    for (int k = 0; k < p.top; ++k) {                      // in the order of the table's row
        const int e = expert_of(p, t, k);
        const T* w = (const T*)p.down + (size_t)e * p.width * p.ff;
        float acc[EV_FEATS];
        warp_dots<T>(w + (size_t)c0 * p.ff, (size_t)p.ff, p.width - c0, p.ff, ms + k * p.ff, lane, acc);
        const float weight = p.pair_weights ? p.pair_weights[(size_t)t * p.top + k] : 1.f;
#pragma unroll
        for (int j = 0; j < EV_FEATS; ++j) total[j] += acc[j] * weight;
    }
#pragma unroll
    for (int j = 0; j < EV_FEATS; ++j)
        if (lane == 0 && c0 + j < p.width) expert_put(p, t, c0 + j, total[j]);
}

// The same two passes for rows that lie on 16-byte boundaries (width and ff multiples of 8).  Bound by the experts' bytes, if enough of
// them are asked for at once: which expert it is is known only when the router is done, so nothing can be fetched ahead, and a
// warp that walks its rows 16 bytes a lane and turn waits out the memory once per turn.  A warp takes FEATS features (gate and up
// rows of each together), a lane asks for EV_BYTES of weights before it uses the first, and the rows of x and mid are read where
// they lie (a block that stages them makes every weight wait for two more trips and a barrier).  FEATS falls from 4 to 1 with the
// pairs, so that one token's experts still spread over the machine.
// Both passes, weights not in L2, before / now: one token of 2 experts of 1,024 x 2,048 33 / 15.5 us, of one of 2,048 x 1,024 26 / 13 us,
// 8 tokens of one of 8 such experts 30 / 23.6 us, 16 tokens of 2 of 16 experts of 1,024 x 2,048 69 / 61 us.
constexpr int EV_BYTES = 256;

template <typename T> struct Eight { uint4 raw[sizeof(T) / 2]; };
template <typename T> __device__ __forceinline__ Eight<T> load_weights(const T* p) {        // read once: past L1
    Eight<T> r;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 2); ++i)
        asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r.raw[i].x), "=r"(r.raw[i].y), "=r"(r.raw[i].z), "=r"(r.raw[i].w) : "l"(reinterpret_cast<const uint4*>(p) + i));
    return r;
}
template <typename T> __device__ __forceinline__ Eight<T> load_eight(const T* p) {
    Eight<T> r;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 2); ++i) r.raw[i] = reinterpret_cast<const uint4*>(p)[i];
    return r;
}
__device__ __forceinline__ void floats_of(const Eight<float>& r, float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        v[4 * i] = __uint_as_float(r.raw[i].x); v[4 * i + 1] = __uint_as_float(r.raw[i].y);
        v[4 * i + 2] = __uint_as_float(r.raw[i].z); v[4 * i + 3] = __uint_as_float(r.raw[i].w);
    }
}
__device__ __forceinline__ void floats_of(const Eight<__nv_bfloat16>& r, float (&v)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r.raw[0]);
#pragma unroll
    for (int j = 0; j < 4; ++j) { v[2 * j] = __low2float(h[j]); v[2 * j + 1] = __high2float(h[j]); }
}

// acc[j] += this lane's part of row[j] . (x times factor), n elements.
template <typename T, int ROWS>
__device__ __forceinline__ void lane_dots(const T* const (&row)[ROWS], const T* x, float factor, int n, int lane, float (&acc)[ROWS]) {
    constexpr int AT_ONCE = EV_BYTES / (ROWS * 8 * (int)sizeof(T)), TURNS = AT_ONCE < 1 ? 1 : AT_ONCE > 8 ? 8 : AT_ONCE;
    for (int i0 = lane * 8; i0 < n; i0 += 256 * TURNS) {
        Eight<T> w[TURNS][ROWS], v[TURNS];
#pragma unroll
        for (int u = 0; u < TURNS; ++u)
            if (i0 + 256 * u < n) {
#pragma unroll
                for (int j = 0; j < ROWS; ++j) w[u][j] = load_weights(row[j] + i0 + 256 * u);
                v[u] = load_eight(x + i0 + 256 * u);
            }
#pragma unroll
        for (int u = 0; u < TURNS; ++u)
            if (i0 + 256 * u < n) {
                float xv[8];
                floats_of(v[u], xv);
#pragma unroll
                for (int i = 0; i < 8; ++i) xv[i] *= factor;
#pragma unroll
                for (int j = 0; j < ROWS; ++j) {
                    float wv[8];
                    floats_of(w[u][j], wv);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[j] += wv[i] * xv[i];
                }
            }
    }
}

// grid (pairs, feature blocks)
template <typename T, int FEATS, bool GATED>
__global__ void __launch_bounds__(EV_WARPS * 32) expert_up_vec_kernel(const ExpertParams p) {
    constexpr int ROWS = GATED ? 2 * FEATS : FEATS;
    pdl_launch_dependents();
    pdl_wait();
    const int pair = blockIdx.x, t = pair / p.top, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int f0 = (blockIdx.y * EV_WARPS + warp) * FEATS;
    if (f0 >= p.ff) return;
    const T* w = (const T*)p.up + (size_t)expert_of(p, t, pair % p.top) * (GATED ? 2 : 1) * p.ff * p.width;
    const T* row[ROWS];
#pragma unroll
    for (int j = 0; j < FEATS; ++j) {
        const int f = min(f0 + j, p.ff - 1);
        row[j] = w + (size_t)f * p.width;
        if (GATED) row[FEATS + j] = w + (size_t)(p.ff + f) * p.width;
    }
    float acc[ROWS] = {};
    lane_dots<T, ROWS>(row, (const T*)p.x + (size_t)t * p.width, p.in_weights ? p.in_weights[pair] : 1.f, p.width, lane, acc);
#pragma unroll
    for (int j = 0; j < ROWS; ++j) acc[j] = warp_sum(acc[j]);
    T* mid = (T*)p.mid + (size_t)pair * p.ff;
#pragma unroll
    for (int j = 0; j < FEATS; ++j)
        if (lane == j && f0 + j < p.ff)
            mid[f0 + j] = from_float<T>(GATED ? gated_value<false>(acc[j], acc[GATED ? FEATS + j : j], p.act, p.limit) : gate_activation<false>(acc[j], p.act));
}

// grid (tokens, column blocks)
template <typename T, int FEATS>
__global__ void __launch_bounds__(EV_WARPS * 32) expert_down_vec_kernel(const ExpertParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = (blockIdx.y * EV_WARPS + warp) * FEATS;
    if (c0 >= p.width) return;
    float total[FEATS] = {};
    for (int k = 0; k < p.top; ++k) {                      // in the order of the table's row
        const T* w = (const T*)p.down + (size_t)expert_of(p, t, k) * p.width * p.ff;
        const T* row[FEATS];
#pragma unroll
        for (int j = 0; j < FEATS; ++j) row[j] = w + (size_t)min(c0 + j, p.width - 1) * p.ff;
        float acc[FEATS] = {};
        lane_dots<T, FEATS>(row, (const T*)p.mid + ((size_t)t * p.top + k) * p.ff, 1.f, p.ff, lane, acc);
        const float weight = p.pair_weights ? p.pair_weights[(size_t)t * p.top + k] : 1.f;
#pragma unroll
        for (int j = 0; j < FEATS; ++j) total[j] += warp_sum(acc[j]) * weight;      // the weight on the finished sum, one rounding a pair
    }
#pragma unroll
    for (int j = 0; j < FEATS; ++j)
        if (lane == j && c0 + j < p.width) expert_put(p, t, c0 + j, total[j]);
}

// Features a warp takes: the most that still give every SM a block.  4 pairs of 2,048 x 1,024 and 4 features in both passes 25.6 us, 2
// 27.7 us, 1 31.7 us; one token of 2 such experts 19.5, 17.4 and 15.5 us (both with cold caches, two launches).
static int feats_for(long long rows, int features) {
    for (int feats = 4; feats > 1; feats /= 2)
        if (rows * ((features + EV_WARPS * feats - 1) / (EV_WARPS * feats)) >= sm_count()) return feats;
    return 1;
}

template <typename T> static int launch_expert_rows(const ExpertParams& p, cudaStream_t s) {
    const dim3 block(EV_WARPS * 32);
    const int pairs = p.n_tokens * p.top;
    const int fu = feats_for(pairs, p.ff), fd = feats_for(p.n_tokens, p.width);
    const dim3 up(pairs, (p.ff + EV_WARPS * fu - 1) / (EV_WARPS * fu)), down(p.n_tokens, (p.width + EV_WARPS * fd - 1) / (EV_WARPS * fd));
#define QT_EXPERT_UP(F) (p.gated ? launch_kernel(expert_up_vec_kernel<T, F, true>, up, block, 0, s, p) : launch_kernel(expert_up_vec_kernel<T, F, false>, up, block, 0, s, p))
    if (fu == 4) QT_EXPERT_UP(4);
    else if (fu == 2) QT_EXPERT_UP(2);
    else QT_EXPERT_UP(1);
#undef QT_EXPERT_UP
    QT_CHECK_LAUNCH("expert_up");
    if (fd == 4) launch_kernel(expert_down_vec_kernel<T, 4>, down, block, 0, s, p);
    else if (fd == 2) launch_kernel(expert_down_vec_kernel<T, 2>, down, block, 0, s, p);
    else launch_kernel(expert_down_vec_kernel<T, 1>, down, block, 0, s, p);
    QT_CHECK_LAUNCH("expert_down");
    return QT_OK;
}

// ----------------------------------------------------------------------------- few tokens: per expert that any of them chose
// The same two passes in bfloat16 for up to 32 pairs, an expert's weights read once for all of its pairs (the passes above read them once
// a pair: 8 tokens of one of 8 experts read twice as many bytes as there are, through L2).  The pairs form groups, of one expert and up to
// eight pairs each; a group's pairs are the N of mma.sync, the weights its M (few_tokens.cuh).  A pair's weight, on the input or on the
// output, multiplies float sums.
constexpr int EG_PAIRS = 32;               // a lane a pair
constexpr int EG_WARPS = 8;
constexpr int EG_STEP = 64;                // K elements of a warp's turn: 16 a lane
constexpr int EG_RANKS = 4;                // most blocks that share K in the second pass

struct PairGroups {
    int expert[EG_PAIRS];
    int pair[EG_PAIRS][8];                 // -1 beyond a group's pairs
    int count;
};
// One warp: groups in the order of their first pairs.
__device__ __forceinline__ void group_pairs(const ExpertParams& p, PairGroups& groups, int lane) {
    const int pairs = p.n_tokens * p.top;
    const int e = lane < pairs ? expert_of(p, lane / p.top, lane % p.top) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, e), before = (1u << lane) - 1u;
    const int rank = __popc(same & before);
    const unsigned leaders = __ballot_sync(0xffffffffu, e >= 0 && rank % 8 == 0);
    unsigned mine = same;                                     // my group's first pair is the (rank / 8 * 8)-th of my expert's
    for (int skip = rank / 8 * 8; skip > 0; --skip) mine &= mine - 1u;
    const int leader = __ffs(mine) - 1, group = __popc(leaders & ((1u << leader) - 1u));
    for (int i = 0; i < 8; ++i) groups.pair[lane][i] = -1;
    __syncwarp();
    if (e >= 0) {
        groups.pair[group][rank % 8] = lane;
        groups.expert[group] = e;
    }
    if (lane == 0) groups.count = __popc(leaders);
}

// grid (feature blocks, pairs): block (i, g) forms 16 features of a gated expert, 32 of another, for the pairs of group g.  (Fewer blocks that walk
// several of these, the next one's weights asked for ahead, took 3 us longer at every size.)
template <bool GATED>
__global__ void __launch_bounds__(EG_WARPS * 32, 2) expert_up_groups_kernel(const ExpertParams p) {
    constexpr int DEPTH = 2, FEATS = GATED ? 16 : 32;
    __shared__ PairGroups groups;
    __shared__ __align__(16) float sums[EG_WARPS][8][36];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (warp == 0) group_pairs(p, groups, lane);
    __syncthreads();
    if ((int)blockIdx.y >= groups.count) return;
    const int f0 = blockIdx.x * FEATS, K = p.width;
    const __nv_bfloat16* w = (const __nv_bfloat16*)p.up + (size_t)groups.expert[blockIdx.y] * (GATED ? 2 : 1) * p.ff * K;
    const int pair = groups.pair[blockIdx.y][g];
    const __nv_bfloat16* x = (const __nv_bfloat16*)p.x + (size_t)(pair < 0 ? 0 : pair / p.top) * K;
    const __nv_bfloat16* row[2][2];                           // rows beyond the last repeat it; their sums are not stored
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            row[r][h] = w + (size_t)(GATED ? r * p.ff + min(f0 + 8 * h + g, p.ff - 1) : min(f0 + 16 * r + 8 * h + g, p.ff - 1)) * K;
    const int turns = (K + EG_STEP - 1) / EG_STEP, mine = (turns - warp + EG_WARPS - 1) / EG_WARPS;
    qt_few::Line a[DEPTH][2][2], b[DEPTH];
    auto ask = [&](int slot, int i) {
        const int k = (warp + i * EG_WARPS) * EG_STEP + 16 * t;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (k < K) a[slot][r][h] = qt_few::load_weight(row[r][h] + k);
                else a[slot][r][h] = qt_few::Line{};
            }
        if (k < K && pair >= 0) b[slot] = qt_few::load_rows(x + k);
        else b[slot] = qt_few::Line{};
    };
    float c[2][4] = {};
#pragma unroll
    for (int u = 0; u < DEPTH; ++u)
        if (u < mine) ask(u, u);
    for (int i0 = 0; i0 < mine; i0 += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
            if (i0 + u >= mine) break;
            qt_few::turn_product<2>(c, a[u], b[u]);
            if (i0 + u + DEPTH < mine) ask(u, i0 + u + DEPTH);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) sums[warp][2 * t + (e & 1)][16 * r + g + 8 * (e >> 1)] = c[r][e];
    __syncthreads();
    if (threadIdx.x >= 64) return;
    const int slot = threadIdx.x / 8, l = threadIdx.x % 8, of = groups.pair[blockIdx.y][slot];
    if (of < 0) return;
    const float weight = p.in_weights ? p.in_weights[of] : 1.f;
    __nv_bfloat16* mid = (__nv_bfloat16*)p.mid + (size_t)of * p.ff;
    if (GATED) {
        float2 gate = make_float2(0.f, 0.f), up = make_float2(0.f, 0.f);
#pragma unroll
        for (int s = 0; s < EG_WARPS; ++s) {
            const float2 gs = *reinterpret_cast<const float2*>(&sums[s][slot][2 * l]), us = *reinterpret_cast<const float2*>(&sums[s][slot][2 * l + 16]);
            gate.x += gs.x; gate.y += gs.y; up.x += us.x; up.y += us.y;
        }
        const int f = f0 + 2 * l;                             // ff is a multiple of 16
        if (f < p.ff)
            *reinterpret_cast<__nv_bfloat162*>(mid + f) = __floats2bfloat162_rn(gated_value<false>(gate.x * weight, up.x * weight, p.act, p.limit),
                                                                                gated_value<false>(gate.y * weight, up.y * weight, p.act, p.limit));
    } else {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < EG_WARPS; ++s) {
            const float4 part = *reinterpret_cast<const float4*>(&sums[s][slot][4 * l]);
            v.x += part.x; v.y += part.y; v.z += part.z; v.w += part.w;
        }
        const int f = f0 + 4 * l;
        if (f < p.ff) {
            *reinterpret_cast<__nv_bfloat162*>(mid + f) = __floats2bfloat162_rn(gate_activation<false>(v.x * weight, p.act), gate_activation<false>(v.y * weight, p.act));
            *reinterpret_cast<__nv_bfloat162*>(mid + f + 2) = __floats2bfloat162_rn(gate_activation<false>(v.z * weight, p.act), gate_activation<false>(v.w * weight, p.act));
        }
    }
}

// grid (blocks of 16 columns x RANKS): a cluster's blocks share K, every block walks all groups; a token's sums meet in the block that
// finishes it.
template <int RANKS>
__global__ void __launch_bounds__(EG_WARPS * 32, 2) expert_down_groups_kernel(const ExpertParams p) {
    constexpr int DEPTH = 4;
    __shared__ PairGroups groups;
    __shared__ __align__(16) float sums[EG_WARPS][EG_PAIRS][16];
    __shared__ __align__(16) float parts[RANKS][EG_PAIRS][16];
    pdl_launch_dependents();
    if (RANKS > 1) cluster_arrive_started();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int rank = blockIdx.x % RANKS, c0 = blockIdx.x / RANKS * 16, K = p.ff, pairs = p.n_tokens * p.top;
    if (warp == 0) group_pairs(p, groups, lane);
    __syncthreads();
    const int first = rank + RANKS * warp, stride = RANKS * EG_WARPS;
    const int turns = (K + EG_STEP - 1) / EG_STEP, per = first < turns ? (turns - first + stride - 1) / stride : 0;   // of a group
    const int mine = per * groups.count;
    qt_few::Line a[DEPTH][1][2], b[DEPTH];
    auto ask = [&](int slot, int i) {                         // turns of the groups one after the other
        const int group = i / per, k = (first + (i - group * per) * stride) * EG_STEP + 16 * t, pair = groups.pair[group][g];
        const __nv_bfloat16* w = (const __nv_bfloat16*)p.down + (size_t)groups.expert[group] * p.width * K + k;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (k < K) a[slot][0][h] = qt_few::load_weight(w + (size_t)min(c0 + 8 * h + g, p.width - 1) * K);
            else a[slot][0][h] = qt_few::Line{};
        }
        if (k < K && pair >= 0) b[slot] = qt_few::load_rows((const __nv_bfloat16*)p.mid + (size_t)pair * K + k);
        else b[slot] = qt_few::Line{};
    };
    float c[1][4] = {};
    auto put = [&](int group) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int pair = groups.pair[group][2 * t + (e & 1)];
            if (pair >= 0) sums[warp][pair][g + 8 * (e >> 1)] = c[0][e];
            c[0][e] = 0.f;
        }
    };
#pragma unroll
    for (int u = 0; u < DEPTH; ++u)
        if (u < mine) ask(u, u);
    for (int i0 = 0; i0 < mine; i0 += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; ++u) {
            const int i = i0 + u;
            if (i >= mine) break;
            qt_few::turn_product<1>(c, a[u], b[u]);
            if (i + DEPTH < mine) ask(u, i + DEPTH);
            if ((i + 1) % per == 0) put(i / per);
        }
    }
    if (per == 0)
        for (int group = 0; group < groups.count; ++group) put(group);
    __syncthreads();
    if (RANKS > 1) cluster_wait_started();
    for (int item = threadIdx.x; item < pairs * 4; item += EG_WARPS * 32) {
        const int pair = item / 4, at = item % 4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < EG_WARPS; ++s) {
            const float4 part = *reinterpret_cast<const float4*>(&sums[s][pair][at]);
            v.x += part.x; v.y += part.y; v.z += part.z; v.w += part.w;
        }
        if (RANKS > 1) qt_few::cluster_store4(&parts[rank][pair][at], (uint32_t)(pair / p.top % RANKS), v);
        else *reinterpret_cast<float4*>(&parts[0][pair][at]) = v;
    }
    if (RANKS > 1) cluster_barrier();
    else __syncthreads();
    for (int item = threadIdx.x; item < (p.n_tokens + RANKS - 1) / RANKS * 16; item += EG_WARPS * 32) {
        const int token = rank + item / 16 * RANKS, col = item % 16;
        if (token >= p.n_tokens || c0 + col >= p.width) continue;
        float total = 0.f;
        for (int k = 0; k < p.top; ++k) {                     // in the order of the table's row
            const int pair = token * p.top + k;
            float v = 0.f;
#pragma unroll
            for (int s = 0; s < RANKS; ++s) v += parts[s][pair][col];
            total += v * (p.pair_weights ? p.pair_weights[pair] : 1.f);
        }
        expert_put(p, token, c0 + col, total);
    }
}

static int launch_expert_groups(const ExpertParams& p, cudaStream_t s) {
    const int feats = p.gated ? 16 : 32;
    const dim3 block(EG_WARPS * 32), up((p.ff + feats - 1) / feats, p.n_tokens * p.top);
    if (p.gated) launch_kernel(expert_up_groups_kernel<true>, up, block, 0, s, p);
    else launch_kernel(expert_up_groups_kernel<false>, up, block, 0, s, p);
    QT_CHECK_LAUNCH("expert_up");
    // as many blocks to a column as leave every warp of theirs a turn of a group
    const int turns = (p.ff + EG_STEP - 1) / EG_STEP, columns = (p.width + 15) / 16;
    if (turns >= EG_RANKS * EG_WARPS) launch_kernel_cluster(expert_down_groups_kernel<EG_RANKS>, dim3(columns * EG_RANKS), block, 0, s, EG_RANKS, p);
    else if (turns >= 2 * EG_WARPS) launch_kernel_cluster(expert_down_groups_kernel<2>, dim3(columns * 2), block, 0, s, 2, p);
    else launch_kernel(expert_down_groups_kernel<1>, dim3(columns), block, 0, s, p);
    QT_CHECK_LAUNCH("expert_down");
    return QT_OK;
}

static int check_experts(const char* name, int n_tokens, int vocab, int top, int experts, int width, int ff, int act) {
    QT_REQUIRE(n_tokens >= 0 && vocab > 0 && top > 0 && experts > 0 && top <= experts, "%s: bad routing sizes T=%d V=%d top=%d E=%d", name, n_tokens, vocab, top, experts);
    QT_REQUIRE(width > 0 && ff > 0, "%s: bad sizes width=%d ff=%d", name, width, ff);
    QT_REQUIRE(act >= 0 && act <= QT_ACT_CAPPED, "%s: unknown activation code %d", name, act);
    return QT_OK;
}

extern "C" int qt_experts_by_pair(const void* x, const int* token_ids, const int* table, const void* up, const void* down, void* mid,
                                  float* out, int dtype, int n_tokens, int vocab, int top, int experts, int width, int ff, int act,
                                  float pair_weight, const float* pair_weights, int gated, float limit, const float* base,
                                  int base_splits, long long base_stride, const float* row_scale, const float* in_weights, void* stream) {
    QT_REQUIRE(gated || act < QT_ACT_COUNT, "experts_by_pair: activation %d needs gated experts", act);
    int rc = check_experts("experts_by_pair", n_tokens, vocab, top, experts, width, ff, act);
    if (rc) return rc;
    if (n_tokens == 0) return QT_OK;
    QT_REQUIRE((size_t)width * 4 <= 200 * 1024 && (size_t)top * ff * 4 <= 200 * 1024, "experts_by_pair: a row of %d or %d x %d floats does not fit shared memory", width, top, ff);
    ExpertParams p{x, token_ids, table, up, down, mid, out, n_tokens, vocab, top, experts, width, ff, act, pair_weight,
                   pair_weights, gated, limit, base, base_splits, (size_t)base_stride, row_scale, in_weights};
    cudaStream_t s = (cudaStream_t)stream;
    const int per_block = EV_WARPS * EV_FEATS;
    return QT_DISPATCH_DTYPE(dtype, "experts_by_pair", {
        const size_t smem_up = (size_t)width * sizeof(float), smem_down = (size_t)top * ff * sizeof(float);
        const dim3 grid_up(n_tokens * top, (ff + per_block - 1) / per_block), grid_down(n_tokens, (width + per_block - 1) / per_block);
        // Per expert where the pairs are at least as many as the experts, so that some share one, and where an expert's bytes outweigh the longer way to
        // them (groups, a cluster's sums).  Both passes, gated, by pair / per expert, us: 8, 16, 32 tokens of one of 8 experts of 1,024 x 2,048 18 / 15, 32 / 24, 53 / 28; of
        // 2,048 x 2,048 29 / 24, 52 / 41, 87 / 44; of 4,096 x 1,536 44 / 29, 73 / 56, 127 / 57; 8, 12, 16 tokens of 2 of 16 of 2,048 x 1,024 33 / 30, 43 / 33, 54 / 38; but of 1,024 x 512
        // 10 / 14, 8 tokens of 4 of 32 of 2,048 x 768 48 / 54.  Above the bound it is the slower form only where there are as many pairs as experts and few share one: 4 tokens of 2
        // of 8 of 2,048 x 1,024 18.4 / 18.9, of 4,096 x 1,024 31 / 33, 8 tokens of 4 of 32 of 2,880 x 2,880 205 / 210.
        if (std::is_same<T, __nv_bfloat16>::value && n_tokens * top <= EG_PAIRS && n_tokens * top >= experts && (long long)width * ff >= (2ll << 20) && width % 16 == 0 && ff % 16 == 0 &&
            (((uintptr_t)up | (uintptr_t)down | (uintptr_t)x | (uintptr_t)mid) & 31) == 0) return launch_expert_groups(p, s);
        // 16-byte loads: rows of both weights, of x and of mid start on 16-byte boundaries
        if (width % 8 == 0 && ff % 8 == 0 && (((uintptr_t)up | (uintptr_t)down | (uintptr_t)x | (uintptr_t)mid) & 15) == 0) return launch_expert_rows<T>(p, s);
        if (smem_up > 48 * 1024) cudaFuncSetAttribute(expert_up_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_up);
        if (smem_down > 48 * 1024) cudaFuncSetAttribute(expert_down_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_down);
        launch_kernel(expert_up_kernel<T>, grid_up, dim3(EV_WARPS * 32), smem_up, s, p);
        QT_CHECK_LAUNCH("expert_up");
        launch_kernel(expert_down_kernel<T>, grid_down, dim3(EV_WARPS * 32), smem_down, s, p);
        QT_CHECK_LAUNCH("expert_down");
        return QT_OK;
    });
}

// ----------------------------------------------------------------------------- many tokens: pairs ordered by expert
// Routing for the tiled products (experts_tc.cu).  One block: count the pairs of every expert, give every expert a
// run of rows padded to whole tiles of `tile_rows`, and give every pair a row in its expert's run.
//   pair_row[pair]     the pair's row in the ordered buffers
//   row_token[row]     the pair whose token's (normed) input the row holds (the token is pair / top), -1 for padding
//   tile_expert[tile]  the expert of the tile's rows, -1 for tiles beyond the last run
// Which row of its run a pair gets depends on the order the threads arrive in; a row's results do not depend on where
// it lies, so the output does not either.
__global__ void __launch_bounds__(1024) expert_route_kernel(const ExpertParams p, int* __restrict__ pair_row, int* __restrict__ row_token,
                                                            int* __restrict__ tile_expert, int tile_rows, int max_tiles) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ int route_smem[];
    int* counts = route_smem;                 // [E]
    int* starts = counts + p.experts;         // [E + 1], in rows
    int* cursor = starts + p.experts + 1;     // [E]
    const int pairs = p.n_tokens * p.top;
    for (int e = threadIdx.x; e < p.experts; e += blockDim.x) { counts[e] = 0; cursor[e] = 0; }
    __syncthreads();
    for (int pair = threadIdx.x; pair < pairs; pair += blockDim.x) atomicAdd(&counts[expert_of(p, pair / p.top, pair % p.top)], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int at = 0;
        for (int e = 0; e < p.experts; ++e) {
            starts[e] = at;
            at += (counts[e] + tile_rows - 1) / tile_rows * tile_rows;
        }
        starts[p.experts] = at;
    }
    __syncthreads();
    const int used_tiles = starts[p.experts] / tile_rows;
    for (int e = threadIdx.x; e < p.experts; e += blockDim.x)
        for (int tile = starts[e] / tile_rows; tile < starts[e + 1] / tile_rows; ++tile) tile_expert[tile] = e;
    for (int tile = used_tiles + threadIdx.x; tile < max_tiles; tile += blockDim.x) tile_expert[tile] = -1;
    for (int row = threadIdx.x; row < max_tiles * tile_rows; row += blockDim.x) row_token[row] = -1;
    __syncthreads();
    for (int pair = threadIdx.x; pair < pairs; pair += blockDim.x) {
        const int e = expert_of(p, pair / p.top, pair % p.top);
        const int row = starts[e] + atomicAdd(&cursor[e], 1);
        pair_row[pair] = row;
        row_token[row] = pair;
    }
}

// ordered[row, :] = x[row_token[row] / top, :] (zeros for padding rows), times the pair's input weight where there is one
// (the product in float, rounded once).  One block per row, 16 bytes per thread and turn.
__global__ void expert_gather_kernel(const uint4* x, const int* row_token, uint4* __restrict__ ordered, int chunks, int top,
                                     const float* in_weights) {
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x, pair = row_token[row], token = pair >= 0 ? pair / top : -1;
    const float w = (in_weights && pair >= 0) ? in_weights[pair] : 1.f;
    for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
        uint4 v = token >= 0 ? x[(size_t)token * chunks + c] : make_uint4(0u, 0u, 0u, 0u);
        if (in_weights) {
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(__low2float(h[j]) * w, __high2float(h[j]) * w);
        }
        ordered[(size_t)row * chunks + c] = v;
    }
}

// out[t, :] = pair_weight * sum_k y[pair_row[t * top + k], :], in float, in the order of k.  Bound by the bytes of the rows; a thread takes V
// neighbouring columns (4 where all rows lie on pieces of that size) and asks for the further term before the experts' rows.  1,999 tokens of 2
// of 16 experts, 2,048 columns, a shared expert beside them: about 10 us; 21 us with one column a thread.
template <typename T, int V>
__global__ void __launch_bounds__(256) expert_combine_kernel(const T* y, const int* pair_row, float* __restrict__ out, int top, int width,
                                      float pair_weight, const float* pair_weights, const float* base,
                                      int base_splits, size_t base_stride, const float* row_scale) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    for (int c = (blockIdx.y * 256 + threadIdx.x) * V; c < width; c += gridDim.y * 256 * V) {
        const size_t at = (size_t)t * width + c;
        float acc[V], more[V];
#pragma unroll
        for (int i = 0; i < V; ++i) acc[i] = more[i] = 0.f;
        if (base) {
            for (int s = 0; s < base_splits; ++s) {
                if constexpr (V == 4) {
                    const float4 b = *reinterpret_cast<const float4*>(base + at + (size_t)s * base_stride);
                    more[0] += b.x; more[1] += b.y; more[2] += b.z; more[3] += b.w;
                } else more[0] += base[at + (size_t)s * base_stride];
            }
        }
        for (int k = 0; k < top; ++k) {
            const T* row = y + (size_t)pair_row[t * top + k] * width + c;
            const float weight = pair_weights ? pair_weights[(size_t)t * top + k] : 1.f;
            if constexpr (V == 1) acc[0] += to_float(row[0]) * weight;
            else if constexpr (sizeof(T) == 4) {
                const float4 r = *reinterpret_cast<const float4*>(row);
                acc[0] += r.x * weight; acc[1] += r.y * weight; acc[2] += r.z * weight; acc[3] += r.w * weight;
            } else {
                const uint2 raw = *reinterpret_cast<const uint2*>(row);
                const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
                acc[0] += __low2float(lo) * weight; acc[1] += __high2float(lo) * weight; acc[2] += __low2float(hi) * weight; acc[3] += __high2float(hi) * weight;
            }
        }
        const float scale = base && row_scale ? row_scale[t] : 1.f;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            if (!pair_weights) acc[i] *= pair_weight;
            if (base) acc[i] += scale * more[i];
        }
        if constexpr (V == 4) *reinterpret_cast<float4*>(out + at) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        else out[at] = acc[0];
    }
}

// A learned router's choice.  logits [splits, T, cols] float (column e < experts: expert e; column `experts`, if
// shared_gate, the logit of a shared expert's gate).  Scores are sigmoid(logit); the `top` largest are chosen (by their
// logits; of equal ones the lower expert first), their weights are the scores over their sum (+ 1e-20) times `scale`, or, without `normalize`, the scores themselves times `scale`.
// `softmax`: the scores are the softmax of the logits over all experts instead.  With `groups` > 1 the experts form that
// many equal runs of neighbours, a group's score is the largest in it, and only the experts of the `keep` best groups (of
// equal ones the lower group first) can be chosen.
// One warp per token; chosen [T, top], weights [T, top], gate [T] = sigmoid of the extra column.
__global__ void __launch_bounds__(128) route_top_kernel(const float* logits, int n_splits, size_t split_stride, int cols,
                                                        int* __restrict__ chosen, float* __restrict__ weights, float* __restrict__ gate,
                                                        int n_tokens, int experts, int top, float scale, int normalize, int softmax, int groups,
                                                        int keep) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float route_scores[];                      // [warps][experts]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= n_tokens) return;
    float* score = route_scores + (size_t)warp * experts;        // the logits: their order is the scores' order, and two logits
    // that differ stay apart where their sigmoids round to the same float
    for (int e = lane; e < experts; e += 32) score[e] = load_sum(logits, (size_t)t * cols + e, n_splits, split_stride);
    if (gate && lane == 0) gate[t] = 1.f / (1.f + expf(-load_sum(logits, (size_t)t * cols + experts, n_splits, split_stride)));
    __syncwarp();
    float highest = 0.f, mass = 1.f;
    if (softmax) {
        highest = -INFINITY;
        for (int e = lane; e < experts; e += 32) highest = fmaxf(highest, score[e]);
        highest = warp_max(highest);
        mass = 0.f;
        for (int e = lane; e < experts; e += 32) mass += expf(score[e] - highest);
        mass = warp_sum(mass);
    }
    if (groups > 1) {
        float* best_of = route_scores + (size_t)(blockDim.x >> 5) * experts + (size_t)warp * groups;     // [groups] of this warp
        const int size = experts / groups;
        for (int g = lane; g < groups; g += 32) {
            float m = -INFINITY;
            for (int e = g * size; e < (g + 1) * size; ++e) m = fmaxf(m, score[e]);
            best_of[g] = m;
        }
        __syncwarp();
        for (int g = lane; g < groups; g += 32) {               // a group is dropped if `keep` groups come before it
            int before = 0;
            for (int o = 0; o < groups; ++o) before += best_of[o] > best_of[g] || (best_of[o] == best_of[g] && o < g);
            if (before >= keep)
                for (int e = g * size; e < (g + 1) * size; ++e) score[e] = -INFINITY;
        }
        __syncwarp();
    }
    float sum = 0.f;
    for (int k = 0; k < top; ++k) {
        float best = -INFINITY;
        int at = experts;
        for (int e = lane; e < experts; e += 32)
            if (score[e] > best || at == experts) { best = score[e]; at = e; }
        for (int off = 16; off > 0; off >>= 1) {
            const float other = __shfl_xor_sync(0xffffffffu, best, off);
            const int where = __shfl_xor_sync(0xffffffffu, at, off);
            if (where < experts && (at == experts || other > best || (other == best && where < at))) { best = other; at = where; }
        }
        const float chosen_score = softmax ? expf(best - highest) / mass : 1.f / (1.f + expf(-best));
        sum += chosen_score;
        if (lane == 0) { chosen[(size_t)t * top + k] = at; weights[(size_t)t * top + k] = chosen_score; score[at] = -INFINITY; }
        __syncwarp();
    }
    if (lane < top) {
        for (int k = lane; k < top; k += 32)
            weights[(size_t)t * top + k] = normalize ? weights[(size_t)t * top + k] / (sum + 1e-20f) * scale : weights[(size_t)t * top + k] * scale;
    }
}

extern "C" int qt_route_top(const float* logits, int n_splits, long long split_stride, int cols, int* chosen, float* weights, float* gate,
                            int n_tokens, int experts, int top, float scale, int normalize, int softmax, int groups, int keep, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && experts > 0 && top > 0 && top <= experts && cols >= experts + (gate ? 1 : 0) && n_splits >= 1,
               "route_top: bad sizes T=%d E=%d top=%d cols=%d", n_tokens, experts, top, cols);
    QT_REQUIRE(groups >= 1 && experts % groups == 0 && keep >= 1 && keep <= groups && top <= keep * (experts / groups),
               "route_top: %d experts out of the best %d of %d groups of %d", top, keep, groups, experts);
    QT_REQUIRE((size_t)8 * experts * sizeof(float) <= 48 * 1024, "route_top: %d experts are too many for a warp's scores in shared memory", experts);
    if (n_tokens == 0) return QT_OK;
    launch_kernel(route_top_kernel, dim3((n_tokens + 3) / 4), dim3(128), (size_t)4 * (experts + groups) * sizeof(float), (cudaStream_t)stream, logits, n_splits,
                  (size_t)split_stride, cols, chosen, weights, gate, n_tokens, experts, top, scale, normalize, softmax, groups, keep);
    QT_CHECK_LAUNCH("route_top");
    return QT_OK;
}

extern "C" int qt_experts_route(const void* x, const int* token_ids, const int* table, void* ordered, int* pair_row, int* row_token,
                                int* tile_expert, int n_tokens, int vocab, int top, int experts, int width, int tile_rows, int max_tiles,
                                const float* in_weights, void* stream) {
    int rc = check_experts("experts_route", n_tokens, vocab, top, experts, width, 1, 0);
    if (rc) return rc;
    if (n_tokens == 0) return QT_OK;
    QT_REQUIRE(width % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)ordered % 16 == 0, "experts_route: rows of 16-byte pieces are needed (width=%d)", width);
    QT_REQUIRE(tile_rows > 0 && (long long)max_tiles * tile_rows >= (long long)n_tokens * top, "experts_route: %d tiles of %d rows do not hold the pairs", max_tiles, tile_rows);
    QT_REQUIRE((3 * (size_t)experts + 1) * sizeof(int) <= 48 * 1024, "experts_route: %d experts are too many for one block's counters", experts);
    ExpertParams p{x, token_ids, table, nullptr, nullptr, nullptr, nullptr, n_tokens, vocab, top, experts, width, 1, 0, 0.f,
                   nullptr, 0, 0.f, nullptr, 1, 0, nullptr, nullptr};
    cudaStream_t s = (cudaStream_t)stream;
    launch_kernel(expert_route_kernel, dim3(1), dim3(1024), (3 * (size_t)experts + 1) * sizeof(int), s, p, pair_row, row_token, tile_expert, tile_rows, max_tiles);
    QT_CHECK_LAUNCH("expert_route");
    launch_kernel(expert_gather_kernel, dim3(max_tiles * tile_rows), dim3(128), 0, s, (const uint4*)x, (const int*)row_token, (uint4*)ordered, width / 8, top, in_weights);
    QT_CHECK_LAUNCH("expert_gather");
    return QT_OK;
}

extern "C" int qt_experts_combine(const void* y, int dtype, const int* pair_row, float* out, int n_tokens, int top, int width, float pair_weight,
                                  const float* pair_weights, const float* base, int base_splits, long long base_stride,
                                  const float* row_scale, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && top > 0 && width > 0, "experts_combine: bad sizes T=%d top=%d width=%d", n_tokens, top, width);
    if (n_tokens == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    return QT_DISPATCH_DTYPE(dtype, "experts_combine", {
        const bool fours = width % 4 == 0 && base_stride % 4 == 0 && (((uintptr_t)y | (uintptr_t)out | (uintptr_t)base) & 15) == 0;
        // few tokens: the columns of a row over several blocks, so that the launch fills the machine
        const int per_block = fours ? 1024 : 256;
        const dim3 grid(n_tokens, n_tokens >= 1024 ? 1u : (unsigned)((width + per_block - 1) / per_block));
        if (fours) launch_kernel(expert_combine_kernel<T, 4>, grid, dim3(256), 0, s, (const T*)y, pair_row, out, top, width, pair_weight, pair_weights, base,
                                 base_splits, (size_t)base_stride, row_scale);
        else launch_kernel(expert_combine_kernel<T, 1>, grid, dim3(256), 0, s, (const T*)y, pair_row, out, top, width, pair_weight, pair_weights, base,
                           base_splits, (size_t)base_stride, row_scale);
        QT_CHECK_LAUNCH("expert_combine");
        return QT_OK;
    });
}

QT_DEFINE_LAST_ERROR(experts)
