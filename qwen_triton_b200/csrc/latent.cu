// Attention through a latent: what stands around the attention kernel of a mixer that caches, per token, one normed
// latent vector c and one rotated key part shared by all heads, and expands keys and values from c per head.
//
// The cache row of a token is [c (rank) | rotated part (rot)], one "kv head" of size rank + rot.  With
// k_h = W_uk_h c and v_h = W_uv_h c the score of head h is q_plain_h . (W_uk_h c) + q_rot_h . k_rot
// = (W_uk_h^T q_plain_h) . c + q_rot_h . k_rot, so the attention kernel runs every head's query
// [W_uk_h^T q_plain_h | q_rot_h] against the cached rows as they are (all heads share the one kv head), its values are
// the first `rank` elements of the same rows, and the head's output is W_uv_h (sum_j p_j c_j).
//
// latent_prepare_kernel   from the first projection's float sums of a token: RMS norm (weight, eps inside the root) of the
//                         query latent -> cq_out; RMS norm of the key/value latent and rotation of the shared key part
//                         by the token's position -> the cache row.
// latent_query_rot_kernel the rotated part of every head's query: rotation by position into the query rows.
// latent_rows_kernel, latent_queries_kernel   the operands of a prompt whose keys and values are formed per head (attention_tc.cu)
// head_product_kernel     Y[t, h, n] = sum_k X[t, h, k] W[h, n, k] for every head with its own matrix (float sums), with
//                         strides for X and Y and optionally times sigmoid(gate[t, h * N + n]) or sigmoid(gate[t, h]).
// head_product_mma_kernel the same on the tensor cores (mma.sync m16n8k16) for bfloat16 matrices and results.
// Rotation: element i of the rotated part turns with element i + rd / 2 by the angle whose cos and sin the table row
// of the position holds (cos | sin, rd columns); elements beyond the first rd pass unchanged.
#include "attention_mma.cuh"

#include <math.h>

using namespace qt;

__device__ __forceinline__ float sum_splits(const float* __restrict__ base, size_t index, int n_splits, size_t split_stride) {
    float acc = base[index];
    for (int s = 1; s < n_splits; ++s) acc += base[index + (size_t)s * split_stride];
    return acc;
}

struct PrepareParams {
    const float* proj; int n_splits; size_t split_stride; int proj_cols;   // columns: query latent (or queries) | key/value latent | rotated part | ...
    const float* q_norm; const float* kv_norm; float eps;
    const float* cos_sin; int rotary_dim, max_pos;
    void* cq_out;                     // [T, q_rank]
    void* cache;                      // [pages, 1, page_tokens, rank + rot]
    const int* token_seq; const int* token_pos; const int* block_table; int max_blocks;
    int q_rank, rank, rot, page_tokens, ring_tokens, write_kv;      // q_rank 0: no query latent
    int at_kv;                        // first column of the key/value latent
};

// one block per token
template <typename TO>
__global__ void __launch_bounds__(256) latent_prepare_kernel(const PrepareParams p) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float scratch[32];
    const int t = blockIdx.x;
    const size_t base = (size_t)t * p.proj_cols;
    if (p.q_rank > 0) {
        float sq = 0.f;
        for (int i = threadIdx.x; i < p.q_rank; i += blockDim.x) {
            const float x = sum_splits(p.proj, base + i, p.n_splits, p.split_stride);
            sq += x * x;
        }
        const float inv = rsqrtf(block_sum(sq, scratch) / (float)p.q_rank + p.eps);
        TO* out = (TO*)p.cq_out + (size_t)t * p.q_rank;
        for (int i = threadIdx.x; i < p.q_rank; i += blockDim.x)
            out[i] = from_float<TO>(sum_splits(p.proj, base + i, p.n_splits, p.split_stride) * inv * p.q_norm[i]);
    }
    if (!p.write_kv) return;
    const int pos = p.token_pos[t];
    const int* table = p.block_table + (size_t)p.token_seq[t] * p.max_blocks;
    TO* row = (TO*)p.cache + cache_offset(table, pos, p.ring_tokens, p.page_tokens, 1, 0, p.rank + p.rot);
    const size_t at = base + p.at_kv;
    float sq = 0.f;
    for (int i = threadIdx.x; i < p.rank; i += blockDim.x) {
        const float x = sum_splits(p.proj, at + i, p.n_splits, p.split_stride);
        sq += x * x;
    }
    const float inv = rsqrtf(block_sum(sq, scratch) / (float)p.rank + p.eps);
    for (int i = threadIdx.x; i < p.rank; i += blockDim.x)
        row[i] = from_float<TO>(sum_splits(p.proj, at + i, p.n_splits, p.split_stride) * inv * p.kv_norm[i]);
    const int half = p.rotary_dim / 2;
    const float* cs = p.cos_sin ? p.cos_sin + (size_t)pos * p.rotary_dim : nullptr;
    for (int i = threadIdx.x; i < p.rot; i += blockDim.x) {
        const float x = sum_splits(p.proj, at + p.rank + i, p.n_splits, p.split_stride);
        float y = x;
        if (cs && i < p.rotary_dim) {
            const int pair = i < half ? i : i - half;
            const float other = sum_splits(p.proj, at + p.rank + (i < half ? i + half : i - half), p.n_splits, p.split_stride);
            y = i < half ? x * cs[pair] - other * cs[half + pair] : x * cs[pair] + other * cs[half + pair];
        }
        row[p.rank + i] = from_float<TO>(y);
    }
}

extern "C" int qt_latent_prepare(const float* proj, int n_splits, long long split_stride, int proj_cols, const float* q_norm,
                                 const float* kv_norm, float eps, const float* cos_sin, int rotary_dim, int max_pos, void* cq_out,
                                 void* cache, int out_dtype, const int* token_seq, const int* token_pos, const int* block_table,
                                 int max_blocks, int n_tokens, int q_rank, int rank, int rot, int page_tokens, int ring_tokens,
                                 int write_kv, int at_kv, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && q_rank >= 0 && at_kv >= q_rank && rank > 0 && rot >= 0 && n_splits >= 1 && eps > 0.f, "latent_prepare: bad sizes");
    QT_REQUIRE(at_kv + (write_kv ? rank + rot : 0) <= proj_cols, "latent_prepare: the latents need %d columns of %d",
               at_kv + (write_kv ? rank + rot : 0), proj_cols);
    QT_REQUIRE(q_rank == 0 || (q_norm && cq_out), "latent_prepare: a query latent needs its weight and a place");
    QT_REQUIRE(rotary_dim >= 0 && rotary_dim % 2 == 0 && rotary_dim <= rot && (rotary_dim == 0 || cos_sin),
               "latent_prepare: %d of %d elements rotate", rotary_dim, rot);
    QT_REQUIRE(!write_kv || (cache && block_table && kv_norm), "latent_prepare: no cache to write to");
    if (n_tokens == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    PrepareParams p{proj, n_splits, (size_t)split_stride, proj_cols, q_norm, kv_norm, eps, rotary_dim ? cos_sin : nullptr, rotary_dim, max_pos,
                    cq_out, cache, token_seq, token_pos, block_table, max_blocks, q_rank, rank, rot, page_tokens, ring_tokens, write_kv, at_kv};
    return QT_DISPATCH_DTYPE(out_dtype, "latent_prepare", {
        launch_kernel(latent_prepare_kernel<T>, dim3(n_tokens), dim3(256), 0, s, p);
        QT_CHECK_LAUNCH("latent_prepare");
        return QT_OK;
    });
}

// ----------------------------------------------------------------------------- the rotated part of the queries
// q [splits, T, q_cols >= heads * (dim + rot)] -> out[t, h, out_offset + i] for i < rot.  One thread per (token, head, element).
template <typename TI, typename TO>
__global__ void latent_query_rot_kernel(const TI* q, int n_splits, size_t split_stride, const float* cos_sin,
                                        int rotary_dim, const int* token_pos, TO* __restrict__ out, long long total,
                                        int heads, int dim, int rot, int q_cols, int out_row, int out_offset) {
    pdl_launch_dependents();
    pdl_wait();
    const int half = rotary_dim / 2;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % rot);
        const long long th = idx / rot;
        const int h = (int)(th % heads);
        const long long t = th / heads;
        const size_t at = (size_t)t * q_cols + (size_t)h * (dim + rot) + dim;
        const float x = load_sum(q, at + i, n_splits, split_stride);
        float y = x;
        if (i < rotary_dim) {
            const float* cs = cos_sin + (size_t)token_pos[t] * rotary_dim;
            const int pair = i < half ? i : i - half;
            const float other = load_sum(q, at + (i < half ? i + half : i - half), n_splits, split_stride);
            y = i < half ? x * cs[pair] - other * cs[half + pair] : x * cs[pair] + other * cs[half + pair];
        }
        out[((size_t)t * heads + h) * out_row + out_offset + i] = from_float<TO>(y);
    }
}

extern "C" int qt_latent_query_rot(const void* q, int in_dtype, int n_splits, long long split_stride, const float* cos_sin, int rotary_dim,
                                   const int* token_pos, void* out, int out_dtype, int n_tokens, int heads, int dim, int rot, int q_cols,
                                   int out_row, int out_offset, void* stream) {
    QT_REQUIRE(q_cols >= heads * (dim + rot), "latent_query_rot: %d heads of %d + %d in %d columns", heads, dim, rot, q_cols);
    QT_REQUIRE(n_tokens >= 0 && heads > 0 && dim >= 0 && rot >= 0 && out_offset >= 0 && out_offset + rot <= out_row, "latent_query_rot: bad sizes");
    QT_REQUIRE(rotary_dim >= 0 && rotary_dim % 2 == 0 && rotary_dim <= rot && (rotary_dim == 0 || cos_sin), "latent_query_rot: %d of %d elements rotate",
               rotary_dim, rot);
    if (n_tokens == 0 || rot == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const long long total = (long long)n_tokens * heads * rot;
    long long blocks = (total + 255) / 256;
    if (blocks > (long long)sm_count() * 16) blocks = (long long)sm_count() * 16;
#define QT_LAUNCH_ROT(TI, TO)                                                                                                      \
    launch_kernel(latent_query_rot_kernel<TI, TO>, dim3((unsigned)blocks), dim3(256), 0, s, (const TI*)q, n_splits, (size_t)split_stride, \
                  cos_sin, rotary_dim, token_pos, (TO*)out, total, heads, dim, rot, q_cols, out_row, out_offset)
    if (in_dtype == QT_F32 && out_dtype == QT_F32) QT_LAUNCH_ROT(float, float);
    else if (in_dtype == QT_F32 && out_dtype == QT_BF16) QT_LAUNCH_ROT(float, __nv_bfloat16);
    else if (in_dtype == QT_BF16 && out_dtype == QT_BF16) QT_LAUNCH_ROT(__nv_bfloat16, __nv_bfloat16);
    else QT_FAIL(QT_ERR_ARG, "latent_query_rot: element types %d/%d", in_dtype, out_dtype);
#undef QT_LAUNCH_ROT
    QT_CHECK_LAUNCH("latent_query_rot");
    return QT_OK;
}

// ----------------------------------------------------------------------------- prompts with keys and values per head
// Queries, keys and values of such a prompt are halves, whose 11 bits are wanted and whose range of 2^-14 .. 65,504 is not that of bfloat16.  So they
// are multiplied by powers of two, which round nothing: the keys and the values of a run of 64 tokens (a tile of the attention) by one each that puts
// the largest they can be into [2^14, 2^15), a query by one that puts its largest element there.  The attention takes them out of its scores and
// weights again.  An element loses bits only where it is 2^-28 and less of its run's bound or of its query's largest.

// The power of two that puts `largest` into [2^14, 2^15), and its inverse; 1 for 0 and for what is not finite.
__device__ __forceinline__ float2 into_halves(float largest) {
    if (!(largest > 0.f && largest < INFINITY)) return make_float2(1.f, 1.f);
    const int e = max(-113, (int)(__float_as_uint(largest) >> 23) - 127 - 14);      // at most 113
    return make_float2(__uint_as_float((uint32_t)(127 - e) << 23), __uint_as_float((uint32_t)(127 + e) << 23));
}

// The cached rows of a step's sequences, all from position 0 on, side by side: rows [64 (seq_start[i] / 64 + i) + position, row], the last run
// of 64 of a sequence filled up with zeros.  A run is a page of the cache; first portions lie within a windowed group's ring, which they never
// go round.  run_scale[run] = {the power of two for its keys, the inverse, the power of two for its values, the logarithm of the inverse}: a key's
// element is at most the largest of the latents (the first `rank` elements) times key_norm, or an element of the shared part behind
// them; a value's at most the largest latent times value_norm.  2,048 tokens of 512 + 64 3.7 us (3.2 us without the largest elements).  grid (runs of the longest sequence, sequences).
constexpr int LR_THREADS = 512;
__global__ void __launch_bounds__(LR_THREADS) latent_rows_kernel(const uint4* cache, uint4* __restrict__ rows, float4* __restrict__ run_scale,
                                                          const int* block_table, int max_blocks, const int* seq_start, int pieces,
                                                          int latent_pieces, float key_norm, float value_norm) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ uint32_t most[2][LR_THREADS / 32];
    const int seq = blockIdx.y, run = blockIdx.x, begin = seq_start[seq], count = seq_start[seq + 1] - begin;
    const int live = min(64, count - run * 64);
    if (live <= 0) return;
    const int page = block_table[(size_t)seq * max_blocks + run];
    const uint4* from = cache + (size_t)page * 64 * pieces;
    uint4* to = rows + (size_t)(begin / 64 + seq + run) * 64 * pieces;
    uint32_t latent = 0, shared = 0;                       // largest magnitudes so far, as bfloat16 bits, of the even and the odd elements
    int at = threadIdx.x % pieces;                         // the piece's place in its row
    const int step = LR_THREADS % pieces;
    for (int i0 = threadIdx.x; i0 < 64 * pieces; i0 += 4 * LR_THREADS) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = i0 + u * LR_THREADS < live * pieces ? from[i0 + u * LR_THREADS] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (i0 + u * LR_THREADS < 64 * pieces) to[i0 + u * LR_THREADS] = v[u];
            const uint32_t here = __vmaxu2(__vmaxu2(v[u].x & 0x7fff7fffu, v[u].y & 0x7fff7fffu), __vmaxu2(v[u].z & 0x7fff7fffu, v[u].w & 0x7fff7fffu));
            if (at < latent_pieces) latent = __vmaxu2(latent, here);
            else shared = __vmaxu2(shared, here);
            at += step;
            if (at >= pieces) at -= pieces;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        latent = __vmaxu2(latent, __shfl_xor_sync(0xffffffffu, latent, off));
        shared = __vmaxu2(shared, __shfl_xor_sync(0xffffffffu, shared, off));
    }
    if ((threadIdx.x & 31) == 0) { most[0][threadIdx.x >> 5] = latent; most[1][threadIdx.x >> 5] = shared; }
    __syncthreads();
    if (threadIdx.x < 32) {
        latent = most[0][threadIdx.x % (LR_THREADS / 32)];
        shared = most[1][threadIdx.x % (LR_THREADS / 32)];
#pragma unroll
        for (int off = LR_THREADS / 64; off > 0; off >>= 1) {
            latent = __vmaxu2(latent, __shfl_xor_sync(0xffffffffu, latent, off));
            shared = __vmaxu2(shared, __shfl_xor_sync(0xffffffffu, shared, off));
        }
        const float most_latent = __uint_as_float(max(latent >> 16, latent & 0xffffu) << 16), most_shared = __uint_as_float(max(shared >> 16, shared & 0xffffu) << 16);
        const float2 keys = into_halves(fmaxf(most_latent * key_norm, most_shared)), values = into_halves(most_latent * value_norm);
        if (threadIdx.x == 0) run_scale[begin / 64 + seq + run] = make_float4(keys.x, keys.y, values.x, (float)((int)(__float_as_uint(values.y) >> 23) - 127));
    }
}

extern "C" int qt_latent_rows(const void* cache, void* rows, float* run_scale, const int* block_table, int max_blocks, const int* seq_start, int n_seqs,
                              int max_tokens, int row, int rank, float key_norm, float value_norm, int page_tokens, int ring_tokens, void* stream) {
    QT_REQUIRE(n_seqs >= 0 && n_seqs <= 65535 && max_tokens >= 0 && row > 0 && row % 8 == 0 && rank >= 0 && rank <= row && rank % 8 == 0 && page_tokens == 64 && ring_tokens % 64 == 0,
               "latent_rows: bad sizes");
    QT_REQUIRE((((uintptr_t)cache | (uintptr_t)rows) & 15) == 0 && run_scale && ((uintptr_t)run_scale & 15) == 0 && (max_tokens + 63) / 64 <= (ring_tokens ? ring_tokens / 64 : max_blocks),
               "latent_rows: %d tokens in %d pages", max_tokens, ring_tokens ? ring_tokens / 64 : max_blocks);
    if (n_seqs == 0 || max_tokens == 0) return QT_OK;
    launch_kernel(latent_rows_kernel, dim3((max_tokens + 63) / 64, n_seqs), dim3(LR_THREADS), 0, (cudaStream_t)stream, (const uint4*)cache, (uint4*)rows, (float4*)run_scale,
                  block_table, max_blocks, seq_start, row / 8, rank / 8, key_norm, value_norm);
    QT_CHECK_LAUNCH("latent_rows");
    return QT_OK;
}

// q [splits, T, q_cols >= heads * (dim + rot)] -> out [T, heads, 64 PIECES] halves: a head's dim elements, its rot elements turned by the
// token's position, zeros behind, all times a power of two whose inverse is q_scale [T, heads].  Eight lanes take a head, PIECES times eight
// neighbouring elements each (all of dim, rot and rotary_dim / 2 are multiples of 8), so that the largest of a head is three shuffles away and no lane
// idles.  2,048 tokens of 16 heads of 128 + 64 6.0 us (8.5 us with a piece a thread and no factors, 11.3 us with a head over 32 lanes, 24 of them live).
__device__ __forceinline__ void sum_eight(const float* p, int n_splits, size_t stride, float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
    for (int s = 0; s < n_splits; ++s) {
        const float4 a = *reinterpret_cast<const float4*>(p + (size_t)s * stride), b = reinterpret_cast<const float4*>(p + (size_t)s * stride)[1];
        v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w; v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
    }
}
__device__ __forceinline__ void sum_eight(const __nv_bfloat16* p, int, size_t, float (&v)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] = __low2float(h[i]); v[2 * i + 1] = __high2float(h[i]); }
}

template <typename TI, int PIECES>
__global__ void __launch_bounds__(256) latent_queries_kernel(const TI* q, int n_splits, size_t split_stride, int q_cols, const float* cos_sin,
                                                             int rotary_dim, const int* token_pos, uint4* __restrict__ out, float* __restrict__ q_scale,
                                                             long long pairs, int heads, int dim, int rot) {
    pdl_launch_dependents();
    pdl_wait();
    const long long th = (long long)blockIdx.x * 32 + threadIdx.x / 8;                       // token and head
    const int l = threadIdx.x % 8, half = rotary_dim / 2;
    const bool live = th < pairs;
    const int h = live ? (int)(th % heads) : 0;
    const long long t = live ? th / heads : 0;
    const TI* head = q + (size_t)t * q_cols + (size_t)h * (dim + rot);
    float v[PIECES][8] = {}, largest = 0.f;
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
        const int c = 8 * (l + 8 * u), i = c - dim;
        if (live && c < dim + rot) sum_eight(head + c, n_splits, split_stride, v[u]);
        if (live && i >= 0 && i < rotary_dim) {
            const bool low = i < half;
            const int pair = low ? i : i - half;
            float other[8], cs[8], sn[8];
            sum_eight(head + (low ? c + half : c - half), n_splits, split_stride, other);
            const float* table = cos_sin + (size_t)token_pos[t] * rotary_dim + pair;
            sum_eight(table, 1, 0, cs);
            sum_eight(table + half, 1, 0, sn);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[u][j] = low ? v[u][j] * cs[j] - other[j] * sn[j] : v[u][j] * cs[j] + other[j] * sn[j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) largest = fmaxf(largest, fabsf(v[u][j]));
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, off));
    if (!live) return;
    const float2 scale = into_halves(largest);
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
        __align__(16) __half rounded[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) rounded[j] = from_float<__half>(v[u][j] * scale.x);
        out[th * (8 * PIECES) + l + 8 * u] = *reinterpret_cast<const uint4*>(rounded);
    }
    if (l == 0) q_scale[th] = scale.y;
}

extern "C" int qt_latent_queries(const void* q, int in_dtype, int n_splits, long long split_stride, int q_cols, const float* cos_sin, int rotary_dim,
                                 const int* token_pos, void* out, float* q_scale, int n_tokens, int heads, int dim, int rot, int out_row, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && heads > 0 && dim > 0 && rot >= 0 && dim + rot <= out_row && (out_row == 128 || out_row == 192) && q_cols >= heads * (dim + rot) && q_scale,
               "latent_queries: bad sizes");
    QT_REQUIRE(dim % 8 == 0 && rot % 8 == 0 && q_cols % 8 == 0 && rotary_dim % 16 == 0 && rotary_dim <= rot && split_stride % 4 == 0 &&
               (((uintptr_t)q | (uintptr_t)out | (uintptr_t)cos_sin) & 15) == 0, "latent_queries: heads of %d + %d (%d turn) are not whole 16-byte pieces", dim, rot, rotary_dim);
    if (n_tokens == 0) return QT_OK;
    const long long pairs = (long long)n_tokens * heads;
    cudaStream_t s = (cudaStream_t)stream;
#define QT_LAUNCH_QUERIES(TI, PIECES)                                                                                                             \
    launch_kernel(latent_queries_kernel<TI, PIECES>, dim3((unsigned)((pairs + 31) / 32)), dim3(256), 0, s, (const TI*)q, n_splits, (size_t)split_stride, \
                  q_cols, cos_sin, rotary_dim, token_pos, (uint4*)out, q_scale, pairs, heads, dim, rot)
    if (in_dtype == QT_F32 && out_row == 128) QT_LAUNCH_QUERIES(float, 2);
    else if (in_dtype == QT_F32) QT_LAUNCH_QUERIES(float, 3);
    else if (out_row == 128) QT_LAUNCH_QUERIES(__nv_bfloat16, 2);
    else QT_LAUNCH_QUERIES(__nv_bfloat16, 3);
#undef QT_LAUNCH_QUERIES
    QT_CHECK_LAUNCH("latent_queries");
    return QT_OK;
}

// ----------------------------------------------------------------------------- a product per head
// grid (n tiles, token tiles, heads); a block of 256 threads forms a tile of HP_TM tokens x HP_TN outputs, K in slices
// of HP_TK through shared memory; a thread owns 2 tokens x 4 outputs.  Float accumulation whatever the element types.
constexpr int HP_TM = 32, HP_TN = 64, HP_TK = 16;

struct HeadProductParams {
    const void* x; int x_splits; size_t x_split_stride; long long x_row, x_head; int x_offset;    // X[t, h, k] at t * x_row + h * x_head + x_offset + k
    const void* w;                                                                                // [heads, N, K]
    void* y; long long y_row, y_head; int y_offset;
    const float* gate; int gate_splits; size_t gate_split_stride; int gate_cols, gate_offset;      // optional: times sigmoid(gate[t, gate_offset + h * gate_head + n * gate_elem])
    int gate_head, gate_elem;      // N and 1 (a gate per element), or 1 and 0 (one per head)
    int n_tokens, heads, n, k;
};

template <typename TI, typename TW, typename TO>
__global__ void __launch_bounds__(256) head_product_kernel(const HeadProductParams p) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float xs[HP_TK][HP_TM + 1];
    __shared__ float wsm[HP_TK][HP_TN + 1];
    const int h = blockIdx.z, t0 = blockIdx.y * HP_TM, n0 = blockIdx.x * HP_TN;
    const TI* x = (const TI*)p.x;
    const TW* w = (const TW*)p.w + (size_t)h * p.n * p.k;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;       // outputs n0 + tx + 16 j (j < 4), tokens t0 + ty + 16 i (i < 2)
    float acc[2][4] = {};
    for (int k0 = 0; k0 < p.k; k0 += HP_TK) {
        for (int i = threadIdx.x; i < HP_TM * HP_TK; i += 256) {
            const int kk = i % HP_TK, tt = i / HP_TK;
            const int t = t0 + tt, k = k0 + kk;
            xs[kk][tt] = (t < p.n_tokens && k < p.k)
                ? load_sum(x, (size_t)((long long)t * p.x_row + (long long)h * p.x_head + p.x_offset + k), p.x_splits, p.x_split_stride) : 0.f;
        }
        for (int i = threadIdx.x; i < HP_TN * HP_TK; i += 256) {
            const int kk = i % HP_TK, nn = i / HP_TK;
            const int n = n0 + nn, k = k0 + kk;
            wsm[kk][nn] = (n < p.n && k < p.k) ? to_float(w[(size_t)n * p.k + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < HP_TK; ++kk) {
            float a[2], b[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = xs[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = wsm[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * b[j];
        }
        __syncthreads();
    }
    TO* y = (TO*)p.y;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int t = t0 + ty + 16 * i;
        if (t >= p.n_tokens) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n >= p.n) continue;
            float v = acc[i][j];
            if (p.gate) {
                const float g = sum_splits(p.gate, (size_t)t * p.gate_cols + p.gate_offset + (size_t)h * p.gate_head + (size_t)n * p.gate_elem, p.gate_splits, p.gate_split_stride);
                v = v / (1.f + expf(-g));
            }
            y[(size_t)((long long)t * p.y_row + (long long)h * p.y_head + p.y_offset + n)] = from_float<TO>(v);
        }
    }
}

// The same product on the tensor cores: bfloat16 matrices and results, X bfloat16 (copied by cp.async) or float partial
// sums (added and rounded to bfloat16 on the way into shared memory).  grid (n tiles, token tiles, heads); four warps
// form a tile of 64 tokens x 64 outputs (16 tokens a warp), K in slices of 64 through a two-stage ring.
constexpr int HM_T = 64, HM_N = 64, HM_K = 64, HM_LDS = HM_K + 8;

template <typename TI>
__global__ void __launch_bounds__(128) head_product_mma_kernel(const HeadProductParams p) {
    using namespace qt_mma;
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) __nv_bfloat16 tiles[2][2][HM_T * HM_LDS];      // [stage][X | W]
    const int h = blockIdx.z, t0 = blockIdx.y * HM_T, n0 = blockIdx.x * HM_N;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const TI* x = (const TI*)p.x;
    const __nv_bfloat16* w = (const __nv_bfloat16*)p.w + (size_t)h * p.n * p.k;
    const int slices = (p.k + HM_K - 1) / HM_K;
    auto issue = [&](int slice) {
        if (slice < slices) {
            const int k0 = slice * HM_K;
            __nv_bfloat16* xs = tiles[slice & 1][0];
            __nv_bfloat16* wt = tiles[slice & 1][1];
            for (int i = tid; i < HM_T * (HM_K / 8); i += 128) {
                const int r = i >> 3, c = (i & 7) * 8;
                const int tok = t0 + r, k = k0 + c;
                __nv_bfloat16* dst = xs + r * HM_LDS + c;
                if constexpr (sizeof(TI) == 2) {
                    if (tok < p.n_tokens && k < p.k) cp_async16(smem_u32(dst), x + (size_t)((long long)tok * p.x_row + (long long)h * p.x_head + p.x_offset + k));
                    else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
                }
                const int n = n0 + r;
                dst = wt + r * HM_LDS + c;
                if (n < p.n && k < p.k) cp_async16(smem_u32(dst), w + (size_t)n * p.k + k);
                else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
            }
            if constexpr (sizeof(TI) == 4) {
                // float partial sums: every load of the slice is issued before the first value is rounded and stored
                constexpr int PER = HM_T * (HM_K / 8) / 128;
                float4 lo[PER], hi[PER];
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const int i = tid + j * 128, tok = t0 + (i >> 3), k = k0 + (i & 7) * 8;
                    lo[j] = hi[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (tok < p.n_tokens && k < p.k) {
                        const float* at = (const float*)p.x + (size_t)((long long)tok * p.x_row + (long long)h * p.x_head + p.x_offset + k);
                        for (int sp = 0; sp < p.x_splits; ++sp) {
                            const float4 a = *reinterpret_cast<const float4*>(at + (size_t)sp * p.x_split_stride);
                            const float4 b = reinterpret_cast<const float4*>(at + (size_t)sp * p.x_split_stride)[1];
                            lo[j].x += a.x; lo[j].y += a.y; lo[j].z += a.z; lo[j].w += a.w;
                            hi[j].x += b.x; hi[j].y += b.y; hi[j].z += b.z; hi[j].w += b.w;
                        }
                    }
                }
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const int i = tid + j * 128;
                    *reinterpret_cast<uint4*>(xs + (i >> 3) * HM_LDS + (i & 7) * 8) =
                        make_uint4(pack_bf16(lo[j].x, lo[j].y), pack_bf16(lo[j].z, lo[j].w), pack_bf16(hi[j].x, hi[j].y), pack_bf16(hi[j].z, hi[j].w));
                }
            }
        }
        cp_async_commit();
    };
    issue(0);
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f; }
    const uint32_t a_off = (uint32_t)((warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * HM_LDS + (lane >> 4) * 8) * 2u;
    const int mi = lane >> 3;
    const uint32_t b_off = (uint32_t)(((mi >> 1) * 8 + (lane & 7)) * HM_LDS + (mi & 1) * 8) * 2u;
    for (int slice = 0; slice < slices; ++slice) {
        issue(slice + 1);
        cp_async_wait<1>();
        __syncthreads();
        const uint32_t xs = smem_u32(tiles[slice & 1][0]), wt = smem_u32(tiles[slice & 1][1]);
#pragma unroll
        for (int ks = 0; ks < HM_K / 16; ++ks) {
            uint32_t a[4];
            ldmatrix_x4(a, xs + a_off + (uint32_t)ks * 32u);
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                uint32_t b[4];
                ldmatrix_x4(b, wt + b_off + (uint32_t)(np * 16 * HM_LDS + ks * 16) * 2u);
                mma_bf16(acc[2 * np], a, b[0], b[1]);
                mma_bf16(acc[2 * np + 1], a, b[2], b[3]);
            }
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    __nv_bfloat16* y = (__nv_bfloat16*)p.y;
    const bool paired = ((p.y_row | p.y_head | (long long)p.y_offset) & 1) == 0;
    if (p.gate) {
        // the gates of all of this thread's results are summed (split by split, the loads of a split independent of one
        // another) before the first result is stored
        float gates[8][4];
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) gates[nt][0] = gates[nt][1] = gates[nt][2] = gates[nt][3] = 0.f;
        for (int sp = 0; sp < p.gate_splits; ++sp) {
            const float* gate = p.gate + (size_t)sp * p.gate_split_stride;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int tok = t0 + warp * 16 + g + 8 * r;
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    const int n = n0 + nt * 8 + 2 * t;
                    const size_t at = (size_t)tok * p.gate_cols + p.gate_offset + (size_t)h * p.gate_head + (size_t)n * p.gate_elem;
                    if (tok < p.n_tokens && n < p.n) gates[nt][2 * r] += gate[at];
                    if (tok < p.n_tokens && n + 1 < p.n) gates[nt][2 * r + 1] += gate[at + p.gate_elem];
                }
            }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] = acc[nt][e] / (1.f + expf(-gates[nt][e]));
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int tok = t0 + warp * 16 + g + 8 * r;
        if (tok >= p.n_tokens) continue;
        __nv_bfloat16* dst = y + (size_t)((long long)tok * p.y_row + (long long)h * p.y_head + p.y_offset);
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const int n = n0 + nt * 8 + 2 * t;
            if (n >= p.n) continue;
            const float v0 = acc[nt][2 * r], v1 = acc[nt][2 * r + 1];
            if (paired && n + 1 < p.n) {
                *reinterpret_cast<uint32_t*>(dst + n) = pack_bf16(v0, v1);
            } else {
                dst[n] = __float2bfloat16_rn(v0);
                if (n + 1 < p.n) dst[n + 1] = __float2bfloat16_rn(v1);
            }
        }
    }
}

// The same for up to 64 tokens (one-token steps).  Bound by latency: a block's operands are a few ten KB, so all of K is asked for at once, the
// weights ahead of the dependency wait (no kernel of a step writes them), the gates with the rows.  A block forms 16 MT tokens x 8 NT outputs; NT
// is small so that the heads' matrices spread over the machine.  32 tokens of 16 heads, 128 x 512 10.3 us (21.7 us through the
// two-stage ring), 512 x 128 from float sums 6.4 us (8.0 us), in a step.
template <typename TI, int MT, int NT>
__global__ void __launch_bounds__(128) head_product_few_kernel(const HeadProductParams p, int k_padded) {
    using namespace qt_mma;
    extern __shared__ __align__(16) __nv_bfloat16 operands[];
    const int ld = k_padded + 8, pieces = k_padded / 8;
    __nv_bfloat16* ws = operands;                        // [8 NT][ld]
    __nv_bfloat16* xs = ws + 8 * NT * ld;                // [16 MT][ld]
    const int h = blockIdx.y, n0 = blockIdx.x * 8 * NT, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const __nv_bfloat16* w = (const __nv_bfloat16*)p.w + (size_t)h * p.n * p.k;
    pdl_launch_dependents();
    for (int i = tid; i < 8 * NT * pieces; i += 128) {
        const int r = i / pieces, c = (i - r * pieces) * 8;
        __nv_bfloat16* dst = ws + r * ld + c;
        if (n0 + r < p.n && c < p.k) cp_async16(smem_u32(dst), w + (size_t)(n0 + r) * p.k + c);
        else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
    }
    pdl_wait();
#pragma unroll 4
    for (int i = tid; i < 16 * MT * pieces; i += 128) {
        const int r = i / pieces, c = (i - r * pieces) * 8;
        __nv_bfloat16* dst = xs + r * ld + c;
        const bool there = r < p.n_tokens && c < p.k;
        const TI* at = (const TI*)p.x + (there ? (long long)r * p.x_row + (long long)h * p.x_head + p.x_offset + c : 0);
        if constexpr (sizeof(TI) == 2) {
            if (there) cp_async16(smem_u32(dst), at);
            else *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
        } else {
            float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
            if (there)
                for (int sp = 0; sp < p.x_splits; ++sp) {
                    const float4 a = *reinterpret_cast<const float4*>(at + (size_t)sp * p.x_split_stride), b = reinterpret_cast<const float4*>(at + (size_t)sp * p.x_split_stride)[1];
                    lo.x += a.x; lo.y += a.y; lo.z += a.z; lo.w += a.w;
                    hi.x += b.x; hi.y += b.y; hi.z += b.z; hi.w += b.w;
                }
            *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(lo.x, lo.y), pack_bf16(lo.z, lo.w), pack_bf16(hi.x, hi.y), pack_bf16(hi.z, hi.w));
        }
    }
    cp_async_commit();
    float gates[NT][4];
    if (p.gate && warp < MT) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) gates[nt][0] = gates[nt][1] = gates[nt][2] = gates[nt][3] = 0.f;
        for (int sp = 0; sp < p.gate_splits; ++sp)
#pragma unroll
            for (int e = 0; e < 4 * NT; ++e) {
                const int tok = warp * 16 + g + 8 * ((e >> 1) & 1), n = n0 + (e >> 2) * 8 + 2 * t + (e & 1);
                if (tok < p.n_tokens && n < p.n)
                    gates[e >> 2][e & 3] += p.gate[(size_t)sp * p.gate_split_stride + (size_t)tok * p.gate_cols + p.gate_offset + (size_t)h * p.gate_head + (size_t)n * p.gate_elem];
            }
    }
    cp_async_wait<0>();
    __syncthreads();
    if (warp >= MT) return;
    float acc[NT][4] = {};
    const uint32_t a_at = smem_u32(xs) + (uint32_t)((warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * ld + (lane >> 4) * 8) * 2u;
    const uint32_t b_at = smem_u32(ws) + (uint32_t)(((lane >> 4) * 8 + (lane & 7)) * ld + ((lane >> 3) & 1) * 8) * 2u;
#pragma unroll 4
    for (int k0 = 0; k0 < k_padded; k0 += 16) {
        uint32_t a[4];
        ldmatrix_x4(a, a_at + (uint32_t)k0 * 2u);
#pragma unroll
        for (int np = 0; np < NT / 2; ++np) {
            uint32_t b[4];
            ldmatrix_x4(b, b_at + (uint32_t)(np * 16 * ld + k0) * 2u);
            mma_bf16(acc[2 * np], a, b[0], b[1]);
            mma_bf16(acc[2 * np + 1], a, b[2], b[3]);
        }
    }
    __nv_bfloat16* y = (__nv_bfloat16*)p.y;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int tok = warp * 16 + g + 8 * (e >> 1), n = n0 + nt * 8 + 2 * t + (e & 1);
            const float v = p.gate ? acc[nt][e] / (1.f + expf(-gates[nt][e])) : acc[nt][e];
            if (tok < p.n_tokens && n < p.n) y[(size_t)((long long)tok * p.y_row + (long long)h * p.y_head + p.y_offset + n)] = __float2bfloat16_rn(v);
        }
}

constexpr int HF_MOST_TOKENS = 64, HF_MOST_K = 512;

// Where all of K at once is the faster form: up to 16 tokens, and up to 32 unless float rows meet the longest K on the most heads.  Every block
// of 32 outputs stages all rows again, so beyond 32 tokens only where that is little (few outputs a head and not too many blocks, or few blocks
// at all).  In microseconds, ring / all at once, T tokens, heads x outputs x K: T 64, 16 x 512 x 128 3.9 / 4.8, 128 x 512 x 128 9.9 / 15.8, 16 x 128 x
// 512 11.4 / 6.2, 64 x 128 x 512 14.1 / 9.7, 128 x 128 x 512 15.8 / 19.1 (from floats 26.9 / 37.4), 8 x 256 x 64 2.6 / 2.4, 16 x 256 x 256 4.2 / 5.7; T 32, 128 x
// 512 x 128 9.6 / 9.3, 128 x 128 x 512 17.0 / 15.0 (from floats 22.5 / 24.5).
static bool few_pays(const HeadProductParams& p, bool floats) {
    const long long blocks = (long long)p.heads * ((p.n + 31) / 32);
    if (p.n_tokens <= 16) return true;
    if (p.n_tokens <= 32) return !floats || p.k <= 128 || blocks * p.k < (1 << 18);
    return blocks <= 64 || (p.k >= 2 * p.n && blocks * p.k <= (1 << 17));
}

template <typename TI, int MT, int NT>
static int launch_head_few(const HeadProductParams& p, cudaStream_t s) {
    const int k_padded = (p.k + 15) / 16 * 16;
    const cudaError_t raised = raise_shared<head_product_few_kernel<TI, MT, NT>>((16 * MT + 8 * NT) * (HF_MOST_K + 8) * 2);
    if (raised != cudaSuccess) QT_FAIL(QT_ERR_LAUNCH, "head_product: cannot raise shared memory: %s", cudaGetErrorString(raised));
    launch_kernel(head_product_few_kernel<TI, MT, NT>, dim3((p.n + 8 * NT - 1) / (8 * NT), p.heads), dim3(128), (size_t)(16 * MT + 8 * NT) * (k_padded + 8) * 2, s, p, k_padded);
    QT_CHECK_LAUNCH("head_product_few");
    return QT_OK;
}
template <typename TI>
static int head_few(const HeadProductParams& p, cudaStream_t s) {
    // 32 outputs a block where that leaves every SM one, else 16
    const bool wide = (long long)((p.n + 31) / 32) * p.heads >= sm_count();
#define QT_HEAD_FEW(MT) return wide ? launch_head_few<TI, MT, 4>(p, s) : launch_head_few<TI, MT, 2>(p, s)
    if (p.n_tokens <= 16) QT_HEAD_FEW(1);
    if (p.n_tokens <= 32) QT_HEAD_FEW(2);
    QT_HEAD_FEW(4);
#undef QT_HEAD_FEW
}

extern "C" int qt_head_product(const void* x, int x_dtype, int x_splits, long long x_split_stride, long long x_row, long long x_head, int x_offset,
                               const void* w, int w_dtype, void* y, int y_dtype, long long y_row, long long y_head, int y_offset,
                               const float* gate, int gate_splits, long long gate_split_stride, int gate_cols, int gate_offset,
                               int gate_per_head, int n_tokens, int heads, int n, int k, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && heads > 0 && n > 0 && k > 0 && x_splits >= 1 && gate_splits >= 1, "head_product: bad sizes");
    QT_REQUIRE(heads <= 65535 && (n_tokens + HP_TM - 1) / HP_TM <= 65535, "head_product: too many heads or tokens for one launch");
    QT_REQUIRE(!gate || gate_offset + heads * (gate_per_head ? 1 : n) <= gate_cols, "head_product: the gate needs %d columns at %d of %d",
               heads * (gate_per_head ? 1 : n), gate_offset, gate_cols);
    if (n_tokens == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    HeadProductParams p{x, x_splits, (size_t)x_split_stride, x_row, x_head, x_offset, w, y, y_row, y_head, y_offset,
                        gate, gate_splits, (size_t)gate_split_stride, gate_cols, gate_offset, gate_per_head ? 1 : n, gate_per_head ? 0 : 1,
                        n_tokens, heads, n, k};
    dim3 grid((n + HP_TN - 1) / HP_TN, (n_tokens + HP_TM - 1) / HP_TM, heads);
    // bfloat16 matrices and results whose rows start on 16 bytes take the tensor cores (QT_B200_HEAD_PRODUCT_MMA=0: never)
    static const bool mma_allowed = [] { const char* env = getenv("QT_B200_HEAD_PRODUCT_MMA"); return !(env && env[0] == '0'); }();
    if (mma_allowed && w_dtype == QT_BF16 && y_dtype == QT_BF16 && k % 8 == 0 && (n_tokens + HM_T - 1) / HM_T <= 65535 &&
        ((x_dtype == QT_F32 && x_row % 4 == 0 && x_head % 4 == 0 && x_offset % 4 == 0 && x_split_stride % 4 == 0 && ((uintptr_t)x & 15) == 0) ||
         (x_dtype == QT_BF16 && x_splits == 1 && x_row % 8 == 0 && x_head % 8 == 0 && x_offset % 8 == 0 && ((uintptr_t)x & 15) == 0)) &&
        ((uintptr_t)w & 15) == 0) {
        if (n_tokens <= HF_MOST_TOKENS && k <= HF_MOST_K && few_pays(p, x_dtype == QT_F32)) return x_dtype == QT_F32 ? head_few<float>(p, s) : head_few<__nv_bfloat16>(p, s);
        dim3 tiles((n + HM_N - 1) / HM_N, (n_tokens + HM_T - 1) / HM_T, heads);
        if (x_dtype == QT_F32) launch_kernel(head_product_mma_kernel<float>, tiles, dim3(128), 0, s, p);
        else launch_kernel(head_product_mma_kernel<__nv_bfloat16>, tiles, dim3(128), 0, s, p);
        QT_CHECK_LAUNCH("head_product_mma");
        return QT_OK;
    }
#define QT_LAUNCH_HP(TI, TW, TO) launch_kernel(head_product_kernel<TI, TW, TO>, grid, dim3(256), 0, s, p)
    if (x_dtype == QT_F32 && w_dtype == QT_F32 && y_dtype == QT_F32) QT_LAUNCH_HP(float, float, float);
    else if (x_dtype == QT_F32 && w_dtype == QT_BF16 && y_dtype == QT_BF16) QT_LAUNCH_HP(float, __nv_bfloat16, __nv_bfloat16);
    else if (x_dtype == QT_BF16 && w_dtype == QT_BF16 && y_dtype == QT_BF16) QT_LAUNCH_HP(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
    else QT_FAIL(QT_ERR_ARG, "head_product: element types %d/%d/%d", x_dtype, w_dtype, y_dtype);
#undef QT_LAUNCH_HP
    QT_CHECK_LAUNCH("head_product");
    return QT_OK;
}

QT_DEFINE_LAST_ERROR(latent)
