// A recurrent mixer: the gated delta rule with one decay per head and key channel, and what surrounds it.
//
// Per head, with a state S [dim, vdim] of float that is carried from token to token of a sequence:
//     S <- diag(g_t) S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
// (o_t is read after token t has been written).  q and k come from kv heads (head h reads kv head h / (heads / kv_heads)),
// are unit vectors per head (q also times dim^-1/2), and q, k, v have passed a short causal convolution per channel and
// SiLU.  Everything here is float whatever the model's element type: the projections before it hand over float sums.
//
// Kernels, in the order of a step:
//   delta_prepare_kernel   convolution (its first taps - 1 inputs from the sequence's kept inputs or from zeros), SiLU, unit
//                          norms, beta = sigmoid(.)
//   conv_keep_kernel       the last taps - 1 raw inputs of every sequence, kept for its next step
//   lowrank_kernel         y = f(W2 (x) + bias) for a projection through a few columns (x is a slice of the first
//                          projection's output): f = -exp(rate_h) softplus(.), the logarithm of the decays, or sigmoid for a gate
//   delta_step_kernel      the recurrence token by token (steps of few tokens per sequence: a state is read and written once
//                          per step anyway, and the kernel is laid out for those bytes); delta_scan_kernel is an older
//                          form of it (QT_B200_DELTA_STEP=0), a column's rows over 8 lanes
//   delta_chunk_prepare_kernel, delta_chunk_walk_kernel (the usual sizes), delta_chunk_scan_kernel
//                          the same recurrence in chunks of 16 tokens for longer steps (see there)
//   gated_head_norm_kernel o / rms(o) * w * gate per head, into the element type of the output projection's input
#include "common.cuh"

#include <math.h>

using namespace qt;

constexpr int MAX_TAPS = 16;

struct PrepareParams {
    const float* proj; int n_splits; size_t split_stride; int proj_cols;    // [splits, T, proj_cols]; columns: q | k | v | beta | ...
    const float* taps;                // [channels, n_taps], the last column is the current token's
    const float* kept;                // [slots + 1, n_taps - 1, channels]: raw inputs of the positions just before the step
    const int* token_seq; const int* token_pos; const int* seq_start; const int* seq_past; const int* slots;
    float* q; float* k; float* v; float* beta;      // [T, kv_heads, dim] x 2, [T, heads, vdim], [T, heads]
    int n_tokens, heads, kv_heads, dim, vdim, n_taps;
    float unit_eps;
};

__device__ __forceinline__ float sigmoidf(float z) { return 1.f / (1.f + expf(-z)); }

// The sum of split-K partial sums in their order, eight loads in flight at a time.
__device__ __forceinline__ float sum_splits(const float* __restrict__ base, size_t index, int n_splits, size_t split_stride) {
    if (n_splits == 1) return base[index];
    float acc = 0.f;
    for (int s0 = 0; s0 < n_splits; s0 += 8) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = s0 + j < n_splits ? base[index + (size_t)(s0 + j) * split_stride] : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc += v[j];
    }
    return acc;
}
__device__ __forceinline__ float softplusf(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

// One warp per (token, item): items 0 .. kv_heads - 1 are the q heads, the next kv_heads the k heads, the next `heads`
// the v heads, the last one all betas of the token.
__global__ void __launch_bounds__(128) delta_prepare_kernel(const PrepareParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int items = 2 * p.kv_heads + p.heads + 1;
    const long long index = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
    if (index >= (long long)p.n_tokens * items) return;
    const int t = (int)(index / items), item = (int)(index % items);
    const size_t row = (size_t)t * p.proj_cols;
    const int channels = 2 * p.kv_heads * p.dim + p.heads * p.vdim;
    if (item == items - 1) {
        for (int h = lane; h < p.heads; h += 32)
            p.beta[(size_t)t * p.heads + h] = sigmoidf(sum_splits(p.proj, row + channels + h, p.n_splits, p.split_stride));
        return;
    }
    const int seq = p.token_seq[t];
    const int local = p.token_pos[t] - p.seq_past[seq];          // tokens of this sequence that the step has run before this one
    const float* kept = p.kept + (size_t)p.slots[seq] * (p.n_taps - 1) * channels;
    const bool is_q = item < p.kv_heads, is_k = !is_q && item < 2 * p.kv_heads;
    const int width = (is_q || is_k) ? p.dim : p.vdim;
    const int c0 = is_q ? item * p.dim : is_k ? p.kv_heads * p.dim + (item - p.kv_heads) * p.dim
                                              : 2 * p.kv_heads * p.dim + (item - 2 * p.kv_heads) * p.vdim;
    float* out = is_q ? p.q + ((size_t)t * p.kv_heads + item) * p.dim
               : is_k ? p.k + ((size_t)t * p.kv_heads + item - p.kv_heads) * p.dim
                      : p.v + ((size_t)t * p.heads + item - 2 * p.kv_heads) * p.vdim;
    float sq = 0.f;
    const float* __restrict__ proj = p.proj;
    const float* __restrict__ taps = p.taps;
    for (int i = lane; i < width; i += 32) {
        const int c = c0 + i;
        float acc = 0.f;
        for (int back0 = 0; back0 < p.n_taps; back0 += 4) {           // four taps at a time: their loads go out together
            float x[4], w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int back = back0 + j;
                x[j] = w[j] = 0.f;
                if (back < p.n_taps) {
                    w[j] = taps[(size_t)c * p.n_taps + p.n_taps - 1 - back];
                    if (back <= local) x[j] = sum_splits(proj, row - (size_t)back * p.proj_cols + c, p.n_splits, p.split_stride);
                    else x[j] = kept[(size_t)(p.n_taps - 1 - (back - local)) * channels + c];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) acc += w[j] * x[j];
        }
        const float y = acc / (1.f + expf(-acc));
        out[i] = y;
        sq += y * y;
    }
    if (is_q || is_k) {
        const float inv = rsqrtf(warp_sum(sq) + p.unit_eps) * (is_q ? rsqrtf((float)p.dim) : 1.f);
        __syncwarp();
        for (int i = lane; i < width; i += 32) out[i] *= inv;
    }
}

// kept[slot] <- the raw inputs of the sequence's last n_taps - 1 positions after this step.  One thread per
// (sequence, channel): it reads what it needs of the old rows before it writes.
__global__ void conv_keep_kernel(const float* proj, int n_splits, size_t split_stride, int proj_cols,
                                 float* __restrict__ kept, const int* seq_start, const int* slots,
                                 int n_seqs, int channels, int n_taps) {
    pdl_launch_dependents();
    pdl_wait();
    const int seq = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    const int row0 = seq_start[seq], count = seq_start[seq + 1] - row0;
    float* mine = kept + (size_t)slots[seq] * (n_taps - 1) * channels + c;
    float value[MAX_TAPS];
    const int rows = n_taps - 1;
    for (int j = 0; j < rows; ++j) {
        const int from = count - rows + j;                       // index among the step's tokens; negative: an older position
        value[j] = from >= 0 ? sum_splits(proj, (size_t)(row0 + from) * proj_cols + c, n_splits, split_stride)
                             : mine[(size_t)(rows + from) * channels];
    }
    for (int j = 0; j < rows; ++j) mine[(size_t)j * channels] = value[j];
}

// out[t, n] = f(sum_r w[r, n] x[t, r] + bias[n]) for a tile of LR_TOKENS tokens and 256 outputs per block.
constexpr int LR_TOKENS = 16;
constexpr int LR_DECAY = 0, LR_SIGMOID = 1, LR_LOG_SIGMOID = 2;

// f of a narrow projection: a decay's logarithm -rate softplus(z), sigmoid(z), or rate * log(sigmoid(z)) (the logarithm of a
// decay that is a power of a sigmoid).
template <int MODE>
__device__ __forceinline__ float lowrank_value(float z, float rate) {
    return MODE == LR_SIGMOID ? sigmoidf(z) : -rate * softplusf(MODE == LR_DECAY ? z : -z);
}

template <int MODE>
__global__ void __launch_bounds__(256) lowrank_kernel(const float* proj, int n_splits, size_t split_stride, int proj_cols,
                                                      int x_offset, int rank, const float* w, const float* bias,
                                                      const float* rate_log, int per_rate, float power, float* __restrict__ out,
                                                      int n_tokens, int n_out) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float xs[];                   // [rank][LR_TOKENS]: a column's 16 tokens side by side
    const int t0 = blockIdx.y * LR_TOKENS;
    const int count = min(LR_TOKENS, n_tokens - t0);
    for (int i = threadIdx.x; i < LR_TOKENS * rank; i += blockDim.x) {
        const int tt = i / rank, r = i % rank;
        xs[r * LR_TOKENS + tt] = tt < count ? sum_splits(proj, (size_t)(t0 + tt) * proj_cols + x_offset + r, n_splits, split_stride) : 0.f;
    }
    __syncthreads();
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= n_out) return;
    float acc[LR_TOKENS];
#pragma unroll
    for (int tt = 0; tt < LR_TOKENS; ++tt) acc[tt] = 0.f;
    for (int r0 = 0; r0 < rank; r0 += 8) {                            // eight weights at a time: their loads go out together
        float wv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) wv[j] = r0 + j < rank ? w[(size_t)(r0 + j) * n_out + n] : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (r0 + j < rank) {
                const float4* x4 = reinterpret_cast<const float4*>(xs + (r0 + j) * LR_TOKENS);
#pragma unroll
                for (int q = 0; q < LR_TOKENS / 4; ++q) {
                    const float4 x = x4[q];
                    acc[4 * q] += wv[j] * x.x; acc[4 * q + 1] += wv[j] * x.y; acc[4 * q + 2] += wv[j] * x.z; acc[4 * q + 3] += wv[j] * x.w;
                }
            }
        }
    }
    const float b = bias ? bias[n] : 0.f;
    const float rate = MODE == LR_DECAY ? expf(rate_log[n / per_rate]) : power;
#pragma unroll
    for (int tt = 0; tt < LR_TOKENS; ++tt) {
        if (tt >= count) break;
        const float z = acc[tt] + b;
        out[(size_t)(t0 + tt) * n_out + n] = lowrank_value<MODE>(z, rate);
    }
}

// The same for a step of few tokens (up to 16 tiles of them): 64 outputs per block, so that many SMs get one, and the
// columns cut into four ranges, one per 64 threads, whose sums meet in shared memory.
template <int MODE>
__global__ void __launch_bounds__(256) lowrank_few_kernel(const float* proj, int n_splits, size_t split_stride, int proj_cols,
                                                          int x_offset, int rank, const float* w, const float* bias,
                                                          const float* rate_log, int per_rate, float power, float* __restrict__ out,
                                                          int n_tokens, int n_out) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float xs[];                                 // [LR_TOKENS][rank], then [4][LR_TOKENS][64] partial sums
    float* part = xs + LR_TOKENS * rank;
    const int t0 = blockIdx.y * LR_TOKENS;
    n_tokens = min(LR_TOKENS, n_tokens - t0);                     // of this tile
    out += (size_t)t0 * n_out;
    for (int i = threadIdx.x; i < LR_TOKENS * rank; i += blockDim.x) {
        const int tt = i / rank, r = i % rank;
        xs[i] = tt < n_tokens ? sum_splits(proj, (size_t)(t0 + tt) * proj_cols + x_offset + r, n_splits, split_stride) : 0.f;
    }
    __syncthreads();
    const int local = threadIdx.x & 63, slice = threadIdx.x >> 6;
    const int n = blockIdx.x * 64 + local;
    const int per = (rank + 3) / 4, r_begin = slice * per, r_end = min(rank, r_begin + per);
    float acc[LR_TOKENS];
#pragma unroll
    for (int tt = 0; tt < LR_TOKENS; ++tt) acc[tt] = 0.f;
    if (n < n_out) {
        for (int r0 = r_begin; r0 < r_end; r0 += 8) {
            float wv[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) wv[j] = r0 + j < r_end ? w[(size_t)(r0 + j) * n_out + n] : 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (r0 + j < r_end) {
#pragma unroll
                    for (int tt = 0; tt < LR_TOKENS; ++tt) acc[tt] += wv[j] * xs[tt * rank + r0 + j];
                }
            }
        }
    }
#pragma unroll
    for (int tt = 0; tt < LR_TOKENS; ++tt) part[(slice * LR_TOKENS + tt) * 64 + local] = acc[tt];
    __syncthreads();
    if (n >= n_out) return;
    const float b = bias ? bias[n] : 0.f;
    const float rate = MODE == LR_DECAY ? expf(rate_log[n / per_rate]) : power;
    for (int tt = slice; tt < n_tokens; tt += 4) {                 // the four ranges' sums in their order
        const float z = part[(0 * LR_TOKENS + tt) * 64 + local] + part[(1 * LR_TOKENS + tt) * 64 + local] +
                        part[(2 * LR_TOKENS + tt) * 64 + local] + part[(3 * LR_TOKENS + tt) * 64 + local] + b;
        out[(size_t)tt * n_out + n] = lowrank_value<MODE>(z, rate);
    }
}

// ----------------------------------------------------------------------------- the recurrence
// grid (column blocks, heads, sequences).  A block of 256 threads owns SCAN_COLS = 32 columns of one head's state; a
// column belongs to 8 neighbouring lanes, lane s of them holding rows s, s + 8, ... (R of them) in registers.  The
// tokens' q, k and decays (shared by the block), and the block's v columns and beta, pass through shared memory in chunks
// of SCAN_CHUNK tokens, the next chunk fetched (cp.async) while this one is worked on.
constexpr int SCAN_COLS = 32;
constexpr int SCAN_LANES = 8;
constexpr int SCAN_CHUNK = 16;

struct ScanParams {
    const float* q; const float* k; const float* v; const float* beta; const float* decay;      // decay: logarithms, [T, heads, dim]
    float* state;                 // [slots + 1, heads, dim, vdim]
    float* out;                   // [T, heads, vdim]
    const int* seq_start; const int* slots;
    int heads, kv_heads, dim, vdim;
};

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int R>
__global__ void __launch_bounds__(SCAN_COLS * SCAN_LANES) delta_scan_kernel(const ScanParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float sm[];
    const int dim = p.dim, vdim = p.vdim;
    const int per_token = 3 * dim + SCAN_COLS + 1;                 // q, k, decay, the block's v columns, beta
    float* buffers[2] = {sm, sm + SCAN_CHUNK * per_token};
    const int head = blockIdx.y, seq = blockIdx.z;
    const int kvh = head / (p.heads / p.kv_heads);
    const int col = threadIdx.x / SCAN_LANES, sub = threadIdx.x % SCAN_LANES;
    const int j = blockIdx.x * SCAN_COLS + col;
    const bool live = j < vdim;
    const int row0 = p.seq_start[seq], count = p.seq_start[seq + 1] - row0;
    float* state = p.state + ((size_t)p.slots[seq] * p.heads + head) * dim * vdim;

    float s[R];
#pragma unroll
    for (int m = 0; m < R; ++m) {
        const int i = sub + SCAN_LANES * m;
        s[m] = (live && i < dim) ? state[(size_t)i * vdim + j] : 0.f;
    }
    auto fetch = [&](int chunk, float* buf) {
        const int first = chunk * SCAN_CHUNK, n = min(SCAN_CHUNK, count - first);
        for (int e = threadIdx.x; e < n * per_token; e += blockDim.x) {
            const int tt = e / per_token, c = e % per_token;
            const size_t t = (size_t)(row0 + first + tt);
            const float* src;
            if (c < dim) src = p.q + (t * p.kv_heads + kvh) * dim + c;
            else if (c < 2 * dim) src = p.k + (t * p.kv_heads + kvh) * dim + (c - dim);
            else if (c < 3 * dim) src = p.decay + (t * p.heads + head) * dim + (c - 2 * dim);
            else if (c < 3 * dim + SCAN_COLS) {
                const int jj = blockIdx.x * SCAN_COLS + (c - 3 * dim);
                src = p.v + (t * p.heads + head) * vdim + (jj < vdim ? jj : vdim - 1);
            } else src = p.beta + t * p.heads + head;
            cp_async4(buf + e, src);
        }
        cp_async_commit();
    };
    const int chunks = (count + SCAN_CHUNK - 1) / SCAN_CHUNK;
    if (chunks > 0) fetch(0, buffers[0]);
    for (int chunk = 0; chunk < chunks; ++chunk) {
        cp_async_wait_all();
        __syncthreads();                                           // this chunk has landed; everyone is done with the other buffer
        if (chunk + 1 < chunks) fetch(chunk + 1, buffers[(chunk + 1) & 1]);
        const float* buf = buffers[chunk & 1];
        const int n = min(SCAN_CHUNK, count - chunk * SCAN_CHUNK);
        for (int tt = 0; tt < n; ++tt) {
            const float* q = buf + tt * per_token;
            const float* k = q + dim;
            const float* g = k + dim;
            const float vj = q[3 * dim + col], beta = q[3 * dim + SCAN_COLS];
            float kk[R];
            float pred = 0.f;
#pragma unroll
            for (int m = 0; m < R; ++m) {
                const int i = sub + SCAN_LANES * m;
                const bool in = i < dim;
                kk[m] = in ? k[i] : 0.f;
                s[m] *= in ? expf(g[i]) : 1.f;                      // `decay` holds logarithms
                pred += s[m] * kk[m];
            }
            pred += __shfl_xor_sync(0xffffffffu, pred, 1);
            pred += __shfl_xor_sync(0xffffffffu, pred, 2);
            pred += __shfl_xor_sync(0xffffffffu, pred, 4);
            const float u = beta * (vj - pred);
            float o = 0.f;
#pragma unroll
            for (int m = 0; m < R; ++m) {
                const int i = sub + SCAN_LANES * m;
                s[m] += kk[m] * u;
                o += s[m] * (i < dim ? q[i] : 0.f);
            }
            o += __shfl_xor_sync(0xffffffffu, o, 1);
            o += __shfl_xor_sync(0xffffffffu, o, 2);
            o += __shfl_xor_sync(0xffffffffu, o, 4);
            if (sub == 0 && live) p.out[((size_t)(row0 + chunk * SCAN_CHUNK + tt) * p.heads + head) * vdim + j] = o;
        }
    }
#pragma unroll
    for (int m = 0; m < R; ++m) {
        const int i = sub + SCAN_LANES * m;
        if (live && i < dim) state[(size_t)i * vdim + j] = s[m];
    }
}

// ----------------------------------------------------------------------------- the recurrence in chunks
// Within a chunk of CH tokens that starts from the state S0, with L_t the sum of the decays' logarithms up to token t
// of the chunk (per key channel), the recurrence unrolls to
//     u_t = beta_t (v_t - S0^T (e^{L_t} k_t) - sum_{s<t} A[t,s] u_s),      A[t,s] = sum_c k_t[c] k_s[c] e^{L_t[c] - L_s[c]}
//     o_t = S0^T (e^{L_t} q_t) + sum_{s<=t} B[t,s] u_s,                    B[t,s] = sum_c q_t[c] k_s[c] e^{L_t[c] - L_s[c]}
//     S   = diag(e^{L_last}) S0 + sum_s (e^{L_last - L_s} k_s) u_s^T
// Every exponent is a sum of logarithms of decays over a range of tokens, so it is <= 0: nothing is divided by a decay.
// What does not depend on the state (the scaled keys and queries and the two triangles) is made for all chunks of all
// heads at once by delta_chunk_prepare_kernel; delta_chunk_scan_kernel then walks the chunks of a sequence with the
// state's columns in registers, and its work per chunk has no chain from token to token but the small triangular
// solve.  All float; the result differs from the token-by-token kernel by rounding only.
constexpr int CH = 16;
constexpr int AB = 2 * CH + 4;      // floats of a token's row of `ab`: its columns of the two triangles, beta, padding to 16 bytes

struct ChunkParams {
    const float* q; const float* k; const float* log_decay;      // [T, kv_heads, dim] x 2, [T, heads, dim]
    float* kt; float* qt; float* kb; float* gc;                    // [T, heads, dim]: e^{L_t} k_t, e^{L_t} q_t, e^{L_last - L_t} k_t; e^{L_last} in a chunk's first row
    const float* beta;                                             // [T, heads]
    // [T, heads, AB], beta at [2 CH] and in front of it, for delta_chunk_scan_kernel, a token s's columns of the triangles: A[t, s] for every
    // t of its chunk (0 unless s < t), then B[t, s] (0 unless s <= t).  solved, for delta_chunk_walk_kernel: a token t's rows, of
    // (I + diag(beta) A)^-1 and of B
    float* ab;
    const int* seq_start;
    int heads, kv_heads, dim, solved;
};

// Sixteen values per lane, summed over the lanes of the warp: lane l gets the sum of value l % 16.
__device__ __forceinline__ float transpose_sum(float (&part)[CH], int lane) {
#pragma unroll
    for (int half = CH / 2; half >= 1; half >>= 1) {
        const bool upper = (lane & half) != 0;
#pragma unroll
        for (int j = 0; j < half; ++j) {
            const float give = upper ? part[j] : part[j + half], keep = upper ? part[j + half] : part[j];
            part[j] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    return part[0] + __shfl_xor_sync(0xffffffffu, part[0], 16);
}

// grid (chunks of the longest sequence, heads, sequences), 128 threads.  The triangles: a warp takes two neighbouring s, its lanes hold
// k_s decayed so far and multiply it by e^{g_t} as t goes on (an exponential per pair and channel took half of the kernel's time:
// 2,048 tokens of 16 heads of 128 97 us, 43 us so).
template <int V> struct Elems { float v[V]; };
template <int V> __device__ __forceinline__ Elems<V> get(const float* p) {
    Elems<V> r;
    if constexpr (V == 4) { const float4 x = *reinterpret_cast<const float4*>(p); r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w; }
    else r.v[0] = *p;
    return r;
}
template <int V> __device__ __forceinline__ void put(float* p, const Elems<V>& r) {
    if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
    else *p = r.v[0];
}

// V: neighbouring channels a thread loads at once (4 where every row starts on a 16-byte boundary)
template <int V>
__global__ void __launch_bounds__(128) delta_chunk_prepare_kernel(const ChunkParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    __shared__ float tri_a[CH][CH + 1], tri_b[CH][CH + 1], inverse[CH][CH + 1], betas[CH];      // [t][s]
    const int dim = p.dim, head = blockIdx.y, seq = blockIdx.z, pieces = dim / V;
    const int kvh = head / (p.heads / p.kv_heads);
    const int row0 = p.seq_start[seq], count = p.seq_start[seq + 1] - row0;
    const int first = blockIdx.x * CH;
    if (first >= count) return;
    const int n = min(CH, count - first);
    float* qs = sm;                       // [CH][dim]
    float* ks = qs + CH * dim;            // [CH][dim]
    float* ls = ks + CH * dim;            // [CH][dim] logarithms of the decays
    float* gs = ls + CH * dim;            // [CH][dim] decays
#pragma unroll 4
    for (int e = threadIdx.x; e < CH * pieces; e += 128) {
        const int tt = e / pieces, c = V * (e - tt * pieces);
        const size_t t = (size_t)(row0 + first + tt);
        Elems<V> q = {}, k = {}, g = {};
        if (tt < n) {
            q = get<V>(p.q + (t * p.kv_heads + kvh) * dim + c);
            k = get<V>(p.k + (t * p.kv_heads + kvh) * dim + c);
            g = get<V>(p.log_decay + (t * p.heads + head) * dim + c);
        }
        put<V>(qs + V * e, q);
        put<V>(ks + V * e, k);
        put<V>(ls + V * e, g);
#pragma unroll
        for (int i = 0; i < V; ++i) g.v[i] = expf(g.v[i]);
        put<V>(gs + V * e, g);
    }
    if (threadIdx.x < CH) betas[threadIdx.x] = threadIdx.x < n ? p.beta[(size_t)(row0 + first + threadIdx.x) * p.heads + head] : 0.f;
    __syncthreads();
    // a channel's running sums, in double: 16 additions and a difference cost nothing here, and every key and query of the walk carries their rounding
    for (int c = threadIdx.x; c < dim; c += 128) {
        double upto[CH];
#pragma unroll
        for (int tt = 0; tt < CH; ++tt) upto[tt] = (tt ? upto[tt - 1] : 0.0) + (double)ls[tt * dim + c];
        const size_t at = ((size_t)(row0 + first) * p.heads + head) * dim + c, row = (size_t)p.heads * dim;
#pragma unroll
        for (int tt = 0; tt < CH; ++tt) {
            if (tt >= n) break;
            const float grow = expf((float)upto[tt]), rest = expf((float)(upto[CH - 1] - upto[tt])), k = ks[tt * dim + c];     // missing tokens add 0
            p.kt[at + tt * row] = grow * k;
            p.qt[at + tt * row] = grow * qs[tt * dim + c];
            p.kb[at + tt * row] = rest * k;
        }
        p.gc[at] = expf((float)upto[CH - 1]);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int s = 2 * warp; s < CH; s += 8) {
        float a0[CH], a1[CH], b0[CH], b1[CH];
#pragma unroll
        for (int t = 0; t < CH; ++t) a0[t] = a1[t] = b0[t] = b1[t] = 0.f;
        for (int c = lane; c < dim; c += 32) {
            float w0 = ks[s * dim + c], w1 = ks[(s + 1) * dim + c];
#pragma unroll
            for (int t = 0; t < CH; ++t) {
                if (t < s) continue;
                const float q = qs[t * dim + c], k = ks[t * dim + c], g = gs[t * dim + c];
                if (t > s) { w0 *= g; a0[t] = fmaf(k, w0, a0[t]); }
                b0[t] = fmaf(q, w0, b0[t]);
                if (t > s + 1) { w1 *= g; a1[t] = fmaf(k, w1, a1[t]); }
                if (t > s) b1[t] = fmaf(q, w1, b1[t]);
            }
        }
        const float ra0 = transpose_sum(a0, lane), ra1 = transpose_sum(a1, lane), rb0 = transpose_sum(b0, lane), rb1 = transpose_sum(b1, lane);
        if (lane < CH) { tri_a[lane][s] = ra0; tri_a[lane][s + 1] = ra1; tri_b[lane][s] = rb0; tri_b[lane][s + 1] = rb1; }
    }
    __syncthreads();
    if (p.solved && warp == 0) {                                            // lane j: column j of the inverse, from the top
        const int j = lane & (CH - 1);
        float x[CH];
#pragma unroll
        for (int t = 0; t < CH; ++t) {
            float sum = 0.f;
#pragma unroll
            for (int s = 0; s < CH; ++s)
                if (s < t) sum = fmaf(tri_a[t][s], x[s], sum);
            x[t] = (t == j ? 1.f : 0.f) - betas[t] * sum;
            if (lane < CH) inverse[t][j] = x[t];
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * 2 * CH; e += blockDim.x) {
        const int tt = e / (2 * CH), c = e % CH;
        const bool second = e % (2 * CH) >= CH;
        float* row = p.ab + ((size_t)(row0 + first + tt) * p.heads + head) * AB;
        if (p.solved) row[e % (2 * CH)] = second ? tri_b[tt][c] : inverse[tt][c];
        else row[e % (2 * CH)] = second ? tri_b[c][tt] : tri_a[c][tt];
        if (c == 0 && !second) row[2 * CH] = betas[tt];
    }
}

struct ChunkScanParams {
    const float* kt; const float* qt; const float* kb; const float* gc; const float* ab;
    const float* v; const float* beta;
    float* state; float* out;
    const int* seq_start; const int* slots;
    int heads, dim, vdim;
};

// grid (column blocks, heads, sequences); threads as in delta_scan_kernel: a column of the state belongs to 8 neighbouring
// lanes, lane s of them holding rows s, s + 8, ...
template <int R>
__global__ void __launch_bounds__(SCAN_COLS * SCAN_LANES) delta_chunk_scan_kernel(const ChunkScanParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float sm[];
    const int dim = p.dim, vdim = p.vdim;
    const int per_token = 3 * dim + 2 * CH + SCAN_COLS + 1;       // kt, qt, kb rows, the A and B rows, the block's v columns, beta
    const int per_chunk = CH * per_token + dim;                   // and the chunk's whole decay
    float* buffers[2] = {sm, sm + per_chunk};
    const int head = blockIdx.y, seq = blockIdx.z;
    const int col = threadIdx.x / SCAN_LANES, sub = threadIdx.x % SCAN_LANES;
    const int j = blockIdx.x * SCAN_COLS + col;
    const bool live = j < vdim;
    const int row0 = p.seq_start[seq], count = p.seq_start[seq + 1] - row0;
    float* state = p.state + ((size_t)p.slots[seq] * p.heads + head) * dim * vdim;

    float s[R];
#pragma unroll
    for (int m = 0; m < R; ++m) {
        const int i = sub + SCAN_LANES * m;
        s[m] = (live && i < dim) ? state[(size_t)i * vdim + j] : 0.f;
    }
    auto fetch = [&](int chunk, float* buf) {
        const int first = chunk * CH, n = min(CH, count - first);
        for (int e = threadIdx.x; e < n * per_token + dim; e += blockDim.x) {
            const float* src;
            float* dst;
            if (e < n * per_token) {
                const int tt = e / per_token, c = e % per_token;
                const size_t at = (size_t)(row0 + first + tt) * p.heads + head;
                if (c < dim) src = p.kt + at * dim + c;
                else if (c < 2 * dim) src = p.qt + at * dim + (c - dim);
                else if (c < 3 * dim) src = p.kb + at * dim + (c - 2 * dim);
                else if (c < 3 * dim + 2 * CH) src = p.ab + at * AB + (c - 3 * dim);
                else if (c < 3 * dim + 2 * CH + SCAN_COLS) {
                    const int jj = blockIdx.x * SCAN_COLS + (c - 3 * dim - 2 * CH);
                    src = p.v + at * vdim + (jj < vdim ? jj : vdim - 1);
                } else src = p.beta + at;
                dst = buf + e;
            } else {
                src = p.gc + ((size_t)(row0 + first) * p.heads + head) * dim + (e - n * per_token);
                dst = buf + CH * per_token + (e - n * per_token);
            }
            cp_async4(dst, src);
        }
        cp_async_commit();
    };
    const int chunks = (count + CH - 1) / CH;
    if (chunks > 0) fetch(0, buffers[0]);
    for (int chunk = 0; chunk < chunks; ++chunk) {
        cp_async_wait_all();
        __syncthreads();
        if (chunk + 1 < chunks) fetch(chunk + 1, buffers[(chunk + 1) & 1]);
        const float* buf = buffers[chunk & 1];
        const int n = min(CH, count - chunk * CH);
        // what the state holds for every token of the chunk: S0^T (e^L k_t) and S0^T (e^L q_t), summed over the 8 lanes of the column
        float pred[CH], read[CH];
#pragma unroll
        for (int tt = 0; tt < CH; ++tt) {
            float a = 0.f, b = 0.f;
            if (tt < n) {
                const float* kt = buf + tt * per_token;
                const float* qt = kt + dim;
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    const int i = sub + SCAN_LANES * m;
                    if (i < dim) { a += kt[i] * s[m]; b += qt[i] * s[m]; }
                }
            }
            pred[tt] = a;
            read[tt] = b;
        }
#pragma unroll
        for (int tt = 0; tt < CH; ++tt) {
            pred[tt] += __shfl_xor_sync(0xffffffffu, pred[tt], 1);
            read[tt] += __shfl_xor_sync(0xffffffffu, read[tt], 1);
            pred[tt] += __shfl_xor_sync(0xffffffffu, pred[tt], 2);
            read[tt] += __shfl_xor_sync(0xffffffffu, read[tt], 2);
            pred[tt] += __shfl_xor_sync(0xffffffffu, pred[tt], 4);
            read[tt] += __shfl_xor_sync(0xffffffffu, read[tt], 4);
        }
        // the triangular solve, the same in each of the column's lanes; pred[t] turns into u_t
#pragma unroll
        for (int tt = 0; tt < CH; ++tt) {
            if (tt < n) {
                const float* row = buf + tt * per_token + 3 * dim;            // the token's columns of A and B, v columns, beta
                const float u = row[2 * CH + SCAN_COLS] * (row[2 * CH + col] - pred[tt]);
                pred[tt] = u;
#pragma unroll
                for (int later = tt + 1; later < CH; ++later)
                    if (later < n) pred[later] += row[later] * u;
#pragma unroll
                for (int later = tt; later < CH; ++later)
                    if (later < n) read[later] += row[CH + later] * u;
            }
        }
        if (sub == 0 && live) {
#pragma unroll
            for (int tt = 0; tt < CH; ++tt)
                if (tt < n) p.out[((size_t)(row0 + chunk * CH + tt) * p.heads + head) * vdim + j] = read[tt];
        }
        // the state behind the chunk
        const float* gc = buf + CH * per_token;
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const int i = sub + SCAN_LANES * m;
            if (i < dim) {
                float acc = gc[i] * s[m];
#pragma unroll
                for (int tt = 0; tt < CH; ++tt)
                    if (tt < n) acc += buf[tt * per_token + 2 * dim + i] * pred[tt];
                s[m] = acc;
            }
        }
    }
#pragma unroll
    for (int m = 0; m < R; ++m) {
        const int i = sub + SCAN_LANES * m;
        if (live && i < dim) state[(size_t)i * vdim + j] = s[m];
    }
}

// The same walk for the usual sizes (dim = 64 P up to 256, vdim a multiple of 16).  A sequence's chunks follow one another, so what counts is
// the time of one chunk: above all its reads of shared memory (ncu, the prompt below: that pipe 80 % busy, FMA 31 %, issue slots 43 %) and the chain from S0 to the next S.  A warp owns two columns of
// the state, a lane 2 P rows of each as P pairs of neighbouring rows (fma.rn.f32x2), so every 16 bytes of a key, a query or a decay that a
// lane reads serve two columns, and everything but the chunk's data stays within the warp.  Per chunk: the sums over the rows, S0^T (e^L
// k) and S0^T (e^L q), are reduced so that lane (h, l) ends with token l of column h (31 exchanges each); r = beta (v - S0^T (e^L k)) and
// u = (I + diag(beta) A)^-1 r pass through shared memory, 16 independent products in the place of a solve from token to
// token; then S.  Chunk data arrives by 16-byte copies under the chunk before; a chunk's missing tokens are zeros, which
// change nothing.  grid (vdim / 16, heads, sequences), 256 threads.  16 heads of 128 x 128, one prompt of 2,048 tokens: 255 us;
// 298 us with four columns a warp (one warp a scheduler, which then issues every third cycle); 451 us with one column over 16
// lanes and the solve passed on by shuffles.
constexpr int WALK_COLS = 16, WALK_THREADS = 256;

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpair(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The first row of a lane's pair m, and a lane's P pairs of neighbouring elements of a row of 64 P.
template <int P> __device__ __forceinline__ int pair_row(int lane, int m) { return P % 2 ? 2 * (lane + 32 * m) : 4 * (lane + 32 * (m / 2)) + 2 * (m & 1); }
template <int P> __device__ __forceinline__ void load_pairs(const float* row, int lane, unsigned long long (&v)[P]) {
    if constexpr (P % 2) {
#pragma unroll
        for (int m = 0; m < P; ++m) v[m] = *reinterpret_cast<const unsigned long long*>(row + 2 * (lane + 32 * m));
    } else {
#pragma unroll
        for (int m = 0; m < P; m += 2) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(row + 4 * (lane + 32 * (m / 2)));
            v[m] = x.x; v[m + 1] = x.y;
        }
    }
}

// sum over the state's rows of rows[t][.] s[.][c] for 16 tokens and 2 columns: lane (h, l) gets token l, column h
template <int P> __device__ __forceinline__ float column_sums(const float* rows, const unsigned long long (&s)[P][2], int lane) {
    float x[CH][2];
#pragma unroll
    for (int t = 0; t < CH; ++t) {
        unsigned long long k[P];
        load_pairs<P>(rows + t * 64 * P, lane, k);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            unsigned long long acc = 0ull;
#pragma unroll
            for (int m = 0; m < P; ++m) acc = fma_pair(k[m], s[m][c], acc);
            const float2 both = unpair(acc);
            x[t][c] = both.x + both.y;
        }
    }
    const bool right = (lane & 16) != 0;
    float y[CH];
#pragma unroll
    for (int t = 0; t < CH; ++t) {
        const float give = right ? x[t][0] : x[t][1], keep = right ? x[t][1] : x[t][0];
        y[t] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
    for (int half = CH / 2; half >= 1; half >>= 1) {
        const bool upper = (lane & half) != 0;
#pragma unroll
        for (int t = 0; t < half; ++t) {
            const float give = upper ? y[t] : y[t + half], keep = upper ? y[t + half] : y[t];
            y[t] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    return y[0];
}

// sum over s of row[s] x[s]
__device__ __forceinline__ float token_sum(const float* row, const float* x) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < CH; s += 4) {
        const float4 w = *reinterpret_cast<const float4*>(row + s), v = *reinterpret_cast<const float4*>(x + s);
        sum[0] = fmaf(w.x, v.x, sum[0]);
        sum[1] = fmaf(w.y, v.y, sum[1]);
        sum[2] = fmaf(w.z, v.z, sum[2]);
        sum[3] = fmaf(w.w, v.w, sum[3]);
    }
    return (sum[0] + sum[1]) + (sum[2] + sum[3]);
}

template <int P>
__global__ void __launch_bounds__(WALK_THREADS) delta_chunk_walk_kernel(const ChunkScanParams p) {
    constexpr int DIM = 64 * P, ROWS = CH * DIM;
    constexpr int PER_CHUNK = 3 * ROWS + CH * AB + CH * WALK_COLS + DIM;     // kt, qt, kb, the tokens' rows of `ab`, v columns, e^{L_last}
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float wanted[WALK_COLS][CH], found[WALK_COLS][CH];     // r and u of the block's columns
    const int vdim = p.vdim, head = blockIdx.y, seq = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = lane >> 4, l = lane & 15;
    const int col = 2 * warp + h, j0 = blockIdx.x * WALK_COLS + 2 * warp;
    const int row0 = p.seq_start[seq], count = p.seq_start[seq + 1] - row0;
    float* state = p.state + ((size_t)p.slots[seq] * p.heads + head) * DIM * vdim + j0;

    unsigned long long s[P][2];
#pragma unroll
    for (int m = 0; m < P; ++m) {
        const float2 a = *reinterpret_cast<const float2*>(state + (size_t)pair_row<P>(lane, m) * vdim);
        const float2 b = *reinterpret_cast<const float2*>(state + (size_t)(pair_row<P>(lane, m) + 1) * vdim);
        s[m][0] = pair_of(a.x, b.x); s[m][1] = pair_of(a.y, b.y);
    }
    auto fetch = [&](int chunk) {
        float* buf = sm + (chunk & 1) * PER_CHUNK;
        const int first = chunk * CH, n = min(CH, count - first);
        const size_t at0 = (size_t)(row0 + first) * p.heads + head;
        auto piece = [&](float* dst, const float* src, int tt) {
            if (tt < n) cp_async16(dst, src);
            else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
        };
#pragma unroll
        for (int i = 0; i < ROWS / 4 / WALK_THREADS; ++i) {
            const int e = threadIdx.x + i * WALK_THREADS, tt = e / (DIM / 4), c = 4 * (e % (DIM / 4));
            const size_t at = (at0 + (size_t)tt * p.heads) * DIM + c;
            piece(buf + 4 * e, p.kt + at, tt);
            piece(buf + ROWS + 4 * e, p.qt + at, tt);
            piece(buf + 2 * ROWS + 4 * e, p.kb + at, tt);
        }
        static_assert(CH * AB / 4 <= WALK_THREADS && CH * WALK_COLS / 4 <= WALK_THREADS && DIM / 4 <= WALK_THREADS, "a piece a thread");
        if (threadIdx.x < CH * AB / 4) {
            const int tt = threadIdx.x / (AB / 4);
            piece(buf + 3 * ROWS + 4 * threadIdx.x, p.ab + (at0 + (size_t)tt * p.heads) * AB + 4 * (threadIdx.x % (AB / 4)), tt);
        }
        if (threadIdx.x < CH * WALK_COLS / 4) {
            const int tt = threadIdx.x / (WALK_COLS / 4);
            piece(buf + 3 * ROWS + CH * AB + 4 * threadIdx.x, p.v + (at0 + (size_t)tt * p.heads) * vdim + blockIdx.x * WALK_COLS + 4 * (threadIdx.x % (WALK_COLS / 4)), tt);
        }
        if (threadIdx.x < DIM / 4) cp_async16(buf + PER_CHUNK - DIM + 4 * threadIdx.x, p.gc + at0 * DIM + 4 * threadIdx.x);
        cp_async_commit();
    };
    const int chunks = (count + CH - 1) / CH;
    if (chunks > 0) fetch(0);
    for (int chunk = 0; chunk < chunks; ++chunk) {
        cp_async_wait_all();
        __syncthreads();                                                    // this chunk has landed; everyone is done with the other buffer
        if (chunk + 1 < chunks) fetch(chunk + 1);
        const float* buf = sm + (chunk & 1) * PER_CHUNK;
        const float* ab = buf + 3 * ROWS + l * AB;                          // token l's rows of the inverse and of B, its beta
        const float pred = column_sums<P>(buf, s, lane);
        wanted[col][l] = ab[2 * CH] * (buf[3 * ROWS + CH * AB + l * WALK_COLS + col] - pred);
        __syncwarp();
        found[col][l] = token_sum(ab, wanted[col]);
        const float o = column_sums<P>(buf + ROWS, s, lane);                // reads the old state
        __syncwarp();
        unsigned long long g[P];
        load_pairs<P>(buf + PER_CHUNK - DIM, lane, g);
#pragma unroll
        for (int m = 0; m < P; ++m)
#pragma unroll
            for (int c = 0; c < 2; ++c) s[m][c] = fma_pair(s[m][c], g[m], 0ull);
#pragma unroll
        for (int t0 = 0; t0 < CH; t0 += 4) {
            const float4 u[2] = {*reinterpret_cast<const float4*>(&found[2 * warp][t0]), *reinterpret_cast<const float4*>(&found[2 * warp + 1][t0])};
            const float us[2][4] = {{u[0].x, u[0].y, u[0].z, u[0].w}, {u[1].x, u[1].y, u[1].z, u[1].w}};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                unsigned long long kb[P];
                load_pairs<P>(buf + 2 * ROWS + (t0 + i) * DIM, lane, kb);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const unsigned long long uu = pair_of(us[c][i], us[c][i]);
#pragma unroll
                    for (int m = 0; m < P; ++m) s[m][c] = fma_pair(kb[m], uu, s[m][c]);
                }
            }
        }
        const float more = token_sum(ab + CH, found[col]);
        if (chunk * CH + l < count) p.out[((size_t)(row0 + chunk * CH + l) * p.heads + head) * vdim + blockIdx.x * WALK_COLS + col] = o + more;
    }
#pragma unroll
    for (int m = 0; m < P; ++m) {
        const float2 x = unpair(s[m][0]), y = unpair(s[m][1]);
        *reinterpret_cast<float2*>(state + (size_t)pair_row<P>(lane, m) * vdim) = make_float2(x.x, y.x);
        *reinterpret_cast<float2*>(state + (size_t)(pair_row<P>(lane, m) + 1) * vdim) = make_float2(x.y, y.y);
    }
}

// out[t, h, :] = o / sqrt(mean(o^2) + eps) * w * gate[t, h, :].  One warp per (token, head).
template <typename TO>
__global__ void __launch_bounds__(128) gated_head_norm_kernel(const float* o, const float* gate,
                                                              const float* w, float eps, TO* __restrict__ out,
                                                              long long items, int vdim) {
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
    if (item >= items) return;
    const float* src = o + item * vdim;
    float sq = 0.f;
    for (int i = lane; i < vdim; i += 32) { const float x = src[i]; sq += x * x; }
    const float inv = rsqrtf(warp_sum(sq) / (float)vdim + eps);
    for (int i = lane; i < vdim; i += 32)
        out[item * vdim + i] = from_float<TO>(src[i] * inv * w[i] * (gate ? gate[item * vdim + i] : 1.f));
}

// ----------------------------------------------------------------------------- the recurrence, few tokens per sequence
// A step of one token (or a few) per sequence costs the state's bytes, so the kernel is laid out for them: a block
// owns STEP_COLS = 32 neighbouring columns of one head's state and threadIdx.x = row group * 32 + column, so a warp reads
// and writes 128 consecutive bytes of a row; a thread keeps RPT consecutive rows of its column in registers, and the
// two sums over rows (the prediction, the read-out) meet in shared memory.  grid (column blocks, heads, sequences).
constexpr int STEP_COLS = 32;

template <int RPT>
__global__ void __launch_bounds__(512) delta_step_kernel(const ScanParams p) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float sm[];
    const int dim = p.dim, vdim = p.vdim;
    const int groups = blockDim.x / STEP_COLS;
    float* ks = sm;                     // [dim]
    float* qs = ks + dim;               // [dim]
    float* gs = qs + dim;               // [dim] decays
    float* sums = gs + dim;             // [groups][STEP_COLS]
    const int head = blockIdx.y, seq = blockIdx.z;
    const int kvh = head / (p.heads / p.kv_heads);
    const int c = threadIdx.x % STEP_COLS, rg = threadIdx.x / STEP_COLS;
    const int j = blockIdx.x * STEP_COLS + c;
    const bool live = j < vdim;
    const int row0 = p.seq_start[seq], count = p.seq_start[seq + 1] - row0;
    float* state = p.state + ((size_t)p.slots[seq] * p.heads + head) * dim * vdim;
    float s[RPT];
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        const int i = rg * RPT + m;
        s[m] = (live && i < dim) ? state[(size_t)i * vdim + j] : 0.f;
    }
    for (int tt = 0; tt < count; ++tt) {
        const size_t t = (size_t)(row0 + tt);
        __syncthreads();                                              // everyone is done with the token before
        for (int i = threadIdx.x; i < dim; i += blockDim.x) {
            ks[i] = p.k[(t * p.kv_heads + kvh) * dim + i];
            qs[i] = p.q[(t * p.kv_heads + kvh) * dim + i];
            gs[i] = expf(p.decay[(t * p.heads + head) * dim + i]);
        }
        const float vj = live ? p.v[(t * p.heads + head) * vdim + j] : 0.f;
        const float beta = p.beta[t * p.heads + head];
        __syncthreads();
        float part = 0.f;
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            const int i = rg * RPT + m;
            if (i < dim) { s[m] *= gs[i]; part += s[m] * ks[i]; }
        }
        sums[rg * STEP_COLS + c] = part;
        __syncthreads();
        float pred = 0.f;
        for (int g = 0; g < groups; ++g) pred += sums[g * STEP_COLS + c];
        const float u = beta * (vj - pred);
        part = 0.f;
#pragma unroll
        for (int m = 0; m < RPT; ++m) {
            const int i = rg * RPT + m;
            if (i < dim) { s[m] += ks[i] * u; part += s[m] * qs[i]; }
        }
        __syncthreads();                                              // the predictions have been read
        sums[rg * STEP_COLS + c] = part;
        __syncthreads();
        if (rg == 0 && live) {
            float o = 0.f;
            for (int g = 0; g < groups; ++g) o += sums[g * STEP_COLS + c];
            p.out[(t * p.heads + head) * vdim + j] = o;
        }
    }
#pragma unroll
    for (int m = 0; m < RPT; ++m) {
        const int i = rg * RPT + m;
        if (live && i < dim) state[(size_t)i * vdim + j] = s[m];
    }
}

template <int RPT>
static int launch_step(const ScanParams& p, int n_seqs, cudaStream_t s) {
    const int groups = (p.dim + RPT - 1) / RPT;
    const size_t smem = ((size_t)3 * p.dim + (size_t)groups * STEP_COLS) * sizeof(float);
    launch_kernel(delta_step_kernel<RPT>, dim3((p.vdim + STEP_COLS - 1) / STEP_COLS, p.heads, n_seqs), dim3(groups * STEP_COLS), smem, s, p);
    QT_CHECK_LAUNCH("delta_step");
    return QT_OK;
}

// ----------------------------------------------------------------------------- entry points
extern "C" int qt_delta_prepare(const float* proj, int n_splits, long long split_stride, int proj_cols, const float* taps,
                                float* kept, const int* token_seq, const int* token_pos, const int* seq_start,
                                const int* seq_past, const int* slots, float* q, float* k, float* v, float* beta, int n_tokens,
                                int n_seqs, int heads, int kv_heads, int dim, int vdim, int n_taps, float unit_eps, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && vdim > 0,
               "delta_prepare: bad sizes T=%d heads=%d kv_heads=%d dim=%d vdim=%d", n_tokens, heads, kv_heads, dim, vdim);
    QT_REQUIRE(n_taps >= 1 && n_taps <= MAX_TAPS, "delta_prepare: a convolution of %d taps (1..%d)", n_taps, MAX_TAPS);
    const int channels = 2 * kv_heads * dim + heads * vdim;
    QT_REQUIRE(proj_cols >= channels + heads && n_splits >= 1, "delta_prepare: a projection of %d columns does not hold q, k, v and beta", proj_cols);
    if (n_tokens == 0) return QT_OK;
    PrepareParams p{proj, n_splits, (size_t)split_stride, proj_cols, taps, kept, token_seq, token_pos, seq_start, seq_past, slots,
                    q, k, v, beta, n_tokens, heads, kv_heads, dim, vdim, n_taps, unit_eps};
    cudaStream_t s = (cudaStream_t)stream;
    const long long items = (long long)n_tokens * (2 * kv_heads + heads + 1);
    launch_kernel(delta_prepare_kernel, dim3((unsigned)((items + 3) / 4)), dim3(128), 0, s, p);
    QT_CHECK_LAUNCH("delta_prepare");
    if (n_taps > 1) {
        launch_kernel(conv_keep_kernel, dim3((channels + 127) / 128, n_seqs), dim3(128), 0, s, proj, n_splits, (size_t)split_stride, proj_cols,
                      kept, seq_start, slots, n_seqs, channels, n_taps);
        QT_CHECK_LAUNCH("conv_keep");
    }
    return QT_OK;
}

template <int MODE>
static int launch_lowrank(const float* proj, int n_splits, size_t split_stride, int proj_cols, int x_offset, int rank, const float* w, const float* bias,
                          const float* rate_log, int per_rate, float power, float* out, int n_tokens, int n_out, cudaStream_t s) {
    const size_t few_smem = ((size_t)LR_TOKENS * rank + 4 * LR_TOKENS * 64) * sizeof(float);
    const unsigned tiles = (unsigned)((n_tokens + LR_TOKENS - 1) / LR_TOKENS);
    if (n_tokens <= 16 * LR_TOKENS && few_smem <= 48 * 1024)
        launch_kernel(lowrank_few_kernel<MODE>, dim3((n_out + 63) / 64, tiles), dim3(256), few_smem, s, proj, n_splits, split_stride, proj_cols, x_offset, rank, w,
                      bias, rate_log, per_rate, power, out, n_tokens, n_out);
    else
        launch_kernel(lowrank_kernel<MODE>, dim3((n_out + 255) / 256, tiles), dim3(256), (size_t)LR_TOKENS * rank * sizeof(float), s, proj, n_splits,
                      split_stride, proj_cols, x_offset, rank, w, bias, rate_log, per_rate, power, out, n_tokens, n_out);
    QT_CHECK_LAUNCH("lowrank");
    return QT_OK;
}

extern "C" int qt_lowrank(const float* proj, int n_splits, long long split_stride, int proj_cols, int x_offset, int rank,
                          const float* w, const float* bias, const float* rate_log, int per_rate, float power, float* out, int n_tokens,
                          int n_out, int mode, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && n_out > 0 && rank > 0 && x_offset >= 0 && x_offset + rank <= proj_cols && n_splits >= 1,
               "lowrank: bad sizes T=%d N=%d rank=%d at column %d of %d", n_tokens, n_out, rank, x_offset, proj_cols);
    QT_REQUIRE(mode == LR_SIGMOID || mode == LR_LOG_SIGMOID || (mode == LR_DECAY && rate_log && per_rate > 0), "lowrank: mode %d", mode);
    QT_REQUIRE((size_t)LR_TOKENS * rank * sizeof(float) <= 48 * 1024, "lowrank: %d columns are too many for a tile in shared memory", rank);
    if (n_tokens == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t stride = (size_t)split_stride;
    if (mode == LR_DECAY) return launch_lowrank<LR_DECAY>(proj, n_splits, stride, proj_cols, x_offset, rank, w, bias, rate_log, per_rate, power, out, n_tokens, n_out, s);
    if (mode == LR_SIGMOID) return launch_lowrank<LR_SIGMOID>(proj, n_splits, stride, proj_cols, x_offset, rank, w, bias, rate_log, per_rate, power, out, n_tokens, n_out, s);
    return launch_lowrank<LR_LOG_SIGMOID>(proj, n_splits, stride, proj_cols, x_offset, rank, w, bias, rate_log, per_rate, power, out, n_tokens, n_out, s);
}

template <int R>
static int launch_scan(const ScanParams& p, int n_seqs, cudaStream_t s) {
    const size_t smem = 2 * (size_t)SCAN_CHUNK * (3 * p.dim + SCAN_COLS + 1) * sizeof(float);
    const cudaError_t raised = raise_shared<delta_scan_kernel<R>>(208 * 1024);
    if (raised != cudaSuccess) QT_FAIL(QT_ERR_LAUNCH, "delta_scan: cannot raise shared memory: %s", cudaGetErrorString(raised));
    launch_kernel(delta_scan_kernel<R>, dim3((p.vdim + SCAN_COLS - 1) / SCAN_COLS, p.heads, n_seqs), dim3(SCAN_COLS * SCAN_LANES), smem, s, p);
    QT_CHECK_LAUNCH("delta_scan");
    return QT_OK;
}

extern "C" int qt_delta_scan(const float* q, const float* k, const float* v, const float* beta, const float* decay, float* state,
                             float* out, const int* seq_start, const int* slots, int n_seqs, int heads, int kv_heads, int dim,
                             int vdim, void* stream) {
    QT_REQUIRE(n_seqs >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && vdim > 0, "delta_scan: bad sizes");
    QT_REQUIRE(dim > 0 && dim <= 512, "delta_scan: %d key channels per head (1..512)", dim);
    QT_REQUIRE(n_seqs <= 65535 && heads <= 65535, "delta_scan: too many sequences or heads for one launch");
    if (n_seqs == 0) return QT_OK;
    ScanParams p{q, k, v, beta, decay, state, out, seq_start, slots, heads, kv_heads, dim, vdim};
    cudaStream_t s = (cudaStream_t)stream;
    static const bool lanes_form = [] { const char* env = getenv("QT_B200_DELTA_STEP"); return env && env[0] == '0'; }();
    if (!lanes_form) {                                                // rows of a column over row groups, 128 bytes of a row per warp
        if (dim <= 64) return launch_step<8>(p, n_seqs, s);
        if (dim <= 256) return launch_step<16>(p, n_seqs, s);
        return launch_step<32>(p, n_seqs, s);
    }
    if (dim <= 32) return launch_scan<4>(p, n_seqs, s);
    if (dim <= 64) return launch_scan<8>(p, n_seqs, s);
    if (dim <= 128) return launch_scan<16>(p, n_seqs, s);
    if (dim <= 256) return launch_scan<32>(p, n_seqs, s);
    return launch_scan<64>(p, n_seqs, s);
}

template <int R>
static int launch_chunk_scan(const ChunkScanParams& p, int n_seqs, cudaStream_t s) {
    const size_t smem = 2 * ((size_t)CH * (3 * p.dim + 2 * CH + SCAN_COLS + 1) + p.dim) * sizeof(float);
    const cudaError_t raised = raise_shared<delta_chunk_scan_kernel<R>>(220 * 1024);
    if (raised != cudaSuccess) QT_FAIL(QT_ERR_LAUNCH, "delta_chunk_scan: cannot raise shared memory: %s", cudaGetErrorString(raised));
    QT_REQUIRE(smem <= 220 * 1024, "delta_chunk_scan: %d key channels per head need more shared memory than a block has", p.dim);
    launch_kernel(delta_chunk_scan_kernel<R>, dim3((p.vdim + SCAN_COLS - 1) / SCAN_COLS, p.heads, n_seqs), dim3(SCAN_COLS * SCAN_LANES), smem, s, p);
    QT_CHECK_LAUNCH("delta_chunk_scan");
    return QT_OK;
}

template <int P>
static int launch_chunk_walk(const ChunkScanParams& p, int n_seqs, cudaStream_t s) {
    const size_t smem = 2 * ((size_t)CH * (3 * 64 * P + AB + WALK_COLS) + 64 * P) * sizeof(float);
    const cudaError_t raised = raise_shared<delta_chunk_walk_kernel<P>>(120 * 1024);
    if (raised != cudaSuccess) QT_FAIL(QT_ERR_LAUNCH, "delta_chunk_walk: cannot raise shared memory: %s", cudaGetErrorString(raised));
    // Blocks start while the kernel before still runs on most SMs; as much shared memory as it takes to keep them from piling up on
    // the first SMs that fall free (646 us in place of 255 us where two or three share an SM and others stand idle).
    const long long blocks = (long long)(p.vdim / WALK_COLS) * p.heads * n_seqs, per_sm = (blocks + sm_count() - 1) / sm_count();
    const size_t spread = (size_t)(228 * 1024) / (size_t)(per_sm + 1);
    const size_t asked = spread > smem && spread <= 120 * 1024 ? spread : smem;
    launch_kernel(delta_chunk_walk_kernel<P>, dim3(p.vdim / WALK_COLS, p.heads, n_seqs), dim3(WALK_THREADS), asked, s, p);
    QT_CHECK_LAUNCH("delta_chunk_walk");
    return QT_OK;
}

// The recurrence in chunks (steps of many tokens per sequence).  Scratch of the caller: kt, qt, kb, gc [T, heads, dim] and
// ab [T, heads, 36], float.  `max_tokens` is the most tokens any sequence of the step has.
extern "C" int qt_delta_scan_chunked(const float* q, const float* k, const float* v, const float* beta, const float* log_decay,
                                     float* state, float* out, float* kt, float* qt, float* kb, float* gc, float* ab,
                                     const int* seq_start, const int* slots, int n_seqs, int max_tokens, int heads, int kv_heads,
                                     int dim, int vdim, void* stream) {
    QT_REQUIRE(n_seqs >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && vdim > 0 && max_tokens >= 0, "delta_scan_chunked: bad sizes");
    QT_REQUIRE(dim > 0 && dim <= 256, "delta_scan_chunked: %d key channels per head (1..256)", dim);
    QT_REQUIRE(n_seqs <= 65535 && heads <= 65535, "delta_scan_chunked: too many sequences or heads for one launch");
    if (n_seqs == 0 || max_tokens == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    static const bool plain_only = [] { const char* env = getenv("QT_B200_DELTA_FAST"); return env && env[0] == '0'; }();
    const bool aligned = (((uintptr_t)kt | (uintptr_t)qt | (uintptr_t)kb | (uintptr_t)gc | (uintptr_t)ab | (uintptr_t)v | (uintptr_t)state | (uintptr_t)out) & 15) == 0;
    const bool walk = !plain_only && aligned && dim % 64 == 0 && dim <= 256 && vdim % WALK_COLS == 0;
    ChunkParams cp{q, k, log_decay, kt, qt, kb, gc, beta, ab, seq_start, heads, kv_heads, dim, walk ? 1 : 0};
    const size_t smem = 4 * (size_t)CH * dim * sizeof(float);
    const bool fours = dim % 4 == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)log_decay) & 15) == 0;
    const cudaError_t raised = fours ? raise_shared<delta_chunk_prepare_kernel<4>>(64 * 1024) : raise_shared<delta_chunk_prepare_kernel<1>>(64 * 1024);
    if (raised != cudaSuccess) QT_FAIL(QT_ERR_LAUNCH, "delta_chunk_prepare: cannot raise shared memory: %s", cudaGetErrorString(raised));
    const dim3 chunk_grid((max_tokens + CH - 1) / CH, heads, n_seqs);
    if (fours) launch_kernel(delta_chunk_prepare_kernel<4>, chunk_grid, dim3(128), smem, s, cp);
    else launch_kernel(delta_chunk_prepare_kernel<1>, chunk_grid, dim3(128), smem, s, cp);
    QT_CHECK_LAUNCH("delta_chunk_prepare");
    ChunkScanParams sp{kt, qt, kb, gc, ab, v, beta, state, out, seq_start, slots, heads, dim, vdim};
    if (walk) {
        if (dim == 64) return launch_chunk_walk<1>(sp, n_seqs, s);
        if (dim == 128) return launch_chunk_walk<2>(sp, n_seqs, s);
        if (dim == 192) return launch_chunk_walk<3>(sp, n_seqs, s);
        return launch_chunk_walk<4>(sp, n_seqs, s);
    }
    if (dim <= 32) return launch_chunk_scan<4>(sp, n_seqs, s);
    if (dim <= 64) return launch_chunk_scan<8>(sp, n_seqs, s);
    if (dim <= 128) return launch_chunk_scan<16>(sp, n_seqs, s);
    return launch_chunk_scan<32>(sp, n_seqs, s);
}

extern "C" int qt_gated_head_norm(const float* o, const float* gate, const float* w, float eps, void* out, int out_dtype,
                                  int n_tokens, int heads, int vdim, void* stream) {
    QT_REQUIRE(n_tokens >= 0 && heads > 0 && vdim > 0, "gated_head_norm: bad sizes");
    if (n_tokens == 0) return QT_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const long long items = (long long)n_tokens * heads;
    return QT_DISPATCH_DTYPE(out_dtype, "gated_head_norm", {
        launch_kernel(gated_head_norm_kernel<T>, dim3((unsigned)((items + 3) / 4)), dim3(128), 0, s, o, gate, w, eps, (T*)out, items, vdim);
        QT_CHECK_LAUNCH("gated_head_norm");
        return QT_OK;
    });
}

QT_DEFINE_LAST_ERROR(delta_rule)
