// The walk of linear_attention.cu for prompts whose memory decays by one number per token and head (constant decay, the
// state-space layer, the matrix memory with exponential gates), all tokens of a chunk at once.
//
// With a chunk of 64 tokens, W_ij = a_{j+1} ... a_i the decay between two of its tokens (1 for i = j) and D_i = a_first ... a_i:
//
//   o_i = D_i S_beforeᵀ q_i + sum_{j <= i} W_ij (q_i · k_j) v_j,      S_after = D_last S_before + sum_j W_{last,j} k_j v_jᵀ
//
// so that the only thing that goes from token to token one after the other is S from chunk to chunk.  Three kernels: what
// every chunk adds to S (a product over its tokens, for all chunks at once); S before every chunk (a multiply-add per chunk
// and entry, all entries at once); and the outputs (three products per chunk, for all chunks at once).  Everything is float32
// multiply-adds as in the walk; decays between tokens are products of the tokens' decays, never quotients or differences of
// logarithms, so that they underflow where the walk's do and are as exact.
//
// What bounds it: the multiply-adds (per chunk and head 2 · 64 · dim · vdim for the state and the queries' product with it,
// 64 · 64 · (dim · column tiles + vdim) inside the chunk), on tiles of 64 tokens x 64 columns or 128 rows x 64 columns, 8 x 4 or
// 8 x 8 outputs per thread.  The walk is a chain 64 times as long on a fraction of the GPU.  B200, three prompts of 1,500, 638 and
// 902 tokens, 6 heads of 128 x 257: 299 us (states 79, scan 23, outputs 197; 240 with keys, values and products side by side in shared
// memory, two blocks an SM), the walk 1,665 us.
#include "common.cuh"
#include "linear_attention.cuh"

namespace mlc {

constexpr int GC_TOKENS = 64;          // tokens of a chunk
constexpr int GC_COLS = 64;            // columns of S per block
constexpr int GC_ROWS = 128;           // rows of S per block of the first kernel
constexpr int GC_THREADS = 128;
constexpr int GC_P = GC_TOKENS + 4;    // floats from row to row of the transposed tiles: rows start 16-byte aligned, and a warp's
                                       // stores of 8 rows x 4 columns hit all banks
constexpr long long GC_MAX_SCRATCH = 512LL << 20;      // floats: beyond 2 GB the walk is taken

// A sequence's first chunk among all chunks of the step: no two sequences' chunks meet.
__device__ __forceinline__ int gc_first(int t0, int seq) { return t0 / GC_TOKENS + seq; }

struct GcArgs {
    GlaArgs a;
    float* states;             // [chunks][H][vdim][dim]: what the chunk adds to S, then S before the chunk
    float* decays;             // [chunks][H]: the chunk's D_last
};

__device__ __forceinline__ float gc_decay(const GlaArgs& a, int t, int head) {
    return a.const_decay != nullptr ? a.const_decay[head] : a.head_decay[(long long)t * a.H + head];
}

__device__ __forceinline__ float gc_value(const GlaArgs& a, int t, int head, int col) {
    float v = col < a.v_cols ? a.vsrc[(long long)t * a.v_stride + a.v_col + head * a.v_cols + col] : col < a.vdim ? 1.0f : 0.0f;
    return a.v_scale != nullptr ? v * a.v_scale[(long long)t * a.H + head] : v;
}

// TOTAL entries from memory into shared memory by the whole block, eight of a thread's loads in flight at a time
template <int TOTAL, typename L, typename S>
__device__ __forceinline__ void gc_stage(L load, S store) {
    static_assert(TOTAL % (8 * GC_THREADS) == 0, "whole rounds");
#pragma unroll 1
    for (int base = threadIdx.x; base < TOTAL; base += 8 * GC_THREADS) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = load(base + u * GC_THREADS);
#pragma unroll
        for (int u = 0; u < 8; ++u) store(base + u * GC_THREADS, v[u]);
    }
}

// grid: (column tiles x row tiles, heads, chunks of the longest sequence x sequences)
__global__ void __launch_bounds__(GC_THREADS)
gla_chunk_states_kernel(GcArgs g, int col_tiles, int max_chunks) {
    __shared__ __align__(16) float ks[GC_TOKENS / 2][GC_ROWS + 4];
    __shared__ __align__(16) float vs[GC_TOKENS / 2][GC_COLS + 4];
    __shared__ __align__(16) float as[GC_TOKENS], ws[GC_TOKENS];
    const GlaArgs& a = g.a;
    const int head = blockIdx.y, seq = blockIdx.z / max_chunks, c = blockIdx.z % max_chunks;
    const int t0 = a.cu_seqlens[seq], t1 = a.cu_seqlens[seq + 1];
    const int c0 = t0 + c * GC_TOKENS, n = min(GC_TOKENS, t1 - c0);
    if (n <= 0) return;
    const int col0 = (blockIdx.x % col_tiles) * GC_COLS, row0 = (blockIdx.x / col_tiles) * GC_ROWS;
    const int chunk = gc_first(t0, seq) + c;
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;           // 8 columns side by side in fours x 16 groups of rows
    if (tid < GC_TOKENS) as[tid] = tid < n ? gc_decay(a, c0 + tid, head) : 1.0f;
    __syncthreads();
    if (tid < GC_TOKENS) {
        float w = 1.0f;
#pragma unroll 16
        for (int l = 0; l < GC_TOKENS; ++l) w *= l > tid ? as[l] : 1.0f;
        ws[tid] = w;
        if (tid == 0 && blockIdx.x == 0) g.decays[(long long)chunk * a.H + head] = w * as[0];
    }
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    const float* kp = a.qk + a.k_col + (head / a.qk_share) * a.dim + row0;
    for (int h = 0; h < n; h += GC_TOKENS / 2) {
        __syncthreads();
        gc_stage<GC_TOKENS / 2 * GC_ROWS>(
            [&](int idx) {
                const int t = idx / GC_ROWS, d = idx % GC_ROWS;
                return (h + t < n && row0 + d < a.dim) ? kp[(long long)(c0 + h + t) * a.qk_stride + d] : 0.0f;
            },
            [&](int idx, float v) { ks[idx / GC_ROWS][idx % GC_ROWS] = v; });
        gc_stage<GC_TOKENS / 2 * GC_COLS>(
            [&](int idx) { return h + idx / GC_COLS < n ? gc_value(a, c0 + h + idx / GC_COLS, head, col0 + idx % GC_COLS) : 0.0f; },
            [&](int idx, float v) { vs[idx / GC_COLS][idx % GC_COLS] = v * ws[h + idx / GC_COLS]; });
        __syncthreads();
#pragma unroll 4
        for (int t = 0; t < GC_TOKENS / 2; ++t) {
            float kr[8], vr[8];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float4 x = *reinterpret_cast<const float4*>(&ks[t][ty * 4 + 64 * i]);
                const float4 y = *reinterpret_cast<const float4*>(&vs[t][tx * 4 + 32 * i]);
                kr[4 * i] = x.x; kr[4 * i + 1] = x.y; kr[4 * i + 2] = x.z; kr[4 * i + 3] = x.w;
                vr[4 * i] = y.x; vr[4 * i + 1] = y.y; vr[4 * i + 2] = y.z; vr[4 * i + 3] = y.w;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(kr[i], vr[j], acc[i][j]);
        }
    }
    float* out = g.states + ((long long)chunk * a.H + head) * a.vdim * a.dim;
    const bool vec = (a.dim & 3) == 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int col = col0 + tx * 4 + 32 * (j >> 2) + (j & 3);
        if (col >= a.vdim) continue;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int row = row0 + ty * 4 + 64 * i;
            float* p = out + (long long)col * a.dim + row;
            if (vec) {
                if (row < a.dim) *reinterpret_cast<float4*>(p) = make_float4(acc[4 * i][j], acc[4 * i + 1][j], acc[4 * i + 2][j], acc[4 * i + 3][j]);
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (row + u < a.dim) p[u] = acc[4 * i + u][j];
            }
        }
    }
}

// An entry of S per thread, from the state before the step through all chunks: what the chunk adds gives way to S before it.
__global__ void __launch_bounds__(256)
gla_chunk_scan_kernel(GcArgs g, long long per_seq) {
    const GlaArgs& a = g.a;
    const int seq = blockIdx.y;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= per_seq) return;
    const int head = (int)(e / ((long long)a.vdim * a.dim));
    const int t0 = a.cu_seqlens[seq], chunks = (a.cu_seqlens[seq + 1] - t0 + GC_TOKENS - 1) / GC_TOKENS;
    const int first = gc_first(t0, seq);
    float* state = a.state + (long long)a.slots[seq] * a.state_stride + e;
    float* p = g.states + (long long)first * per_seq + e;
    const float* d = g.decays + (long long)first * a.H + head;
    float S = *state;
    constexpr int AHEAD = 8;
    for (int c = 0; c < chunks; c += AHEAD) {
        float u[AHEAD], w[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int at = min(c + i, chunks - 1);
            u[i] = p[(long long)at * per_seq];
            w[i] = d[(long long)at * a.H];
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (c + i < chunks) {
                p[(long long)(c + i) * per_seq] = S;
                S = fmaf(w[i], S, u[i]);
            }
        }
    }
    if (chunks > 0) *state = S;
}

// dst[d][t] = src[t][d] for `n` rows of `width` floats with a stride: four rows x eight entries per warp and pass, which is one
// 32-byte sector per row on the way in and all banks on the way out
template <typename F>
__device__ __forceinline__ void gc_transpose(float* dst, int n, int width, F value) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int dl = lane & 7, tl = lane >> 3;
    for (int t = warp * 4 + tl; t < GC_TOKENS; t += GC_THREADS / 8) {
        for (int d0 = dl; d0 < width; d0 += 64) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = (t < n && d0 + 8 * u < width) ? value(t, d0 + 8 * u) : 0.0f;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (d0 + 8 * u < width) dst[(d0 + 8 * u) * GC_P + t] = v[u];
        }
    }
}

// grid: (column tiles, heads, chunks of the longest sequence x sequences).  A thread: 8 tokens (two fours) x 4 neighbours.
// One region of shared memory holds first S before the chunk, then the keys, then the weighted products of queries and keys
// and the values: three blocks of dim 128 share an SM, and one's loads hide behind another's products.
__host__ __device__ constexpr int gc_region_floats(int dim) { return (dim > 2 * GC_TOKENS ? dim : 2 * GC_TOKENS) * GC_P; }

__global__ void __launch_bounds__(GC_THREADS)
gla_chunk_outputs_kernel(GcArgs g, int max_chunks) {
    extern __shared__ __align__(16) float gc_smem[];
    const GlaArgs& a = g.a;
    float* const region = gc_smem;                     // S [dim][columns], keys [dim][tokens], then the two below
    float* const PT = region;                          // [token j][GC_P tokens i]
    float* const vs = region + GC_TOKENS * GC_P;       // [token][GC_P columns]
    float* const qT = region + gc_region_floats(a.dim);        // [dim][GC_P]
    float* const as = qT + a.dim * GC_P;               // [64] decays
    float* const Ds = as + GC_TOKENS;                  // [64] decays from the chunk's first token to token i
    const int head = blockIdx.y, seq = blockIdx.z / max_chunks, c = blockIdx.z % max_chunks;
    const int t0 = a.cu_seqlens[seq], t1 = a.cu_seqlens[seq + 1];
    const int c0 = t0 + c * GC_TOKENS, n = min(GC_TOKENS, t1 - c0);
    if (n <= 0) return;
    const int col0 = blockIdx.x * GC_COLS, cols = min(GC_COLS, a.vdim - col0);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    if (tid < GC_TOKENS) as[tid] = tid < n ? gc_decay(a, c0 + tid, head) : 1.0f;
    const float* qp = a.qk + a.q_col + (head / a.qk_share) * a.dim + (long long)c0 * a.qk_stride;
    const float* kp = a.qk + a.k_col + (head / a.qk_share) * a.dim + (long long)c0 * a.qk_stride;
    const float* sp = g.states + ((long long)(gc_first(t0, seq) + c) * a.H + head) * a.vdim * a.dim + (long long)col0 * a.dim;
    gc_transpose(qT, n, a.dim, [&](int t, int d) { return qp[(long long)t * a.qk_stride + d] * a.q_scale; });
    gc_transpose(region, cols, a.dim, [&](int t, int d) { return sp[(long long)t * a.dim + d]; });
    __syncthreads();
    if (tid < GC_TOKENS) {
        float w = 1.0f;
#pragma unroll 16
        for (int l = 0; l < GC_TOKENS; ++l) w *= l <= tid ? as[l] : 1.0f;
        Ds[tid] = w;
    }
    auto product = [&](float (&acc)[8][4], const float* A, const float* B, int depth) {      // acc[i][j] += sum_d A[d][i] B[d][j]
#pragma unroll 4
        for (int d = 0; d < depth; ++d) {
            const float4 x0 = *reinterpret_cast<const float4*>(A + d * GC_P + ty * 4), x1 = *reinterpret_cast<const float4*>(A + d * GC_P + ty * 4 + 32);
            const float4 y = *reinterpret_cast<const float4*>(B + d * GC_P + tx * 4);
            const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[i][0] = fmaf(x[i], y.x, acc[i][0]);
                acc[i][1] = fmaf(x[i], y.y, acc[i][1]);
                acc[i][2] = fmaf(x[i], y.z, acc[i][2]);
                acc[i][3] = fmaf(x[i], y.w, acc[i][3]);
            }
        }
    };
    auto token_of = [&](int i) { return ty * 4 + 32 * (i >> 2) + (i & 3); };
    float out[8][4], qk[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) out[i][j] = qk[i][j] = 0.0f;
    product(out, qT, region, a.dim);                   // S_beforeᵀ q_i
    __syncthreads();                                   // S has been read, the decays are there
    gc_transpose(region, n, a.dim, [&](int t, int d) { return kp[(long long)t * a.qk_stride + d]; });
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float D = Ds[token_of(i)];
#pragma unroll
        for (int j = 0; j < 4; ++j) out[i][j] *= D;
    }
    __syncthreads();
    product(qk, qT, region, a.dim);                    // q_i · k_j
    // times the decays W_ij: per column the product from the column's next token to the thread's first, then on token by token;
    // a token that does not see the other gets a zero whatever their product is
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i0 = token_of(4 * half);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = tx * 4 + j;
            float w = 1.0f;
#pragma unroll 4
            for (int l = col + 1; l < i0; ++l) w *= as[l];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i0 + i > col) w *= as[i0 + i];
                const bool sees = i0 + i >= col && w != 0.0f;
                qk[4 * half + i][j] = sees ? w * qk[4 * half + i][j] : 0.0f;
            }
        }
    }
    __syncthreads();                                   // the keys have been read
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(PT + (tx * 4 + j) * GC_P + token_of(4 * half)) =
                make_float4(qk[4 * half][j], qk[4 * half + 1][j], qk[4 * half + 2][j], qk[4 * half + 3][j]);
    gc_stage<GC_TOKENS * GC_COLS>([&](int idx) { return idx / GC_COLS < n ? gc_value(a, c0 + idx / GC_COLS, head, col0 + idx % GC_COLS) : 0.0f; },
                                  [&](int idx, float v) { vs[idx / GC_COLS * GC_P + idx % GC_COLS] = v; });
    __syncthreads();
    // The weighted products times the values, each token over the tokens up to itself: half the work, and a value that is not a
    // number reaches no token before its own.
    auto add = [&](int first, const float4& x, const float4& y) {
        const float xi[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            out[first + i][0] = fmaf(xi[i], y.x, out[first + i][0]);
            out[first + i][1] = fmaf(xi[i], y.y, out[first + i][1]);
            out[first + i][2] = fmaf(xi[i], y.z, out[first + i][2]);
            out[first + i][3] = fmaf(xi[i], y.w, out[first + i][3]);
        }
    };
    const float* const pt = PT + ty * 4;
    const float* const vt = vs + tx * 4;
    const int full0 = min(n, ty * 4), full1 = min(n, ty * 4 + 32);
#pragma unroll 4
    for (int j = 0; j < full0; ++j) {
        const float4 y = *reinterpret_cast<const float4*>(vt + j * GC_P);
        add(0, *reinterpret_cast<const float4*>(pt + j * GC_P), y);
        add(4, *reinterpret_cast<const float4*>(pt + j * GC_P + 32), y);
    }
#pragma unroll 4
    for (int j = full0; j < full1; ++j)
        add(4, *reinterpret_cast<const float4*>(pt + j * GC_P + 32), *reinterpret_cast<const float4*>(vt + j * GC_P));
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int u = 0; u < 4; ++u) {                  // the four tokens among themselves
            const int j = ty * 4 + 32 * half + u;
            const float4 y = *reinterpret_cast<const float4*>(vt + j * GC_P);
#pragma unroll
            for (int i = u; i < 4; ++i) {
                const float x = PT[j * GC_P + ty * 4 + 32 * half + i];
                float (&o)[4] = out[4 * half + i];
                o[0] = fmaf(x, y.x, o[0]);
                o[1] = fmaf(x, y.y, o[1]);
                o[2] = fmaf(x, y.z, o[2]);
                o[3] = fmaf(x, y.w, o[3]);
            }
        }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = token_of(i);
        if (t >= n) continue;
        float* o = a.out + (long long)(c0 + t) * a.H * a.vdim + (long long)head * a.vdim + col0 + tx * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (tx * 4 + j < cols) o[j] = out[i][j];
    }
}

long long gla_chunk_floats(int n_seqs, int n_tokens, int max_q_len, int H, int dim, int vdim) {
    // A run of 32 tokens takes the walk about as long as three launches take (from there on gla_chunks_pay in
    // kernels/bindings.py says which of the two is the sooner).
    if (max_q_len <= 32 || n_seqs <= 0 || H <= 0 || H > 65535 || dim <= 0 || dim > 256 || vdim <= 0) return 0;
    const long long max_chunks = (max_q_len + GC_TOKENS - 1) / GC_TOKENS;
    if (max_chunks * n_seqs > 65535) return 0;
    const long long chunks = n_tokens / GC_TOKENS + n_seqs, need = chunks * H * ((long long)dim * vdim + 4);
    return need <= GC_MAX_SCRATCH ? need : 0;
}

int gla_chunks(GlaArgs a, int n_seqs, int n_tokens, int max_q_len, float* scratch, cudaStream_t s) {
    const int max_chunks = (max_q_len + GC_TOKENS - 1) / GC_TOKENS;
    const long long chunks = n_tokens / GC_TOKENS + n_seqs, per_seq = (long long)a.H * a.dim * a.vdim;
    GcArgs g{a, scratch, scratch + chunks * per_seq};
    const int col_tiles = (a.vdim + GC_COLS - 1) / GC_COLS, row_tiles = (a.dim + GC_ROWS - 1) / GC_ROWS;
    gla_chunk_states_kernel<<<dim3(col_tiles * row_tiles, a.H, max_chunks * n_seqs), GC_THREADS, 0, s>>>(g, col_tiles, max_chunks);
    MLC_LAUNCH_CHECK();
    gla_chunk_scan_kernel<<<dim3((unsigned)((per_seq + 255) / 256), n_seqs), 256, 0, s>>>(g, per_seq);
    MLC_LAUNCH_CHECK();
    const size_t smem = ((size_t)gc_region_floats(a.dim) + a.dim * GC_P + 2 * GC_TOKENS) * sizeof(float);
    static size_t allowed = 48 * 1024;
    if (smem > allowed) {
        constexpr size_t most = ((size_t)gc_region_floats(256) + 256 * GC_P + 2 * GC_TOKENS) * sizeof(float);
        static_assert(most <= 227 * 1024, "shared memory of a block");
        cudaError_t e = cudaFuncSetAttribute(gla_chunk_outputs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return (int)e;
        allowed = most;
    }
    gla_chunk_outputs_kernel<<<dim3(col_tiles, a.H, max_chunks * n_seqs), GC_THREADS, smem, s>>>(g, max_chunks);
    MLC_LAUNCH_CHECK();
    return 0;
}

}  // namespace mlc
