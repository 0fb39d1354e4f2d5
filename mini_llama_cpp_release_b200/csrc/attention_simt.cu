// Attention over the paged cache in plain float32 arithmetic (no tensor cores), for any
// element type of the cache and any head size up to 512 (a second instance of the kernel, with
// twice the accumulators, takes the sizes above 256).  It is the whole-model 32-bit
// path's attention and the yardstick the tensor-core kernels are checked against.
//
// One kernel serves prompts, continuation chunks and single decoded tokens: a step gives
// each sequence q_len new tokens at positions start_pos .. start_pos + q_len - 1, their
// keys and values are already in the cache, and a token at position p reads keys
// lo(p) .. p, with lo(p) = 0 or p - window + 1, and beside a window the first `keep_first`
// keys of the sequence, which stay visible at any distance (at their true positions).  With `chunk` the mask is one of
// chunks instead: lo(p) = (p / chunk) * chunk, counted from the sequence's first position.  With `softcap` a score
// becomes softcap * tanh(score / softcap) before the softmax.  The reference computes the same thing
// one (head, position) at a time: score = (q·k)·1/sqrt(hd), max, exp, sum, weighted sum
// of values (src/forward.cpp:585-611; src/ops.cpp:43-70); query head h reads kv head
// h / (H/KV) (src/forward.cpp:524-526).  Here a block holds up to 16 (token, head) rows
// that share one kv head, streams 32-key tiles through shared memory and keeps a running
// maximum and sum per row; long key ranges can be split over blocks, whose partial
// (max, sum, weighted values) are merged by a second kernel.
#include "common.cuh"

namespace mlc {

constexpr int ATT_ROWS = 16;       // (token, head) rows per block
constexpr int ATT_WARPS = 4;
constexpr int ATT_ROWS_PER_WARP = ATT_ROWS / ATT_WARPS;
constexpr int ATT_TILE = 32;       // keys per tile: one per lane
constexpr int ATT_MAX_HD = 512;

struct AttnArgs {
    const void* q;            // [N][H][hd]
    void* out;                // [N][H][hd]
    const int* cu_seqlens;    // [B+1] token offsets of this step
    const int* start_pos;     // [B] tokens cached before this step
    float* part_ml;           // [N*H][n_splits][2]   (n_splits > 1)
    float* part_o;            // [N*H][n_splits][hd]
    const float* sinks;       // [H] or null: exp(sinks[h]) joins the softmax denominator of head h, once, with no value
    float scale;
    int q_heads;
    int group;                // query heads per kv head
    int window;               // 0: all keys
    int keep_first;           // with a window: keys at positions below this stay visible whatever the distance
    int chunk;                // > 0: a token at position p reads only the keys from (p / chunk) * chunk on (a mask of chunks)
    float softcap;            // > 0: score <- softcap * tanh(score / softcap), after the scale
    int tokens_per_block;     // TQ
    int heads_per_block;      // GH, TQ*GH <= 16
    int head_chunks;          // ceil(group / GH)
    int n_splits;
};

// Floats from one row of a tile to the next: whole 16-byte pieces, an odd number of them, so that the lanes of a warp, each
// reading a piece of a key of its own, hit all banks.  What lies between a row's end and its last whole piece is zero.
__host__ __device__ __forceinline__ int att_pitch(int hd) { return 4 * (((hd + 3) / 4) | 1); }

// What bounds it: with the few rows of a decode step, the chain of a tile's loads, scores, softmax and weighted values; so
// loads are 16 bytes, the next tile's are in flight while a tile is used, and a key's (a value's) entries pass a lane's
// registers once for all four rows of its warp.  B200, float32, 3 sequences of about 100 keys, 14 heads of 64 on 2: 82 us a
// launch with entry-by-entry loads and a row at a time, now 22.
// Up to 128 entries a head the accumulators are half as many and an SM holds four blocks, not three.  64 sequences of 200 keys,
// 8 heads of 80 on 8, where only the first of a block's warps has a row: 72 us as it was at first, 83 when all warps multiplied and
// an SM held three, now 66; 2,048 tokens, 16 heads of 128 on 4: 3,866, 1,665, now 1,372.
template <typename T, int ATT_ACC>        // ATT_ACC: output entries a lane holds per row, head size <= 32 * ATT_ACC
__global__ void __launch_bounds__(ATT_WARPS * 32, ATT_ACC <= 4 || (sizeof(T) == 2 && ATT_ACC <= 8) ? 4 : 3)
attention_simt_kernel(AttnArgs a, PagedKV c) {
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ float smem[];
    const int hd = c.head_dim;
    const int ld = att_pitch(hd);                  // a row's floats in shared memory
    float* Qs = smem;                              // [16][ld]
    float* Ks = Qs + ATT_ROWS * ld;                // [32][ld]
    float* Vs = Ks + ATT_TILE * ld;                // [32][ld]
    __shared__ long long key_off[ATT_TILE];
    __shared__ __align__(16) float Ps[ATT_WARPS][ATT_TILE][ATT_ROWS_PER_WARP];   // a warp's probabilities of a tile

    const int b = blockIdx.z;
    int y = blockIdx.y;
    const int split = y % a.n_splits;  y /= a.n_splits;
    const int chunk = y % a.head_chunks;  y /= a.head_chunks;
    const int kvh = y;
    const int tok0 = blockIdx.x * a.tokens_per_block;
    const int seq_tok0 = a.cu_seqlens[b];
    const int q_len = a.cu_seqlens[b + 1] - seq_tok0;
    if (tok0 >= q_len) return;
    const int start = a.start_pos[b];
    const int n_tok = min(a.tokens_per_block, q_len - tok0);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T* q = (const T*)a.q;

    // stage the block's query rows
    for (int idx = threadIdx.x; idx < ATT_ROWS * ld; idx += blockDim.x) {
        const int r = idx / ld, d = idx % ld;
        const int t = r / a.heads_per_block, hg = chunk * a.heads_per_block + r % a.heads_per_block;
        float v = 0.0f;
        if (t < n_tok && hg < a.group && d < hd) {
            const long long row = (long long)(seq_tok0 + tok0 + t) * a.q_heads + (kvh * a.group + hg);
            v = to_float(q[row * hd + d]);
        }
        Qs[idx] = v;
    }

    // key range of the block and of this split
    const int p_first = start + tok0, p_last = start + tok0 + n_tok - 1;
    const int lo_block = (a.chunk > 0) ? (p_first / a.chunk) * a.chunk : (a.window > 0) ? max(0, p_first - a.window + 1) : 0;
    const int tile_begin = lo_block / ATT_TILE, tile_end = p_last / ATT_TILE + 1;
    // tiles of kept first keys that lie before the window's first tile are walked ahead of it: the walk's tile number
    // v stands for tile v below `head_tiles`, and for tile_begin + (v - head_tiles) from there on
    const int keep = (a.window > 0) ? a.keep_first : 0;
    const int head_tiles = min(tile_begin, (keep + ATT_TILE - 1) / ATT_TILE);
    const int walk = head_tiles + tile_end - tile_begin;
    const int per_split = (walk + a.n_splits - 1) / a.n_splits;
    const int my_begin = split * per_split;
    const int my_end = min(walk, my_begin + per_split);

    float m[ATT_ROWS_PER_WARP], l[ATT_ROWS_PER_WARP], acc[ATT_ROWS_PER_WARP][ATT_ACC];
    int row_lo[ATT_ROWS_PER_WARP], row_hi[ATT_ROWS_PER_WARP];
    bool row_ok[ATT_ROWS_PER_WARP];
#pragma unroll
    for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) {
        const int r = warp * ATT_ROWS_PER_WARP + i;
        const int t = r / a.heads_per_block, hg = chunk * a.heads_per_block + r % a.heads_per_block;
        row_ok[i] = (t < n_tok) && (hg < a.group);
        row_hi[i] = start + tok0 + t;
        row_lo[i] = (a.chunk > 0) ? (row_hi[i] / a.chunk) * a.chunk : (a.window > 0) ? max(0, row_hi[i] - a.window + 1) : 0;
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int k = 0; k < ATT_ACC; ++k) acc[i][k] = 0.0f;
    }

    bool any_row = false;                          // the same for the whole warp
#pragma unroll
    for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) any_row |= row_ok[i];

    const T* kp = (const T*)c.k_pool;
    const T* vp = (const T*)c.v_pool;
    auto tile_of = [&](int v) { return v < head_tiles ? v : tile_begin + (v - head_tiles); };
    // a float32 cache whose rows are whole 16-byte pieces: a thread's pieces of the next tile wait in registers
    const bool wide = sizeof(T) == 4 && ATT_ACC <= 8 && (hd & 3) == 0 && ((((uintptr_t)kp) | ((uintptr_t)vp)) & 15) == 0 && (c.entry_offset & 3) == 0;
    constexpr int PIECES = ATT_ACC <= 8 ? 4 : 1;      // up to 64 entries per head: 32 keys x 16 pieces on 128 threads
    const int row_pieces = hd >> 2;
    const bool ahead = wide && hd <= 64;
    float4 kr[PIECES], vr[PIECES];
    auto offset_of = [&](int tile, int j) -> long long {
        const int kpos = tile * ATT_TILE + j;
        return ((kpos >= lo_block || kpos < keep) && kpos <= p_last) ? paged_offset(c, b, kpos, kvh) : -1;
    };
    auto fetch = [&](int v) {
        const int tile = tile_of(v);
#pragma unroll
        for (int u = 0; u < PIECES; ++u) {
            const int idx = threadIdx.x + u * ATT_WARPS * 32, j = idx / row_pieces, d = (idx - j * row_pieces) * 4;
            kr[u] = vr[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const long long off = j < ATT_TILE ? offset_of(tile, j) : -1;
            if (off >= 0) {
                kr[u] = *reinterpret_cast<const float4*>((const float*)kp + off + d);
                vr[u] = *reinterpret_cast<const float4*>((const float*)vp + off + d);
            }
        }
    };
    if (ahead && my_begin < my_end) fetch(my_begin);
    for (int v = my_begin; v < my_end; ++v) {
        const int tile = tile_of(v);
        __syncthreads();   // previous tile's readers are done (and Qs is staged)
        if (ahead) {
#pragma unroll
            for (int u = 0; u < PIECES; ++u) {
                const int idx = threadIdx.x + u * ATT_WARPS * 32, j = idx / row_pieces, d = (idx - j * row_pieces) * 4;
                if (j < ATT_TILE) {
                    *reinterpret_cast<float4*>(Ks + j * ld + d) = kr[u];
                    *reinterpret_cast<float4*>(Vs + j * ld + d) = vr[u];
                }
            }
            if (v + 1 < my_end) fetch(v + 1);
        } else {
            if (threadIdx.x < ATT_TILE) key_off[threadIdx.x] = offset_of(tile, threadIdx.x);
            __syncthreads();
            if (wide) {
                for (int idx = threadIdx.x; idx < ATT_TILE * row_pieces; idx += blockDim.x) {
                    const int j = idx / row_pieces, d = (idx - j * row_pieces) * 4;
                    const long long off = key_off[j];
                    float4 kv = make_float4(0.0f, 0.0f, 0.0f, 0.0f), vv = kv;
                    if (off >= 0) {
                        kv = *reinterpret_cast<const float4*>((const float*)kp + off + d);
                        vv = *reinterpret_cast<const float4*>((const float*)vp + off + d);
                    }
                    *reinterpret_cast<float4*>(Ks + j * ld + d) = kv;
                    *reinterpret_cast<float4*>(Vs + j * ld + d) = vv;
                }
            } else {
                for (int idx = threadIdx.x; idx < ATT_TILE * ld; idx += blockDim.x) {
                    const int j = idx / ld, d = idx % ld;
                    const long long off = key_off[j];
                    float kv = 0.0f, vv = 0.0f;
                    if (off >= 0 && d < hd) {
                        kv = to_float(kp[off + d]);
                        vv = to_float(vp[off + d]);
                    }
                    Ks[idx] = kv;
                    Vs[idx] = vv;
                }
            }
        }
        __syncthreads();
        // A single token of few heads a kv head: most warps have no row.
        if (!any_row) continue;

        // scores of the warp's four rows against the lane's key, each summed in ascending order of the entries
        const int kpos = tile * ATT_TILE + lane;
        float dot[ATT_ROWS_PER_WARP];
#pragma unroll
        for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) dot[i] = 0.0f;
        const float* const qw = Qs + warp * ATT_ROWS_PER_WARP * ld;
        const float* const kl = Ks + lane * ld;
#pragma unroll 4
        for (int d = 0; d < hd; d += 4) {
            const float4 kk = *reinterpret_cast<const float4*>(kl + d);
            float4 qq[ATT_ROWS_PER_WARP];
#pragma unroll
            for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) qq[i] = *reinterpret_cast<const float4*>(qw + i * ld + d);
            // row after row, not term after term: the multiply-adds of one sum wait for one another
#pragma unroll
            for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) dot[i] = fmaf(qq[i].x, kk.x, dot[i]);
#pragma unroll
            for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) dot[i] = fmaf(qq[i].y, kk.y, dot[i]);
#pragma unroll
            for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) dot[i] = fmaf(qq[i].z, kk.z, dot[i]);
#pragma unroll
            for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) dot[i] = fmaf(qq[i].w, kk.w, dot[i]);
        }
        bool any = false, apart = false;               // apart: a row sees nothing of a tile that another row of the warp sees
        float corr[ATT_ROWS_PER_WARP];
#pragma unroll
        for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) {
            const bool in_range = row_ok[i] && (kpos >= row_lo[i] || kpos < keep) && kpos <= row_hi[i];
            float s = -INFINITY;
            if (in_range) {
                s = dot[i] * a.scale;
                if (a.softcap > 0.0f) s = a.softcap * tanhf(s / a.softcap);
            }
            const float tile_max = warp_max(s);
            float p = 0.0f;
            corr[i] = 1.0f;
            if (tile_max != -INFINITY) {              // the same for the whole warp
                const float m_new = fmaxf(m[i], tile_max);
                p = in_range ? expf(s - m_new) : 0.0f;
                corr[i] = (m[i] == -INFINITY) ? 0.0f : expf(m[i] - m_new);
                l[i] = l[i] * corr[i] + warp_sum(p);
                m[i] = m_new;
                any = true;
            } else if (row_ok[i]) {
                corr[i] = -1.0f;                      // (no factor of a sum is negative)
                apart = true;
            }
            Ps[warp][lane][i] = p;
        }
        __syncwarp();
        if (!any) continue;
        if (apart) {
            // Row by row, so that a row that sees nothing of the tile takes nothing from it, not even a zero times an
            // infinite value of a later token.  Such tiles are the few at the edges of the rows' masks.  (A predicate per row in
            // the loop below instead: 2,048 tokens, float32, 16 heads of 128 on 4, 2,081 us, 1,372 so.)
#pragma unroll
            for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) {
                if (corr[i] < 0.0f || !row_ok[i]) continue;
#pragma unroll
                for (int k = 0; k < ATT_ACC; ++k) acc[i][k] *= corr[i];
#pragma unroll 1
                for (int j = 0; j < ATT_TILE; ++j) {
                    const float pj = Ps[warp][j][i];
#pragma unroll
                    for (int k = 0; k < ATT_ACC; ++k) {
                        const int d = lane + 32 * k;
                        if (d < hd) acc[i][k] = fmaf(pj, Vs[j * ld + d], acc[i][k]);
                    }
                }
            }
            continue;
        }
#pragma unroll
        for (int i = 0; i < ATT_ROWS_PER_WARP; ++i)
#pragma unroll
            for (int k = 0; k < ATT_ACC; ++k) acc[i][k] *= corr[i];
#pragma unroll 4
        for (int j = 0; j < ATT_TILE; ++j) {
            const float4 pj = *reinterpret_cast<const float4*>(&Ps[warp][j][0]);
            const float* vl = Vs + j * ld;
#pragma unroll
            for (int k = 0; k < ATT_ACC; ++k) {
                const int d = lane + 32 * k;
                if (d < hd) {
                    const float vv = vl[d];
                    acc[0][k] = fmaf(pj.x, vv, acc[0][k]);
                    acc[1][k] = fmaf(pj.y, vv, acc[1][k]);
                    acc[2][k] = fmaf(pj.z, vv, acc[2][k]);
                    acc[3][k] = fmaf(pj.w, vv, acc[3][k]);
                }
            }
        }
    }

    // results
#pragma unroll
    for (int i = 0; i < ATT_ROWS_PER_WARP; ++i) {
        if (!row_ok[i]) continue;
        const int r = warp * ATT_ROWS_PER_WARP + i;
        const int t = r / a.heads_per_block, hg = chunk * a.heads_per_block + r % a.heads_per_block;
        const long long row = (long long)(seq_tok0 + tok0 + t) * a.q_heads + (kvh * a.group + hg);
        if (a.n_splits == 1) {
            T* o = (T*)a.out + row * hd;
            const float sink = a.sinks != nullptr ? expf(a.sinks[kvh * a.group + hg] - m[i]) : 0.0f;
            const float inv = 1.0f / (l[i] + sink);
#pragma unroll
            for (int k = 0; k < ATT_ACC; ++k) {
                const int d = lane + 32 * k;
                if (d < hd) o[d] = from_float<T>(acc[i][k] * inv);
            }
        } else {
            const long long pr = row * a.n_splits + split;
            if (lane == 0) {
                a.part_ml[pr * 2] = m[i];
                a.part_ml[pr * 2 + 1] = l[i];
            }
#pragma unroll
            for (int k = 0; k < ATT_ACC; ++k) {
                const int d = lane + 32 * k;
                if (d < hd) a.part_o[pr * hd + d] = acc[i][k];
            }
        }
    }
}

// Merge the partial results of the key splits of each (token, head) row; one warp per row.
// The lanes first share out the splits (maximum, weights, sum), then the output dims; the
// loads of a lane do not depend on each other, so they are in flight together.
template <typename T>
__global__ void attention_combine_kernel(const float* __restrict__ part_ml, const float* __restrict__ part_o,
                                         long long n_rows, int n_splits, int hd, const float* __restrict__ sinks, int q_heads,
                                         T* __restrict__ out) {
    grid_launch_dependents();
    grid_dependency_wait();
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n_rows) return;
    const int lane = threadIdx.x & 31;
    const float* ml = part_ml + row * n_splits * 2;
    float M = -INFINITY;
    for (int s = lane; s < n_splits; s += 32) M = fmaxf(M, __ldg(ml + 2 * s));
    M = warp_max(M);
    float L = 0.0f;
    for (int s = lane; s < n_splits; s += 32) {
        const float ms = __ldg(ml + 2 * s);
        if (ms != -INFINITY) L += __ldg(ml + 2 * s + 1) * expf(ms - M);
    }
    L = warp_sum(L);
    if (sinks != nullptr) L += expf(sinks[row % q_heads] - M);      // rows are (token, head) pairs, heads fastest
    const float inv = 1.0f / L;
    const float* po = part_o + row * n_splits * hd;
    for (int d = lane; d < hd; d += 32) {
        float o = 0.0f;
#pragma unroll 8
        for (int s = 0; s < n_splits; ++s) {
            const float ms = __ldg(ml + 2 * s);
            const float w = (ms != -INFINITY) ? expf(ms - M) : 0.0f;
            const float v = __ldg(po + (long long)s * hd + d);
            o += (w != 0.0f) ? v * w : 0.0f;           // an empty split's values were never written
        }
        out[row * hd + d] = from_float<T>(o * inv);
    }
}

}  // namespace mlc

// The launch shared by every entry point of the split-key attention (the ordinary one below and the one that keeps
// its scratch inside the library): checks, the plan of heads and tokens per block, the two kernels.
// n_splits > 1 needs part_ml (n_tokens*q_heads*n_splits*2 floats) and part_o (n_tokens*q_heads*n_splits*hd).
namespace mlc {
static int launch_attention_simt(const void* q, void* out, int dtype, const int* cu_seqlens, const int* start_pos,
                                 int n_seqs, int n_tokens, int max_q_len, int q_heads, int kv_heads, int hd, float scale,
                                 int window, int n_splits, float* part_ml, float* part_o, void* k_pool, void* v_pool,
                                 const int* page_table, long long entry_offset, int pages_per_seq, int page_size,
                                 cudaStream_t s, const float* sinks = nullptr, int keep_first = 0, int chunk = 0,
                                 float softcap = 0.0f) {
    if (n_seqs <= 0 || n_tokens <= 0) return 0;
    if (hd <= 0 || hd > ATT_MAX_HD || q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads != 0) return MLC_ERR_BAD_SIZE;
    if (n_splits < 1 || (n_splits > 1 && (part_ml == nullptr || part_o == nullptr))) return MLC_ERR_BAD_SIZE;
    if (n_seqs > 65535) return MLC_ERR_BAD_SIZE;
    if (chunk < 0 || (chunk > 0 && window > 0) || softcap < 0.0f) return MLC_ERR_UNSUPPORTED;
    if (dtype != MLC_DTYPE_F32 && dtype != MLC_DTYPE_BF16) return MLC_ERR_BAD_DTYPE;
    AttnArgs a;
    a.q = q;
    a.out = out;
    a.cu_seqlens = cu_seqlens;
    a.start_pos = start_pos;
    a.part_ml = part_ml;
    a.part_o = part_o;
    a.sinks = sinks;
    a.scale = scale;
    a.q_heads = q_heads;
    a.group = q_heads / kv_heads;
    a.window = window;
    a.keep_first = keep_first < 0 ? 0 : keep_first;
    a.chunk = chunk;
    a.softcap = softcap;
    a.heads_per_block = a.group < ATT_ROWS ? a.group : ATT_ROWS;
    a.tokens_per_block = ATT_ROWS / a.heads_per_block;
    a.head_chunks = (a.group + a.heads_per_block - 1) / a.heads_per_block;
    a.n_splits = n_splits;
    const long long gy = (long long)kv_heads * a.head_chunks * n_splits;
    if (gy > 65535) return MLC_ERR_BAD_SIZE;
    PagedKV c{k_pool, v_pool, page_table, entry_offset, pages_per_seq, page_size, kv_heads, hd};
    dim3 grid((max_q_len + a.tokens_per_block - 1) / a.tokens_per_block, (unsigned)gy, n_seqs);
    const size_t smem = (size_t)(ATT_ROWS + 2 * ATT_TILE) * att_pitch(hd) * sizeof(float);
    cudaError_t e;
    // one instance per element type and accumulator count; each remembers how much shared memory it was allowed
#define MLC_SIMT_LAUNCH(T, ACC)                                                                                          \
    do {                                                                                                                 \
        static size_t allowed = 48 * 1024;                                                                               \
        if (smem > allowed) {                                                                                            \
            e = cudaFuncSetAttribute(attention_simt_kernel<T, ACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            if (e != cudaSuccess) return (int)e;                                                                         \
            allowed = smem;                                                                                              \
        }                                                                                                                \
        launch_pdl(attention_simt_kernel<T, ACC>, grid, dim3(ATT_WARPS * 32), smem, s, a, c);                                          \
    } while (0)
    if (dtype == MLC_DTYPE_F32) {
        if (hd <= 128) MLC_SIMT_LAUNCH(float, 4);
        else if (hd <= 256) MLC_SIMT_LAUNCH(float, 8);
        else MLC_SIMT_LAUNCH(float, 16);
    } else {
        if (hd <= 256) MLC_SIMT_LAUNCH(bf16, 8);
        else MLC_SIMT_LAUNCH(bf16, 16);
    }
#undef MLC_SIMT_LAUNCH
    MLC_LAUNCH_CHECK();
    // With one split the first kernel has written `out` itself and no scratch was touched; with more, every
    // (row, split) pair of the scratch was written above before the merge reads it.
    if (n_splits > 1) {
        const long long n_rows = (long long)n_tokens * q_heads;
        const unsigned blocks = (unsigned)((n_rows + 3) / 4);
        if (dtype == MLC_DTYPE_F32)
            attention_combine_kernel<float><<<blocks, 128, 0, s>>>(part_ml, part_o, n_rows, n_splits, hd, sinks, q_heads, (float*)out);
        else
            attention_combine_kernel<bf16><<<blocks, 128, 0, s>>>(part_ml, part_o, n_rows, n_splits, hd, sinks, q_heads, (bf16*)out);
        MLC_LAUNCH_CHECK();
    }
    return 0;
}
}  // namespace mlc

#ifndef MLC_KERNELS_ONLY   // a file that includes this one for its kernels defines its own entry points
using namespace mlc;

// q, out: [n_tokens][q_heads][hd] of `dtype`; the cache pools hold the same type.  sinks: null, or one float per query
// head whose exponential is added to that head's softmax denominator (a key that is always seen and has no value).
// max_q_len: the longest sequence of this step (sizes the grid).  n_splits > 1 needs
// part_ml (n_tokens*q_heads*n_splits*2 floats) and part_o (n_tokens*q_heads*n_splits*hd).
extern "C" int mlc_attention_simt(const void* q, void* out, int dtype, const int* cu_seqlens,
                                  const int* start_pos, int n_seqs, int n_tokens, int max_q_len, int q_heads,
                                  int kv_heads, int hd, float scale, int window, int n_splits, float* part_ml,
                                  float* part_o, void* k_pool, void* v_pool, const int* page_table,
                                  long long entry_offset, int pages_per_seq, int page_size, const float* sinks, int keep_first,
                                  int chunk, float softcap, void* stream) {
    return launch_attention_simt(q, out, dtype, cu_seqlens, start_pos, n_seqs, n_tokens, max_q_len, q_heads, kv_heads, hd,
                                 scale, window, n_splits, part_ml, part_o, k_pool, v_pool, page_table, entry_offset,
                                 pages_per_seq, page_size, (cudaStream_t)stream, sinks, keep_first, chunk, softcap);
}

// Merge partial results that another attention kernel left in part_ml / part_o
// (maxima in natural-log units, sums and weighted values relative to them).
extern "C" int mlc_attention_combine(const float* part_ml, const float* part_o, long long n_rows, int n_splits,
                                     int hd, const float* sinks, int q_heads, void* out, int dtype, void* stream) {
    if (n_rows <= 0) return 0;
    if (n_splits < 1 || hd <= 0 || (sinks != nullptr && q_heads <= 0)) return MLC_ERR_BAD_SIZE;
    const unsigned blocks = (unsigned)((n_rows + 3) / 4);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    if (dtype == MLC_DTYPE_F32)
        e = launch_pdl(attention_combine_kernel<float>, dim3(blocks), dim3(128), 0, s, part_ml, part_o, n_rows, n_splits, hd, sinks, q_heads, (float*)out);
    else if (dtype == MLC_DTYPE_BF16)
        e = launch_pdl(attention_combine_kernel<bf16>, dim3(blocks), dim3(128), 0, s, part_ml, part_o, n_rows, n_splits, hd, sinks, q_heads, (bf16*)out);
    else
        return MLC_ERR_BAD_DTYPE;
    return e == cudaSuccess ? 0 : (int)e;
}
#endif  // MLC_KERNELS_ONLY
