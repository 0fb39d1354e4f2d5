// y[token][row] = sum_k W[row][k] · h[token][k] for up to 32 tokens, with the norm that precedes the product and the
// epilogue that follows it in the same kernel.
//
// A product of so few tokens is a stream of weights with next to no arithmetic, and a decode step is a chain of a hundred
// and more of them: what counts is how soon the weights are asked for and how short the way from the last activation of
// the kernel before to the first result is.  So a block asks for its first ring of weight tiles before the wait for the
// kernel before (they depend on nothing) and holds them in shared memory; after the wait a warp needs one trip to L2 for
// its activations, a few products with mma.sync and one exchange through shared memory.
//
// A block owns tiles of 16 rows of W, RT neighbours at a time.  K is cut into units of 64 elements and dealt out to the
// block's warps, UW units each, so that a warp's share of the activations stays in its registers as B fragments for all of
// the block's tiles.  A lane copies with cp.async what it will multiply itself, 16 bytes of a row at a time, into a place
// of its own: no barrier stands between the copy and its use, and a warp's accesses hit all banks.  The 16 bytes hold the
// elements of two k16 steps in an order of their own, the same order for W and h: the sum over k does not care.  The
// warps' partial sums of RT tiles meet in shared memory, are added in the order of the warps, and the epilogue runs with
// one thread per output.
//
// With NORM the activations are the float32 residual stream x and the product is of its RMS norm: the fragments are
// bf16(x·gain), the squares are summed along the way, and the sum over k is multiplied by 1/sqrt(mean(x²) + eps) in
// float32 (src/ops.cpp:19-41).  The rounding to 16 bits is relative, so it costs what rounding the finished norm costs.
//
// What bounds it, B200, one kernel of a chain in a graph, weights from HBM, 8 rows (in brackets the norm's kernel and the
// tcgen05 form that it stands in for): Q/K/V of 1,152 x 896 with its norm 2.5 us (6.6), output product of 896 x 896 1.6 us
// (2.3), gate/up of 9,728 x 896 with its norm 5.2 us = 3.4 TB/s (7.5), down of 896 x 4,864 2.7 us = 3.2 TB/s (3.5): the
// boundary between two kernels (about 1 us) and the trip to L2 for the activations; gate/up of 37,888 x 3,584 44.9 us =
// 6.0 TB/s (48.1): memory.  With the weights held in registers instead of shared memory gate/up took 5.1 us but down 3.5 us
// and the 1,536-wide gate/up 11.6 against 10.6 us.  From 9 rows on the products and the activations' conversion show:
// gate/up 6.4 us at 16 rows (7.5), 9.1 us at 24 (8.9: not taken).
//
// Epilogues as in gemm_tcgen05.cu: STORE, SILU_MUL (rows alternate gate_j, up_j), QKV (rows of a head alternate dim i,
// dim i + hd/2: bias, rotation, cache write), ADD (into the float32 stream: by one block per output where the K range is
// whole, with atomic adds where it is split over blockIdx.y).
#include "gemm_few.cuh"

namespace mlc {

enum { FEW_STORE = 0, FEW_SILU_MUL = 1, FEW_QKV = 2, FEW_ADD = 3 };

struct FewArgs {
    const void* x;             // [n_tok][K]: bfloat16, with NORM float32
    const float* gain;         // NORM: [K]
    float eps;
    const bf16* w;             // [n_out][K]
    void* out;
    int out_dtype;
    int n_tok, n_out, K;
    int units_per_split;       // units of K a block takes: blockIdx.y · units_per_split ...
    int tiles;                 // ceil(n_out / 16)
    const float* bias;         // QKV
    const int* positions;
    const int* tok_seq;
    const float2* rope;
    int rope_positions;
    int q_heads, kv_heads, hd;
    PagedKV cache;
    int glu_kind;              // SILU_MUL
    float glu_limit, glu_alpha;
};

// NT: tiles of 8 tokens; UW: units of K per warp; RT: tiles of 16 rows between two barriers, which is also the depth of the
// ring of weight tiles.
template <int NT, int UW, int RT, int EPI, bool NORM>
__global__ void __launch_bounds__(32 * FEW_MAX_WARPS, 1) gemm_few_kernel(FewArgs g) {
    constexpr int TOKENS = 8 * NT;
    constexpr int TILE_U4 = UW * 4 * 32;                                       // 16-byte pieces of a warp's part of a weight tile
    extern __shared__ uint4 few_smem[];
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gq = lane >> 2, t = lane & 3;
    uint4* const ring = few_smem + warp * RT * TILE_U4 + lane;                 // [warps][RT][UW][4][32]
    float* const red = reinterpret_cast<float*>(few_smem + warps * RT * TILE_U4);   // [warps][RT][TOKENS][FEW_PITCH]
    float* const squares = red + warps * RT * TOKENS * FEW_PITCH;              // [warps][TOKENS], NORM only
    long long* const tok_off = reinterpret_cast<long long*>(squares + (NORM ? FEW_MAX_WARPS * TOKENS : 0));   // [TOKENS], QKV only
    int* const tok_pos = reinterpret_cast<int*>(tok_off + TOKENS);             // [TOKENS], QKV only

    const int n_units = g.K / FEW_UNIT;
    const int unit0 = blockIdx.y * g.units_per_split + warp;
    const int unit_end = min(n_units, ((int)blockIdx.y + 1) * g.units_per_split);

    grid_launch_dependents();
    // the warp's part of weight tile `tile` on its way into slot `slot`: per unit rows gq and gq + 8, each k 0-31 and 32-63
    const unsigned ring_at = (unsigned)__cvta_generic_to_shared(ring);
    auto ask = [&](int slot, int tile) {
        if (tile < g.tiles) {
            const int r = tile * FEW_ROWS + gq;
            const bf16* p = g.w + (long long)min(r, g.n_out - 1) * g.K + unit0 * FEW_UNIT + t * 8;
            const bf16* q = g.w + (long long)min(r + 8, g.n_out - 1) * g.K + unit0 * FEW_UNIT + t * 8;
#pragma unroll
            for (int i = 0; i < UW; ++i) {
                if (unit0 + i * warps < unit_end) {
                    const unsigned at = ring_at + (slot * TILE_U4 + i * 128) * 16;
                    const int k = i * warps * FEW_UNIT;
                    few_copy16(at, p + k);
                    few_copy16(at + 512, q + k);
                    few_copy16(at + 1024, p + k + 32);
                    few_copy16(at + 1536, q + k + 32);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int r = 0; r < RT; ++r) ask(r, blockIdx.x * RT + r);
    if (NORM) {                // the gain's lines on their way into L2: 64 floats a unit are two lines
#pragma unroll
        for (int i = 0; i < UW; ++i) {
            const int unit = unit0 + i * warps;
            if (unit < unit_end && lane < 2) few_prefetch_l2(g.gain + unit * FEW_UNIT + 32 * lane);
        }
    }
    if (EPI == FEW_QKV) {
        // the step's description was complete before the step's first kernel
        for (int k = threadIdx.x; k < TOKENS; k += blockDim.x) {
            int p = 0;
            long long off = 0;
            if (k < g.n_tok) {
                p = __ldg(g.positions + k);
                if (g.kv_heads > 0) off = paged_offset(g.cache, __ldg(g.tok_seq + k), p, 0);
            }
            tok_pos[k] = p;
            tok_off[k] = off;
        }
        __syncthreads();
    }
    // what the epilogue of this thread's first output wants beside the sum: asked for ahead as well
    const int o_tok = (threadIdx.x >> 4) & (TOKENS - 1), o_row = (blockIdx.x * RT + threadIdx.x / (16 * TOKENS)) * FEW_ROWS + (threadIdx.x & 15);
    const bool o_ok = threadIdx.x < RT * TOKENS * FEW_ROWS && o_tok < g.n_tok && o_row < g.n_out;
    float pre_bias = 0.0f, pre_add = 0.0f;
    float2 pre_cs = make_float2(1.0f, 0.0f);
    auto bias_of = [&](int row) { return (g.bias != nullptr && row < g.n_out) ? __ldg(g.bias + row) : 0.0f; };
    auto rotation_of = [&](int tok, int row) {
        const int head = row / g.hd;
        if (g.rope == nullptr || head >= g.q_heads + g.kv_heads) return make_float2(1.0f, 0.0f);
        return __ldg(g.rope + (long long)min(tok_pos[tok], g.rope_positions - 1) * (g.hd >> 1) + ((row % g.hd) >> 1));
    };
    if (EPI == FEW_QKV && o_ok) pre_bias = bias_of(o_row);
    grid_dependency_wait();
    if (EPI == FEW_QKV && o_ok) pre_cs = rotation_of(o_tok, o_row);          // behind the wait: this step may have made the table longer
    const bool adds_alone = EPI == FEW_ADD && gridDim.y == 1;
    if (adds_alone && o_ok) pre_add = __ldcg((const float*)g.out + (long long)o_tok * g.n_out + o_row);

    // ---------------- the warp's activations as B fragments: token gq (+ 8 per n-tile), k = unit · 64 + half · 32 + 8t ... + 7
    unsigned b[UW][NT][8];
    float sq[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) sq[n] = 0.0f;
    if (!NORM) {
#pragma unroll
        for (int i = 0; i < UW; ++i) {
            const int unit = unit0 + i * warps;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int tok = n * 8 + gq;
                uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
                if (unit < unit_end && tok < g.n_tok) {
                    const bf16* p = (const bf16*)g.x + (long long)tok * g.K + unit * FEW_UNIT + t * 8;
                    lo = __ldcg(reinterpret_cast<const uint4*>(p));
                    hi = __ldcg(reinterpret_cast<const uint4*>(p + 32));
                }
                b[i][n][0] = lo.x; b[i][n][1] = lo.y; b[i][n][2] = lo.z; b[i][n][3] = lo.w;
                b[i][n][4] = hi.x; b[i][n][5] = hi.y; b[i][n][6] = hi.z; b[i][n][7] = hi.w;
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < UW; ++i) {
            const int unit = unit0 + i * warps;
            float4 gn[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) gn[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const int k0 = unit * FEW_UNIT + t * 8;
            if (unit < unit_end) {
#pragma unroll
                for (int j = 0; j < 4; ++j) gn[j] = __ldg(reinterpret_cast<const float4*>(g.gain + k0 + (j >> 1) * 32 + (j & 1) * 4));
            }
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int tok = n * 8 + gq;
                float4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (unit < unit_end && tok < g.n_tok) {
                    const float* p = (const float*)g.x + (long long)tok * g.K + k0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = __ldcg(reinterpret_cast<const float4*>(p + (j >> 1) * 32 + (j & 1) * 4));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sq[n] = fmaf(v[j].x, v[j].x, fmaf(v[j].y, v[j].y, fmaf(v[j].z, v[j].z, fmaf(v[j].w, v[j].w, sq[n]))));
                    b[i][n][2 * j] = few_pack(v[j].x * gn[j].x, v[j].y * gn[j].y);
                    b[i][n][2 * j + 1] = few_pack(v[j].z * gn[j].z, v[j].w * gn[j].w);
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            sq[n] += __shfl_xor_sync(0xffffffffu, sq[n], 1);
            sq[n] += __shfl_xor_sync(0xffffffffu, sq[n], 2);
            if (t == 0) squares[warp * TOKENS + n * 8 + gq] = sq[n];
        }
    }

    for (int tile = blockIdx.x * RT; tile < g.tiles; tile += gridDim.x * RT) {
        float acc[RT][NT][4];
#pragma unroll
        for (int r = 0; r < RT; ++r) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[r][n][e] = 0.0f;
            few_wait_copies<RT - 1>();
#pragma unroll
            for (int i = 0; i < UW; ++i) {
                if (unit0 + i * warps < unit_end) {
                    const uint4* const at = ring + r * TILE_U4 + i * 128;
                    const uint4 p0 = at[0], q0 = at[32], p1 = at[64], q1 = at[96];
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        few_mma(acc[r][n], p0.x, q0.x, p0.y, q0.y, b[i][n][0], b[i][n][1]);
                        few_mma(acc[r][n], p0.z, q0.z, p0.w, q0.w, b[i][n][2], b[i][n][3]);
                        few_mma(acc[r][n], p1.x, q1.x, p1.y, q1.y, b[i][n][4], b[i][n][5]);
                        few_mma(acc[r][n], p1.z, q1.z, p1.w, q1.w, b[i][n][6], b[i][n][7]);
                    }
                }
            }
            ask(r, tile + gridDim.x * RT + r);             // behind the products that have read the slot
        }
        if (tile != blockIdx.x * RT) __syncthreads();      // the sums of the tiles before have been read
#pragma unroll
        for (int r = 0; r < RT; ++r) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float* const at = red + ((warp * RT + r) * TOKENS + n * 8 + 2 * t) * FEW_PITCH + gq;
                at[0] = acc[r][n][0];
                at[FEW_PITCH] = acc[r][n][1];
                at[8] = acc[r][n][2];
                at[FEW_PITCH + 8] = acc[r][n][3];
            }
        }
        __syncthreads();
        const bool first_tile = tile == blockIdx.x * RT;
        // one thread per output: 16 rows of a token on neighbouring lanes; a warp's two tokens are neighbours
        for (int o = threadIdx.x; o < RT * TOKENS * FEW_ROWS; o += blockDim.x) {
            const int rt = o / (TOKENS * FEW_ROWS), tok = (o >> 4) & (TOKENS - 1), r = o & 15, row = (tile + rt) * FEW_ROWS + r;
            if ((tok & ~1) >= g.n_tok || tile + rt >= g.tiles) continue;          // the same for the whole warp
            float v = 0.0f;
#pragma unroll 4
            for (int k = 0; k < warps; ++k) v += red[((k * RT + rt) * TOKENS + tok) * FEW_PITCH + r];
            if (NORM) {
                float s = 0.0f;
#pragma unroll 4
                for (int k = 0; k < warps; ++k) s += squares[k * TOKENS + tok];
                v *= rsqrtf(s / (float)g.K + g.eps);
            }
            const bool ok = tok < g.n_tok && row < g.n_out;
            const bool ahead = first_tile && o == threadIdx.x;
            if (EPI == FEW_STORE) {
                if (ok) {
                    const long long at = (long long)tok * g.n_out + row;
                    if (g.out_dtype == MLC_DTYPE_F32) ((float*)g.out)[at] = v;
                    else ((bf16*)g.out)[at] = __float2bfloat16_rn(v);
                }
            } else if (EPI == FEW_ADD) {
                if (ok) {
                    float* const p = (float*)g.out + (long long)tok * g.n_out + row;
                    if (adds_alone) *p = (ahead ? pre_add : __ldcg(p)) + v;
                    else atomicAdd(p, v);
                }
            } else if (EPI == FEW_SILU_MUL) {
                const float up = __shfl_xor_sync(0xffffffffu, v, 1);
                if (ok && (r & 1) == 0) {
                    const float act = g.glu_kind == 0 ? glu_act<0>(v, up, 0.0f, 0.0f)
                                      : g.glu_kind == 1 ? glu_act<1>(v, up, 0.0f, 0.0f)
                                                        : glu_act<2>(v, up, g.glu_limit, g.glu_alpha);
                    const long long at = (long long)tok * (g.n_out >> 1) + (row >> 1);
                    if (g.out_dtype == MLC_DTYPE_F32) ((float*)g.out)[at] = act;
                    else ((bf16*)g.out)[at] = __float2bfloat16_rn(act);
                }
            } else {
                const int half = g.hd >> 1, head = row / g.hd, within = row % g.hd;
                const bool second = (within & 1) != 0;
                const float y0 = v + (ahead ? pre_bias : bias_of(row));
                const float other = __shfl_xor_sync(0xffffffffu, y0, 1);
                if (ok) {
                    const float2 cs = ahead ? pre_cs : rotation_of(tok, row);
                    const float y = second ? other * cs.y + y0 * cs.x : y0 * cs.x - other * cs.y;
                    const int d = (within >> 1) + (second ? half : 0);
                    const bool is_q = head < g.q_heads, is_k = !is_q && head < g.q_heads + g.kv_heads;
                    const int kvh = is_k ? head - g.q_heads : head - g.q_heads - g.kv_heads;
                    void* const to = is_q ? g.out : is_k ? g.cache.k_pool : g.cache.v_pool;
                    const long long at = is_q ? ((long long)tok * g.q_heads + head) * g.hd + d
                                              : tok_off[tok] + (long long)kvh * g.cache.page_size * g.hd + d;
                    if (g.out_dtype == MLC_DTYPE_F32) ((float*)to)[at] = y;
                    else ((bf16*)to)[at] = __float2bfloat16_rn(y);
                }
            }
        }
    }
}

template <int NT, int UW, int RT, int EPI, bool NORM>
static int launch_few(const FewArgs& g, int blocks, int splits, int warps, cudaStream_t s) {
    const size_t smem = (size_t)warps * RT * UW * 2048 + sizeof(float) * (warps * RT * 8 * NT * FEW_PITCH + (NORM ? FEW_MAX_WARPS * 8 * NT : 0)) +
                        (EPI == FEW_QKV ? 8 * NT * (sizeof(long long) + sizeof(int)) : 0);
    if (smem > 227 * 1024) return MLC_ERR_BAD_SIZE;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<NT, UW, RT, EPI, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int groups = (g.tiles + RT - 1) / RT;
    cudaError_t e = launch_pdl(gemm_few_kernel<NT, UW, RT, EPI, NORM>, dim3(blocks < groups ? blocks : groups, splits), dim3(32 * warps), smem, s, g);
    return e == cudaSuccess ? 0 : (int)e;
}

template <int NT, int UW, int RT>
static int launch_few_epilogue(const FewArgs& g, int epilogue, bool norm, int blocks, int splits, int warps, cudaStream_t s) {
    if (epilogue == FEW_ADD) return norm ? MLC_ERR_UNSUPPORTED : launch_few<NT, UW, RT, FEW_ADD, false>(g, blocks, splits, warps, s);
    if (epilogue == FEW_STORE)
        return norm ? launch_few<NT, UW, RT, FEW_STORE, true>(g, blocks, splits, warps, s) : launch_few<NT, UW, RT, FEW_STORE, false>(g, blocks, splits, warps, s);
    if (epilogue == FEW_SILU_MUL)
        return norm ? launch_few<NT, UW, RT, FEW_SILU_MUL, true>(g, blocks, splits, warps, s) : launch_few<NT, UW, RT, FEW_SILU_MUL, false>(g, blocks, splits, warps, s);
    return norm ? launch_few<NT, UW, RT, FEW_QKV, true>(g, blocks, splits, warps, s) : launch_few<NT, UW, RT, FEW_QKV, false>(g, blocks, splits, warps, s);
}

template <int NT>
static int launch_few_shape(const FewArgs& g, int uw, int rt, int epilogue, bool norm, int blocks, int splits, int warps, cudaStream_t s) {
    switch (uw * 8 + rt) {     // what gemm_few_plan in kernels/bindings.py gives, and the shapes beside those that a caller's own plan may name
        case 9: return launch_few_epilogue<NT, 1, 1>(g, epilogue, norm, blocks, splits, warps, s);
        case 10: return launch_few_epilogue<NT, 1, 2>(g, epilogue, norm, blocks, splits, warps, s);
        case 11: if constexpr (NT == 1) return launch_few_epilogue<NT, 1, 3>(g, epilogue, norm, blocks, splits, warps, s); break;
        case 17: return launch_few_epilogue<NT, 2, 1>(g, epilogue, norm, blocks, splits, warps, s);
        case 18: return launch_few_epilogue<NT, 2, 2>(g, epilogue, norm, blocks, splits, warps, s);
        case 25: if constexpr (NT <= 2) return launch_few_epilogue<NT, 3, 1>(g, epilogue, norm, blocks, splits, warps, s); break;
        case 33: if constexpr (NT <= 2) return launch_few_epilogue<NT, 4, 1>(g, epilogue, norm, blocks, splits, warps, s); break;
    }
    return MLC_ERR_BAD_SIZE;
}

}  // namespace mlc

using namespace mlc;

// x: bfloat16 [n_tok][K] (gain null), or float32 [n_tok][K] whose RMS norm with `gain` and `eps` is multiplied; w: bfloat16
// [n_out][K]; n_tok <= 32, K a multiple of 64, everything 16-byte aligned.  epilogue: 0 out [n_tok][n_out], 1 out
// [n_tok][n_out/2], 2 out = q [n_tok][q_heads·hd] with k and v in the cache, 3 out (float32 [n_tok][n_out]) += (bfloat16 x).
// warps (up to 16) of a block, units = units of 64 elements of K per warp, row_tiles = tiles of 16 rows
// at a time (the shapes that launch_few_shape lists), blocks: how many walk the tiles, splits: how many share the K range (epilogue 3 only): warps · units · splits · 64 >= K.
extern "C" int mlc_gemm_few(const void* x, const float* gain, float eps, const void* w, void* out, int out_dtype, int n_tok, int n_out,
                            int K, int epilogue, int warps, int units, int row_tiles, int blocks, int splits, const float* bias, const int* positions,
                            const int* tok_seq, const void* rope_table, int rope_positions, int q_heads, int kv_heads, int hd,
                            void* k_pool, void* v_pool, const int* page_table, long long entry_offset, int pages_per_seq, int page_size,
                            int glu_kind, float glu_limit, float glu_alpha, void* stream) {
    if (n_tok <= 0 || n_out <= 0) return 0;
    if (n_tok > 32 || K <= 0 || K % FEW_UNIT || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)gain) & 15)) return MLC_ERR_BAD_SIZE;
    if (out_dtype != MLC_DTYPE_F32 && out_dtype != MLC_DTYPE_BF16) return MLC_ERR_BAD_DTYPE;
    if (epilogue < 0 || epilogue > 3) return MLC_ERR_UNSUPPORTED;
    if (epilogue == FEW_ADD && out_dtype != MLC_DTYPE_F32) return MLC_ERR_BAD_DTYPE;
    if (warps < 1 || warps > FEW_MAX_WARPS || blocks < 1 || splits < 1 || (splits > 1 && epilogue != FEW_ADD)) return MLC_ERR_BAD_SIZE;
    if (glu_kind < 0 || glu_kind > 2 || (glu_kind == 2 && !(glu_limit > 0.0f))) return MLC_ERR_UNSUPPORTED;
    if (epilogue == FEW_SILU_MUL && (n_out & 1)) return MLC_ERR_BAD_SIZE;
    FewArgs g{};
    g.x = x; g.gain = gain; g.eps = eps; g.w = (const bf16*)w; g.out = out; g.out_dtype = out_dtype;
    g.n_tok = n_tok; g.n_out = n_out; g.K = K;
    const int n_units = K / FEW_UNIT;
    g.units_per_split = (n_units + splits - 1) / splits;
    if ((long long)g.units_per_split > (long long)warps * units || (splits - 1) * g.units_per_split >= n_units) return MLC_ERR_BAD_SIZE;
    g.tiles = (n_out + FEW_ROWS - 1) / FEW_ROWS;
    g.glu_kind = glu_kind; g.glu_limit = glu_limit; g.glu_alpha = glu_alpha;
    g.hd = 2;
    if (epilogue == FEW_QKV) {
        if (hd <= 0 || (hd & 1) || n_out != (q_heads + 2 * kv_heads) * hd || positions == nullptr) return MLC_ERR_BAD_SIZE;
        if (kv_heads > 0 && (tok_seq == nullptr || k_pool == nullptr || v_pool == nullptr || page_table == nullptr)) return MLC_ERR_BAD_SIZE;
        g.bias = bias; g.positions = positions; g.tok_seq = tok_seq; g.rope = (const float2*)rope_table; g.rope_positions = rope_positions;
        g.q_heads = q_heads; g.kv_heads = kv_heads; g.hd = hd;
        g.cache = PagedKV{k_pool, v_pool, page_table, entry_offset, pages_per_seq, page_size, kv_heads, hd};
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (n_tok <= 8) return launch_few_shape<1>(g, units, row_tiles, epilogue, gain != nullptr, blocks, splits, warps, s);
    if (n_tok <= 16) return launch_few_shape<2>(g, units, row_tiles, epilogue, gain != nullptr, blocks, splits, warps, s);
    return launch_few_shape<4>(g, units, row_tiles, epilogue, gain != nullptr, blocks, splits, warps, s);
}
