// What the two prompt forms of the tcgen05 product share (tokens as the M operand: gemm_tcgen05_rows.cu with one SM
// per tile, gemm_tcgen05_pair.cu with a pair of SMs): the arguments, and what an epilogue thread does with 32 columns
// of its token's accumulator row.
#pragma once

#include "tcgen05.cuh"

namespace mlc {

enum { R_EPI_STORE = 0, R_EPI_SILU_MUL = 1, R_EPI_QKV = 2, R_EPI_ADD = 3 };

struct RowsArgs {
    void* out;
    int out_dtype;
    int n_out;                 // rows of W = columns of the product; a multiple of 16
    int n_tok;
    int k_blocks;              // ceil(K / 64)
    int m_tiles, n_tiles;
    int n_first;               // tiles of one token tile follow one another (1), or those of one tile of W's rows (0)
    int n_splits;              // blocks that share out a tile's K range (ADD only); 1: none
    int k_blocks_per_split;
    int* status;
    // QKV epilogue
    const float* bias;         // [n_out] in the stored row order, or null
    const int* positions;      // [tokens]
    const int* tok_seq;        // [tokens]
    const float2* rope;        // [positions][hd/2] cos, sin; or null
    int rope_positions;
    int q_heads, kv_heads, hd;
    PagedKV cache;
    // grouped form (one-SM kernel only): every token tile of 128 rows multiplies by the matrix of its own group, group e's
    // n_out rows starting at row e * n_out of W.  tile_group [m_tiles]: the tile's group, negative: the tile is skipped.
    // The table comes from a kernel before this one, so nothing is asked for ahead of the wait for that kernel.
    const int* tile_group;
    // STORE only: an activation applied to the product before it is stored (0 none, 1 silu, 2 gelu with erf, 3 gelu with
    // the tanh approximation), in float32
    int act;
    // SILU_MUL only: which gated unit the epilogue forms from the alternating gate and up columns (0 SiLU, 1 the tanh form of
    // GELU, 2 clamped with `glu_limit` and `glu_alpha`: see glu_act)
    int glu_kind;
    float glu_limit, glu_alpha;
};

// One activation over a chunk of accumulator columns.  The kind is tested once per chunk, outside the unrolled loop: with
// the test inside, the loop's body holds all three functions, is not unrolled, and the chunk is indexed through local
// memory (a product with an activation then took 1.7 times the time of the same product without one).
template <int ACT>
__device__ __forceinline__ float rows_activation(float z) {
    if constexpr (ACT == 1) return z / (1.0f + expf(-z));
    else if constexpr (ACT == 2) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752440f));
    else return 0.5f * z * (1.0f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z)));
}

__device__ __forceinline__ void rows_activate(float (&v)[32], int act) {
    if (act == 1) {
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = rows_activation<1>(v[u]);
    } else if (act == 2) {
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = rows_activation<2>(v[u]);
    } else {
#pragma unroll
        for (int u = 0; u < 32; ++u) v[u] = rows_activation<3>(v[u]);
    }
}

constexpr int R_BM = 128;
constexpr int R_BK = 64;
constexpr int R_A_BYTES = R_BM * R_BK * 2;

__device__ __forceinline__ unsigned pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<unsigned*>(&h);
}

// Tile number t of a product.  Consecutive blocks take tiles that share one operand's piece, which is then fetched from memory
// once by all of them together, while the other operand is walked whole for each such piece, out of L2 if it stays there
// (n_first: the shared pieces are x's).
struct TileWalk {
    int m, n, split;
};
__device__ __forceinline__ TileWalk tile_walk(const RowsArgs& g, int t) {
    TileWalk w;
    const int inner = g.n_first ? g.n_tiles : g.m_tiles, outer = g.n_first ? g.m_tiles : g.n_tiles;
    const int i = t % inner, r = t / inner, o = r % outer;
    w.m = g.n_first ? o : i;
    w.n = g.n_first ? i : o;
    w.split = r / outer;
    return w;
}

// Whether a product's walk shares x's pieces and goes through W for each of them (n_first).  An adding product's does where x has
// more rows than W: its output is fetched and written in L2 too, and consecutive blocks then work on the same tokens' rows.  B200,
// us, W's pieces shared and x's: 2,048 x 512 16,384 tokens 66.0, 59.7; 896 x 4,864 8,191 63.7, 60.7, 16,384 141, 121; whole prompts
// of the 0.5B sizes of 2,048 tokens 2,366, 2,349 (1,000 to 4,500 tokens by themselves the other way, by 2 %).  The others' does
// where x does not stay in L2 from one piece of W to the next, beyond some 60 MB, half of the 126 MB that two dies share: STORE
// 4,096 x 4,096 8,191 (67 MB) 203, 198, 16,384 424, 351; QKV 4,608 x 3,584 8,191 (59 MB) 265, 267, 16,384 641, 548; but QKV
// 1,536 x 512 2,048 14.8, 17.4; STORE 1,152 x 896 16,384 (29 MB) 31.8, 34.0.
static bool walk_shares_x(long long n_tok, long long n_out, long long K, int epilogue) {
    return n_tok > n_out && (epilogue == R_EPI_ADD || n_tok * K * 2 > 60000000);
}

// A warp's 32 tokens x 32 accumulator columns on their way into the float32 stream through `buf`, 4 KiB of shared memory of the
// warp's own: a thread writes its token's 128 bytes (16-byte pieces in the order of the 128-byte swizzle, so that eight lanes hit
// all banks), one lane hands the tile to TMA, which adds a line at a time; 16-byte atomic adds by the threads themselves touch 32
// lines an instruction.  B200, us, those adds and these, the same walk: 896 x 4,864 512 tokens 8.7, 7.9, 2,048 18.2, 17.2; 896 x
// 896 8,191 19.7, 15.9; 1,536 x 1,536 2,048 19.7, 17.4; 2,048 x 512 8,191 36.9, 26.6.
constexpr int R_OUT_BYTES = 32 * 32 * 4;
__device__ __forceinline__ void rows_tile_add(const CUtensorMap* map, const float (&v)[32], unsigned buf, int lane, int n, int tok0) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(buf + lane * 128 + ((u ^ (lane & 7)) << 4)), "f"(v[4 * u]),
                     "f"(v[4 * u + 1]), "f"(v[4 * u + 2]), "f"(v[4 * u + 3]) : "memory");
    fence_async_shared();
    __syncwarp();
    if (lane == 0) {
        tma_add_2d(map, n, tok0, buf);
        tma_store_commit();
    }
}

// One token's 32 (or, at the matrix's edge, 16) accumulator columns n .. n+31 leave the block.  `second`: the upper 16
// exist too.  STORE: y as float32 or bfloat16; SILU_MUL: columns alternate gate_j, up_j and gate·sigmoid(gate)·up goes to [token][n/2].
template <int EPI>
__device__ __forceinline__ void rows_epilogue_chunk(const RowsArgs& g, const float (&vin)[32], int tok, int n, bool second) {
    float v[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) v[u] = vin[u];
    if (EPI == R_EPI_STORE && g.act != 0) rows_activate(v, g.act);
    if (EPI == R_EPI_STORE) {
        if (g.out_dtype == MLC_DTYPE_BF16) {
            uint4* dst = reinterpret_cast<uint4*>((bf16*)g.out + (long long)tok * g.n_out + n);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (u < 2 || second)
                    dst[u] = make_uint4(pack2(v[8 * u], v[8 * u + 1]), pack2(v[8 * u + 2], v[8 * u + 3]),
                                        pack2(v[8 * u + 4], v[8 * u + 5]), pack2(v[8 * u + 6], v[8 * u + 7]));
        } else {
            float4* dst = reinterpret_cast<float4*>((float*)g.out + (long long)tok * g.n_out + n);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < 4 || second) dst[u] = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
        }
    } else {                                          // SILU_MUL: columns alternate gate_j, up_j
        float act[16];
        // the kind is tested once per chunk, outside the unrolled loops
        if (g.glu_kind == 0) {
#pragma unroll
            for (int u = 0; u < 16; ++u) act[u] = glu_act<0>(v[2 * u], v[2 * u + 1], 0.0f, 0.0f);
        } else if (g.glu_kind == 1) {
#pragma unroll
            for (int u = 0; u < 16; ++u) act[u] = glu_act<1>(v[2 * u], v[2 * u + 1], 0.0f, 0.0f);
        } else {
#pragma unroll
            for (int u = 0; u < 16; ++u) act[u] = glu_act<2>(v[2 * u], v[2 * u + 1], g.glu_limit, g.glu_alpha);
        }
        const long long at = (long long)tok * (g.n_out >> 1) + (n >> 1);
        if (g.out_dtype == MLC_DTYPE_BF16) {
            uint4* dst = reinterpret_cast<uint4*>((bf16*)g.out + at);
            dst[0] = make_uint4(pack2(act[0], act[1]), pack2(act[2], act[3]), pack2(act[4], act[5]), pack2(act[6], act[7]));
            if (second) dst[1] = make_uint4(pack2(act[8], act[9]), pack2(act[10], act[11]), pack2(act[12], act[13]), pack2(act[14], act[15]));
        } else {
            float4* dst = reinterpret_cast<float4*>((float*)g.out + at);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (u < 2 || second) dst[u] = make_float4(act[4 * u], act[4 * u + 1], act[4 * u + 2], act[4 * u + 3]);
        }
    }
}

}  // namespace mlc
