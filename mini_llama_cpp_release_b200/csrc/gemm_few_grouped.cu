// The few-row product of gemm_few.cu for experts: y[row] = W[expert of the row's run] · x[row] where up to 16 (token, choice)
// pairs stand in runs, one per chosen expert (the order moe_plan makes, with runs padded to `group_rows`).
//
// All chosen experts' tiles of W form one list, experts in order, and a block walks an equal, unbroken share of it: how many
// experts were chosen is known on the device alone, and a share of the list spans two or three of them at most.  Where the
// expert changes, the warps fetch that run's rows as B fragments; the ring of weight tiles runs on across the change.  With `src_tok` the rows are
// gathered on the way (row r of a run is row src_tok[r] of x), which saves the kernel that would lay them out.
//
// What bounds it: the chosen experts' weights.  B200, 8 tokens of which each takes one of 8 experts of 1,536 x 4,480 (5.3 chosen
// on average), in brackets tiles of 128 tokens: gate/up 30 us = 4.8 TB/s (33 and 3 for the gather), down 22 us = 3.3 TB/s (57:
// its 64 tiles left most SMs idle).
#include "gemm_few.cuh"

namespace mlc {

struct GroupedFewArgs {
    const bf16* x;             // rows of K: [groups][group_rows], or any with src_tok
    const int* src_tok;        // [groups * group_rows] or null: a row's row of x, negative: padding
    const bf16* w;             // [E][n_out][K]
    const int* tile_group;     // [groups] a run's expert; the runs come first, then -1
    void* out;                 // [groups * group_rows][n_out or n_out / 2]
    int out_dtype;
    int groups, group_rows, n_out, K;
    int tiles;                 // ceil(n_out / 16)
    int glu_kind;
    float glu_limit, glu_alpha;
};

// Two units a warp and two tiles at a time: up to 12 warps' rings leave room for a second block on an SM, whose loads are
// under way while the first block's sums meet; the registers are held down to allow it.
template <int NT, int UW, int RT, bool SILU>
__global__ void __launch_bounds__(UW == 2 && NT == 1 ? 384 : 32 * FEW_MAX_WARPS, UW == 2 && NT == 1 ? 2 : 1)
gemm_few_grouped_kernel(GroupedFewArgs g) {
    constexpr int TOKENS = 8 * NT;
    constexpr int TILE_U4 = UW * 4 * 32;
    extern __shared__ uint4 few_smem[];
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gq = lane >> 2, t = lane & 3;
    uint4* const ring = few_smem + warp * RT * TILE_U4 + lane;                      // [warps][RT][UW][4][32]
    float* const red = reinterpret_cast<float*>(few_smem + warps * RT * TILE_U4);   // [warps][RT][TOKENS][FEW_PITCH]
    const int n_units = g.K / FEW_UNIT;

    // The plan: complete before the kernel before this one began, unless that was the plan itself (`src_tok`: no kernel has
    // laid the rows out in between).  In the first case the weights are asked for ahead of the wait; in the second the kernel
    // after this one may begin only behind the wait, so that it in turn finds the plan complete.
    if (g.src_tok != nullptr) grid_dependency_wait();
    grid_launch_dependents();
    const int run_expert = lane < g.groups ? __ldcg(g.tile_group + lane) : -1;      // lane r: the expert of run r
    const int active = __popc(__ballot_sync(0xffffffffu, run_expert >= 0));
    const int per_group = (g.tiles + RT - 1) / RT;                                  // items: RT neighbouring tiles of an expert
    const long long total = (long long)active * per_group;
    const int lo = (int)(total * blockIdx.x / gridDim.x), hi = (int)(total * (blockIdx.x + 1) / gridDim.x);

    const unsigned ring_at = (unsigned)__cvta_generic_to_shared(ring);
    auto ask = [&](int slot, int item) {
        const int grp = item / per_group, tile = (item - grp * per_group) * RT + slot;
        const int expert = __shfl_sync(0xffffffffu, run_expert, grp & 31);
        if (item < hi && tile < g.tiles) {
            const bf16* w = g.w + (long long)expert * g.n_out * g.K;
            const int r = tile * FEW_ROWS + gq;
            const bf16* p = w + (long long)min(r, g.n_out - 1) * g.K + warp * FEW_UNIT + t * 8;
            const bf16* q = w + (long long)min(r + 8, g.n_out - 1) * g.K + warp * FEW_UNIT + t * 8;
#pragma unroll
            for (int i = 0; i < UW; ++i) {
                if (warp + i * warps < n_units) {
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
    for (int r = 0; r < RT; ++r) ask(r, lo);
    if (g.src_tok == nullptr) grid_dependency_wait();

    unsigned b[UW][NT][8];
    int have = -1;
    for (int item = lo; item < hi; ++item) {
        const int grp = item / per_group, tile = (item - grp * per_group) * RT;
        if (grp != have) {                                 // the same for the whole block
            have = grp;
            const bf16* row[NT];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int at = grp * g.group_rows + n * 8 + gq;
                long long src = at;
                if (g.src_tok != nullptr) src = n * 8 + gq < g.group_rows ? __ldcg(g.src_tok + at) : -1;
                row[n] = src >= 0 && n * 8 + gq < g.group_rows ? g.x + src * g.K : nullptr;
            }
#pragma unroll
            for (int i = 0; i < UW; ++i) {
                const int unit = warp + i * warps;
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    uint4 lo4 = make_uint4(0u, 0u, 0u, 0u), hi4 = lo4;
                    if (unit < n_units && row[n] != nullptr) {
                        const bf16* p = row[n] + unit * FEW_UNIT + t * 8;
                        lo4 = __ldcg(reinterpret_cast<const uint4*>(p));
                        hi4 = __ldcg(reinterpret_cast<const uint4*>(p + 32));
                    }
                    b[i][n][0] = lo4.x; b[i][n][1] = lo4.y; b[i][n][2] = lo4.z; b[i][n][3] = lo4.w;
                    b[i][n][4] = hi4.x; b[i][n][5] = hi4.y; b[i][n][6] = hi4.z; b[i][n][7] = hi4.w;
                }
            }
        }
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
                if (warp + i * warps < n_units) {
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
            ask(r, item + 1);                              // behind the products that have read the slot
        }
        if (item != lo) __syncthreads();                   // the sums of the tiles before have been read
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
        // one thread per output: 16 rows of a token on neighbouring lanes, a warp's two tokens are neighbours
        for (int o = threadIdx.x; o < RT * TOKENS * FEW_ROWS; o += blockDim.x) {
            const int rt = o / (TOKENS * FEW_ROWS), tok = (o >> 4) & (TOKENS - 1), r = o & 15, row = (tile + rt) * FEW_ROWS + r;
            if ((tok & ~1) >= g.group_rows || tile + rt >= g.tiles) continue;      // the same for the whole warp
            float v = 0.0f;
#pragma unroll 4
            for (int k = 0; k < warps; ++k) v += red[((k * RT + rt) * TOKENS + tok) * FEW_PITCH + r];
            const bool ok = tok < g.group_rows && row < g.n_out;
            const long long out_row = (long long)grp * g.group_rows + tok;
            if (SILU) {
                const float up = __shfl_xor_sync(0xffffffffu, v, 1);
                if (ok && (r & 1) == 0) {
                    const float act = g.glu_kind == 0 ? glu_act<0>(v, up, 0.0f, 0.0f)
                                      : g.glu_kind == 1 ? glu_act<1>(v, up, 0.0f, 0.0f)
                                                        : glu_act<2>(v, up, g.glu_limit, g.glu_alpha);
                    const long long at = out_row * (g.n_out >> 1) + (row >> 1);
                    if (g.out_dtype == MLC_DTYPE_F32) ((float*)g.out)[at] = act;
                    else ((bf16*)g.out)[at] = __float2bfloat16_rn(act);
                }
            } else if (ok) {
                const long long at = out_row * g.n_out + row;
                if (g.out_dtype == MLC_DTYPE_F32) ((float*)g.out)[at] = v;
                else ((bf16*)g.out)[at] = __float2bfloat16_rn(v);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int NT, int UW, int RT, bool SILU>
static int launch_grouped(const GroupedFewArgs& g, int warps, int n_sms, cudaStream_t s) {
    const size_t smem = (size_t)warps * RT * UW * 2048 + sizeof(float) * warps * RT * 8 * NT * FEW_PITCH;
    if (smem > 227 * 1024) return MLC_ERR_BAD_SIZE;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_few_grouped_kernel<NT, UW, RT, SILU>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    static int resident[FEW_MAX_WARPS + 1] = {0};          // blocks an SM holds: one or two, by the ring's size
    if (resident[warps] == 0) {
        int n = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, gemm_few_grouped_kernel<NT, UW, RT, SILU>, 32 * warps, smem);
        if (e != cudaSuccess) return (int)e;
        resident[warps] = n < 1 ? 1 : n > 2 ? 2 : n;
    }
    const long long items = (long long)g.groups * ((g.tiles + RT - 1) / RT), most = (long long)n_sms * resident[warps];
    cudaError_t e = launch_pdl(gemm_few_grouped_kernel<NT, UW, RT, SILU>, dim3((unsigned)(items < most ? items : most)), dim3(32 * warps), smem, s, g);
    return e == cudaSuccess ? 0 : (int)e;
}

template <int NT, bool SILU>
static int launch_grouped_shape(const GroupedFewArgs& g, int warps, int uw, int n_sms, cudaStream_t s) {
    if (uw == 1) return launch_grouped<NT, 1, NT == 1 ? 3 : 2, SILU>(g, warps, n_sms, s);
    if (uw == 2) return launch_grouped<NT, 2, 2, SILU>(g, warps, n_sms, s);
    if (uw == 3) return launch_grouped<NT, 3, 1, SILU>(g, warps, n_sms, s);
    if (uw == 4) return launch_grouped<NT, 4, 1, SILU>(g, warps, n_sms, s);
    if (uw == 5) return launch_grouped<NT, 5, 1, SILU>(g, warps, n_sms, s);
    return MLC_ERR_BAD_SIZE;
}

}  // namespace mlc

using namespace mlc;

// The largest K the grouped few-row product takes: 16 warps of five units of 64.
constexpr int GROUPED_FEW_MAX_K = FEW_MAX_WARPS * 5 * FEW_UNIT;
extern "C" int mlc_gemm_few_grouped_max_k() { return GROUPED_FEW_MAX_K; }

// x: bfloat16 rows of K; w: bfloat16 [E][n_out][K]; tile_group: int [groups], the experts of the runs, then -1 (its values are
// not checked: moe_plan's); src_tok: null (x is [groups * group_rows][K]; then the kernel that made tile_group has to have
// ended before the kernel before this one began), or int [groups * group_rows].  out [groups * group_rows][n_out], with silu
// [..][n_out / 2] from rows of w that alternate gate, up; padding rows of a run get the product of a row of zeros (of whatever
// x holds there, without src_tok), rows of no run are not written.  groups <= 32, group_rows <= 16, K a multiple of 64, everything 16-byte aligned.
extern "C" int mlc_gemm_few_grouped(const void* x, const int* src_tok, const void* w, const int* tile_group, void* out, int out_dtype,
                                    int groups, int group_rows, int n_out, int K, int silu, int glu_kind, float glu_limit,
                                    float glu_alpha, int n_sms, void* stream) {
    if (groups <= 0 || n_out <= 0) return 0;
    if (groups > 32 || group_rows < 1 || group_rows > 16 || K < FEW_UNIT || K % FEW_UNIT || K > GROUPED_FEW_MAX_K || n_sms < 1 ||
        (((uintptr_t)x | (uintptr_t)w) & 15))
        return MLC_ERR_BAD_SIZE;
    if (out_dtype != MLC_DTYPE_F32 && out_dtype != MLC_DTYPE_BF16) return MLC_ERR_BAD_DTYPE;
    if (tile_group == nullptr || (silu && (n_out & 1))) return MLC_ERR_BAD_SIZE;
    if (glu_kind < 0 || glu_kind > 2 || (glu_kind == 2 && !(glu_limit > 0.0f))) return MLC_ERR_UNSUPPORTED;
    GroupedFewArgs g{(const bf16*)x, src_tok, (const bf16*)w, tile_group, out, out_dtype, groups, group_rows, n_out, K,
                     (n_out + FEW_ROWS - 1) / FEW_ROWS, glu_kind, glu_limit, glu_alpha};
    const int units = K / FEW_UNIT;
    int uw = (units + FEW_MAX_WARPS - 1) / FEW_MAX_WARPS;
    if (uw == 2 && group_rows <= 8 && units > 24) uw = 3;            // (that instance has 12 warps at most)
    const int warps = (units + uw - 1) / uw;
    cudaStream_t s = (cudaStream_t)stream;
    if (group_rows <= 8) return silu ? launch_grouped_shape<1, true>(g, warps, uw, n_sms, s) : launch_grouped_shape<1, false>(g, warps, uw, n_sms, s);
    return silu ? launch_grouped_shape<2, true>(g, warps, uw, n_sms, s) : launch_grouped_shape<2, false>(g, warps, uw, n_sms, s);
}
