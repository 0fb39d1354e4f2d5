// y[M][N] = x[M][K] · W[N][K]ᵀ with float32 multiply-adds on the CUDA cores: the linear
// layer of the whole-model 32-bit path, and the fallback for operand types the
// tensor-core kernels do not take.  No tensor-core mode of any precision is involved.
//
// The reference's linear is y = W·x for one row x, W row-major [out, in]
// (src/matmul_optimized.cpp:40-54, 210-224); its CUDA path calls cublasSgemm with one
// row (src/cuda_matmul.cpp:216-233).  Here any number of rows runs at once.
//
// One order of summation for every shape.  K is cut into chunks of 256; inside a chunk the
// terms are added in ascending k into one accumulator that starts at zero (fused
// multiply-adds); the chunks' sums are then added in ascending order into a total that
// starts at zero.  Every kernel below produces exactly this sum for every output element,
// so a token's result does not depend, bit for bit, on how many other tokens ran with it
// or on which kernel took the step.
//
// Three shapes of work:
//   many rows (prompts)   tiles of 128 x 128 or 64 x 64 outputs, 8 x 8 or 4 x 4 per thread; operands come in
//                         16-byte loads into registers one K step ahead and go through a
//                         double-buffered shared-memory tile;
//   few rows (decoding)   of a float32 matrix whose rows are 16-byte aligned: a stream of weights with almost no
//                         arithmetic, `linear_few_kernel` below;
//   few rows, other types or alignments   tiles of 16 rows x 64 columns.
// Where the tiles alone would leave SMs idle, each block of the tiled kernel takes one chunk of K for its tile and
// leaves the chunk's sums in scratch memory, and a second kernel adds the chunks in order.
// 256 rows of x, B200, in brackets 128 x 128 tiles without chunks: 9,728 x 896 149 us (266), 896 x 4,864 84 us (715).
// The tiled kernels start in the ordinary way.  Blocks that were launched while the kernel before ran came to lie several on the SMs
// that were free first: 64 x 64 tiles of 700 x 1,536 x 8,960 1,356 us so and 815 in the ordinary way, 16 x 64 tiles of 1 x
// 9,728 x 898 53 and 30.
#include "tcgen05.cuh"      // mbarriers with bounded waits, TMA tile loads, tensor maps, shared-memory addresses of a cluster's blocks

namespace mlc {

constexpr int LS_BK = 16;
constexpr int LS_CHUNK = 256;          // a multiple of LS_BK

// Four consecutive elements of a row as floats; `vec` says that 4-element groups of every row are aligned for one load.
template <typename T>
__device__ __forceinline__ float4 load4(const T* __restrict__ base, long long row, int K, int k, bool row_ok, bool vec);

template <>
__device__ __forceinline__ float4 load4<float>(const float* __restrict__ base, long long row, int K, int k, bool row_ok, bool vec) {
    if (!row_ok || k >= K) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float* p = base + row * K + k;
    if (vec && k + 3 < K) return __ldg(reinterpret_cast<const float4*>(p));
    float4 v = make_float4(p[0], 0.0f, 0.0f, 0.0f);
    if (k + 1 < K) v.y = p[1];
    if (k + 2 < K) v.z = p[2];
    if (k + 3 < K) v.w = p[3];
    return v;
}

template <>
__device__ __forceinline__ float4 load4<bf16>(const bf16* __restrict__ base, long long row, int K, int k, bool row_ok, bool vec) {
    if (!row_ok || k >= K) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const bf16* p = base + row * K + k;
    if (vec && k + 3 < K) {
        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(p));
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
        return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
    }
    float4 v = make_float4(__bfloat162float(p[0]), 0.0f, 0.0f, 0.0f);
    if (k + 1 < K) v.y = __bfloat162float(p[1]);
    if (k + 2 < K) v.z = __bfloat162float(p[2]);
    if (k + 3 < K) v.w = __bfloat162float(p[3]);
    return v;
}

template <typename T> __device__ __forceinline__ bool rows_vectorizable(const T* base, int K) {
    return (K & 3) == 0 && (reinterpret_cast<uintptr_t>(base) & (4 * sizeof(T) - 1)) == 0;
}

// A tile of BM x BN outputs, TM x TN per thread, over the K range [k_begin, k_end) (whole chunks, but for the matrix's
// end).  `total` starts at zero and gets each chunk's sum in turn.  PARTIAL: the range is one chunk and its sum goes to
// part[chunk][M][N] instead of y.
template <typename TX, typename TW, typename TY, int BM, int BN, int TM, int TN, bool PARTIAL>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
linear_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TY* __restrict__ y, float* __restrict__ part,
                   int M, int N, int K) {
    constexpr int THREADS = (BM / TM) * (BN / TN);
    constexpr int XV = (BM * (LS_BK / 4) + THREADS - 1) / THREADS;       // 16-byte loads per thread and K step
    constexpr int WV = (BN * (LS_BK / 4) + THREADS - 1) / THREADS;
    __shared__ __align__(16) float xs[2][LS_BK][BM + 4];
    __shared__ __align__(16) float ws[2][LS_BK][BN + 4];
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int k_begin = PARTIAL ? blockIdx.z * LS_CHUNK : 0;
    const int k_end = PARTIAL ? min(K, k_begin + LS_CHUNK) : K;
    const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
    // a thread's rows and columns in groups of up to four side by side, the groups spread over the tile: neighbouring
    // threads' 16-byte reads of a group are neighbours in shared memory and hit all banks once
    constexpr int GM = TM < 4 ? TM : 4, GN = TN < 4 ? TN : 4;
    auto row_of = [&](int i) { return (i / GM) * (BM / (TM / GM)) + ty * GM + i % GM; };
    auto col_of = [&](int j) { return (j / GN) * (BN / (TN / GN)) + tx * GN + j % GN; };
    const bool x_vec = rows_vectorizable(x, K), w_vec = rows_vectorizable(w, K);

    // the totals of the 64 x 64 tile of 8 x 8 per thread lie in shared memory, a column per thread: its blocks are small, and
    // what hides their loads is how many of them an SM's registers hold
    constexpr bool PARKED = !PARTIAL && BM == 64 && TM == 8;
    __shared__ float parked[PARKED ? TM * TN : 1][PARKED ? THREADS : 1];
    float total[PARKED ? 1 : TM][PARKED ? 1 : TN], acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            acc[i][j] = 0.0f;
            if constexpr (PARKED) parked[i * TN + j][threadIdx.x] = 0.0f;
            else total[i][j] = 0.0f;
        }

    float4 xr[XV], wr[WV];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int v = 0; v < XV; ++v) {
            const int idx = threadIdx.x + v * THREADS, row = idx / (LS_BK / 4), kq = (idx % (LS_BK / 4)) * 4;
            xr[v] = load4<TX>(x, m0 + row, K, k0 + kq, idx < BM * (LS_BK / 4) && m0 + row < M && k0 + kq < k_end, x_vec);
        }
#pragma unroll
        for (int v = 0; v < WV; ++v) {
            const int idx = threadIdx.x + v * THREADS, row = idx / (LS_BK / 4), kq = (idx % (LS_BK / 4)) * 4;
            wr[v] = load4<TW>(w, n0 + row, K, k0 + kq, idx < BN * (LS_BK / 4) && n0 + row < N && k0 + kq < k_end, w_vec);
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int v = 0; v < XV; ++v) {
            const int idx = threadIdx.x + v * THREADS, row = idx / (LS_BK / 4), kq = (idx % (LS_BK / 4)) * 4;
            if (idx < BM * (LS_BK / 4)) {
                xs[buf][kq][row] = xr[v].x; xs[buf][kq + 1][row] = xr[v].y; xs[buf][kq + 2][row] = xr[v].z; xs[buf][kq + 3][row] = xr[v].w;
            }
        }
#pragma unroll
        for (int v = 0; v < WV; ++v) {
            const int idx = threadIdx.x + v * THREADS, row = idx / (LS_BK / 4), kq = (idx % (LS_BK / 4)) * 4;
            if (idx < BN * (LS_BK / 4)) {
                ws[buf][kq][row] = wr[v].x; ws[buf][kq + 1][row] = wr[v].y; ws[buf][kq + 2][row] = wr[v].z; ws[buf][kq + 3][row] = wr[v].w;
            }
        }
    };

    fetch(k_begin);
    stash(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += LS_BK) {
        const bool more = k0 + LS_BK < k_end;
        if (more) fetch(k0 + LS_BK);                         // the next step's operands travel while this one is multiplied
        const int steps = min(LS_BK, k_end - k0);            // no term beyond K is ever added
#pragma unroll 4
        for (int kk = 0; kk < steps; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = xs[buf][kk][row_of(i)];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = ws[buf][kk][col_of(j)];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (!PARTIAL && ((k0 + LS_BK) % LS_CHUNK == 0 || !more)) {       // a chunk is complete
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    if constexpr (PARKED) parked[i * TN + j][threadIdx.x] += acc[i][j];
                    else total[i][j] += acc[i][j];
                    acc[i][j] = 0.0f;
                }
        }
        if (more) {
            stash(buf ^ 1);
            __syncthreads();
            buf ^= 1;
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + row_of(i);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + col_of(j);
            if (n >= N) continue;
            if constexpr (PARTIAL) part[((long long)blockIdx.z * M + m) * N + n] = acc[i][j];
            else if constexpr (PARKED) y[(long long)m * N + n] = from_float<TY>(parked[i * TN + j][threadIdx.x]);
            else y[(long long)m * N + n] = from_float<TY>(total[i][j]);
        }
    }
}

// y = the chunks' sums added in ascending order into a total that starts at zero.
template <typename TY>
__global__ void linear_simt_add_chunks_kernel(const float* __restrict__ part, TY* __restrict__ y, long long MN, int n_chunks) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= MN) return;
    float total = 0.0f;
#pragma unroll 8
    for (int c = 0; c < n_chunks; ++c) total += part[(long long)c * MN + i];
    y[i] = from_float<TY>(total);
}

// ------------------------------------------------------------------ up to 16 rows of x, float32 operands, aligned rows
// The order of summation wants one thread to walk a chunk of K, 256 multiply-adds that wait for one another, so the chunks go
// to different warps: a warp takes 32 rows of W, one per lane, TOKENS rows of x and one chunk (or `pw` of them one after the
// other), and the chunks' sums meet in shared memory, where they are added in ascending order; beyond eight warps' worth of
// chunks the blocks of a cluster share them out and read one another's sums.  Neither a scratch array nor a second kernel is
// needed.
// Weights and tokens come by TMA into a ring of a warp's own, in boxes of 32 floats a row (seen as 64 16-bit elements, the
// width of the other kernels' boxes) whose 16-byte pieces are swapped by the row's number modulo 8: a warp's reads, one row
// per lane, hit all banks; the tokens' reads are broadcasts.  Warps do not wait for one another before the end of a tile,
// and the ring runs on from tile to tile.
// What bounds it: memory for large matrices; for small ones the launch, the first trip to memory and a chunk's chain (1,024
// cycles at least); from nine rows on the tokens' reads.  B200, one kernel of a chain in a graph, 3 rows, in brackets tiles of
// 16 x 64 with the chunks' sums in scratch memory and a second kernel: 1,152 x 896 5.4 us, 896 x 896 5.4, 896 x 4,864 8.5,
// 9,728 x 896 8.2 (17 and 2 for the second kernel on the average of the four), 151,936 x 896 84 us = 6.5 TB/s (257).  With a ring of four
// stages an SM holds one block instead of two: 9,728 x 896 12.1 us, 151,936 x 896 95.
constexpr int LF_BOX = 32;              // elements of K in a stage
constexpr int LF_ROW_BYTES = 128;
constexpr int LF_ROWS = 32;
constexpr int LF_SLOTS = 3;
constexpr int LF_MAX_WARPS = 8;
constexpr int LF_MAX_CLUSTER = 8;
constexpr int LF_MAX_PW = 4;

__host__ __device__ constexpr int lf_slot_bytes(int tokens) { return LF_ROWS * LF_ROW_BYTES + (tokens + 7) / 8 * 1024; }      // boxes begin on 1024-byte boundaries

__device__ __forceinline__ float load_cluster_float(unsigned cluster_addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
    return v;
}

template <typename TY, int TOKENS>
__global__ void __launch_bounds__(32 * LF_MAX_WARPS)
linear_few_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, TY* __restrict__ y, int M, int N,
                  int K, int n_chunks, int pw, int cluster, int tiles, int* status) {
    constexpr int SLOT_BYTES = lf_slot_bytes(TOKENS), W_BYTES = LF_ROWS * LF_ROW_BYTES;
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    extern __shared__ unsigned char lf_smem[];
    unsigned char* const smem = lf_smem + ((1024u - (smem_u32(lf_smem) & 1023u)) & 1023u);
    unsigned char* const ring = smem + warp * LF_SLOTS * SLOT_BYTES;                                // [SLOTS][W box, x box]
    float* const sums = reinterpret_cast<float*>(smem + warps * LF_SLOTS * SLOT_BYTES);             // [2][warps * pw][TOKENS][LF_ROWS]
    __shared__ __align__(8) unsigned long long full_bars[LF_MAX_WARPS * LF_SLOTS];
    const unsigned ring_at = smem_u32(ring), bars = smem_u32(full_bars) + 8u * (unsigned)(warp * LF_SLOTS);
    const int rank = cluster > 1 ? (int)cluster_rank() : 0;
    const int first_tile = blockIdx.x / cluster, tile_step = gridDim.x / cluster;
    const int chunk0 = (rank * warps + warp) * pw, chunk1 = min(n_chunks, chunk0 + pw);
    const int k_begin = chunk0 * LS_CHUNK, k_end = min(K, chunk1 * LS_CHUNK);
    const int stages = k_end > k_begin ? (k_end - k_begin + LF_BOX - 1) / LF_BOX : 0;               // of one tile
    const int my_tiles = first_tile < tiles ? (tiles - first_tile + tile_step - 1) / tile_step : 0;
    const int total_stages = my_tiles * stages;

    grid_launch_dependents();
    int ask_tile = first_tile, ask_stage = 0;
    auto ask = [&](int slot, bool weights, bool tokens) {
        const int c = 2 * (k_begin + ask_stage * LF_BOX);
        const unsigned at = ring_at + (unsigned)(slot * SLOT_BYTES), bar = bars + 8u * (unsigned)slot;
        if (weights) {
            mbar_expect_tx(bar, W_BYTES + TOKENS * LF_ROW_BYTES);
            tma_load_2d(at, &map_w, c, ask_tile * LF_ROWS, bar);
        }
        if (tokens) tma_load_2d(at + W_BYTES, &map_x, c, 0, bar);
    };
    auto next = [&]() {
        if (++ask_stage == stages) {
            ask_stage = 0;
            ask_tile += tile_step;
        }
    };
    const int early = min(LF_SLOTS, total_stages);
    if (lane == 0) {
        for (int s = 0; s < LF_SLOTS; ++s) mbar_init(bars + 8u * s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int s = 0; s < early; ++s, next()) ask(s, true, false);          // the weights depend on nothing
    }
    __syncwarp();
    grid_dependency_wait();
    if (lane == 0) {
        ask_tile = first_tile;
        ask_stage = 0;
        for (int s = 0; s < early; ++s, next()) ask(s, false, true);
    }

    int slot = 0, round = 0, done = 0, asked = early, parity = 0;     // stages used and asked for, of all tiles
    bool ok = true;
    for (int tile = first_tile; tile < tiles; tile += tile_step, parity ^= 1) {
        float* const mine = sums + ((parity * warps + warp) * pw) * TOKENS * LF_ROWS;
        float acc[TOKENS];
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) acc[t] = 0.0f;
        for (int s = 0; s < stages && ok; ++s) {
            ok = __all_sync(0xffffffffu, mbar_wait(bars + 8u * (unsigned)slot, (unsigned)round & 1u, status, 61));
            if (!ok) break;
            const unsigned char* const wr = ring + slot * SLOT_BYTES + lane * LF_ROW_BYTES;
            const unsigned char* const xr = ring + slot * SLOT_BYTES + W_BYTES;
            float4 wv[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) wv[q] = *reinterpret_cast<const float4*>(wr + ((q ^ (lane & 7)) << 4));
            // what lies beyond K has arrived as zeros, which change no sum
#pragma unroll
            for (int q = 0; q < 8; ++q) {
#pragma unroll
                for (int g = 0; g < TOKENS; g += 4) {
                    float4 xv[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) xv[t] = *reinterpret_cast<const float4*>(xr + (g + t) * LF_ROW_BYTES + ((q ^ ((g + t) & 7)) << 4));
                    // token after token, not term after term: the multiply-adds of one sum wait for one another
#pragma unroll
                    for (int t = 0; t < 4; ++t) acc[g + t] = fmaf(xv[t].x, wv[q].x, acc[g + t]);
#pragma unroll
                    for (int t = 0; t < 4; ++t) acc[g + t] = fmaf(xv[t].y, wv[q].y, acc[g + t]);
#pragma unroll
                    for (int t = 0; t < 4; ++t) acc[g + t] = fmaf(xv[t].z, wv[q].z, acc[g + t]);
#pragma unroll
                    for (int t = 0; t < 4; ++t) acc[g + t] = fmaf(xv[t].w, wv[q].w, acc[g + t]);
                }
            }
            if ((s + 1) % (LS_CHUNK / LF_BOX) == 0 || s + 1 == stages) {       // a chunk is complete
#pragma unroll
                for (int t = 0; t < TOKENS; ++t) {
                    mine[((s / (LS_CHUNK / LF_BOX)) * TOKENS + t) * LF_ROWS + lane] = acc[t];
                    acc[t] = 0.0f;
                }
            }
            __syncwarp();                                            // the slot has been read
            if (lane == 0 && done + LF_SLOTS < total_stages) {
                ask(slot, true, true);
                next();
                ++asked;
            }
            ++done;
            if (++slot == LF_SLOTS) {
                slot = 0;
                ++round;
            }
        }
        // the other set of sums takes the next tile's, so one barrier a tile is enough
        const bool all_ok = __syncthreads_and(ok);
        if (cluster == 1 && all_ok) {
            for (int o = threadIdx.x; o < TOKENS * LF_ROWS; o += blockDim.x) {
                const int n = tile * LF_ROWS + o % LF_ROWS, m = o / LF_ROWS;
                if (m >= M || n >= N) continue;
                const float* const at = sums + parity * warps * pw * TOKENS * LF_ROWS + o;
                float total = 0.0f;
#pragma unroll 8
                for (int c = 0; c < n_chunks; ++c) total += at[c * TOKENS * LF_ROWS];
                y[(long long)m * N + n] = from_float<TY>(total);
            }
        }
        ok = all_ok;
    }
    // A wait ran out: nobody leaves while a copy into its shared memory may still be under way (bounded waits again).
    if (!ok && lane == 0) {
        for (; done < asked; ++done) {
            mbar_wait(bars + 8u * (unsigned)slot, (unsigned)round & 1u, status, 61);
            if (++slot == LF_SLOTS) {
                slot = 0;
                ++round;
            }
        }
    }
    if (cluster > 1) {                                               // one tile per cluster; its blocks share out the outputs
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const unsigned sums_at = smem_u32(sums);
        const int per = warps * pw;
        for (int o = rank * blockDim.x + threadIdx.x; o < TOKENS * LF_ROWS; o += cluster * blockDim.x) {
            const int n = first_tile * LF_ROWS + o % LF_ROWS, m = o / LF_ROWS;
            if (m >= M || n >= N || !ok) continue;
            float total = 0.0f;
#pragma unroll 8
            for (int c = 0; c < n_chunks; ++c) {
                const int r = c / per;
                total += load_cluster_float(cluster_map(sums_at + (unsigned)((c - r * per) * TOKENS * LF_ROWS + o) * 4u, r));
            }
            y[(long long)m * N + n] = from_float<TY>(total);
        }
        // nobody leaves while another block may still read its sums
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// K's chunks over the warps of a block, the blocks of a cluster and, only beyond those, a warp's time.
struct FewPlan { int warps, cluster, pw; };
static FewPlan few_plan(int K) {
    const int n_chunks = (K + LS_CHUNK - 1) / LS_CHUNK;
    const int pw = (n_chunks + LF_MAX_WARPS * LF_MAX_CLUSTER - 1) / (LF_MAX_WARPS * LF_MAX_CLUSTER), shares = (n_chunks + pw - 1) / pw;
    const int cluster = (shares + LF_MAX_WARPS - 1) / LF_MAX_WARPS;
    return FewPlan{(shares + cluster - 1) / cluster, cluster, pw};
}

template <typename TY, int TOKENS>
static int launch_few(const float* x, const float* w, TY* y, int M, int N, int K, int* status, int n_sms, cudaStream_t s) {
    const int tiles = (N + LF_ROWS - 1) / LF_ROWS, n_chunks = (K + LS_CHUNK - 1) / LS_CHUNK;
    const FewPlan p = few_plan(K);
    static_assert((size_t)LF_MAX_WARPS * (LF_SLOTS * lf_slot_bytes(TOKENS) + 2 * (TOKENS > 8 ? 1 : LF_MAX_PW) * TOKENS * LF_ROWS * sizeof(float)) + 2048 <= 227 * 1024, "shared memory of a block");
    const size_t smem = (size_t)p.warps * (LF_SLOTS * lf_slot_bytes(TOKENS) + 2 * p.pw * TOKENS * LF_ROWS * sizeof(float)) + 1024 /* alignment slack */;
    if (smem + 1024 > 227 * 1024) return MLC_ERR_BAD_SIZE;           // (takes_few has seen to it)
    CUtensorMap mx, mw;
    int rc = cached_map_2d(&mx, x, M, 2LL * K, 64, TOKENS);
    if (rc) return rc;
    rc = cached_map_2d(&mw, w, N, 2LL * K, 64, LF_ROWS);
    if (rc) return rc;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(linear_few_kernel<TY, TOKENS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const long long resident = (long long)n_sms * (long long)(227 * 1024 / (smem + 1024));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.cluster > 1 ? (long long)tiles * p.cluster : tiles < resident ? tiles : resident));
    cfg.blockDim = dim3(32 * p.warps);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.cluster > 1 ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, linear_few_kernel<TY, TOKENS>, mx, mw, y, M, N, K, n_chunks, p.pw, p.cluster, tiles, status);
    return e == cudaSuccess ? 0 : (int)e;
}

// Whether the product takes the kernel above.
static bool takes_few(int x_dtype, int w_dtype, const void* x, const void* w, int M, int K) {
    return x_dtype == MLC_DTYPE_F32 && w_dtype == MLC_DTYPE_F32 && M <= 16 && (K & 3) == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 &&
           few_plan(K).pw <= (M > 8 ? 1 : LF_MAX_PW);
}

template <typename TY>
static int launch_few_rows(const float* x, const float* w, TY* y, int M, int N, int K, int* status, int n_sms, cudaStream_t s) {
    if (M <= 4) return launch_few<TY, 4>(x, w, y, M, N, K, status, n_sms, s);
    if (M <= 8) return launch_few<TY, 8>(x, w, y, M, N, K, status, n_sms, s);
    return launch_few<TY, 16>(x, w, y, M, N, K, status, n_sms, s);
}

// The form of a product of more than 16 rows.  Lone blocks take 37 us a chunk of K with 128 x 128 tiles, 22 with 64 x 64 tiles of
// 8 x 8 per thread and 13 with 64 x 64 tiles of 4 x 4 (four warps a scheduler instead of one half), B200; a GPU full of
// them 31, 37 and 31 TFLOP/s.  So
//   TILES_128    more than 64 rows (64 rows of a 128-row tile are work for nothing: 64 x 151,936 x 896 1,170 us, 64 x 64 tiles
//                527) where such tiles fill the GPU four times over;
//   TILES_4X4    one or two chunks of K and at most three tiles an SM, where a lone block's time is what counts (64 x 500 x 300
//                18 us, 8 x 8 per thread 28, in chunks 31; 700 x 2,000 x 128 17, 21);
//   CHUNKS       single chunks of K a block and a second kernel that adds them, where whole tiles would fill less than 78 % of
//                their waves of six an SM (9,728 columns of K = 896, whole and in chunks: 256 rows, 608 tiles 160, 149 us; 300 rows,
//                760 tiles 169, 176; 400 rows, 1,064 tiles 294, 238; 700 rows, 1,672 tiles 333, 383);
//   TILES        whole tiles otherwise.
enum TileForm { TILES_128, TILES, TILES_4X4, CHUNKS };
struct TilePlan { TileForm form; long long scratch; };
constexpr long long LS_MAX_SCRATCH = 32LL << 20;          // floats: 128 MB
static TilePlan tile_plan(int M, int N, int K, int n_sms) {
    const long long t128 = (long long)((M + 127) / 128) * ((N + 127) / 128), t64 = (long long)((M + 63) / 64) * ((N + 63) / 64);
    const int n_chunks = (K + LS_CHUNK - 1) / LS_CHUNK;
    if ((M > 64 && t128 >= 4LL * n_sms) || (M + 63) / 64 > 65535) return TilePlan{TILES_128, 0};
    if (n_chunks <= 2 && t64 <= 3LL * n_sms) return TilePlan{TILES_4X4, 0};
    const long long need = (long long)n_chunks * M * N, slots = 6LL * n_sms, waves = (t64 + slots - 1) / slots;
    if (n_chunks > 1 && n_chunks <= 65535 && 100 * t64 < 78 * waves * slots && need <= LS_MAX_SCRATCH) return TilePlan{CHUNKS, need};
    return TilePlan{TILES, 0};
}

template <typename TX, typename TW, typename TY>
static int launch_linear(const void* x, const void* w, void* y, float* scratch, long long scratch_floats, int M, int N, int K,
                         int* status, int n_sms, cudaStream_t s) {
    const TX* xp = (const TX*)x;
    const TW* wp = (const TW*)w;
    TY* yp = (TY*)y;
    const int n_chunks = (K + LS_CHUNK - 1) / LS_CHUNK;
    const long long MN = (long long)M * N;
    bool chunks = false;
    if (M > 16) {
        const TilePlan p = tile_plan(M, N, K, n_sms);
        chunks = p.form == CHUNKS && scratch != nullptr && scratch_floats >= p.scratch;
        const dim3 g64((N + 63) / 64, (M + 63) / 64, chunks ? n_chunks : 1);
        if (p.form == TILES_128) {
            dim3 grid((N + 127) / 128, (M + 127) / 128);
            if (grid.y > 65535) return MLC_ERR_BAD_SIZE;
            linear_simt_kernel<TX, TW, TY, 128, 128, 8, 8, false><<<grid, 256, 0, s>>>(xp, wp, yp, nullptr, M, N, K);
        } else if (chunks) {
            linear_simt_kernel<TX, TW, TY, 64, 64, 8, 8, true><<<g64, 64, 0, s>>>(xp, wp, yp, scratch, M, N, K);
        } else if (p.form == TILES_4X4) {
            linear_simt_kernel<TX, TW, TY, 64, 64, 4, 4, false><<<g64, 256, 0, s>>>(xp, wp, yp, nullptr, M, N, K);
        } else {
            linear_simt_kernel<TX, TW, TY, 64, 64, 8, 8, false><<<g64, 64, 0, s>>>(xp, wp, yp, nullptr, M, N, K);
        }
    } else {
        if constexpr (sizeof(TX) == 4 && sizeof(TW) == 4) {
            if (takes_few(MLC_DTYPE_F32, MLC_DTYPE_F32, x, w, M, K)) return launch_few_rows<TY>(xp, wp, yp, M, N, K, status, n_sms, s);
        }
        const int tiles = (N + 63) / 64;
        // few tiles: a block per (tile, chunk) and a second kernel that adds the chunks, if the caller gave room for them
        chunks = tiles < 4 * n_sms && n_chunks > 1 && n_chunks <= 65535 && scratch != nullptr && scratch_floats >= n_chunks * MN;
        if (chunks) {
            dim3 grid(tiles, 1, n_chunks);
            linear_simt_kernel<TX, TW, TY, 16, 64, 2, 4, true><<<grid, 128, 0, s>>>(xp, wp, yp, scratch, M, N, K);
        } else {
            dim3 grid(tiles, 1);
            linear_simt_kernel<TX, TW, TY, 16, 64, 2, 4, false><<<grid, 128, 0, s>>>(xp, wp, yp, nullptr, M, N, K);
        }
    }
    MLC_LAUNCH_CHECK();
    if (chunks) {
        linear_simt_add_chunks_kernel<TY><<<(unsigned)((MN + 255) / 256), 256, 0, s>>>(scratch, yp, MN, n_chunks);
        MLC_LAUNCH_CHECK();
    }
    return 0;
}

}  // namespace mlc

using namespace mlc;

// Floats of scratch memory a product of these sizes can use (0: none): room for each K chunk's sums when the tiles alone
// are few.  Without it the product still runs, with fewer blocks.
extern "C" long long mlc_linear_simt_scratch_floats(const void* x, int x_dtype, const void* w, int w_dtype, int M, int N, int K, int n_sms) {
    if (M <= 0 || N <= 0 || K <= LS_CHUNK || n_sms < 1) return 0;
    if (M > 16) return tile_plan(M, N, K, n_sms).scratch;
    if (takes_few(x_dtype, w_dtype, x, w, M, K) || (N + 63) / 64 >= 4 * n_sms) return 0;
    return (long long)((K + LS_CHUNK - 1) / LS_CHUNK) * M * N;
}

// x [M][K] of x_dtype, w [N][K] of w_dtype, y [M][N] of y_dtype; all row-major and dense.  scratch: null, or
// `scratch_floats` floats of device memory (see mlc_linear_simt_scratch_floats).  status: one int on the device, 0 before the
// call; a bounded wait that ran out leaves 61 there.
extern "C" int mlc_linear_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* y, int y_dtype,
                               int M, int N, int K, float* scratch, long long scratch_floats, int* status, int n_sms, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || n_sms < 1 || status == nullptr) return MLC_ERR_BAD_SIZE;
    if ((x_dtype | w_dtype | y_dtype) & ~1) return MLC_ERR_BAD_DTYPE;
    cudaStream_t s = (cudaStream_t)stream;
    const int code = x_dtype * 4 + w_dtype * 2 + y_dtype;
    switch (code) {
        case 0: return launch_linear<float, float, float>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
        case 1: return launch_linear<float, float, bf16>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
        case 2: return launch_linear<float, bf16, float>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
        case 3: return launch_linear<float, bf16, bf16>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
        case 4: return launch_linear<bf16, float, float>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
        case 5: return launch_linear<bf16, float, bf16>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
        case 6: return launch_linear<bf16, bf16, float>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
        case 7: return launch_linear<bf16, bf16, bf16>(x, w, y, scratch, scratch_floats, M, N, K, status, n_sms, s);
    }
    return MLC_ERR_BAD_DTYPE;
}
