// Pieces shared by the few-row products (gemm_few.cu, gemm_few_grouped.cu).
#pragma once

#include "common.cuh"

namespace mlc {

constexpr int FEW_UNIT = 64;              // elements of K: a 128-byte line of a row of W
constexpr int FEW_ROWS = 16;              // rows of W in a tile
constexpr int FEW_PITCH = 20;             // floats from one token's 16 partial sums to the next: the four stores of a warp hit 32 banks each
constexpr int FEW_MAX_WARPS = 16;

__device__ __forceinline__ void few_copy16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void few_prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ void few_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ unsigned few_pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&v);
}

template <int N> __device__ __forceinline__ void few_wait_copies() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

}  // namespace mlc
