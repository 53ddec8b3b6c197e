// Warp-level building blocks of the binarised-network layers: the 1-bit tensor-core MMA
// wrapper, fragment conventions and small bit helpers.  Everything here is warp-scoped (no
// block barriers), so the layer loops built on it run unchanged inside any grid: a plain
// launch of the library's own kernels, or a caller's persistent cooperative kernel.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace tcbnn {

// mma.sync m16n8k256 on 1-bit operands, AND + popcount, int32 accumulate.
// Fragment ownership (lane = 4*g + t):
//   a0: row g,   k-slice t of the first 128 bits     a1: row g+8, same slice
//   a2: row g,   k-slice t of the second 128 bits    a3: row g+8, same slice
//   b0: col g,   k-slice t of the first 128 bits     b1: col g,   second 128 bits
//   c0: (g, 2t)  c1: (g, 2t+1)  c2: (g+8, 2t)  c3: (g+8, 2t+1)
// A popcount does not care which physical word feeds which slice as long as both operands
// agree, so callers feed a0/a2 (and b0/b1) from one 64-bit load of two adjacent words.
__device__ __forceinline__ void mma_b1_and(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                           uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k256.row.col.s32.b1.b1.s32.and.popc "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint2 ldg64(const uint32_t* p) {
    return __ldg(reinterpret_cast<const uint2*>(p));
}
// A load of what an earlier launch wrote, in a kernel that may have been set up while that launch was
// still running (griddepcontrol): not through the read-only path, whose data has to stay the same for as
// long as the kernel lives -- a line of a buffer that is used again may be in L1 from before.
// (volatile keeps it behind the wait; without a memory clobber it may still be issued ahead of stores: as plain
// loads, ResNet-18 at batch 1024 1937 -> 2012 us.)
__device__ __forceinline__ uint32_t ld_dep(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_dep(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_dep(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_dep(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ int4 ld_dep(const int4* p) {
    int4 v;
    asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ int quad_sum(int v) {   // sum over the 4 lanes sharing g
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}
__device__ __forceinline__ uint32_t quad_or(uint32_t v) {
    v |= __shfl_xor_sync(0xffffffffu, v, 1);
    v |= __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}

// Global warp index / warp count of the running grid (1-D grid, 1-D block).
__device__ __forceinline__ int grid_warp() { return blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); }
__device__ __forceinline__ int grid_warps() { return gridDim.x * (blockDim.x >> 5); }

}  // namespace tcbnn
