// Warp and block primitives shared by the tree kernels: shuffles for every row type
// and the named barrier of a warp group.
#pragma once

#include <cuda_runtime.h>

#include "hwt_df64.cuh"

namespace hwt {

// Width-w warp shuffles for every row type (df64 moves as two floats).
template <typename T>
__device__ __forceinline__ T shfl_up(T v, unsigned d, int w) { return __shfl_up_sync(0xffffffffu, v, d, w); }
template <typename T>
__device__ __forceinline__ T shfl_down(T v, unsigned d, int w) { return __shfl_down_sync(0xffffffffu, v, d, w); }
__device__ __forceinline__ df64 shfl_up(df64 v, unsigned d, int w)
{
    return df64_make(__shfl_up_sync(0xffffffffu, v.hi, d, w), __shfl_up_sync(0xffffffffu, v.lo, d, w));
}
__device__ __forceinline__ df64 shfl_down(df64 v, unsigned d, int w)
{
    return df64_make(__shfl_down_sync(0xffffffffu, v.hi, d, w), __shfl_down_sync(0xffffffffu, v.lo, d, w));
}

template <typename T>
__device__ __forceinline__ T shfl_xor(T v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ df64 shfl_xor(df64 v, int m)
{
    return df64_make(__shfl_xor_sync(0xffffffffu, v.hi, m), __shfl_xor_sync(0xffffffffu, v.lo, m));
}

// Named barrier `id` over the `nthreads` threads of one tree's warp group (id 0
// with the whole block is __syncthreads).
__device__ __forceinline__ void tree_barrier(int id, int nthreads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Warps that price one tree together: `nthreads` threads from `base`, synchronised
// by named barrier `bar`.
struct Group {
    int base, nthreads, bar;
};

// A block's time since t_start, added to its SM's (one thread).  By SM, not by block: the
// general and the polynomial path's kernels share the SMs, one block of either at a time on
// each, and block i of one may follow block k of the other.
__device__ __forceinline__ void add_busy(unsigned long long *sm_busy, unsigned long long t_start)
{
    unsigned long long t_end;
    unsigned sm;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    atomicAdd(&sm_busy[sm % gridDim.x], t_end - t_start);
}

// The next warp task of a queue (all lanes).
__device__ __forceinline__ int draw_task(int32_t *counter)
{
    int t = 0;
    if ((threadIdx.x & 31) == 0) t = atomicAdd(counter, 1);
    return __shfl_sync(0xffffffffu, t, 0);
}

// A warp's first task of n.  Dealt queues (the counter starts past the dealt tasks): task i
// goes to warp i / grid of block i % grid, so that few tasks use every SM and the
// heaviest start on different SMs; drawn, the first blocks' 16 warps took them all
// (1,000 options: 32 of 152 SMs).  Queues behind group trees or beside the general path's
// kernel are drawn from the start (a block may start late, or still be busy), by no more
// warps of a block than give every block its share (480 options in double-float
// mode, two of them stepped through: 0.23 -> 0.15 ms).  n or more: no task.
__device__ __forceinline__ int first_task(int dealt, int n, int32_t *counter)
{
    const int warp = (int)(threadIdx.x >> 5), blocks = (int)gridDim.x;
    if (dealt) return warp * blocks + (int)blockIdx.x;
    return warp * blocks < n ? draw_task(counter) : n;
}

}  // namespace hwt
