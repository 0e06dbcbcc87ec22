// wd_reduce.cuh -- warp/block reduction helpers shared by the BLAS and
// solver kernels.  Partials are FP64; block size WD_RED_THREADS.
#pragma once
#include "wd_kernels.h"

__device__ __forceinline__ double wd_warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Block sums of N values; thread 0 holds them on return.  The threads' values
// go through shared memory to the first warp, which adds T / 32 of them per
// lane before its shuffles: T / 32 + 5 warp-wide FP64 additions per value
// instead of 5 in every warp, on a pipe that takes 16 cycles for each.
template <int T, int N>
__device__ __forceinline__ void wd_block_sum(const double (&v)[N], double (&total)[N])
{
    __shared__ double sw[N][T];
    __syncthreads();  // a previous call's readers are done
#pragma unroll
    for (int n = 0; n < N; ++n) sw[n][threadIdx.x] = v[n];
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
            double s = sw[n][threadIdx.x];
#pragma unroll
            for (int i = 1; i < T / 32; ++i) s += sw[n][threadIdx.x + 32 * i];
            total[n] = wd_warp_sum(s);
        }
    }
}

// Block-reduce (a, b) and write one partial per block.
__device__ __forceinline__ void wd_block_partial(double a, double b, double2 *partial)
{
    double t[2];
    wd_block_sum<WD_RED_THREADS, 2>({a, b}, t);
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(t[0], t[1]);
}
__device__ __forceinline__ void wd_block_partial(double a, double2 *partial)
{
    double t[1];
    wd_block_sum<WD_RED_THREADS, 1>({a}, t);
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(t[0], 0.0);
}

// Grid-wide sums of N values with no waiting: each block adds its threads' v
// and writes N partials; the block that finishes last in its group of
// kRedGroup (a one-shot atomic counter, which it resets to 0) folds the
// group's partials, and the one that finishes the last group folds the groups,
// both in a fixed order, so the totals do not depend on which blocks those
// are.  (One fold over all blocks left its T threads a chain of loads each:
// 0.05 ms for 41,472 blocks of 128 threads, 0.2 ms for 82,944 of 64.)
// Returns true in thread 0 of the last block, with the totals in total.  T =
// threads per block (a multiple of 32); every thread of the block must call
// it; the grid is one- or two-dimensional.
template <int T, int N>
__device__ __forceinline__ bool wd_grid_sum_n(const double (&v)[N], WdRed red, double (&total)[N])
{
    __shared__ int last;
    const int blocks = gridDim.x * gridDim.y, block = blockIdx.y * gridDim.x + blockIdx.x;
    const int groups = (blocks + kRedGroup - 1) / kRedGroup, group = block / kRedGroup;
    double t[N];
    wd_block_sum<T, N>(v, t);
    // level 0: this block into its group; level 1: its group into the total
    double *out = red.partial;
    int slot = block, first = group * kRedGroup;
    int count = min(kRedGroup, blocks - first);
    unsigned *counter = red.counters + 1 + group;
#pragma unroll 1
    for (int level = 0; level < 2; ++level) {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int n = 0; n < N; ++n) out[(size_t)slot * N + n] = t[n];
            __threadfence();
            last = atomicAdd(counter, 1u) == (unsigned)count - 1;
            if (last) *counter = 0;
        }
        __syncthreads();
        if (!last) return false;
        __threadfence();
#pragma unroll
        for (int n = 0; n < N; ++n) t[n] = 0.0;
#pragma unroll 4
        for (int i = threadIdx.x; i < count; i += T)
#pragma unroll
            for (int n = 0; n < N; ++n) t[n] += __ldcg(out + (size_t)(first + i) * N + n);
        wd_block_sum<T, N>(t, total);
        if (groups == 1) break;
#pragma unroll
        for (int n = 0; n < N; ++n) t[n] = total[n];
        out = red.partial + (size_t)blocks * N;
        slot = group, first = 0, count = groups;
        counter = red.counters;
    }
    return threadIdx.x == 0;
}

template <int T>
__device__ __forceinline__ bool wd_grid_sum(double v, WdRed red, double *total)
{
    double t[1];
    if (!wd_grid_sum_n<T, 1>({v}, red, t)) return false;
    *total = t[0];
    return true;
}
