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
// and writes N partials; the block that finishes last (a one-shot atomic
// counter, which it resets to 0) folds the partials in a fixed order, so the
// totals do not depend on which block that is.  Returns true in thread 0 of
// that block, with the totals in total.  T = threads per block (a multiple of
// 32); every thread of the block must call it; partial holds N doubles per
// block of the (one- or two-dimensional) grid.
template <int T, int N>
__device__ __forceinline__ bool wd_grid_sum_n(const double (&v)[N], double *partial, unsigned *counter,
                                              double (&total)[N])
{
    __shared__ int last;
    const int blocks = gridDim.x * gridDim.y, block = blockIdx.y * gridDim.x + blockIdx.x;
    double t[N];
    wd_block_sum<T, N>(v, t);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int n = 0; n < N; ++n) partial[(size_t)block * N + n] = t[n];
        __threadfence();
        last = atomicAdd(counter, 1u) == (unsigned)blocks - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
#pragma unroll
    for (int n = 0; n < N; ++n) t[n] = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < blocks; i += T)
#pragma unroll
        for (int n = 0; n < N; ++n) t[n] += __ldcg(partial + (size_t)i * N + n);
    wd_block_sum<T, N>(t, total);
    if (threadIdx.x != 0) return false;
    *counter = 0;
    return true;
}

template <int T>
__device__ __forceinline__ bool wd_grid_sum(double v, double *partial, unsigned *counter, double *total)
{
    double t[1];
    if (!wd_grid_sum_n<T, 1>({v}, partial, counter, t)) return false;
    *total = t[0];
    return true;
}
