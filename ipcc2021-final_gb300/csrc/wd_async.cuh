// wd_async.cuh -- per-thread asynchronous copies global -> shared memory
// (cp.async, LDGSTS) for kernels that stage the next direction's operands
// while they compute the current one.  Each copy moves one 4-, 8- or 16-byte
// element; both addresses must be aligned to its size.  A thread's copies
// become visible to that thread after cp.async.wait_group retires their
// group; other threads also need a barrier after that wait.  The FP16 and
// double-float hops read back only their own copies.  The fixed-point hop
// shares a site's link between the two threads of a pair: there the
// __syncwarp after the wait makes the partner's copies visible, and keeps a
// slot from being overwritten while the partner still reads it.
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ unsigned wd_smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// L1-allocating copy of BYTES = 4, 8 or 16
template <int BYTES>
__device__ __forceinline__ void wd_cp_async_ca(void *smem, const void *gmem)
{
    static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async copies 4, 8 or 16 bytes");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(wd_smem_addr(smem)), "l"(gmem), "n"(BYTES)
                 : "memory");
}
// L2-only copy of 16 bytes (data read once)
__device__ __forceinline__ void wd_cp_async_cg16(void *smem, const void *gmem)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(wd_smem_addr(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void wd_cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// wait until at most N of this thread's committed groups are still pending
template <int N>
__device__ __forceinline__ void wd_cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Programmatic dependent launch: a kernel launched with wd_launch_pdl may start
// while its predecessor in the stream finishes.  It calls wd_pdl_wait before it
// touches memory (a no-op under an ordinary launch), which returns once the
// predecessor has completed, and from that point lets its own successor start
// the same way (pdl = false: an ordinary launch).  Its operands are neither
// marked const __restrict__ nor read with __ldg: both promise data that is
// constant over the kernel's life, which begins before the predecessor has
// written them (without them: FP32 and FP16 solves 0.2-1.3 % slower).  ahead: the successor may
// start before the wait already.  That piles up kernels ahead of the running
// one, which spread unevenly over the SMs where a grid does not fill them (a
// fixed-point hop at 8^4: 6.5 us instead of 4.9), but is the better order for
// the FP64 solver's full grids (CG at 16^3x32: 7.07 ms instead of 7.26).
// It hides the launch itself: a fixed-point hop at 4^4 takes 3.4 us in a row of
// them instead of 6.2, at 8^3x16 5.8 instead of 8.2, at 16^3x32 25.8 instead of 28.7.
__device__ __forceinline__ void wd_pdl_wait(bool ahead = false)
{
    if (ahead) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!ahead) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
inline void wd_launch_pdl(bool pdl, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                          A... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// The same for the other hops, by the number of their blocks.  Up to a block
// per SM (FP32 hop at 8^3x16 3.6 instead of 6.2 us) and from several waves on
// (24^4 16.4 instead of 18.4 us; double-float at 16^3x32 25.2 instead of 27.5)
// the early launch gains; in between it is unevenly spread (double-float CG at
// 12^3x16 2.45 instead of 2.19 ms), and the largest grids lose by it (82,944
// blocks: an FP16 solve at 48^3x96 145.7 instead of 140.8 ms).
inline bool wd_pdl_early(int blocks) { return blocks <= 152 || (blocks >= 1000 && blocks <= 10000); }
template <class... P, class... A>
inline void wd_launch_early(void (*kernel)(P...), int blocks, int threads, cudaStream_t stream, A... args)
{
    wd_launch_pdl(wd_pdl_early(blocks), kernel, blocks, threads, 0, stream, args...);
}
