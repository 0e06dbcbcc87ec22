// wd_async.cuh -- per-thread asynchronous copies global -> shared memory
// (cp.async, LDGSTS) for kernels that stage the next direction's operands
// while they compute the current one.  Each copy moves one 4-, 8- or 16-byte
// element; both addresses must be aligned to its size.  A thread's copies
// become visible to that thread after cp.async.wait_group retires their
// group; other threads would also need a barrier (the kernels using these
// read back only their own copies).
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
// predecessor has completed, and at that point lets its own successor start
// the same way (pdl = false: an ordinary launch).  It hides the launch itself:
// a fixed-point hop at 4^4 takes 3.5 us in a row of them instead of 6.2, at
// 8^3x16 6.7 instead of 8.2, at 16^3x32 25.8 instead of 28.7.
__device__ __forceinline__ void wd_pdl_wait()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
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
