// wd_pinned.h -- which host arrays the layout kernels may reach themselves.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime_api.h>

// The address at which kernels reach pinned host memory in 16-byte accesses,
// or null.  The layout kernels then read or write it themselves, so the
// conversion rides on the transfer instead of following or preceding it
// through the staging buffer (32^3x64 on pinned arrays: field download 2.22
// -> 2.09 ms, upload 2.05 -> 1.92, links 9.3 -> 7.8).  Pageable memory keeps
// the copy: pages that were never touched fault one by one from the device
// (118 ms for a fresh 403 MB array against 17).
// The last byte is looked at too: what begins in a pinned range and ends
// outside it is for the copy to take or to refuse.
inline void *wd_pinned_view(const void *p, size_t bytes)
{
    cudaPointerAttributes a, z;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess ||
        cudaPointerGetAttributes(&z, (const char *)p + bytes - 1) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || !a.devicePointer || ((uintptr_t)a.devicePointer & 15)) return nullptr;
    if (z.type != cudaMemoryTypeHost || z.devicePointer != (char *)a.devicePointer + bytes - 1) return nullptr;
    return a.devicePointer;
}
