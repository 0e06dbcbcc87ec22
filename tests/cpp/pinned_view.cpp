// wd_pinned_view against a runtime that holds one pinned range: 1000 bytes
// from host address 0x10000, at device address 0x90000.
#include <cstdio>
#include "wd_pinned.h"

static int errors;
extern "C" cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    const uintptr_t h = (uintptr_t)p;
    *a = cudaPointerAttributes{};
    if (h >= 0xf0000) return cudaErrorInvalidValue;
    if (h < 0x10000 || h >= 0x10000 + 1000) return cudaSuccess;  // type 0: unregistered
    a->type = cudaMemoryTypeHost;
    a->devicePointer = (void *)(h - 0x10000 + 0x90000);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

static void expect(uintptr_t host, size_t bytes, uintptr_t device)
{
    const uintptr_t got = (uintptr_t)wd_pinned_view((const void *)host, bytes);
    if (got == device) return;
    std::printf("%lx + %zu: %lx, not %lx\n", (unsigned long)host, bytes, (unsigned long)got, (unsigned long)device);
    ++errors;
}

int main()
{
    expect(0x10000, 1000, 0x90000);
    expect(0x10010, 984, 0x90010);
    expect(0x10000, 1, 0x90000);
    expect(0x10000, 1001, 0);   // ends one byte outside
    expect(0x10000, 5000, 0);
    expect(0x10008, 16, 0);     // no 16-byte address
    expect(0xfff0, 32, 0);      // begins outside
    expect(0xf0000, 16, 0);     // the runtime knows nothing of it
    expect(0x10000, 0xe0010, 0);
    return errors != 0;
}
