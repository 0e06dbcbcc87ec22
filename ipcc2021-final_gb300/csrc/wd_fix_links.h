// wd_fix_links.h -- who may use and who may free a lattice's fixed-point links.
//
// They are a second copy of the links that only makes FP64 hops faster, so any
// context that runs out of device memory takes back the copies of every
// lattice on its device, also of lattices that other contexts, on other
// threads, are using.  One lock orders the two: a launch holds it shared from
// its look at wd_lattice::gauge_fix until the kernels are in the stream, and a
// copy is freed under it held alone, after the device has finished what was
// launched.  Nothing that allocates through the context (wd_malloc) may run
// under it.  An uncontended shared lock is some 20 ns of a launch's 3 us.
#pragma once
#include <mutex>
#include <shared_mutex>
#include "wd_internal.cuh"

std::shared_mutex &wd_fix_mutex();
using WdFixShared = std::shared_lock<std::shared_mutex>;
using WdFixAlone = std::unique_lock<std::shared_mutex>;

// The lattice has its fixed-point links, built now if they fit, are wanted and
// have room.  Not to be called under the lock (and the copy may be gone again
// by the time the caller looks).
bool wd_fix_ensure(wd_context *ctx, const wd_lattice *lat);
// The lattice's links are about to change: the copy is no longer theirs
void wd_fix_outdate(wd_lattice *lat);
// Frees one lattice's copy, if it has one
void wd_drop_fix(wd_lattice *lat);
// Frees the copies of every lattice on a device; true if there were any
bool wd_release_fix(int device);
// Bytes the lattice holds for its copy now (0: none)
size_t wd_fix_bytes(const wd_lattice *lat);
// Device memory was freed: copies that were refused are tried again
void wd_memory_freed();
