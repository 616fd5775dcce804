// block_cache.hpp -- memory of closed sets, kept for the next ones.
//
// cudaMalloc, cudaFree and cudaMallocHost synchronise with the device and take
// the driver's locks: 0.4 to 1.5 ms each on an idle B200 host, up to 100 ms on
// a shared one, where a whole small batch runs for 4 ms.  A program that
// creates set after set gets the blocks of the sets it has closed.
//
// Kept, per device: at most kCacheDeviceBytes of device memory and
// kCachePinnedBytes of pinned memory, in at most kCacheBlocks blocks each.  A
// set may get a block up to an eighth larger than it needs, or up to twice while
// all that is in use beyond the need stays within kCacheSlackBytes.
// Larger or later blocks go back to the driver at once, and so does all that is
// kept when an allocation of the library's on the device fails (retry_trimmed)
// or the program asks (lulesh_release_memory).  A block is put back only when
// no work on it can be pending, so any stream may have it next: the set's
// stream has been synchronised, and nobody else knows the memory.  A set whose
// pointers a caller holds, or whose kernels a caller's graph holds, may still
// be at work on a stream the library does not know; its blocks go to the
// driver, whose cudaFree waits for the device (lulesh_set::handed_out).
// Blocks are kept by context, and those of a context that cudaDeviceReset has
// ended are never looked at again.  Thread-safe.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace lulesh {

constexpr size_t kCacheDeviceBytes = size_t(512) << 20;
constexpr size_t kCachePinnedBytes = size_t(1) << 20;
constexpr size_t kCacheBlocks = 64;
constexpr size_t kCacheSlackBytes = size_t(128) << 20;  // of blocks over an eighth too large

struct Block {
    void *p = nullptr;
    size_t bytes = 0, asked = 0;     // of the block, and of it what was asked for
    unsigned long long context = 0;  // id of the context it lives in, 0 not known
    int device = 0;
    bool pinned = false;
};

// On the current device; the contents are whatever they were.
cudaError_t block_get(Block *b, size_t bytes, bool pinned = false);
// Nothing may be pending on the block; *b is emptied.  Any current device.
void block_put(Block *b);
// The block to the driver, after all work on its device; *b is emptied.
void block_free(Block *b);
// All that is kept in the current context to the driver; false if nothing was.
bool block_trim();

// alloc(), and once more without the kept blocks where it was short of memory
template <class Alloc>
inline cudaError_t retry_trimmed(const Alloc &alloc)
{
    const cudaError_t e = alloc();
    if (e != cudaErrorMemoryAllocation || !block_trim()) return e;
    (void)cudaGetLastError();
    return alloc();
}

template <class T>
inline cudaError_t device_malloc(T **p, size_t bytes)
{
    return retry_trimmed([&] { return cudaMalloc(reinterpret_cast<void **>(p), bytes); });
}

}  // namespace lulesh
