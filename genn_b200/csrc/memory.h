// Where a runner's memory comes from.
//
// Building a model allocates a dozen arrays and as many tables, and parameter sweeps build models all the time.  On a B200 a
// cudaMalloc costs 10 - 350 us, a cudaFree as much, page-locking a few KB 1.6 ms, and the first touch of fresh pageable
// memory 2 us per page (a 40 MB array: 20 ms of a pull whose transfer takes 0.75).  Hence: device memory from a
// stream-ordered pool of the library's own (per device, at most POOL_KEEP bytes kept while nobody uses them, everything
// beyond goes back when it is freed), page-locked blocks from a cache (at most HOST_KEEP bytes idle), and large pulls
// copied out of page-locked chunks by several threads.  All of it may be called from any thread.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace b200
{
constexpr size_t POOL_KEEP = (size_t)1 << 30;
constexpr size_t POOL_MOST = (size_t)128 << 20;     // a larger allocation is one of its own: a pool maps new memory more slowly
constexpr size_t HOST_KEEP = (size_t)32 << 20;

// Device memory of the current device, usable in the order of `stream`.
cudaError_t poolAllocBytes(void **p, size_t bytes, cudaStream_t stream);
cudaError_t poolFree(void *p, cudaStream_t stream);

template<typename T>
cudaError_t poolAlloc(T **p, size_t bytes, cudaStream_t stream)
{
    void *q = nullptr;
    const cudaError_t e = poolAllocBytes(&q, bytes, stream);
    *p = static_cast<T*>(q);
    return e;
}

// Page-locked memory.
cudaError_t hostAcquire(void **p, size_t bytes);
void hostRelease(void *p);

// Copies `count` elements of `elemBytes` (1, 2 or 4; `widen`: stored as 32-bit values) from the device behind what `stream`
// holds, and waits.
cudaError_t pullLarge(void *host, const void *device, size_t count, unsigned int elemBytes, bool widen, int deviceIndex, cudaStream_t stream);
}   // namespace b200
