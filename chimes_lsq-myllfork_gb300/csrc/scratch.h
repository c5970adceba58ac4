// Per-call device scratch shared by the host orchestration files.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "model.h"

namespace cg {

void cuda_check(cudaError_t e, const char* what);
#define CK(x) ::cg::cuda_check((x), #x)

// The stream-ordered pool that per-call scratch comes from: one per device, made on
// first use (with that device current) and kept until the process exits.  It keeps
// up to 32 GiB of freed scratch mapped across synchronisations; a pool that returns
// freed memory to the driver at every synchronisation has to map each row block's
// work lists again, which cost tens of milliseconds per block of a streamed
// assembly when the rest of device memory was busy.
cudaMemPool_t scratch_pool(int device);
// Return the pool's unused memory to the driver: before sizing a cache from the device's
// free memory, and for callers that share the GPU with another allocator (cg_session_tune
// "release_memory").
void scratch_pool_trim(int device);

// One stream-ordered allocation from the current device's scratch pool (cudaFreeAsync
// returns it).  The default pool gives freed memory back to the driver at every
// synchronisation, and a call that synchronises pays for mapping it again each time.
template <typename T>
T* scratch_alloc(size_t n, cudaStream_t st) {
    int dev = 0;
    void* p = nullptr;
    CK(cudaGetDevice(&dev));
    CK(cudaMallocFromPoolAsync(&p, std::max<size_t>(n * sizeof(T), 8), scratch_pool(dev), st));
    return static_cast<T*>(p);
}

// Device memory of an object that outlives a call or is shared by streams: its owner may use
// it on any stream once the allocating stream has been synchronised, and it goes back when
// nothing on the device can use it any more.  Up to POOL_BLOCK from the scratch pool: cudaMalloc
// and cudaFree of a dozen arrays took half of a call on a small system, and one pair takes 120
// us (1 MiB) to 274 us (256 MiB) where the pool takes 5.  Larger blocks by cudaMalloc, so that
// the driver has them back at once: 0.5 to 1.1 ms (512 MiB, 2 GiB) beside work on as much data.
// Copies to the host run at the same rate out of either (193 GB/s from 64 MiB on).
constexpr size_t POOL_BLOCK = size_t(256) << 20;
void* pool_alloc(size_t bytes, cudaStream_t st);
void pool_free(std::vector<void*>& ptrs);   // synchronises the device first

// Arrays laid out one behind the other, 256-byte aligned: take() adds up the sizes while
// there is no base, and hands out the places once there is.
struct Layout {
    unsigned char* base = nullptr;
    size_t used = 0;
    template <typename T>
    T* take(size_t n) {
        const size_t off = (used + 255) / 256 * 256;
        used = off + std::max<size_t>(n, 1) * sizeof(T);
        return base ? reinterpret_cast<T*>(base + off) : nullptr;
    }
};

// Per-call scratch: stream-ordered device allocations from scratch_pool() released
// at the end of the call, or -- for the no-allocation entry point -- a bump
// allocator over the static device array below (256-byte aligned sub-buffers,
// capacity checked).
struct Scratch {
    cudaStream_t s;
    unsigned char* base = nullptr;
    size_t cap = 0, used = 0;
    std::vector<void*> ptrs;
    cudaMemPool_t pool = nullptr;
    explicit Scratch(cudaStream_t st) : s(st) {
        int dev = 0;
        CK(cudaGetDevice(&dev));
        pool = scratch_pool(dev);
    }
    Scratch(cudaStream_t st, void* static_base, size_t capacity)
        : s(st), base(reinterpret_cast<unsigned char*>(static_base)), cap(capacity) {}
    template <typename T>
    T* get(size_t n) {
        const size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
        if (base) {
            const size_t off = (used + 255) & ~size_t(255);
            if (off + bytes > cap)
                throw Error(4, "input exceeds the no-allocation scratch capacity of " +
                                   std::to_string(cap >> 20) + " MiB; use cg_assemble_device");
            used = off + bytes;
            return reinterpret_cast<T*>(base + off);
        }
        void* p = nullptr;
        CK(cudaMallocFromPoolAsync(&p, bytes, pool, s));
        ptrs.push_back(p);
        return reinterpret_cast<T*>(p);
    }
    ~Scratch() {
        for (void* p : ptrs) cudaFreeAsync(p, s);
    }
};


}  // namespace cg
