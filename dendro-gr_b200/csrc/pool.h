// Scratch for calls that may run on any stream and thread at once and so must
// not share a handle's buffers.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <mutex>

namespace bssn {

// A stream-ordered memory pool on the device that is current at its first
// allocation.  At most `keep` bytes stay reserved while unused; more goes back
// to the system at the next synchronisation, all of it with the pool.
class ScratchPool {
public:
    explicit ScratchPool(size_t keep) : keep_(keep) {}
    ~ScratchPool();
    ScratchPool(const ScratchPool&) = delete;
    ScratchPool& operator=(const ScratchPool&) = delete;
    // A buffer for the caller alone, ordered on s.  BSSN_ENOMEM, with nothing
    // enqueued, while s is being captured (the graph would record the
    // allocation) or when there is no memory; a later call tries again.
    int alloc(void** p, size_t bytes, cudaStream_t s);

private:
    std::mutex mu_;
    cudaMemPool_t pool_ = nullptr;
    size_t keep_;
};

// Bytes the library's own pool of each device keeps (the split scratch of the
// largest block).
constexpr size_t kPoolKeepBytes = size_t(160) << 20;

// The library's pool of the current device.
int pool_alloc(void** p, size_t bytes, cudaStream_t s);
// Returns a buffer of any pool.
int pool_free(void* p, cudaStream_t s);

}  // namespace bssn
