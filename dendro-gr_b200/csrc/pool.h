// Scratch for calls that may run on any stream and thread at once and so must
// not share a handle's buffers.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <mutex>
#include <vector>

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

// One buffer that grows.  A buffer that a captured launch may have recorded is
// kept when a larger one takes its place, until the object goes, so that the
// graph stays valid; any other is freed.  A growth that fails leaves a buffer of
// the old size.
class GrowingScratch {
public:
    GrowingScratch() = default;
    ~GrowingScratch();
    GrowingScratch(const GrowingScratch&) = delete;
    GrowingScratch& operator=(const GrowingScratch&) = delete;
    // Makes the buffer hold at least `bytes` (outside stream captures).
    int grow(size_t bytes);
    size_t bytes() const { return bytes_; }
    // The buffer, for launches on s.
    double* on(cudaStream_t s);

private:
    double* p_ = nullptr;
    size_t bytes_ = 0;
    bool captured_ = false;
    std::vector<double*> kept_;
};

// Bytes the library's own pool of each device keeps (the split scratch of the
// largest block).
constexpr size_t kPoolKeepBytes = size_t(160) << 20;

// The library's pool of the current device.
int pool_alloc(void** p, size_t bytes, cudaStream_t s);
// Returns a buffer of any pool.
int pool_free(void* p, cudaStream_t s);

}  // namespace bssn
