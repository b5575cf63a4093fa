// Stream-ordered scratch pools.
#include "pool.h"

#include <map>

#include "bssn_b200.h"
#include "bssn_common.cuh"

namespace bssn {

namespace {

// The calling thread may create and allocate while another thread captures a
// graph in the global mode, which forbids both to every thread and would be
// spoilt by them; nothing here touches a captured stream.
struct OutsideCaptures {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace

int ScratchPool::alloc(void** p, size_t bytes, cudaStream_t s) {
    *p = nullptr;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {  // the legacy stream while another one captures
        cudaGetLastError();
        return BSSN_ENOMEM;
    }
    if (cap != cudaStreamCaptureStatusNone) return BSSN_ENOMEM;
    OutsideCaptures outside;
    std::lock_guard<std::mutex> lock(mu_);
    if (!pool_) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        if (cudaGetDevice(&props.location.id) != cudaSuccess || cudaMemPoolCreate(&pool_, &props) != cudaSuccess) {
            cudaGetLastError();
            pool_ = nullptr;
            return BSSN_ENOMEM;
        }
        uint64_t keep = keep_;
        if (cudaMemPoolSetAttribute(pool_, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) cudaGetLastError();
    }
    if (cudaMallocFromPoolAsync(p, bytes, pool_, s) != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return BSSN_ENOMEM;
    }
    return 0;
}

ScratchPool::~ScratchPool() {
    if (pool_) cudaMemPoolDestroy(pool_);
}

int pool_alloc(void** p, size_t bytes, cudaStream_t s) {
    // never destroyed: calls may come from any thread until the process ends
    static std::mutex& mu = *new std::mutex;
    static std::map<int, ScratchPool*>& pools = *new std::map<int, ScratchPool*>;
    *p = nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return BSSN_ENOMEM;
    }
    ScratchPool* pool;
    {
        std::lock_guard<std::mutex> lock(mu);
        ScratchPool*& q = pools[dev];
        if (!q) q = new ScratchPool(kPoolKeepBytes);
        pool = q;
    }
    return pool->alloc(p, bytes, s);
}

int pool_free(void* p, cudaStream_t s) {
    OutsideCaptures outside;
    return cuda_status(cudaFreeAsync(p, s));
}

}  // namespace bssn
