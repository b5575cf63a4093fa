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

int GrowingScratch::grow(size_t bytes) {
    if (bytes <= bytes_) return 0;
    auto make = [](size_t n) {
        void* p = nullptr;
        if (cudaMalloc(&p, n) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return static_cast<double*>(p);
    };
    double* p = make(bytes);
    if (p) {
        if (captured_)
            kept_.push_back(p_);
        else
            cudaFree(p_);
    } else {
        if (captured_ || !p_) return BSSN_ENOMEM;
        // both do not fit at once: the old one goes first
        cudaFree(p_);
        p = make(bytes);
        if (!p) {
            p_ = make(bytes_);
            if (!p_) bytes_ = 0;
            return BSSN_ENOMEM;
        }
    }
    p_ = p;
    bytes_ = bytes;
    captured_ = false;
    return 0;
}

double* GrowingScratch::on(cudaStream_t s) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess)
        cudaGetLastError();  // the legacy stream while another one captures: the launch reports it
    else if (cap != cudaStreamCaptureStatusNone)
        captured_ = true;
    return p_;
}

GrowingScratch::~GrowingScratch() {
    if (p_) cudaFree(p_);
    for (double* p : kept_) cudaFree(p);
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
