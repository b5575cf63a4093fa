// The scratch pools and the growing scratch over a fake of the CUDA calls they
// make: a pool that could not be created once is created by a later call, a
// captured stream gets nothing, and the thread's capture mode is put back; a
// buffer that a captured launch may hold outlives its successors, any other is
// freed, and a failed growth leaves a buffer of the old size.
#include <stdio.h>
#include <stdlib.h>

#include <map>

#include "pool.h"
#include "bssn_b200.h"

static int creates, create_fails, mallocs, malloc_fails, frees, destroys;
static bool capturing, implicit;
static size_t room = 100;  // bytes of the device
static std::map<void*, size_t> live;
static cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal, mode_at_create;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return implicit ? cudaErrorStreamCaptureImplicit : cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
    const cudaStreamCaptureMode t = mode;
    mode = *m;
    *m = t;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    creates++;
    mode_at_create = mode;
    if (create_fails > 0) {
        create_fails--;
        return cudaErrorMemoryAllocation;
    }
    *p = (cudaMemPool_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { destroys++; free(p); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t) {
    mallocs++;
    if (malloc_fails > 0) {
        malloc_fails--;
        return cudaErrorMemoryAllocation;
    }
    *p = malloc(1);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    if (n > room) return cudaErrorMemoryAllocation;
    *p = malloc(1);
    room -= n;
    live[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    room += live.at(p);
    live.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { frees++; free(p); return cudaSuccess; }
}

#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    void* p = nullptr;
    create_fails = 1;
    CHECK(bssn::pool_alloc(&p, 8, nullptr) == BSSN_ENOMEM && !p && mallocs == 0);
    CHECK(bssn::pool_alloc(&p, 8, nullptr) == 0 && p && creates == 2 && mallocs == 1);
    CHECK(mode_at_create == cudaStreamCaptureModeRelaxed && mode == cudaStreamCaptureModeGlobal);
    CHECK(bssn::pool_free(p, nullptr) == 0 && frees == 1);
    malloc_fails = 1;
    CHECK(bssn::pool_alloc(&p, 8, nullptr) == BSSN_ENOMEM && !p);
    CHECK(bssn::pool_alloc(&p, 8, nullptr) == 0 && p && creates == 2);
    CHECK(bssn::pool_free(p, nullptr) == 0);
    const int m = mallocs;
    capturing = true;
    CHECK(bssn::pool_alloc(&p, 8, nullptr) == BSSN_ENOMEM && !p);
    capturing = false;
    implicit = true;
    CHECK(bssn::pool_alloc(&p, 8, nullptr) == BSSN_ENOMEM && !p);
    implicit = false;
    CHECK(mallocs == m && mode == cudaStreamCaptureModeGlobal);
    {
        bssn::ScratchPool own(64);
        capturing = true;
        CHECK(own.alloc(&p, 8, nullptr) == BSSN_ENOMEM && creates == 2);
        capturing = false;
        CHECK(own.alloc(&p, 8, nullptr) == 0 && creates == 3);
        CHECK(bssn::pool_free(p, nullptr) == 0);
    }
    CHECK(destroys == 1);
    {
        bssn::GrowingScratch g;
        CHECK(g.on(nullptr) == nullptr && g.grow(10) == 0 && g.bytes() == 10 && g.grow(5) == 0 && live.size() == 1);
        CHECK(g.grow(20) == 0 && live.size() == 1 && live.count(g.on(nullptr)));
        // 20 + 90 do not fit beside each other: the old buffer goes first
        CHECK(g.grow(90) == 0 && g.bytes() == 90 && live.size() == 1);
        // 200 do not fit at all: a buffer of the old size stays
        CHECK(g.grow(200) == BSSN_ENOMEM && g.bytes() == 90 && live.size() == 1 && live.count(g.on(nullptr)));
    }
    CHECK(live.empty() && room == 100);
    {
        bssn::GrowingScratch g;
        CHECK(g.grow(10) == 0);
        capturing = true;
        double* held = g.on(nullptr);
        capturing = false;
        CHECK(g.grow(20) == 0 && live.count(held) && live.size() == 2 && g.on(nullptr) != held);
        CHECK(g.grow(30) == 0 && live.count(held) && live.size() == 2);  // the 20 bytes nobody captured went
        capturing = true;
        held = g.on(nullptr);
        capturing = false;
        CHECK(g.grow(80) == BSSN_ENOMEM && g.on(nullptr) == held && g.bytes() == 30);  // 10 + 30 held: no room
    }
    CHECK(live.empty() && room == 100);
    printf("ok\n");
    return 0;
}
