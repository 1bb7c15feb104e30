// Device memory of the library, taken from one memory pool per GPU in stream order.
//
// An engine makes about thirty allocations, and cudaMalloc and cudaFree map and unmap pages, wait for the whole
// device and - on a host that others use - now and then take milliseconds: creating, filling and destroying an
// engine for two million ratings spent 5 of its 14 ms in them.  The pool keeps up to kKeep bytes of freed memory
// mapped for the next allocation (of this process; beyond that, memory goes back to the system as soon as it is
// free); mascot_release_scratch returns the rest.  The driver serialises pools internally, so engines on several
// threads and streams can share one; memory freed on one stream reaches another only after the work that used it.
//
// Buffers above kLarge still come from cudaMalloc: they live as long as an engine, would fill the pool's bound at once,
// and unmapping 2 GB of pool memory took 40 to 80 ms where cudaFree took 6.
//
// Where the process sees more than one GPU, memory comes from cudaMalloc instead: programs copy item rows between
// GPUs (mascot_item_rows), and a pool's memory is not mapped on peers.
#include <cuda_runtime.h>

#include <mutex>
#include <set>

#include "handle.h"

namespace mascot {

namespace {

constexpr size_t kKeep = 1ull << 30;
constexpr size_t kLarge = 256ull << 20;
constexpr int kDevices = 64;
std::mutex g_mutex;
std::set<void*> g_plain;                          // what cudaMalloc gave
cudaMemPool_t g_pools[kDevices] = {};

bool one_gpu() {
    static const int gpus = [] { int n = 0; return cudaGetDeviceCount(&n) == cudaSuccess ? n : 0; }();
    return gpus <= 1;
}

cudaError_t current_pool(cudaMemPool_t* pool) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= kDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_pools[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        e = cudaMemPoolCreate(&g_pools[dev], &props);
        if (e != cudaSuccess) { g_pools[dev] = nullptr; return e; }
        unsigned long long keep = kKeep;
        cudaMemPoolSetAttribute(g_pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
    }
    *pool = g_pools[dev];
    return cudaSuccess;
}

}  // namespace

cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t st) {
    cudaError_t e;
    if (bytes > kLarge || !one_gpu()) {
        e = cudaMalloc(p, bytes);
        if (e == cudaSuccess) { std::lock_guard<std::mutex> lock(g_mutex); g_plain.insert(*p); }
        return e;
    }
    cudaMemPool_t pool = nullptr;
    e = current_pool(&pool);
    return e == cudaSuccess ? cudaMallocFromPoolAsync(p, bytes, pool, st) : e;
}

void pool_free(void* p, cudaStream_t st) {
    bool plain;
    { std::lock_guard<std::mutex> lock(g_mutex); plain = g_plain.erase(p) > 0; }
    if (plain) cudaFree(p);
    else cudaFreeAsync(p, st);
}

void pool_trim() {
    cudaMemPool_t pool = nullptr;
    if (current_pool(&pool) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
}

}  // namespace mascot
