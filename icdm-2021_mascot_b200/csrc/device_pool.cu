// Device memory of the library, taken from one memory pool per GPU in stream order.
//
// An engine makes about thirty allocations, and cudaMalloc and cudaFree map and unmap pages, wait for the whole
// device and - on a host that others use - now and then take milliseconds: creating, filling and destroying an
// engine for two million ratings spent 5 of its 14 ms in them.  (A process pays once for its first pool: 7 to 10 ms.)  The pool keeps up to kKeep bytes of freed memory
// mapped for the next allocation (of this process; beyond that, memory goes back to the system as soon as it is
// free); mascot_release_scratch and mascot_release_cached return the rest.  The driver serialises pools internally, so engines on several
// threads and streams can share one; memory freed on one stream reaches another only after the work that used it.
//
// Buffers above kLarge still come from cudaMalloc.  What an engine frees beyond kKeep is unmapped, and pool memory is slow
// there: 6 ms for 1 GiB (36 on a busy host) where cudaMalloc and cudaFree together take 1.6 (3.6).  Up to kLarge the
// buffers of one engine fit kKeep together: at 9M ratings the set-up's scratch is 256 MiB and the rest as much again.
// One buffer beyond the line costs a job 1.0 to 1.6 ms: 4 epochs of 9M, 11M and 16M ratings from creation to factors take
// 15.3, 16.1 and 18.4 ms, with a line of 1 GiB 14.2, 15.1 and 16.9.
//
// Where the process sees more than one GPU, memory comes from cudaMalloc instead: programs copy item rows between
// GPUs (mascot_item_rows), and a pool's memory is not mapped on peers.  Where it sees one of several, another process may ask
// for the rows, and cudaIpcGetMemHandle refuses pool memory: rows whose address a caller asks for move to cudaMalloc's.
#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <vector>

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

// Pinned blocks of Results: a few for the whole process, whatever number of engines and threads there are.
constexpr size_t kBlockFloats = 16384;            // 64 KiB: block sums of 8.4M ratings
constexpr int kBlocks = 8;
struct PinnedBlock { float* mem; bool busy; };
std::vector<PinnedBlock> g_blocks;

// Memory of Results whose caller gave up waiting (a group of engines that was dissolved): a kernel behind `after` still
// writes into it.  It serves nobody else until the event has passed; without an event it never does.
struct Abandoned { float* mem; bool pinned; cudaEvent_t after; };
std::vector<Abandoned> g_abandoned;

// With g_mutex held: pinned blocks that are free again, and device memory that may be freed now.
void sweep_abandoned(std::vector<float*>* device) {
    for (size_t j = 0; j < g_abandoned.size();) {
        const Abandoned a = g_abandoned[j];
        // freeing device memory may wait for the whole device: only where the caller asks for memory back
        if ((!a.pinned && !device) || !a.after || cudaEventQuery(a.after) != cudaSuccess) { cudaGetLastError(); j++; continue; }
        cudaEventDestroy(a.after);
        if (a.pinned) { for (PinnedBlock& b : g_blocks) if (b.mem == a.mem) b.busy = false; }
        else device->push_back(a.mem);
        g_abandoned.erase(g_abandoned.begin() + (long)j);
    }
}

float* take_block() {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_abandoned.empty()) sweep_abandoned(nullptr);
    for (PinnedBlock& b : g_blocks) if (!b.busy) { b.busy = true; return b.mem; }
    if (g_blocks.size() >= (size_t)kBlocks) return nullptr;
    float* mem = nullptr;
    if (cudaHostAlloc(reinterpret_cast<void**>(&mem), kBlockFloats * sizeof(float), cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    g_blocks.push_back(PinnedBlock{mem, true});
    return mem;
}

}  // namespace

Results::Results(size_t floats, cudaStream_t st) : n_(floats), st_(st) {
    if (floats < kBlockFloats) pinned_ = take_block();
    if (pinned_) { reinterpret_cast<uint32_t*>(pinned_)[n_] = 0; return; }
    status_ = dev_alloc(&dev_, n_ + 1, st_);
    if (status_ == cudaSuccess) status_ = cudaMemsetAsync(dev_ + n_, 0, sizeof(uint32_t), st_);
}

Results::~Results() {
    if (status_ == cudaSuccess && !waited_) {      // the kernel may still be queued
        Abandoned a{pinned_ ? pinned_ : dev_, pinned_ != nullptr, nullptr};
        if (cudaEventCreateWithFlags(&a.after, cudaEventDisableTiming) != cudaSuccess) a.after = nullptr;
        else if (cudaEventRecord(a.after, st_) != cudaSuccess) { cudaEventDestroy(a.after); a.after = nullptr; }
        std::lock_guard<std::mutex> lock(g_mutex);
        g_abandoned.push_back(a);
        return;
    }
    dev_free(dev_, st_);
    if (!pinned_) return;
    std::lock_guard<std::mutex> lock(g_mutex);
    for (PinnedBlock& b : g_blocks) if (b.mem == pinned_) b.busy = false;
}

cudaError_t Results::wait() {
    cudaError_t e = cudaSuccess;
    if (!pinned_) {
        host_.resize(n_ + 1);
        e = cudaMemcpyAsync(host_.data(), dev_, sizeof(float) * (n_ + 1), cudaMemcpyDeviceToHost, st_);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
    waited_ = e == cudaSuccess;
    return e;
}

void release_results() {
    std::vector<float*> device;
    { std::lock_guard<std::mutex> lock(g_mutex); sweep_abandoned(&device); }
    for (float*& p : device) dev_free(p, nullptr);
    std::lock_guard<std::mutex> lock(g_mutex);
    for (size_t j = 0; j < g_blocks.size();) {
        if (g_blocks[j].busy) { j++; continue; }
        cudaFreeHost(g_blocks[j].mem);
        g_blocks.erase(g_blocks.begin() + (long)j);
    }
}

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

cudaError_t pool_make_plain(void** p, size_t bytes, cudaStream_t st) {
    { std::lock_guard<std::mutex> lock(g_mutex); if (!*p || g_plain.count(*p)) return cudaSuccess; }
    void* own = nullptr;
    cudaError_t e = cudaMalloc(&own, bytes);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(own, *p, bytes, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { cudaFree(own); return e; }
    cudaFreeAsync(*p, st);
    *p = own;
    std::lock_guard<std::mutex> lock(g_mutex);
    g_plain.insert(own);
    return cudaSuccess;
}

void pool_trim() {
    cudaMemPool_t pool = nullptr;
    if (current_pool(&pool) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
}

cudaError_t pool_trim_all() {
    int before = 0;
    cudaError_t e = cudaSuccess;
    bool moved = false;
    for (int dev = 0; dev < kDevices; dev++) {
        cudaMemPool_t pool;
        { std::lock_guard<std::mutex> lock(g_mutex); pool = g_pools[dev]; }
        if (!pool) continue;
        if (!moved) { e = cudaGetDevice(&before); moved = true; }
        if (e == cudaSuccess) e = cudaSetDevice(dev);
        if (e == cudaSuccess) e = cudaDeviceSynchronize();      // what was freed behind queued work is idle after it
        if (e == cudaSuccess) e = cudaMemPoolTrimTo(pool, 0);
    }
    if (moved) { const cudaError_t back = cudaSetDevice(before); if (e == cudaSuccess) e = back; }
    return e;
}

}  // namespace mascot
