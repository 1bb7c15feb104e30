// The few CUDA runtime calls that device_pool.cu, host_copy.cu and shard.cu make, on the host: streams that can be stuck,
// events behind them, memory from malloc.  A call that would wait for a stuck stream says so and ends the program with
// status 3, where the real one would wait for good.
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>

struct FakeStream { bool stuck = false; };
struct FakeEvent { const FakeStream* behind = nullptr; };

inline FakeStream g_legacy;                       // the default stream
inline FakeStream* fake(cudaStream_t st) { return st ? reinterpret_cast<FakeStream*>(st) : &g_legacy; }
inline cudaStream_t real(FakeStream* s) { return reinterpret_cast<cudaStream_t>(s); }
inline std::mutex g_fake_mutex;
inline std::set<FakeStream*> g_streams;
inline std::set<void*> g_device, g_pinned, g_registered;      // live allocations
inline int g_gpus = 1;

inline void fake_wait(const FakeStream* s, const char* who) {
    if (s && s->stuck) { std::printf("%s would wait for a stream that makes no progress\n", who); std::fflush(stdout); std::_Exit(3); }
}
inline void fake_wait_all(const char* who) { for (FakeStream* s : g_streams) fake_wait(s, who); }

extern "C" {
inline cudaError_t fake_alloc(void** p, size_t n) { std::lock_guard<std::mutex> l(g_fake_mutex); *p = std::malloc(n ? n : 1); g_device.insert(*p); return cudaSuccess; }
inline cudaError_t fake_release(void* p) { std::lock_guard<std::mutex> l(g_fake_mutex); g_device.erase(p); std::free(p); return cudaSuccess; }

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = g_gpus; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaMalloc(void** p, size_t n) { return fake_alloc(p, n); }
cudaError_t cudaFree(void* p) { fake_wait_all("cudaFree"); return fake_release(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*) { *pool = reinterpret_cast<cudaMemPool_t>(8); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return fake_alloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return fake_release(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { std::lock_guard<std::mutex> l(g_fake_mutex); *p = std::calloc(1, n); g_pinned.insert(*p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::lock_guard<std::mutex> l(g_fake_mutex); g_pinned.erase(p); std::free(p); return cudaSuccess; }
cudaError_t cudaHostRegister(void* p, size_t, unsigned) { std::lock_guard<std::mutex> l(g_fake_mutex); g_registered.insert(p); return cudaSuccess; }
cudaError_t cudaHostUnregister(void* p) { std::lock_guard<std::mutex> l(g_fake_mutex); g_registered.erase(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { std::memset(a, 0, sizeof *a); a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) { FakeStream* s = new FakeStream(); g_streams.insert(s); *st = real(s); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t st) { g_streams.erase(fake(st)); return cudaSuccess; }      // events may still look at it
cudaError_t cudaStreamQuery(cudaStream_t st) { return fake(st)->stuck ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) { fake_wait(fake(st), "cudaStreamSynchronize"); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { fake_wait_all("cudaDeviceSynchronize"); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
    if (kind == cudaMemcpyDeviceToHost) fake_wait(fake(st), "a copy into pageable memory");
    std::memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind) { std::memcpy(to, from, n); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(new FakeEvent()); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<FakeEvent*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) { reinterpret_cast<FakeEvent*>(e)->behind = fake(st); return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) { const FakeStream* s = reinterpret_cast<FakeEvent*>(e)->behind; return s && s->stuck ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { fake_wait(reinterpret_cast<FakeEvent*>(e)->behind, "cudaEventSynchronize"); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
}
