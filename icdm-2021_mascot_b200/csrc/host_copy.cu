// Pageable copies.  A rating array, a factor matrix or an order map comes from or goes to ordinary memory of the
// caller, and cudaMemcpy moves such buffers with one host thread through the driver's own staging: measured on a
// 16-core B200 host 11 GB/s up, 15 GB/s down into memory that has been touched and 4.6 GB/s into fresh pages, where
// that thread also takes the page faults - against 55 GB/s of the link from pinned memory.  Here up to eight threads
// (down, above 64 MB, twelve) move the data between the caller's memory and a pinned ring while the copy engine works on
// other parts of the ring, so the host side runs at several cores' bandwidth and the faults are taken in parallel.  Up:
// 4 MB 15 -> 22 GB/s, 36 MB 12 -> 41, 480 MB 11 -> 51; down into fresh pages 4.6 -> 38.
//
// The first large copy of a process makes the ring: 24 MiB touched in 4 to 5 ms, registered in 1 to 10.
#include "host_copy.h"

#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "host_cores.h"

namespace mascot {

namespace {

constexpr int kMaxUp = 8;                         // 8 threads: 63 GB/s of memcpy on that host, 4: 48, 16: 51
constexpr int kMaxThreads = 12;                   // down, where page faults cost as much as the copy: 8 threads 42 GB/s, 12: 52
constexpr size_t kSlot = 1u << 20;                // long enough for the link's bandwidth, short enough to overlap
constexpr int kSlots = 2 * kMaxThreads;
constexpr int kMaxRings = 2;                      // rings of a process: 2 x 24 MiB of pinned memory at most
constexpr size_t kDirect = 192u << 10;            // below this the driver's copy is as fast

// The helper threads of a ring.  Starting eight threads costs more than copying 4 MB, and waking parked ones takes most
// of a millisecond on a virtual machine (16 MB up: 1.3 ms after parked threads, 0.45 after awake ones).  Copies come in
// groups - both factor matrices, then the test set - so a helper stays awake for kAwake after its last work, giving its
// core to whoever asks for it, and parks then.  (Under a CPU quota there are no more helpers than it pays for.)
class Team {
public:
    ~Team() {
        { std::lock_guard<std::mutex> lock(mu_); quit_ = true; round_++; }
        start_.notify_all();
        for (std::thread& t : threads_) t.join();
    }
    // Runs work(0 .. threads - 1), work(0) on the caller's thread; returns when all are done.
    void run(int threads, const std::function<void(int)>& work) {
        try { while ((int)threads_.size() < threads - 1) { const int id = (int)threads_.size() + 1; threads_.emplace_back([this, id] { loop(id); }); } }
        catch (...) {}                             // no more threads to be had: those that exist do the work
        const int helpers = std::min((int)threads_.size(), threads - 1);
        if (helpers > 0) {
            bool parked;
            { std::lock_guard<std::mutex> lock(mu_); work_ = &work; helpers_ = helpers; running_ = helpers; round_++; parked = parked_ > 0; }
            if (parked) start_.notify_all();
        }
        work(0);
        while (running_.load(std::memory_order_acquire) > 0) std::this_thread::yield();
    }

private:
    static constexpr std::chrono::milliseconds kAwake{4};
    void loop(int id) {
        unsigned long seen = 0;
        for (;;) {
            const auto parking = std::chrono::steady_clock::now() + kAwake;
            while (round_.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < parking) std::this_thread::yield();
            const std::function<void(int)>* work = nullptr;
            {
                std::unique_lock<std::mutex> lock(mu_);
                if (round_ == seen) {
                    parked_++;
                    start_.wait(lock, [&] { return round_ != seen; });
                    parked_--;
                }
                if (quit_) return;
                seen = round_;
                if (id <= helpers_) work = work_;
            }
            if (!work) continue;
            (*work)(id);
            running_.fetch_sub(1, std::memory_order_release);
        }
    }
    std::mutex mu_;
    std::condition_variable start_;
    std::vector<std::thread> threads_;
    const std::function<void(int)>* work_ = nullptr;      // of round `round_`, for the helpers 1 .. helpers_
    int helpers_ = 0, parked_ = 0;
    std::atomic<unsigned long> round_{0};
    std::atomic<int> running_{0};
    bool quit_ = false;
};

struct Ring {
    unsigned char* mem = nullptr;
    cudaEvent_t done[kSlots] = {};                // last use of each slot
    int device = -1;
    bool busy = false;
    Team team;
};

std::mutex g_mutex;
std::vector<Ring*> g_rings;

void drop_events(Ring* r) {
    for (cudaEvent_t& e : r->done) if (e) { cudaEventSynchronize(e); cudaEventDestroy(e); e = nullptr; }
    r->device = -1;
}

// The events of a ring belong to one device; a ring that served another device gets new ones.
bool bind(Ring* r, int device) {
    if (r->device == device) return true;
    drop_events(r);
    for (cudaEvent_t& e : r->done) if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); return false; }
    r->device = device;
    return true;
}

// A ring of this process that nobody uses, or null when both are in use (or pinned memory is short): the caller
// then takes the driver's copy.
Ring* take_ring(int device) {
    std::lock_guard<std::mutex> lock(g_mutex);
    Ring* found = nullptr;
    for (Ring* r : g_rings) if (!r->busy && (!found || r->device == device)) found = r;
    if (!found && g_rings.size() < (size_t)kMaxRings) {
        Ring* r = new Ring();
        // pages of 2 MiB where the system has them: 38 GB/s down into fresh pages against 25 from cudaHostAlloc's memory
        r->mem = static_cast<unsigned char*>(std::aligned_alloc(2u << 20, kSlot * kSlots));
        if (r->mem) { madvise(r->mem, kSlot * kSlots, MADV_HUGEPAGE); std::memset(r->mem, 0, kSlot * kSlots); }
        if (!r->mem || cudaHostRegister(r->mem, kSlot * kSlots, cudaHostRegisterPortable) != cudaSuccess) {
            cudaGetLastError();
            std::free(r->mem);
            delete r;
            return nullptr;
        }
        g_rings.push_back(r);
        found = r;
    }
    if (!found || !bind(found, device)) return nullptr;
    found->busy = true;
    return found;
}

void give_ring(Ring* r) {
    std::lock_guard<std::mutex> lock(g_mutex);
    r->busy = false;
}

int host_threads(size_t bytes, int most) {
    static const int cores = usable_cores();
    // waking a thread costs about ten microseconds: half a megabyte each at least
    return (int)std::max<size_t>(1, std::min<size_t>({(size_t)cores, (size_t)most, bytes >> 19}));
}

// Maps the whole pages of a buffer that is about to be written, in one call instead of a fault per page (fresh 4 KB pages,
// 8 threads: 28 GB/s against 19).  Where the kernel does not know the call, the pages come with the faults.
void populate(unsigned char* host, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
    const uintptr_t page = 4096, from = (reinterpret_cast<uintptr_t>(host) + page - 1) & ~(page - 1), to = (reinterpret_cast<uintptr_t>(host) + bytes) & ~(page - 1);
    if (to > from) madvise(reinterpret_cast<void*>(from), to - from, MADV_POPULATE_WRITE);
#endif
}

bool is_pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type != cudaMemoryTypeUnregistered;
}

// The spans of a download cut into pieces of at most a slot, two of which (a block) a thread takes in one go.  With
// whole slots the blocks start at multiples of 2 MiB of the host address, so that two threads never fault the same
// large page: 38 GB/s into fresh pages against 26 with single pieces.
struct Piece { unsigned char* host; unsigned char* dev; size_t bytes; };
constexpr size_t kPerBlock = 2;
std::vector<Piece> blocks(const CopySpan* spans, int n, size_t piece) {
    const size_t block = kPerBlock * piece;
    std::vector<Piece> out;
    for (int s = 0; s < n; s++) {
        unsigned char* host = static_cast<unsigned char*>(spans[s].host);
        unsigned char* dev = static_cast<unsigned char*>(spans[s].dev);
        size_t left = spans[s].bytes;
        while (left) {
            size_t in_block = std::min(left, block - (piece == kSlot ? reinterpret_cast<uintptr_t>(host) % block : 0));
            left -= in_block;
            for (size_t k = 0; k < kPerBlock; k++) {                   // the second piece of a short block may be empty
                const size_t b = std::min(in_block, piece);
                out.push_back(Piece{host, dev, b});
                host += b; dev += b; in_block -= b;
            }
        }
    }
    return out;
}

}  // namespace

cudaError_t copy_to_device(void* dev, const void* host, size_t bytes, cudaStream_t st) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    Ring* const ring = bytes < kDirect || is_pinned(host) ? nullptr : take_ring(device);
    if (!ring) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    // The ring is used in parts of a quarter: a copy costs the engine 4.5 us whatever its size (pieces of 256 KB: 29
    // GB/s from pinned memory, 1 MB: 43, 4 MB: 49).  The threads fill a part together, and whoever finishes it sends it.
    const int threads = host_threads(bytes, kMaxUp);
    constexpr size_t kFill = 256u << 10, kParts = 4, kMostPart = kSlot * kSlots / kParts;
    const size_t part = std::min(kMostPart, std::max<size_t>((bytes / kParts + kFill - 1) / kFill * kFill, 4 * kFill));
    const size_t parts = (bytes + part - 1) / part, fills = part / kFill;
    std::vector<std::atomic<int>> left(parts);             // pieces of each part that are still to be filled; -1: sent
    for (size_t c = 0; c < parts; c++) left[c] = (int)((std::min(part, bytes - c * part) + kFill - 1) / kFill);
    std::atomic<size_t> next{0};
    std::atomic<int> error{0};
    ring->team.run(threads, [&](int) {
        cudaError_t r = cudaSetDevice(device);
        for (size_t ready = ~(size_t)0; !error.load(std::memory_order_relaxed);) {
            const size_t i = next.fetch_add(1), c = i / fills, in = i % fills * kFill;
            if (c >= parts) break;
            const size_t len = std::min(part, bytes - c * part);
            if (in >= len) continue;
            unsigned char* const mem = ring->mem + c % kParts * kMostPart;
            if (c != ready) {                                   // what this quarter of the ring held before - of an earlier call, too - has to be gone
                while (c >= kParts && left[c - kParts].load(std::memory_order_acquire) >= 0 && !error.load(std::memory_order_relaxed)) std::this_thread::yield();
                if (r == cudaSuccess && !error.load()) r = cudaEventSynchronize(ring->done[c % kParts]);
                ready = c;
            }
            if (r == cudaSuccess) std::memcpy(mem + in, static_cast<const unsigned char*>(host) + c * part + in, std::min(kFill, len - in));
            if (r == cudaSuccess && left[c].fetch_sub(1, std::memory_order_acq_rel) == 1) {
                r = cudaMemcpyAsync(static_cast<unsigned char*>(dev) + c * part, mem, len, cudaMemcpyHostToDevice, st);
                if (r == cudaSuccess) r = cudaEventRecord(ring->done[c % kParts], st);
                if (r == cudaSuccess) left[c].store(-1, std::memory_order_release);
            }
            if (r != cudaSuccess) error = (int)r;
        }
    });
    give_ring(ring);                               // copies still in flight are waited for at the next use
    return (cudaError_t)error.load();
}

cudaError_t copy_to_host(const CopySpan* spans, int n_spans, cudaStream_t st) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    size_t bytes = 0;
    bool pinned = true;
    for (int s = 0; s < n_spans; s++) {
        bytes += spans[s].bytes;
        pinned = pinned && (spans[s].bytes == 0 || is_pinned(spans[s].host));
    }
    Ring* const ring = bytes < kDirect || pinned ? nullptr : take_ring(device);
    if (!ring) {
        for (int s = 0; s < n_spans && e == cudaSuccess; s++)
            if (spans[s].bytes) e = cudaMemcpyAsync(spans[s].host, spans[s].dev, spans[s].bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    // 36 MB are as fast with eight threads as with twelve; small pieces are populated no faster than faulted.
    const int threads = host_threads(bytes, bytes < (64u << 20) ? kMaxUp : kMaxThreads);
    const bool ahead = bytes >= (16u << 20);
    for (cudaEvent_t& ev : ring->done) if (e == cudaSuccess) e = cudaEventSynchronize(ev);      // the last parts of an upload before this
    if (e != cudaSuccess) { give_ring(ring); return e; }
    const std::vector<Piece> pieces = blocks(spans, n_spans, std::min(kSlot, std::max<size_t>(bytes / (4 * threads), 128u << 10)));
    std::atomic<size_t> next{0};
    std::atomic<int> error{0};
    ring->team.run(threads, [&](int t) {
        cudaError_t r = cudaSetDevice(device);
        auto request = [&](size_t c, int slot) {
            if (!pieces[c].bytes) return;
            r = cudaEventSynchronize(ring->done[slot]);
            if (r == cudaSuccess) r = cudaMemcpyAsync(ring->mem + kSlot * slot, pieces[c].dev, pieces[c].bytes, cudaMemcpyDeviceToHost, st);
            if (r == cudaSuccess) r = cudaEventRecord(ring->done[slot], st);
        };
        size_t c = r == cudaSuccess ? next.fetch_add(kPerBlock) : pieces.size();
        if (c < pieces.size()) request(c, 2 * t);
        while (r == cudaSuccess && c < pieces.size()) {
            const size_t after = (c + 1) % kPerBlock ? c + 1 : next.fetch_add(kPerBlock);
            const int slot = 2 * t + (int)(c & 1);
            if (after < pieces.size()) { request(after, slot ^ 1); if (r != cudaSuccess) break; }
            if (pieces[c].bytes) {
                if (ahead) populate(pieces[c].host, pieces[c].bytes);
                r = cudaEventSynchronize(ring->done[slot]);
                if (r == cudaSuccess) std::memcpy(pieces[c].host, ring->mem + kSlot * slot, pieces[c].bytes);
            }
            c = after;
        }
        if (r != cudaSuccess) error = (int)r;
    });
    give_ring(ring);
    return (cudaError_t)error.load();
}

void release_copy_rings() {
    std::lock_guard<std::mutex> lock(g_mutex);
    for (size_t j = 0; j < g_rings.size();) {
        if (g_rings[j]->busy) { j++; continue; }
        drop_events(g_rings[j]);
        cudaHostUnregister(g_rings[j]->mem);
        std::free(g_rings[j]->mem);
        delete g_rings[j];
        g_rings.erase(g_rings.begin() + (long)j);
    }
}

}  // namespace mascot
