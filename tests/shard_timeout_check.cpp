// A sharded evaluation whose peer never answers, on the host: shard.cu and device_pool.cu against fake_cudart.h and a fake
// NCCL.  argv[1]: the collective that never ends ("gather" or "reduce"); argv[2]: test ratings; argv[3]: visible GPUs.
#include "fake_cudart.h"

#include <nccl.h>

#include <string>

#include "handle.h"

static FakeStream* g_hung = nullptr;
static std::string g_mode;
static float* g_written = nullptr;                // where the queued evaluation kernel will write

static ncclResult_t hang(const char* what, cudaStream_t st) {
    if (g_mode == what) { g_hung = fake(st); g_hung->stuck = true; }
    return ncclSuccess;
}
static ncclResult_t comm_init(ncclComm_t* c, int, ncclUniqueId, int) { *c = reinterpret_cast<ncclComm_t>(8); return ncclSuccess; }
static ncclResult_t comm_done(ncclComm_t) { return ncclSuccess; }          // an aborted communicator's kernels end some time later
static ncclResult_t async_error(ncclComm_t, ncclResult_t* r) { *r = ncclSuccess; return ncclSuccess; }
static const char* error_string(ncclResult_t) { return "fake"; }
static ncclResult_t unique_id(ncclUniqueId*) { return ncclSuccess; }
static ncclResult_t group() { return ncclSuccess; }
static ncclResult_t transfer(const void*, size_t, ncclDataType_t, int, ncclComm_t, cudaStream_t) { return ncclSuccess; }
static ncclResult_t receive(void*, size_t, ncclDataType_t, int, ncclComm_t, cudaStream_t) { return ncclSuccess; }
static ncclResult_t all_reduce(const void*, void*, size_t, ncclDataType_t, ncclRedOp_t, ncclComm_t, cudaStream_t st) { return hang("reduce", st); }
static ncclResult_t all_gather(const void*, void*, size_t, ncclDataType_t, ncclComm_t, cudaStream_t st) { return hang("gather", st); }

extern "C" void* dlopen(const char*, int) noexcept { return reinterpret_cast<void*>(8); }
extern "C" int dlclose(void*) noexcept { return 0; }
extern "C" char* dlerror() noexcept { return nullptr; }
extern "C" void* dlsym(void*, const char* name) noexcept {
    const std::string n(name);
    if (n == "ncclGetUniqueId") return reinterpret_cast<void*>(&unique_id);
    if (n == "ncclCommInitRank") return reinterpret_cast<void*>(&comm_init);
    if (n == "ncclCommDestroy" || n == "ncclCommAbort") return reinterpret_cast<void*>(&comm_done);
    if (n == "ncclCommGetAsyncError") return reinterpret_cast<void*>(&async_error);
    if (n == "ncclGetErrorString") return reinterpret_cast<void*>(&error_string);
    if (n == "ncclGroupStart" || n == "ncclGroupEnd") return reinterpret_cast<void*>(&group);
    if (n == "ncclSend") return reinterpret_cast<void*>(&transfer);
    if (n == "ncclRecv") return reinterpret_cast<void*>(&receive);
    if (n == "ncclAllReduce") return reinterpret_cast<void*>(&all_reduce);
    return reinterpret_cast<void*>(&all_gather);
}

// what shard.cu needs of the rest of the library
namespace mascot {
cudaError_t launch_rmse(int, const Stream& t, Arena, Arena, float* out, cudaStream_t) {
    g_written = out;
    for (uint64_t b = 0; b < (t.n + 511) / 512; b++) out[b] = 1.f;
    return cudaSuccess;
}
cudaError_t launch_reduce_stats(float*, int, size_t, size_t, cudaStream_t) { return cudaSuccess; }
int setup_ratings(mascot_handle*, const SetupRequest&) { return MASCOT_OK; }
int train_range(mascot_handle*, float, uint32_t, size_t, bool, LaunchShape*, uint32_t*, uint64_t) { return MASCOT_OK; }
int fetch_stats(mascot_handle*, uint32_t*) { return MASCOT_OK; }
int apply_stats(mascot_handle*, uint32_t, uint32_t*, uint32_t*, uint32_t*) { return MASCOT_OK; }
uint64_t algorithmic_bytes(const mascot_handle*) { return 0; }
float lr_at(const mascot_config&, uint32_t) { return 0.f; }
bool is_check_epoch(const mascot_config&, uint32_t) { return false; }
size_t stats_floats(const mascot_handle*) { return 0; }
int fail(mascot_handle* h, int code, const std::string& msg) { if (h) h->err = msg; return code; }
NvtxRange::NvtxRange(const char*) {}
NvtxRange::~NvtxRange() {}
}  // namespace mascot

int main(int, char** argv) {
    using namespace mascot;
    g_gpus = std::atoi(argv[3]);
    const uint64_t n_test = (uint64_t)std::atoll(argv[2]);
    mascot_handle h;
    std::memset(&h.cfg, 0, sizeof h.cfg);
    h.K = 64; h.n_test = n_test; h.have_ratings = h.have_factors = true;
    h.ilay.rows_per_part = 1; h.iprec.assign(1, 1);
    static float rows[4 * 64];
    h.Q.f32 = rows;
    cudaStreamCreateWithFlags(&h.stream, 0);
    const char id[MASCOT_COMM_ID_BYTES] = {};
    if (mascot_shard_init(&h, id, 0, 2, 1, 50) != MASCOT_OK) { std::printf("no group: %s\n", h.err.c_str()); return 1; }
    double rmse = 0;
    g_mode = "";
    int rc = mascot_shard_eval_rmse(&h, &rmse);
    std::printf("answered rc %d rmse %.6f\n", rc, rmse);
    g_mode = argv[1];
    rc = mascot_shard_eval_rmse(&h, &rmse);
    std::printf("hung rc %d\n", rc);
    // the kernel that writes into g_written is still queued behind the collective: nobody else may get that memory
    cudaStream_t other;
    cudaStreamCreateWithFlags(&other, 0);
    int reused = 0;
    const size_t floats = (n_test + 511) / 512;
    // (plain device memory of somebody else may wait for the device when it is freed: not tried while that hangs)
    for (int j = 0; j < 3 && (g_gpus == 1 || g_pinned.count(g_written)); j++) { Results r(floats, other); reused += r.device() == g_written; r.wait(); }
    if (g_mode == "gather") std::printf("given away %d alive %d\n", reused, (int)(g_pinned.count(g_written) + g_device.count(g_written)));
    release_results();
    if (g_mode == "gather") std::printf("kept by a release %d\n", (int)(g_pinned.count(g_written) + g_device.count(g_written)));
    if (g_hung) g_hung->stuck = false;             // the aborted collective has ended, the kernel has run
    { Results r(floats, other); r.wait(); }
    release_results();
    std::printf("left pinned %d\n", (int)g_pinned.size());
    shard_destroy(&h);
    std::printf("left device %d\n", (int)g_device.size());
    return 0;
}
