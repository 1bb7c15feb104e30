// libmascot: host control code behind the C ABI of include/mascot.h.
//
// One handle = one GPU, one stream, one host control thread (like the reference: a single thread
// driving the default stream with a synchronisation after each epoch, mf_methods.cu:239).  The
// m-quantization set-up (degree sort, maps, coded stream: setup.cu) and everything per epoch run on the device; the host
// cuts the groups from the sorted degrees, and the small group statistics travel back on check epochs.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include "../../include/mascot.h"
#include "handle.h"
#include "host_copy.h"

using namespace mascot;

namespace {

thread_local std::string g_create_error;

}  // namespace

void mascot::set_global_error(const char* msg) { g_create_error = msg ? msg : ""; }

mascot::NvtxRange::NvtxRange(const char* name) { nvtxRangePushA(name); }
mascot::NvtxRange::~NvtxRange() { nvtxRangePop(); }

// L2 residency for the item factors (north of L2-sized models the item side is what every rating of a
// run re-reads): a persisting access-policy window on the engine's stream over the arena that holds the
// binary16 item rows (or the fp32 one for fp32 variants).  The carve-out is a per-process limit of the
// device, not a GPU setting: it is restored when the engine goes away.
int mascot::l2_window_install(mascot_handle* h) {
    if (!h->cfg.l2_item_window || h->l2_window_set) return MASCOT_OK;
    int dev = h->cfg.device, max_persist = 0, max_window = 0;
    CU(h, cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, dev));
    CU(h, cudaDeviceGetAttribute(&max_window, cudaDevAttrMaxAccessPolicyWindowSize, dev));
    void* base = h->Q.f16 ? (void*)h->Q.f16 : (void*)h->Q.f32;
    const size_t bytes = (size_t)h->irows * h->K * (h->Q.f16 ? sizeof(__half) : sizeof(float));
    if (!base || !bytes || max_persist <= 0 || max_window <= 0) return MASCOT_OK;
    CU(h, cudaDeviceGetLimit(&h->l2_limit_before, cudaLimitPersistingL2CacheSize));
    const size_t carve = std::min<size_t>((size_t)max_persist, bytes);
    CU(h, cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, carve));
    cudaStreamAttrValue attr;
    std::memset(&attr, 0, sizeof attr);
    attr.accessPolicyWindow.base_ptr = base;
    attr.accessPolicyWindow.num_bytes = std::min<size_t>(bytes, (size_t)max_window);
    attr.accessPolicyWindow.hitRatio = (float)std::min(1.0, (double)carve / (double)attr.accessPolicyWindow.num_bytes);
    attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    CU(h, cudaStreamSetAttribute(h->stream, cudaStreamAttributeAccessPolicyWindow, &attr));
    h->l2_window_set = true;
    return MASCOT_OK;
}

void mascot::l2_window_remove(mascot_handle* h) {
    if (!h->l2_window_set) return;
    cudaStreamAttrValue attr;
    std::memset(&attr, 0, sizeof attr);
    attr.accessPolicyWindow.num_bytes = 0;            // an empty window switches the policy off
    cudaStreamSetAttribute(h->stream, cudaStreamAttributeAccessPolicyWindow, &attr);
    cudaCtxResetPersistingL2Cache();
    cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, h->l2_limit_before);
    h->l2_window_set = false;
}

double mascot::now_us() {
    return std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

int mascot::fail(mascot_handle* h, int code, const std::string& msg) {
    if (h) h->err = msg; else g_create_error = msg;
    return code;
}

namespace mascot {

void free_ratings(mascot_handle* h) {
    dev_free(h->tr_r, h->stream); dev_free(h->tr_u, h->stream); dev_free(h->tr_i, h->stream); dev_free(h->tr_src, h->stream);
    dev_free(h->te_r, h->stream); dev_free(h->te_u, h->stream); dev_free(h->te_i, h->stream);
    dev_free(h->P.f16, h->stream); dev_free(h->P.f32, h->stream); dev_free(h->Q.f16, h->stream); dev_free(h->Q.f32, h->stream);
    dev_free(h->d_uprec_row, h->stream); dev_free(h->d_iprec_row, h->stream); dev_free(h->d_ugroup, h->stream); dev_free(h->d_igroup, h->stream);
    dev_free(h->d_umap, h->stream); dev_free(h->d_imap, h->stream); dev_free(h->d_stats, h->stream);
    h->have_ratings = h->have_factors = false;
}

// mf_methods.cu:94-97: evaluated in double, stored as float.

float lr_at(const mascot_config& c, uint32_t e) {
    return (float)((double)c.learning_rate / (1.0 + ((double)c.decay * std::pow((double)e, 1.5))));
}

// mf_methods.cu:168-175: first check at epoch index 5, then every `interval`, never the last epoch.
bool is_check_epoch(const mascot_config& c, uint32_t e) {
    const uint32_t start_idx = 5;
    const uint32_t it = c.interval ? c.interval : 1;
    return e >= start_idx && (e % it == start_idx % it) && (c.epoch - 1 != e);
}

// split_group_based_equal_size_not_strict_ret_end_idx (preprocess_utils.h:101-213): target size
// T = ceil(N / requested); walk the distinct degrees upward counting entities; close a group at the
// last entity of a degree class once the count reaches T; always close one at the top degree.
void make_groups(const std::vector<uint32_t>& cnt_sorted, uint32_t requested, std::vector<uint32_t>& end_idx) {
    end_idx.clear();
    const uint32_t n = (uint32_t)cnt_sorted.size();
    if (!n) return;
    const uint32_t threshold = (uint32_t)std::ceil((float)n / (float)(requested ? requested : 1));
    const uint32_t max_cnt = cnt_sorted[n - 1];
    uint32_t acc = 0, pos = 0, prev = 0;
    while (pos < n) {
        const uint32_t c = cnt_sorted[pos];
        uint32_t last = pos;
        while (last + 1 < n && cnt_sorted[last + 1] == c) last++;
        if (c >= 1) {   // the reference's walk starts at degree 1 (preprocess_utils.h:139)
            acc += last - prev + 1;
            if (acc >= threshold) { end_idx.push_back(last); acc = 0; }
            else if (c == max_cnt) end_idx.push_back(last);
            prev = last + 1;
        }
        pos = last + 1;
    }
    if (end_idx.empty() || end_idx.back() != n - 1) end_idx.push_back(n - 1);   // only when every degree is 0
}

// bytes the update rule moves per epoch: every rating reads and writes k elements on each side
uint64_t algorithmic_bytes(const mascot_handle* h) {
    double per_side[2] = {0, 0};
    for (int side = 0; side < 2; side++) {
        const std::vector<uint64_t>& deg = side == 0 ? h->udeg_sum : h->ideg_sum;
        const std::vector<uint8_t>& prec = side == 0 ? h->uprec : h->iprec;
        for (size_t g = 0; g < deg.size(); g++) {
            // MPT / AFP / MuPPET keep fp32 masters; fp16-stored groups move 2 bytes per element
            per_side[side] += (double)deg[g] * (prec[g] ? 4.0 : 2.0);
        }
    }
    double total = 2.0 * h->K * (per_side[0] + per_side[1]);
    if (h->n_train_accounted && h->n_train != h->n_train_accounted) total *= (double)h->n_train / (double)h->n_train_accounted;
    return (uint64_t)total;
}

// MuPPET's ladder of pass widths (mf_methods.cu:597).
int muppet_width_at(int idx) {
    static const int widths[5] = {8, 12, 14, 16, 32};
    return widths[idx < 0 ? 0 : (idx < 4 ? idx : 4)];
}

size_t stats_floats(const mascot_handle* h) {
    return (size_t)(h->uend.size() + h->iend.size()) * (h->K + 1);
}

// Encodes an uploaded rating array into the structure-of-arrays stream, segment by segment: the
// seeded permutation and the item-sorted windows never cross a segment boundary.
cudaError_t encode_segments(mascot_handle* h, const mascot_rating* d_src, const std::vector<uint64_t>& seg, bool shuffle,
                            float* r, uint32_t* u, uint32_t* i, uint32_t* src_idx) {
    for (size_t sgm = 0; sgm + 1 < seg.size(); sgm++) {
        const uint64_t off = seg[sgm], n = seg[sgm + 1] - off;
        cudaError_t e = launch_encode_stream(d_src + off, n, shuffle, h->cfg.seed + 0x9e3779b97f4a7c15ull * sgm, h->d_umap, h->d_imap,
                                             h->d_uprec_row, h->d_iprec_row, h->n_users, h->n_items, h->irows, h->d_err_flag,
                                             r + off, u + off, i + off, src_idx ? src_idx + off : nullptr, (uint32_t)off, h->stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// The groups g .. last fp16 -> fp32 (precision_switching.h:12-27): widen their rows into the fp32 arena and flip
// the per-row precision bytes; the stream ids are re-tagged afterwards by recode_side().
int promote_groups(mascot_handle* h, bool users, size_t g, size_t last) {
    const std::vector<uint32_t>& end = users ? h->uend : h->iend;
    std::vector<uint8_t>& prec = users ? h->uprec : h->iprec;
    uint8_t* prow = users ? h->d_uprec_row : h->d_iprec_row;
    const uint32_t b = g ? end[g - 1] + 1 : 0, e = end[last] + 1;
    CU(h, launch_promote_rows(h->K, users ? h->P : h->Q, prow, users ? h->ulay : h->ilay, b, e, h->stream));
    std::fill(prec.begin() + (long)g, prec.begin() + (long)last + 1, (uint8_t)1);
    return MASCOT_OK;
}

int recode_side(mascot_handle* h, bool users) {
    const uint8_t* prow = users ? h->d_uprec_row : h->d_iprec_row;
    CU(h, launch_recode(users ? h->tr_u : h->tr_i, h->n_train, prow, h->stream));
    CU(h, launch_recode(users ? h->te_u : h->te_i, h->n_test, prow, h->stream));
    return MASCOT_OK;
}

int need_scratch(mascot_handle* h, size_t bytes) {
    if (h->scratch_bytes >= bytes) return MASCOT_OK;
    dev_free(h->d_scratch, h->stream); h->scratch_bytes = 0;
    CU(h, pool_alloc(&h->d_scratch, bytes, h->stream));
    h->scratch_bytes = bytes;
    return MASCOT_OK;
}

int need_copy_stream(mascot_handle* h) {
    if (h->copy_stream) return MASCOT_OK;
    for (int b = 0; b < 2; b++) {
        if (!h->ev_copied[b]) CU(h, cudaEventCreateWithFlags(&h->ev_copied[b], cudaEventDisableTiming));
        if (!h->ev_free[b]) CU(h, cudaEventCreateWithFlags(&h->ev_free[b], cudaEventDisableTiming));
    }
    CU(h, cudaStreamCreateWithFlags(&h->copy_stream, cudaStreamNonBlocking));
    return MASCOT_OK;
}

bool any_fp32_group(const mascot_handle* h) {
    for (uint8_t p : h->uprec) if (p) return true;
    for (uint8_t p : h->iprec) if (p) return true;
    return false;
}

// Scratch of a re-ordering: pieces that are carved off one after the other.  The first call sizes it (base null), the second lays it out.
struct SortSpace {
    unsigned char* base = nullptr;
    size_t off = 0;
    float* r; uint32_t *u, *i, *src;       // the re-ordered arrays
    uint64_t* seg;                         // the segment offsets
    template <typename T> T* take(size_t count) {
        T* const p = reinterpret_cast<T*>(base + off);
        off += (sizeof(T) * count + 255) / 256 * 256;
        return p;
    }
    void arrays(size_t n, size_t nseg) {
        r = take<float>(n); u = take<uint32_t>(n); i = take<uint32_t>(n); src = take<uint32_t>(n);
        seg = take<uint64_t>(nseg + 1);
    }
};
static int take_reordered(mascot_handle* h, const SortSpace& sp) {
    const size_t n = h->n_train;
    CU(h, cudaMemcpyAsync(h->tr_r, sp.r, sizeof(float) * n, cudaMemcpyDeviceToDevice, h->stream));
    CU(h, cudaMemcpyAsync(h->tr_u, sp.u, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, h->stream));
    CU(h, cudaMemcpyAsync(h->tr_i, sp.i, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, h->stream));
    if (h->tr_src) CU(h, cudaMemcpyAsync(h->tr_src, sp.src, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, h->stream));
    return MASCOT_OK;
}

// Sorts every window of 2^run_window_log2 positions of the coded stream by item (longer runs of equal items), inside each
// segment.  Called once after a stream was encoded.  The single-worker deterministic mode keeps the caller's order.
static int sort_windows(mascot_handle* h, int run_window_log2) {
    const uint64_t n = h->n_train;
    const int nseg = (int)h->seg_off.size() - 1;
    int seg_bits = 0;
    while ((1ll << seg_bits) < nseg) seg_bits++;
    const size_t temp_bytes = stream_sort_temp_bytes(n, seg_bits, run_window_log2, h->irows), key_bytes = stream_sort_key_bytes(n, seg_bits, run_window_log2, h->irows);
    SortSpace sp;
    unsigned char *key_a, *key_b, *temp;
    uint32_t *idx_a, *idx_b;
    auto lay_out = [&]() {
        sp.off = 0;
        key_a = sp.take<unsigned char>(key_bytes * n); key_b = sp.take<unsigned char>(key_bytes * n);
        idx_a = sp.take<uint32_t>(n); idx_b = sp.take<uint32_t>(n);
        sp.arrays(n, nseg);
        temp = sp.take<unsigned char>(temp_bytes);
    };
    lay_out();
    int rc = need_scratch(h, sp.off);
    if (rc != MASCOT_OK) return rc;
    sp.base = static_cast<unsigned char*>(h->d_scratch);
    lay_out();
    CU(h, cudaMemcpyAsync(sp.seg, h->seg_off.data(), sizeof(uint64_t) * (nseg + 1), cudaMemcpyHostToDevice, h->stream));
    CU(h, launch_stream_sort(h->tr_r, h->tr_u, h->tr_i, h->tr_src, n, sp.seg, nseg, seg_bits, run_window_log2, h->irows, key_a, key_b, idx_a, idx_b,
                             temp, temp_bytes, sp.r, sp.u, sp.i, sp.src, h->stream));
    if ((rc = take_reordered(h, sp)) != MASCOT_OK) return rc;
    CU(h, cudaStreamSynchronize(h->stream));
    return MASCOT_OK;
}

// Makes the ratings of each precision class contiguous inside every segment - the order inside a class is the order before - and
// records the class boundaries.  Called after the
// precision bits of the ids changed (promotion + recode) or after a stream was encoded while promoted groups exist.
static int partition_by_class(mascot_handle* h) {
    const uint64_t n = h->n_train;
    const size_t nseg = h->seg_off.size() - 1;
    h->cls_off.assign(nseg * 5, 0);
    if (n == 0) return MASCOT_OK;
    std::vector<uint32_t> first_tile(nseg + 1), first(nseg * 4);
    const uint32_t tiles = class_tiles(h->seg_off.data(), (int)nseg, first_tile.data());
    const size_t temp_bytes = class_partition_temp_bytes(tiles);
    SortSpace sp;
    uint32_t *d_first_tile, *d_first, *counts, *starts;
    unsigned char* temp;
    auto lay_out = [&]() {
        sp.off = 0;
        sp.arrays(n, nseg);
        d_first_tile = sp.take<uint32_t>(nseg + 1); d_first = sp.take<uint32_t>(nseg * 4);
        counts = sp.take<uint32_t>(4 * (size_t)tiles); starts = sp.take<uint32_t>(4 * (size_t)tiles);
        temp = sp.take<unsigned char>(temp_bytes);
    };
    lay_out();
    int rc = need_scratch(h, sp.off);
    if (rc != MASCOT_OK) return rc;
    sp.base = static_cast<unsigned char*>(h->d_scratch);
    lay_out();
    CU(h, cudaMemcpyAsync(sp.seg, h->seg_off.data(), sizeof(uint64_t) * (nseg + 1), cudaMemcpyHostToDevice, h->stream));
    CU(h, cudaMemcpyAsync(d_first_tile, first_tile.data(), sizeof(uint32_t) * (nseg + 1), cudaMemcpyHostToDevice, h->stream));
    CU(h, launch_class_partition(h->tr_r, h->tr_u, h->tr_i, h->tr_src, n, sp.seg, d_first_tile, (int)nseg, tiles,
                                 counts, starts, temp, temp_bytes, d_first, sp.r, sp.u, sp.i, sp.src, h->stream));
    if ((rc = take_reordered(h, sp)) != MASCOT_OK) return rc;
    CU(h, cudaMemcpyAsync(first.data(), d_first, sizeof(uint32_t) * first.size(), cudaMemcpyDeviceToHost, h->stream));
    CU(h, cudaStreamSynchronize(h->stream));
    for (size_t j = 0; j < nseg; j++) {
        for (int c = 0; c < 4; c++) h->cls_off[j * 5 + c] = first[j * 4 + c];
        h->cls_off[j * 5 + 4] = h->seg_off[j + 1];
    }
    return MASCOT_OK;
}

// The stream is partitioned when that pays: mixed-precision trainer, more than one worker, at least
// one promoted group, and sizes the sort key and the 32-bit permutation can express.
bool wants_partition(const mascot_handle* h) {
    if (!(h->grouped && !h->cfg.deterministic && any_fp32_group(h) && h->n_train < (1ull << 32) && (h->seg_off.size() - 1) * 4 <= 65536)) return false;
    // Measured on one B200, ms per epoch with one launch per class and with one that reads each id's precision bit: 100M
    // ratings, a fifth of the groups promoted 10.0 and 13.6 to 14.2; 252M, 40 % of them 34.0 and 36 to 40.  In between the one
    // launch is faster - 63M, 40 % promoted 9.2 and 9.0; 40M 7.1 and 5.5; k=64, 100M 13.0 and 7.2 - but leaves a test RMSE
    // that is 0.1 % higher after four epochs (0.57343 against 0.57262 at 40M).
    return h->cfg.no_class_partition != 1;
}

int partition_all(mascot_handle* h) {
    h->partitioned = false;
    if (!wants_partition(h)) return MASCOT_OK;
    const int rc = partition_by_class(h);
    if (rc == MASCOT_OK) h->partitioned = true;
    return rc;
}

// log2 of the item-sorted run windows of the resident stream; 0 = none beyond the encode kernel's own windows.
// The configured length (default 2^20) is shortened to the largest power of two that keeps two properties:
//   * a window is no longer than the ratings all workers of a launch hold at one time (workers x K ratings, the
//     longest run of one ticket): with longer windows every worker is on the same few items at once, and since item rows are
//     plain stores most of their updates are lost (100M-rating set, 8,288 workers: windows of 2^20 and 2^22
//     converge like the unsorted stream, 2^24 needs twice the epochs);
//   * when statistics are sampled, the sampled tail of every launched range (sample_ratio of a segment) spans
//     at least four windows, so that every item group is met there in proportion.
int run_window_log2(const mascot_handle* h) {
    if (h->cfg.deterministic || !h->cfg.shuffle || h->n_train == 0 || h->n_train >= (1ull << 32) || (h->seg_off.size() - 1) * 4 > 65536) return 0;
    uint32_t w = h->cfg.run_window_log2 ? std::min<uint32_t>(h->cfg.run_window_log2, 32) : 20;
    uint64_t limit = (uint64_t)worker_count(h, h->n_train) * h->K;
    const bool sampled = h->kind == KIND_MIXED || h->kind == KIND_SWITCH || h->kind == KIND_MUPPET;
    if (sampled && h->cfg.sample_ratio > 0.f) {
        uint64_t shortest = ~0ull;
        for (size_t sg = 0; sg + 1 < h->seg_off.size(); sg++)
            if (h->seg_off[sg + 1] > h->seg_off[sg]) shortest = std::min<uint64_t>(shortest, h->seg_off[sg + 1] - h->seg_off[sg]);
        limit = std::min<uint64_t>(limit, (uint64_t)((double)shortest * h->cfg.sample_ratio / 4.0));
    }
    while (w > 12 && (1ull << w) > limit) w--;
    return w <= 12 ? 0 : (int)w;
}

int muppet_bits(const mascot_handle* h);

// Loads and configures the update-kernel instantiations the first epochs will launch (the CUDA runtime loads
// a kernel at its first use, which otherwise costs the first epoch a few milliseconds).  The instantiations
// for promoted rows are left to their first use.
int warm_kernels(mascot_handle* h) {
    if (!h->n_train) return MASCOT_OK;
    Stream s; s.r = h->tr_r; s.u = h->tr_u; s.i = h->tr_i; s.n = h->n_train;
    const unsigned workers = worker_count(h, h->n_train);
    const RowClass cls = any_fp32_group(h) ? ROWCLASS_ANY : ROWCLASS_HH;
    SampleStats st = SampleStats();
    const bool sampled = h->kind == KIND_MIXED || h->kind == KIND_SWITCH || h->kind == KIND_MUPPET;
    for (int with_stats = 0; with_stats <= (sampled ? 1 : 0); with_stats++)
        CU(h, launch_train(h->K, h->kind, s, h->P, h->Q, 0.f, 0.f, with_stats ? &st : nullptr, cls, workers, nullptr, muppet_bits(h), 0,
                           h->cfg.plain_user_stores == 0, h->hot_user_shift, h->n_train, h->stream, nullptr));
    return MASCOT_OK;
}

// Sorts the freshly encoded resident stream by item inside its run windows.
int sort_run_windows(mascot_handle* h) {
    const int w = run_window_log2(h);
    if (w == 0 || h->n_train == 0) return MASCOT_OK;
    NvtxRange range("mascot: item-sorted run windows");
    return sort_windows(h, w);
}

float reference_rmse_from_partials(const Results& part, uint64_t n) {
    float sum = 0;                                  // rmse.h:183-186: float accumulation in block order
    for (float v : part) sum += v;
    return (float)std::sqrt(sum / (double)n);       // rmse.h:188, returned through a float
}

}  // namespace

extern "C" {

int mascot_abi_info(uint32_t* abi_version, uint32_t* config_bytes, uint32_t* epoch_stats_bytes) {
    if (abi_version) *abi_version = MASCOT_ABI_VERSION;
    if (config_bytes) *config_bytes = (uint32_t)sizeof(mascot_config);
    if (epoch_stats_bytes) *epoch_stats_bytes = (uint32_t)sizeof(mascot_epoch_stats);
    return MASCOT_OK;
}

int mascot_config_default(mascot_config* cfg) {
    if (!cfg) return MASCOT_ERR_BAD_ARG;
    std::memset(cfg, 0, sizeof(*cfg));
    cfg->lambda = 0.015f; cfg->learning_rate = 0.01f; cfg->decay = 0.1f; cfg->sample_ratio = 0.01f;
    cfg->error_threshold = 0.001f; cfg->interval = 1; cfg->user_group_num = 10; cfg->item_group_num = 10;
    cfg->k = 128; cfg->num_workers = 2048; cfg->epoch = 50; cfg->thread_block_size = 128; cfg->version = 7;
    cfg->shuffle = 1; cfg->seed = 1; cfg->device = 0;
    return MASCOT_OK;
}

const char* mascot_status_string(int s) {
    switch (s) {
        case MASCOT_OK: return "ok";
        case MASCOT_ERR_BAD_ARG: return "bad argument";
        case MASCOT_ERR_CUDA: return "CUDA error";
        case MASCOT_ERR_OOM: return "out of memory";
        case MASCOT_ERR_STATE: return "call order violated";
        case MASCOT_ERR_NO_DEVICE: return "no usable CUDA device";
        case MASCOT_ERR_TIMEOUT: return "timed out";
        case MASCOT_ERR_UNSUPPORTED: return "unsupported";
        case MASCOT_ERR_COMM: return "communication failure";
    }
    return "unknown status";
}

const char* mascot_last_error(const mascot_handle* h) { return h ? h->err.c_str() : g_create_error.c_str(); }

int mascot_create(const mascot_config* cfg, mascot_handle** out) {
    if (!cfg || !out) return fail(nullptr, MASCOT_ERR_BAD_ARG, "null config or output pointer");
    *out = nullptr;
    if (cfg->k != 64 && cfg->k != 128) return fail(nullptr, MASCOT_ERR_BAD_ARG, "k must be 64 or 128");
    if (cfg->epoch == 0) return fail(nullptr, MASCOT_ERR_BAD_ARG, "epoch count must be positive");
    TrainKind kind;
    switch (cfg->version) {
        case MASCOT_V_MASCOT: kind = KIND_MIXED; break;
        case MASCOT_V_SGD: kind = KIND_FP32; break;
        case MASCOT_V_MPT: kind = KIND_MPT; break;
        case MASCOT_V_MEMQUANT: kind = KIND_MEMQUANT; break;
        case MASCOT_V_NAIVE: kind = KIND_MIXED; break;
        case MASCOT_V_SWITCH_ONLY: kind = KIND_SWITCH; break;
        case MASCOT_V_MUPPET: kind = KIND_MUPPET; break;
        case MASCOT_V_AFP: kind = KIND_AFP; break;
        default: return fail(nullptr, MASCOT_ERR_BAD_ARG, "unknown training variant");
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return fail(nullptr, MASCOT_ERR_NO_DEVICE, "no CUDA device is visible; libmascot has no CPU path");
    }
    if (cfg->device < 0 || cfg->device >= ndev) return fail(nullptr, MASCOT_ERR_NO_DEVICE, "requested CUDA device does not exist");
    mascot_handle* h = new (std::nothrow) mascot_handle();
    if (!h) return fail(nullptr, MASCOT_ERR_OOM, "host allocation failed");
    h->cfg = *cfg; h->K = (int)cfg->k; h->kind = kind; h->grouped = (cfg->version == MASCOT_V_MASCOT || cfg->version == MASCOT_V_NAIVE);
    h->mup_idx = cfg->is_yahoo ? 1 : 0;            // mf_methods.cu:600-601
    for (int j = 0; j < 5; j++) if (cfg->muppet_width == (uint32_t)muppet_width_at(j)) h->mup_idx = j;
    h->lr.resize(cfg->epoch);
    for (uint32_t e = 0; e < cfg->epoch; e++) h->lr[e] = lr_at(*cfg, e);
    cudaError_t e = cudaSetDevice(cfg->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    for (int j = 0; j < 4 && e == cudaSuccess; j++) e = cudaEventCreate(&h->ev[j]);
    if (e == cudaSuccess) e = dev_alloc(&h->counters.d_slots, 4, h->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(h->counters.d_slots, 0, 4 * sizeof(unsigned long long), h->stream);
    if (e != cudaSuccess) {
        std::string msg = std::string("CUDA set-up failed: ") + cudaGetErrorString(e);
        mascot_destroy(h);
        return fail(nullptr, MASCOT_ERR_CUDA, msg);
    }
    *out = h;
    return MASCOT_OK;
}

int mascot_destroy(mascot_handle* h) {
    if (!h) return MASCOT_OK;
    cudaSetDevice(h->cfg.device);
    l2_window_remove(h);
    free_ratings(h);
    shard_destroy(h);
    if (h->stream) cudaStreamSynchronize(h->stream);       // the staging buffers below are freed on the other stream
    dev_free(h->d_scratch, h->stream); dev_free(h->counters.d_slots, h->stream); dev_free(h->d_err_flag, h->stream);
    for (auto& ev : h->ev) if (ev) cudaEventDestroy(ev);
    for (int b = 0; b < 2; b++) {
        if (h->ev_copied[b]) cudaEventDestroy(h->ev_copied[b]);
        if (h->ev_free[b]) cudaEventDestroy(h->ev_free[b]);
        dev_free(h->d_stage[b], h->copy_stream);
    }
    if (h->copy_stream) cudaStreamDestroy(h->copy_stream);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return MASCOT_OK;
}

int mascot_set_ratings(mascot_handle* h, const mascot_rating* train, uint64_t n_train,
                       const mascot_rating* test, uint64_t n_test, uint32_t n_users, uint32_t n_items) {
    return mascot_set_ratings_sharded(h, train, n_train, nullptr, 1, test, n_test, n_users, n_items, nullptr, nullptr);
}

int mascot_set_ratings_sharded(mascot_handle* h, const mascot_rating* train, uint64_t n_train,
                               const uint64_t* segment_offsets, uint32_t n_segments,
                               const mascot_rating* test, uint64_t n_test, uint32_t n_users, uint32_t n_items,
                               const uint32_t* user_degree, const uint32_t* item_degree) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (h->shard) return fail(h, MASCOT_ERR_STATE, "this engine belongs to a sharded group: use mascot_shard_set_ratings");
    SetupRequest rq;
    rq.train = train; rq.n_train = n_train; rq.segment_offsets = segment_offsets; rq.n_segments = n_segments;
    rq.test = test; rq.n_test = n_test; rq.n_users = n_users; rq.n_items = n_items;
    rq.user_degree = user_degree; rq.item_degree = item_degree;
    return setup_ratings(h, rq);
}

int mascot_reload_train(mascot_handle* h, const mascot_rating* train, uint64_t n_train) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!train && n_train) return fail(h, MASCOT_ERR_BAD_ARG, "null rating array");
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    if (n_train >= (1ull << 32)) return fail(h, MASCOT_ERR_BAD_ARG, "too many ratings (limit 2^32 - 1 per engine)");
    CU(h, cudaSetDevice(h->cfg.device));
    if (n_train != h->n_train) {
        CU(h, reserve(h, &h->tr_r, n_train)); CU(h, reserve(h, &h->tr_u, n_train)); CU(h, reserve(h, &h->tr_i, n_train));
        CU(h, reserve(h, &h->tr_src, n_train));
        h->n_train = n_train;
        h->seg_off.assign({0, n_train});           // a stream of another length is one segment
        h->stream_is_new();
    }
    if (!n_train) return MASCOT_OK;
    const size_t bytes = sizeof(mascot_rating) * n_train, sort_at = (bytes + 255) / 256 * 256;
    const int run_window = run_window_log2(h), nseg = (int)h->seg_off.size() - 1;
    const size_t sort_bytes = source_sort_bytes(n_train, h->seg_off.data(), nseg, run_window, h->irows);
    int rc = need_scratch(h, sort_at + sort_bytes);
    if (rc != MASCOT_OK) return rc;
    CU(h, cudaMemsetAsync(h->d_err_flag, 0, sizeof(uint32_t), h->stream));
    CU(h, copy_to_device(h->d_scratch, train, bytes, h->stream));
    if (sort_bytes)
        CU(h, launch_source_sort(h->d_scratch, n_train, h->seg_off.data(), nseg, h->cfg.seed, run_window, h->irows, h->d_umap, h->d_imap, h->d_uprec_row, h->d_iprec_row,
                                 h->n_users, h->n_items, h->d_err_flag, static_cast<unsigned char*>(h->d_scratch) + sort_at, nullptr, h->tr_r, h->tr_u, h->tr_i, h->tr_src, h->stream));
    else
        CU(h, encode_segments(h, static_cast<const mascot_rating*>(h->d_scratch), h->seg_off, h->cfg.shuffle != 0,
                              h->tr_r, h->tr_u, h->tr_i, h->tr_src));
    uint32_t bad = 0;
    CU(h, cudaMemcpyAsync(&bad, h->d_err_flag, sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream));
    h->stream_is_new();
    if (!sort_bytes && (rc = sort_run_windows(h)) != MASCOT_OK) return rc;
    if ((rc = partition_all(h)) != MASCOT_OK) return rc;      // the new stream carries the current precisions
    CU(h, cudaStreamSynchronize(h->stream));
    if (bad) return fail(h, MASCOT_ERR_BAD_ARG, "training rating with id out of range (replaced by zero ratings of row 0; reload a valid array)");
    return MASCOT_OK;
}

static int scatter_from_device(mascot_handle* h, const float* dP, const float* dQ) {
    const double t0 = now_us();
    const bool through_half = (h->kind == KIND_MPT);   // MPT masters start from fp16 values (mf_methods.cu:730-733)
    CU(h, launch_scatter_factors(h->K, dP, h->n_users, h->d_umap, through_half, h->P.f16, h->P.f32, h->stream));
    CU(h, launch_scatter_factors(h->K, dQ, h->n_items, h->d_imap, through_half, h->Q.f16, h->Q.f32, h->stream));
    CU(h, cudaStreamSynchronize(h->stream));
    h->timings.copy_to_grouped_us += now_us() - t0;
    h->have_factors = true;
    return l2_window_install(h);
}

// Both factor matrices as fp32 rows in the scratch buffer: what set_factors uploads, init_factors fills and
// get_factors collects.
static int factor_scratch(mascot_handle* h, float** dP, float** dQ) {
    const size_t pu = ((size_t)h->n_users * h->K + 63) / 64 * 64, qi = (size_t)h->n_items * h->K;
    const int rc = need_scratch(h, sizeof(float) * (pu + qi));
    if (rc != MASCOT_OK) return rc;
    *dP = static_cast<float*>(h->d_scratch);
    *dQ = *dP + pu;
    return MASCOT_OK;
}

int mascot_set_factors(mascot_handle* h, const float* P, const float* Q) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!P || !Q) return fail(h, MASCOT_ERR_BAD_ARG, "null factor matrix");
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    CU(h, cudaSetDevice(h->cfg.device));
    float *dP = nullptr, *dQ = nullptr;
    const int rc = factor_scratch(h, &dP, &dQ);
    if (rc != MASCOT_OK) return rc;
    CU(h, copy_to_device(dP, P, sizeof(float) * (size_t)h->n_users * h->K, h->stream));
    CU(h, copy_to_device(dQ, Q, sizeof(float) * (size_t)h->n_items * h->K, h->stream));
    return scatter_from_device(h, dP, dQ);
}

int mascot_init_factors(mascot_handle* h) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    CU(h, cudaSetDevice(h->cfg.device));
    float *dP = nullptr, *dQ = nullptr;
    const int rc = factor_scratch(h, &dP, &dQ);
    if (rc != MASCOT_OK) return rc;
    CU(h, launch_init_normal(dP, (size_t)h->n_users * h->K, h->cfg.seed, 1, h->stream));
    CU(h, launch_init_normal(dQ, (size_t)h->n_items * h->K, h->cfg.seed, 2, h->stream));
    return scatter_from_device(h, dP, dQ);
}

}  // extern "C"

namespace mascot {

unsigned worker_count(const mascot_handle* h, uint64_t n) {
    // -wg 0 = automatic: one worker per 8192 ratings keeps the sequential depth per worker - and with
    // it the convergence per epoch - at the level of the reference's tuned runs; the launch caps the
    // count at what the GPU can keep resident.  Small sets (under 1.5M ratings) would leave most SMs
    // idle at that rate: they get one worker per 512 ratings, at most 1536 (measured on the 0.8M-rating
    // configuration: final RMSE still below the reference's, three times the throughput of 512 workers).
    if (h->cfg.deterministic) return 1u;
    if (h->cfg.num_workers) return h->cfg.num_workers;
    if (h->shard) return shard_worker_count(h);
    if (n < 1500000) return (unsigned)std::min<uint64_t>(std::max<uint64_t>(n / 512, 512), 1536);
    uint64_t w = std::min<uint64_t>(std::max<uint64_t>(n / 8192, 512), 1u << 20);
    return (unsigned)w;
}

// Width of MuPPET's forward and backward pass this epoch (mf_methods.cu:597, 623-624).
int muppet_bits(const mascot_handle* h) { return muppet_width_at(h->mup_idx); }

// MuPPET's switching rule after epoch e (mf_methods.cu:586-595, 660-695): over the last three epochs,
// gradient diversity = sum of the sampled squared gradient norms / squared norm of the summed sampled
// updates; when the largest diversity seen since the last switch exceeds the current one by more than a
// decaying threshold, the next wider format is used from the next epoch on.
void muppet_policy(mascot_handle* h, uint32_t epoch) {
    const int K = h->K, e = (int)epoch, resolution = 3;
    const float alpha = 1.0f, beta = 1.5f, lambda_thr = 0.3f;
    const float threshold = alpha + (beta * std::exp(-1 * lambda_thr * (e)));
    if ((int)h->mup_norms_epoch.size() <= e) { h->mup_norms_epoch.resize(e + 1, 0.f); h->mup_sums_epoch.resize((size_t)(e + 1) * K, 0.f); }
    h->mup_norms_epoch[e] = h->h_stats[(size_t)2 * K];                       // nsum_p[0]
    std::copy(h->h_stats.begin(), h->h_stats.begin() + K, h->mup_sums_epoch.begin() + (size_t)e * K);
    if (e - h->mup_switched_epoch < resolution) return;
    float norms = 0.f, sq = 0.f;
    std::vector<float> acc(K, 0.f);
    for (int w = e - resolution + 1; w <= e; w++) {
        norms += h->mup_norms_epoch[w];
        for (int d = 0; d < K; d++) acc[d] += h->mup_sums_epoch[(size_t)w * K + d];
    }
    for (int d = 0; d < K; d++) sq += powf(acc[d], 2);
    const float diversity = norms / sq;
    h->mup_max_diversity = h->mup_max_diversity < diversity ? diversity : h->mup_max_diversity;
    const float ratio = h->mup_max_diversity / diversity;
    if (ratio > threshold && ++h->mup_violations == 1) {
        if (h->mup_idx < 4) h->mup_idx++;
        h->mup_switched_epoch = e;
        h->mup_max_diversity = -1.f;
        h->mup_violations = 0;
    }
}

int promote_groups(mascot_handle* h, bool users, size_t g, size_t last);
int recode_side(mascot_handle* h, bool users);

// Whole-model switching trainer after a check epoch (mf_methods.cu:1515-1545): error = squared norm of
// the summed sampled updates / sum of their squared norms, relative to its value at epoch index 5;
// above the threshold every row is widened to fp32 and the fp32 trainer takes over.
int switch_only_policy(mascot_handle* h, uint32_t epoch, uint32_t* promoted_u, uint32_t* promoted_i) {
    const int K = h->K;
    float sq = 0.f;
    for (int d = 0; d < K; d++) sq += powf(h->h_stats[d], 2);
    float error = sq / h->h_stats[(size_t)2 * K];
    error = error / h->switch_initial_error;
    h->uerr[0] = error; h->ierr[0] = error;
    if (epoch == 5) h->switch_initial_error = error;
    if (epoch > 5 && error > h->cfg.error_threshold) {
        int rc;
        if ((rc = promote_groups(h, true, 0, 0)) != MASCOT_OK) return rc;
        if ((rc = promote_groups(h, false, 0, 0)) != MASCOT_OK) return rc;
        if ((rc = recode_side(h, true)) != MASCOT_OK) return rc;
        if ((rc = recode_side(h, false)) != MASCOT_OK) return rc;
        h->switched_to_fp32 = true;
        *promoted_u = 1; *promoted_i = 1;
    }
    return MASCOT_OK;
}

SampleStats stats_view(mascot_handle* h) {
    const int ug = (int)h->uend.size(), ig = (int)h->iend.size(), K = h->K;
    SampleStats st;
    st.ugroup = h->d_ugroup; st.igroup = h->d_igroup; st.ug = ug; st.ig = ig;
    st.gsum_p = h->d_stats; st.gsum_q = st.gsum_p + (size_t)ug * K;
    st.nsum_p = st.gsum_q + (size_t)ig * K; st.nsum_q = st.nsum_p + ug;
    st.copies = h->stats_copies; st.copy_stride = h->stats_stride;
    st.first_sample_pos = 0;
    return st;
}

// Runs the update kernel over stream positions [begin, end), all of whose ratings are of row class
// `cls`.  With `collect`, the last sample_ratio of the range (mf_methods.cu:102-103, 173-174) goes
// through the statistics kernel - a second launch, so that only the sampled fraction pays for the
// statistics.  `whole`: ratings of the epoch or segment that the range is a part of, for which the workers were counted.
int train_span(mascot_handle* h, float lr, uint32_t epoch, uint64_t begin, uint64_t end, RowClass cls, bool collect,
               LaunchShape* shape, uint32_t* launches, unsigned workers, uint64_t whole, cudaStream_t stream, WorkCounters* counters) {
    if (end <= begin) return MASCOT_OK;
    const uint64_t n = end - begin;
    // after its switch the whole-model switching trainer is the plain fp32 trainer (sgd_kernel.h:296-326)
    const TrainKind kind = (h->kind == KIND_SWITCH && h->switched_to_fp32) ? KIND_FP32 : h->kind;
    Stream s; s.r = h->tr_r + begin; s.u = h->tr_u + begin; s.i = h->tr_i + begin; s.n = n;
    uint64_t head = n;
    if (collect) {
        const uint64_t sample_num = (uint64_t)((float)n * h->cfg.sample_ratio);
        head = n - std::min<uint64_t>(sample_num, n);
    }
    if (head > 0) {
        Stream sa = s; sa.n = head;
        CU(h, launch_train(h->K, kind, sa, h->P, h->Q, lr, h->cfg.lambda, nullptr, cls, workers,
                           counters, muppet_bits(h), (int)epoch, h->cfg.plain_user_stores == 0, h->hot_user_shift, whole, stream, shape));
        (*launches)++;
    }
    if (head < n) {
        Stream sb; sb.r = s.r + head; sb.u = s.u + head; sb.i = s.i + head; sb.n = n - head;
        const SampleStats st = stats_view(h);
        LaunchShape tail_shape;            // the caller is told the shape of the plain launch when there is one
        CU(h, launch_train(h->K, kind, sb, h->P, h->Q, lr, h->cfg.lambda, &st, cls, workers,
                           counters, muppet_bits(h), (int)epoch, h->cfg.plain_user_stores == 0, h->hot_user_shift, whole, stream, head > 0 ? &tail_shape : shape));
        (*launches)++;
    }
    return MASCOT_OK;
}

// One segment of the stream: a single launch while every row is binary16 (or when the stream is not
// partitioned: the launch then reads each id's precision bit), else one launch per non-empty precision
// class, one after the other.  (Running the classes side by side on streams of their own, each with a
// share of the workers, was measured too: 15.7 ms per promoted epoch on the 100M-rating set against 14.0 ms
// one after the other.)  On a check epoch every launched range contributes its own sampled tail.  `policy_n` (0 = the segment's
// own length) is the stream length the automatic worker count is taken from.
int train_range(mascot_handle* h, float lr, uint32_t epoch, size_t segment, bool collect, LaunchShape* shape, uint32_t* launches,
                uint64_t policy_n) {
    const uint64_t begin = h->seg_off[segment], end = h->seg_off[segment + 1];
    if (!policy_n) policy_n = end - begin;
    const unsigned workers = worker_count(h, policy_n);
    if (!h->partitioned)
        return train_span(h, lr, epoch, begin, end, any_fp32_group(h) ? ROWCLASS_ANY : ROWCLASS_HH, collect, shape, launches, workers, policy_n,
                          h->stream, &h->counters);
    const uint64_t* off = &h->cls_off[segment * 5];
    for (int c = 0; c < 4; c++) {
        const int rc = train_span(h, lr, epoch, off[c], off[c + 1], (RowClass)c, collect, shape, launches, workers, policy_n, h->stream, &h->counters);
        if (rc != MASCOT_OK) return rc;
    }
    return MASCOT_OK;
}

// Folds the private accumulator sets and brings the sums to the host in LOGICAL element order.
int fetch_stats(mascot_handle* h, uint32_t* launches) {
    const int ug = (int)h->uend.size(), ig = (int)h->iend.size(), K = h->K;
    const double t0 = now_us();
    if (h->stats_copies > 1) {
        CU(h, launch_reduce_stats(h->d_stats, h->stats_copies, h->stats_stride, stats_floats(h), h->stream));
        if (launches) (*launches)++;
    }
    std::vector<float> raw(stats_floats(h));
    CU(h, cudaMemcpyAsync(raw.data(), h->d_stats, sizeof(float) * raw.size(), cudaMemcpyDeviceToHost, h->stream));
    CU(h, cudaStreamSynchronize(h->stream));
    for (size_t g = 0; g < (size_t)(ug + ig); g++)
        for (int p = 0; p < K; p++) h->h_stats[g * K + logical_of_phys(K, p)] = raw[g * K + p];
    std::copy(raw.begin() + (size_t)(ug + ig) * K, raw.end(), h->h_stats.begin() + (size_t)(ug + ig) * K);
    h->timings.error_computation_us += now_us() - t0;
    return MASCOT_OK;
}

// Group errors from the sums in h->h_stats and the switching that follows (mf_methods.cu:325-393,
// precision_switching.h:8-51).
int apply_stats(mascot_handle* h, uint32_t epoch, uint32_t* promoted_u, uint32_t* promoted_i, uint32_t* launches) {
    NvtxRange range("mascot: group errors and precision switching");
    const int ug = (int)h->uend.size(), ig = (int)h->iend.size(), K = h->K;
    const double t_err = now_us();
    auto errors = [&](int groups, const float* gsum, const float* nsum, const std::vector<uint8_t>& prec,
                      const std::vector<float>& initial, std::vector<float>& err) {
        for (int g = 0; g < groups; g++) {
            if (prec[g]) { err[g] = -1.f; continue; }
            float num = 0.f;
            for (int d = 0; d < K; d++) num += powf(gsum[(size_t)g * K + d], 2);
            const float den = nsum[g];
            err[g] = (num / den) / initial[g];
        }
    };
    const float* gs_p = h->h_stats.data(); const float* gs_q = gs_p + (size_t)ug * K;
    const float* ns_p = gs_q + (size_t)ig * K; const float* ns_q = ns_p + ug;
    errors(ug, gs_p, ns_p, h->uprec, h->init_uerr, h->uerr);
    errors(ig, gs_q, ns_q, h->iprec, h->init_ierr, h->ierr);
    if (epoch == 5) { h->init_uerr = h->uerr; h->init_ierr = h->ierr; }   // mf_methods.cu:381-388
    h->timings.error_computation_us += now_us() - t_err;
    if (epoch > 5) {
        int rc;
        const double t_sw = now_us();
        for (int side = 0; side < 2; side++) {
            const bool users = side == 0;
            const std::vector<uint8_t>& prec = users ? h->uprec : h->iprec;
            const std::vector<float>& err = users ? h->uerr : h->ierr;
            uint32_t& count = users ? *promoted_u : *promoted_i;
            // neighbouring groups are one range of rows: a launch for each run of them
            for (size_t g = 0; g < prec.size(); g++) {
                size_t last = g;
                auto due = [&](size_t j) { return j < prec.size() && err[j] > h->cfg.error_threshold && !prec[j]; };
                if (!due(g)) continue;
                while (due(last + 1)) last++;
                if ((rc = promote_groups(h, users, g, last)) != MASCOT_OK) return rc;
                count += (uint32_t)(last - g + 1); if (launches) (*launches)++;
                g = last;
            }
            if (count) {
                if ((rc = recode_side(h, users)) != MASCOT_OK) return rc;
                if (launches) (*launches) += 2;
            }
        }
        if (*promoted_u + *promoted_i) {
            if ((rc = partition_all(h)) != MASCOT_OK) return rc;
            if (launches && h->partitioned) (*launches) += 4;
            CU(h, cudaStreamSynchronize(h->stream));
        }
        h->timings.precision_switching_us += now_us() - t_sw;
    }
    return MASCOT_OK;
}

}  // namespace

extern "C" {

int mascot_is_check_epoch(const mascot_handle* h, uint32_t epoch) {
    return (h && h->grouped && is_check_epoch(h->cfg, epoch)) ? 1 : 0;
}

int mascot_stats_begin(mascot_handle* h) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    CU(h, cudaSetDevice(h->cfg.device));
    CU(h, cudaMemsetAsync(h->d_stats, 0, sizeof(float) * h->stats_stride * h->stats_copies, h->stream));   // mf_methods.cu:178-182
    return MASCOT_OK;
}

int mascot_train_segment(mascot_handle* h, uint32_t epoch, uint32_t segment, uint32_t collect_stats, mascot_epoch_stats* out) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings || !h->have_factors) return fail(h, MASCOT_ERR_STATE, "ratings and factors must be set before training");
    if (segment + 1 >= h->seg_off.size()) return fail(h, MASCOT_ERR_BAD_ARG, "segment index out of range");
    CU(h, cudaSetDevice(h->cfg.device));
    const float lr = epoch < h->lr.size() ? h->lr[epoch] : lr_at(h->cfg, epoch);
    LaunchShape shape; uint32_t launches = 0;
    CU(h, cudaEventRecord(h->ev[0], h->stream));
    const int rc = train_range(h, lr, epoch, segment, collect_stats && h->grouped, &shape, &launches);
    if (rc != MASCOT_OK) return rc;
    CU(h, cudaEventRecord(h->ev[3], h->stream));
    if (out) {
        CU(h, cudaEventSynchronize(h->ev[3]));
        std::memset(out, 0, sizeof(*out));
        out->updates = h->seg_off[segment + 1] - h->seg_off[segment]; out->lr = lr; out->kernel_launches = launches;
        out->workers = shape.workers; out->error_check = (collect_stats && h->grouped) ? 1 : 0;
        cudaEventElapsedTime(&out->kernel_ms, h->ev[0], h->ev[3]);
        out->total_ms = out->kernel_ms;
    }
    return MASCOT_OK;
}

int mascot_stats_fetch(mascot_handle* h, float* grad_sum_p, float* grad_sum_q, float* norm_sum_p, float* norm_sum_q) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    CU(h, cudaSetDevice(h->cfg.device));
    const int rc = fetch_stats(h, nullptr);
    if (rc != MASCOT_OK) return rc;
    return mascot_get_sample_stats(h, grad_sum_p, grad_sum_q, norm_sum_p, norm_sum_q);
}

int mascot_stats_apply(mascot_handle* h, uint32_t epoch, const float* grad_sum_p, const float* grad_sum_q,
                       const float* norm_sum_p, const float* norm_sum_q, uint32_t* promoted_user_groups, uint32_t* promoted_item_groups) {
    if (!h || !grad_sum_p || !grad_sum_q || !norm_sum_p || !norm_sum_q) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings || !h->have_factors) return fail(h, MASCOT_ERR_STATE, "ratings and factors must be set first");
    CU(h, cudaSetDevice(h->cfg.device));
    const size_t ug = h->uend.size(), ig = h->iend.size(), K = h->K;
    float* s = h->h_stats.data();
    std::copy(grad_sum_p, grad_sum_p + ug * K, s);
    std::copy(grad_sum_q, grad_sum_q + ig * K, s + ug * K);
    std::copy(norm_sum_p, norm_sum_p + ug, s + (ug + ig) * K);
    std::copy(norm_sum_q, norm_sum_q + ig, s + (ug + ig) * K + ug);
    uint32_t pu = 0, pi = 0;
    const int rc = apply_stats(h, epoch, &pu, &pi, nullptr);
    if (rc != MASCOT_OK) return rc;
    CU(h, cudaStreamSynchronize(h->stream));
    if (promoted_user_groups) *promoted_user_groups = pu;
    if (promoted_item_groups) *promoted_item_groups = pi;
    return MASCOT_OK;
}

int mascot_train_epoch(mascot_handle* h, uint32_t epoch, mascot_epoch_stats* out) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (h->shard) return fail(h, MASCOT_ERR_STATE, "this engine belongs to a sharded group: use mascot_shard_train_epoch");
    if (!h->have_ratings || !h->have_factors) return fail(h, MASCOT_ERR_STATE, "ratings and factors must be set before training");
    NvtxRange range("mascot_train_epoch");
    CU(h, cudaSetDevice(h->cfg.device));
    const float lr = epoch < h->lr.size() ? h->lr[epoch] : lr_at(h->cfg, epoch);
    const bool muppet = h->kind == KIND_MUPPET;
    const int bits_this_epoch = muppet ? muppet_bits(h) : 0;
    // MuPPET samples every epoch (its statistics feed the width policy), MASCOT on its check epochs
    const bool switch_only = h->kind == KIND_SWITCH;
    const bool check = muppet || ((h->grouped || (switch_only && !h->switched_to_fp32)) && is_check_epoch(h->cfg, epoch));
    uint32_t launches = 0, promoted_u = 0, promoted_i = 0;
    const uint64_t bytes_this_epoch = algorithmic_bytes(h);    // with the precisions the kernel is about to see
    // An epoch without statistics is its update kernels: two events time both the kernels and the whole (each event and
    // each reading of one costs the host one to two microseconds, of the 160 of an epoch of the smallest configuration).
    if (check) CU(h, cudaEventRecord(h->ev[0], h->stream));
    if (check) CU(h, cudaMemsetAsync(h->d_stats, 0, sizeof(float) * h->stats_stride * h->stats_copies, h->stream));   // mf_methods.cu:178-182
    CU(h, cudaEventRecord(h->ev[1], h->stream));
    LaunchShape shape;
    int rc;
    for (size_t sgm = 0; sgm + 1 < h->seg_off.size(); sgm++)
        if ((rc = train_range(h, lr, epoch, sgm, check, &shape, &launches)) != MASCOT_OK) return rc;
    if (check && h->stats_copies > 1) {
        CU(h, launch_reduce_stats(h->d_stats, h->stats_copies, h->stats_stride, stats_floats(h), h->stream));
        launches++;
    }
    CU(h, cudaEventRecord(h->ev[2], h->stream));
    if (check) {
        const int saved = h->stats_copies;
        h->stats_copies = 1;                      // already folded above, inside the timed kernel span
        rc = fetch_stats(h, nullptr);
        h->stats_copies = saved;
        if (rc != MASCOT_OK) return rc;
        if (muppet) muppet_policy(h, epoch);
        else if (switch_only) { if ((rc = switch_only_policy(h, epoch, &promoted_u, &promoted_i)) != MASCOT_OK) return rc; }
        else if ((rc = apply_stats(h, epoch, &promoted_u, &promoted_i, &launches)) != MASCOT_OK) return rc;
    }
    if (check) CU(h, cudaEventRecord(h->ev[3], h->stream));
    CU(h, cudaEventSynchronize(h->ev[check ? 3 : 2]));
    float kernel_ms = 0.f, total_ms = 0.f;
    if (cudaEventElapsedTime(&kernel_ms, h->ev[1], h->ev[2]) == cudaSuccess) h->timings.update_us += 1e3 * kernel_ms;
    total_ms = kernel_ms;
    if (check && out) cudaEventElapsedTime(&total_ms, h->ev[0], h->ev[3]);
    if (out) {
        std::memset(out, 0, sizeof(*out));
        out->updates = h->n_train; out->lr = lr; out->error_check = check ? 1 : 0; out->pass_bits = (uint32_t)bits_this_epoch;
        out->promoted_user_groups = promoted_u; out->promoted_item_groups = promoted_i; out->kernel_launches = launches;
        out->algorithmic_bytes = bytes_this_epoch;
        out->workers = shape.workers;
        out->kernel_ms = kernel_ms;
        out->total_ms = total_ms;
    }
    return MASCOT_OK;
}

int mascot_train_epoch_streamed(mascot_handle* h, uint32_t epoch, const mascot_rating* train, uint64_t n_train, mascot_epoch_stats* out) {
    if (!h || (!train && n_train)) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings || !h->have_factors) return fail(h, MASCOT_ERR_STATE, "ratings and factors must be set before training");
    if (h->kind == KIND_AFP) return fail(h, MASCOT_ERR_UNSUPPORTED, "the AFP trainer keeps its per-worker state for a whole epoch: use mascot_train_epoch");
    if (h->shard) return fail(h, MASCOT_ERR_STATE, "this engine belongs to a sharded group: use mascot_shard_train_epoch");
    CU(h, cudaSetDevice(h->cfg.device));
    constexpr uint64_t kPiece = 8ull << 20;           // ratings per piece (96 MiB of input)
    { const int rc_stream = need_copy_stream(h); if (rc_stream != MASCOT_OK) return rc_stream; }
    const uint64_t piece = std::min<uint64_t>(kPiece, std::max<uint64_t>(n_train, 1));
    if (h->stage_ratings < piece) {
        for (int b = 0; b < 2; b++) dev_free(h->d_stage[b], h->copy_stream);
        h->stage_ratings = 0;
        for (int b = 0; b < 2; b++) CU(h, dev_alloc(&h->d_stage[b], piece, h->copy_stream));
        h->stage_ratings = piece;
    }
    if (n_train != h->n_train) {
        CU(h, reserve(h, &h->tr_r, n_train)); CU(h, reserve(h, &h->tr_u, n_train)); CU(h, reserve(h, &h->tr_i, n_train));
        CU(h, reserve(h, &h->tr_src, n_train));
        h->n_train = n_train;
    }
    CU(h, cudaMemsetAsync(h->d_err_flag, 0, sizeof(uint32_t), h->stream));
    // The pieces become the segments of the resident stream (seeded permutation inside each piece).  Beyond two of them some are
    // smaller (multiples of 4096, the encoding kernel's windows).  Binary16 rows are coded and trained in 0.6 of the time of their
    // copy: what follows the end of the copy counts, and the last pieces are halves of what is left (27M ratings, MASCOT 6.91 -> 6.37 ms
    // per epoch, k=64 6.65 -> 6.07, fp16 storage 6.90 -> 6.35).  MuPPET takes longer than the copy: what comes before its start counts,
    // and its first pieces are an eighth, a quarter and a half (9.50 -> 9.02).  Trainers with fp32 rows take about as long as the copy
    // and lose in more launches what they gain (SGD 7.63, either way or both 7.60 to 7.73; promoted groups 7.78 and 7.86).
    const bool binary16 = (h->kind == KIND_MIXED || h->kind == KIND_MEMQUANT || h->kind == KIND_SWITCH) && !any_fp32_group(h);
    h->seg_off.clear();
    for (uint64_t off = 0, c = 0; off < n_train; c++) {
        h->seg_off.push_back(off);
        const uint64_t left = n_train - off;
        uint64_t len = std::min(piece, left);
        if (n_train > 2 * piece && !h->cfg.deterministic) {
            if (h->kind == KIND_MUPPET && c < 3) len = piece >> (3 - c);
            else if (binary16 && left <= 2 * piece && left > piece / 4) len = (left / 2 + 4095) / 4096 * 4096;
        }
        off += len;
    }
    h->seg_off.push_back(n_train);
    // The pieces are not partitioned by precision class: finding the class boundaries needs a read-back,
    // i.e. a host wait per piece, which would stall the upload pipeline.  With promoted groups every piece
    // runs the instantiation that reads each id's precision bit; its extra cost hides behind the upload.
    h->stream_is_new();

    const float lr = epoch < h->lr.size() ? h->lr[epoch] : lr_at(h->cfg, epoch);
    const bool muppet = h->kind == KIND_MUPPET;
    const int bits_this_epoch = muppet ? muppet_bits(h) : 0;
    const bool switch_only = h->kind == KIND_SWITCH;
    const bool check = muppet || ((h->grouped || (switch_only && !h->switched_to_fp32)) && is_check_epoch(h->cfg, epoch));
    uint32_t launches = 0, promoted_u = 0, promoted_i = 0;
    const uint64_t bytes_this_epoch = algorithmic_bytes(h);
    CU(h, cudaEventRecord(h->ev[0], h->stream));
    if (check) CU(h, cudaMemsetAsync(h->d_stats, 0, sizeof(float) * h->stats_stride * h->stats_copies, h->stream));
    CU(h, cudaEventRecord(h->ev[1], h->stream));
    LaunchShape shape;
    int rc;
    for (size_t c = 0; c + 1 < h->seg_off.size(); c++) {
        const int b = (int)(c & 1);
        const uint64_t off = h->seg_off[c], len = h->seg_off[c + 1] - off;
        if (c >= 2) CU(h, cudaStreamWaitEvent(h->copy_stream, h->ev_free[b], 0));
        CU(h, copy_to_device(h->d_stage[b], train + off, sizeof(mascot_rating) * len, h->copy_stream));
        CU(h, cudaEventRecord(h->ev_copied[b], h->copy_stream));
        CU(h, cudaStreamWaitEvent(h->stream, h->ev_copied[b], 0));
        CU(h, launch_encode_stream(h->d_stage[b], len, h->cfg.shuffle != 0, h->cfg.seed + 0x9e3779b97f4a7c15ull * c, h->d_umap, h->d_imap,
                                   h->d_uprec_row, h->d_iprec_row, h->n_users, h->n_items, h->irows, h->d_err_flag,
                                   h->tr_r + off, h->tr_u + off, h->tr_i + off, h->tr_src ? h->tr_src + off : nullptr, (uint32_t)off, h->stream));
        launches++;
        CU(h, cudaEventRecord(h->ev_free[b], h->stream));
        if ((rc = train_range(h, lr, epoch, c, check, &shape, &launches, n_train)) != MASCOT_OK) return rc;
    }
    if (check && h->stats_copies > 1) {
        CU(h, launch_reduce_stats(h->d_stats, h->stats_copies, h->stats_stride, stats_floats(h), h->stream));
        launches++;
    }
    CU(h, cudaEventRecord(h->ev[2], h->stream));
    if (check) {
        const int saved = h->stats_copies;
        h->stats_copies = 1;
        rc = fetch_stats(h, nullptr);
        h->stats_copies = saved;
        if (rc != MASCOT_OK) return rc;
        if (muppet) muppet_policy(h, epoch);
        else if (switch_only) { if ((rc = switch_only_policy(h, epoch, &promoted_u, &promoted_i)) != MASCOT_OK) return rc; }
        else if ((rc = apply_stats(h, epoch, &promoted_u, &promoted_i, &launches)) != MASCOT_OK) return rc;
    }
    uint32_t bad = 0;
    CU(h, cudaMemcpyAsync(&bad, h->d_err_flag, sizeof(uint32_t), cudaMemcpyDeviceToHost, h->stream));
    CU(h, cudaEventRecord(h->ev[3], h->stream));
    CU(h, cudaEventSynchronize(h->ev[3]));
    if (bad) return fail(h, MASCOT_ERR_BAD_ARG, "training rating with id out of range (it was trained as a zero rating of row 0)");
    if (out) {
        std::memset(out, 0, sizeof(*out));
        out->updates = n_train; out->lr = lr; out->error_check = check ? 1 : 0; out->pass_bits = (uint32_t)bits_this_epoch;
        out->promoted_user_groups = promoted_u; out->promoted_item_groups = promoted_i; out->kernel_launches = launches;
        out->algorithmic_bytes = bytes_this_epoch;
        out->workers = shape.workers;
        cudaEventElapsedTime(&out->kernel_ms, h->ev[1], h->ev[2]);
        cudaEventElapsedTime(&out->total_ms, h->ev[0], h->ev[3]);
    }
    { float kms = 0.f; if (cudaEventElapsedTime(&kms, h->ev[1], h->ev[2]) == cudaSuccess) h->timings.update_us += 1e3 * kms; }
    return MASCOT_OK;
}

int mascot_item_rows(mascot_handle* h, uint32_t row_begin, uint32_t row_end, void** f16_ptr, uint64_t* f16_bytes,
                     void** f32_ptr, uint64_t* f32_bytes) {
    if (!h || row_end < row_begin) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    if (row_end > h->n_items) return fail(h, MASCOT_ERR_BAD_ARG, "item row range out of bounds");
    if (h->ilay.parts > 1) return fail(h, MASCOT_ERR_UNSUPPORTED, "the items of a sharded engine are laid out block by block, not by sorted index");
    CU(h, cudaSetDevice(h->cfg.device));
    const void* const before[2] = {h->Q.f16, h->Q.f32};
    CU(h, pool_make_plain(reinterpret_cast<void**>(&h->Q.f16), h->reserved[&h->Q.f16], h->stream));
    CU(h, pool_make_plain(reinterpret_cast<void**>(&h->Q.f32), h->reserved[&h->Q.f32], h->stream));
    if (h->l2_window_set && (h->Q.f16 != before[0] || h->Q.f32 != before[1])) {
        l2_window_remove(h);
        const int rc = l2_window_install(h);
        if (rc != MASCOT_OK) return rc;
    }
    const size_t b = (size_t)row_begin * h->K, n = (size_t)(row_end - row_begin) * h->K;
    if (f16_ptr) *f16_ptr = h->Q.f16 ? (void*)(h->Q.f16 + b) : nullptr;
    if (f16_bytes) *f16_bytes = h->Q.f16 ? n * sizeof(__half) : 0;
    if (f32_ptr) *f32_ptr = h->Q.f32 ? (void*)(h->Q.f32 + b) : nullptr;
    if (f32_bytes) *f32_bytes = h->Q.f32 ? n * sizeof(float) : 0;
    return MASCOT_OK;
}

int mascot_get_timings(mascot_handle* h, mascot_timings* out) {
    if (!h || !out) return MASCOT_ERR_BAD_ARG;
    *out = h->timings;
    return MASCOT_OK;
}

int mascot_get_worker_count(mascot_handle* h, uint32_t* workers) {
    if (!h || !workers) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    *workers = worker_count(h, h->n_train);
    return MASCOT_OK;
}

int mascot_release_scratch(mascot_handle* h) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    CU(h, cudaSetDevice(h->cfg.device));
    CU(h, cudaStreamSynchronize(h->stream));
    dev_free(h->d_scratch, h->stream); h->scratch_bytes = 0;
    CU(h, cudaStreamSynchronize(h->stream));
    pool_trim();
    release_copy_rings();
    release_results();
    return MASCOT_OK;
}

int mascot_release_cached(void) {
    release_copy_rings();
    release_results();
    CU(nullptr, pool_trim_all());
    return MASCOT_OK;
}

int mascot_sync(mascot_handle* h) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    CU(h, cudaSetDevice(h->cfg.device));
    CU(h, cudaStreamSynchronize(h->stream));
    return MASCOT_OK;
}

int mascot_get_stream(mascot_handle* h, void** stream) {
    if (!h || !stream) return MASCOT_ERR_BAD_ARG;
    *stream = (void*)h->stream;
    return MASCOT_OK;
}

int mascot_eval_sq_error(mascot_handle* h, double* sum_sq, uint64_t* count) {
    if (!h || !sum_sq || !count) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings || !h->have_factors) return fail(h, MASCOT_ERR_STATE, "ratings and factors must be set before evaluation");
    *sum_sq = 0; *count = h->n_test;
    if (!h->n_test) return MASCOT_OK;
    CU(h, cudaSetDevice(h->cfg.device));
    Stream t; t.r = h->te_r; t.u = h->te_u; t.i = h->te_i; t.n = h->n_test;
    Results sums((h->n_test + 511) / 512, h->stream);
    CU(h, sums.status());
    CU(h, launch_rmse(h->K, t, h->P, h->Q, sums.device(), h->stream));
    CU(h, sums.wait());
    double s = 0;
    for (float v : sums) s += (double)v;
    *sum_sq = s;
    return MASCOT_OK;
}

int mascot_eval_rmse(mascot_handle* h, double* rmse) {
    if (!h || !rmse) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings || !h->have_factors) return fail(h, MASCOT_ERR_STATE, "ratings and factors must be set before evaluation");
    if (!h->n_test) return fail(h, MASCOT_ERR_STATE, "no test ratings were given");
    CU(h, cudaSetDevice(h->cfg.device));
    Stream t; t.r = h->te_r; t.u = h->te_u; t.i = h->te_i; t.n = h->n_test;
    Results sums((h->n_test + 511) / 512, h->stream);
    CU(h, sums.status());
    CU(h, launch_rmse(h->K, t, h->P, h->Q, sums.device(), h->stream));
    CU(h, sums.wait());
    *rmse = (double)reference_rmse_from_partials(sums, h->n_test);
    return MASCOT_OK;
}

int mascot_get_factors(mascot_handle* h, float* P, float* Q, int order) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!h->have_factors) return fail(h, MASCOT_ERR_STATE, "no factors yet");
    if (order != 0 && order != 1) return fail(h, MASCOT_ERR_BAD_ARG, "order must be 0 or 1");
    CU(h, cudaSetDevice(h->cfg.device));
    float *dP = nullptr, *dQ = nullptr;
    const int rc = factor_scratch(h, &dP, &dQ);
    if (rc != MASCOT_OK) return rc;
    CopySpan spans[2];
    int n = 0;
    if (P) {
        CU(h, launch_gather_factors(h->K, h->P, h->d_uprec_row, h->n_users, order == 0 ? h->d_umap : nullptr, h->ulay, dP, h->stream));
        spans[n++] = CopySpan{P, dP, sizeof(float) * (size_t)h->n_users * h->K};
    }
    if (Q) {
        CU(h, launch_gather_factors(h->K, h->Q, h->d_iprec_row, h->n_items, order == 0 ? h->d_imap : nullptr, h->ilay, dQ, h->stream));
        spans[n++] = CopySpan{Q, dQ, sizeof(float) * (size_t)h->n_items * h->K};
    }
    CU(h, copy_to_host(spans, n, h->stream));
    return MASCOT_OK;
}

int mascot_get_group_info(mascot_handle* h, int side, uint32_t* n_groups, uint32_t* end_idx, uint8_t* precision, float* error) {
    if (!h || (side != 0 && side != 1)) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    const std::vector<uint32_t>& end = side == 0 ? h->uend : h->iend;
    const std::vector<uint8_t>& prec = side == 0 ? h->uprec : h->iprec;
    const std::vector<float>& err = side == 0 ? h->uerr : h->ierr;
    if (n_groups) *n_groups = (uint32_t)end.size();
    if (end_idx) std::copy(end.begin(), end.end(), end_idx);
    if (precision) std::copy(prec.begin(), prec.end(), precision);
    if (error) std::copy(err.begin(), err.end(), error);
    return MASCOT_OK;
}

// id -> sorted index of both sides (either may be null), from the device's id -> arena row maps
static cudaError_t sorted_indices(mascot_handle* h, uint32_t* users, uint32_t* items) {
    if (h->sorted_space) {
        CopySpan spans[2];
        int n = 0;
        if (users) spans[n++] = CopySpan{users, h->d_umap, sizeof(uint32_t) * h->n_users};
        if (items) spans[n++] = CopySpan{items, h->d_imap, sizeof(uint32_t) * h->n_items};
        const cudaError_t e = copy_to_host(spans, n, h->stream);
        if (e != cudaSuccess) return e;
    }
    auto finish = [&](uint32_t* v, uint32_t n, const RowLayout& L) {
        if (!v || (h->sorted_space && L.parts <= 1)) return;           // the row is the sorted index
        for (uint32_t e = 0; e < n; e++) v[e] = h->sorted_space ? sorted_of_row(L, v[e]) : e;
    };
    finish(users, h->n_users, h->ulay);
    finish(items, h->n_items, h->ilay);
    return cudaSuccess;
}

int mascot_get_index_maps(mascot_handle* h, uint32_t* user2sorted, uint32_t* item2sorted) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    CU(h, cudaSetDevice(h->cfg.device));
    CU(h, sorted_indices(h, user2sorted, item2sorted));
    return MASCOT_OK;
}

int mascot_promote_group(mascot_handle* h, int side, uint32_t group) {
    if (!h || (side != 0 && side != 1)) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings || !h->have_factors) return fail(h, MASCOT_ERR_STATE, "ratings and factors must be set first");
    if (!h->grouped) return fail(h, MASCOT_ERR_UNSUPPORTED, "only the MASCOT variant stores groups in switchable precision");
    const bool users = side == 0;
    std::vector<uint8_t>& prec = users ? h->uprec : h->iprec;
    if (group >= prec.size()) return fail(h, MASCOT_ERR_BAD_ARG, "group index out of range");
    if (prec[group]) return MASCOT_OK;
    CU(h, cudaSetDevice(h->cfg.device));
    int rc = promote_groups(h, users, group, group);
    if (rc == MASCOT_OK) rc = recode_side(h, users);
    if (rc == MASCOT_OK) rc = partition_all(h);
    if (rc != MASCOT_OK) return rc;
    CU(h, cudaStreamSynchronize(h->stream));
    return MASCOT_OK;
}

int mascot_get_sample_stats(mascot_handle* h, float* grad_sum_p, float* grad_sum_q, float* norm_sum_p, float* norm_sum_q) {
    if (!h) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    const size_t ug = h->uend.size(), ig = h->iend.size(), K = h->K;
    const float* s = h->h_stats.data();
    if (grad_sum_p) std::copy(s, s + ug * K, grad_sum_p);
    if (grad_sum_q) std::copy(s + ug * K, s + (ug + ig) * K, grad_sum_q);
    if (norm_sum_p) std::copy(s + (ug + ig) * K, s + (ug + ig) * K + ug, norm_sum_p);
    if (norm_sum_q) std::copy(s + (ug + ig) * K + ug, s + (ug + ig) * K + ug + ig, norm_sum_q);
    return MASCOT_OK;
}

int mascot_get_test_ratings(mascot_handle* h, mascot_rating* out, int order) {
    if (!h || !out) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    if (order != 0 && order != 1) return fail(h, MASCOT_ERR_BAD_ARG, "order must be 0 or 1");
    CU(h, cudaSetDevice(h->cfg.device));
    const uint64_t n = h->n_test;
    std::vector<float> r(n); std::vector<uint32_t> u(n), i(n);
    const CopySpan spans[3] = {{r.data(), h->te_r, sizeof(float) * n}, {u.data(), h->te_u, sizeof(uint32_t) * n}, {i.data(), h->te_i, sizeof(uint32_t) * n}};
    CU(h, copy_to_host(spans, 3, h->stream));
    std::vector<uint32_t> s2u, s2i;
    if (order == 0 && h->sorted_space) {
        s2u.resize(h->n_users); s2i.resize(h->n_items);
        std::vector<uint32_t> u2s(h->n_users), i2s(h->n_items);
        CU(h, sorted_indices(h, u2s.data(), i2s.data()));
        for (uint32_t e = 0; e < h->n_users; e++) s2u[u2s[e]] = e;
        for (uint32_t e = 0; e < h->n_items; e++) s2i[i2s[e]] = e;
    }
    for (uint64_t j = 0; j < n; j++) {
        // the stream holds arena rows: back to sorted indices, then (order 0) to the caller's ids
        uint32_t uu = sorted_of_row(h->ulay, u[j] & kIdMask), ii = sorted_of_row(h->ilay, i[j] & kIdMask);
        if (!s2u.empty()) { uu = s2u[uu]; ii = s2i[ii]; }
        out[j].r = r[j]; out[j].u = uu; out[j].i = ii;
    }
    return MASCOT_OK;
}

int mascot_stream_source_index(const mascot_handle* h, uint64_t pos, uint64_t* src) {
    if (!h || !src) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings || pos >= h->n_train) return MASCOT_ERR_BAD_ARG;
    if (!h->cfg.shuffle) { *src = pos; return MASCOT_OK; }
    if (!h->tr_src) return MASCOT_ERR_UNSUPPORTED;       // streams of 2^32 ratings or more keep no map
    uint32_t v = 0;
    if (cudaSetDevice(h->cfg.device) != cudaSuccess ||
        cudaMemcpy(&v, h->tr_src + pos, sizeof(v), cudaMemcpyDeviceToHost) != cudaSuccess) return MASCOT_ERR_CUDA;
    *src = v;
    return MASCOT_OK;
}

int mascot_get_stream_order(mascot_handle* h, uint32_t* src_out) {
    if (!h || !src_out) return MASCOT_ERR_BAD_ARG;
    if (!h->have_ratings) return fail(h, MASCOT_ERR_STATE, "mascot_set_ratings must come first");
    if (!h->tr_src) return fail(h, MASCOT_ERR_UNSUPPORTED, "streams of 2^32 ratings or more keep no order map");
    CU(h, cudaSetDevice(h->cfg.device));
    const CopySpan span{src_out, h->tr_src, sizeof(uint32_t) * h->n_train};
    CU(h, copy_to_host(&span, 1, h->stream));
    return MASCOT_OK;
}

int mascot_rmse_device(const float* d_P, const float* d_Q, uint32_t k, const mascot_rating* d_test, uint64_t n_test, double* rmse) {
    if (!d_P || !d_Q || !d_test || !rmse || !n_test) return fail(nullptr, MASCOT_ERR_BAD_ARG, "null pointer or empty test set");
    if (k != 64 && k != 128) return fail(nullptr, MASCOT_ERR_BAD_ARG, "k must be 64 or 128");
    Results sums((n_test + 511) / 512, nullptr);
    CU(nullptr, sums.status());
    CU(nullptr, launch_rmse_plain((int)k, d_test, n_test, d_P, d_Q, 0, 0, sums.device(), nullptr, nullptr));
    CU(nullptr, sums.wait());
    *rmse = (double)reference_rmse_from_partials(sums, n_test);
    return MASCOT_OK;
}

int mascot_rmse_host(const float* P, uint32_t n_users, const float* Q, uint32_t n_items, uint32_t k,
                     const mascot_rating* test, uint64_t n_test, int device, double* rmse) {
    if (!P || !Q || !test || !rmse || !n_test || !n_users || !n_items) return fail(nullptr, MASCOT_ERR_BAD_ARG, "null pointer or empty input");
    if (k != 64 && k != 128) return fail(nullptr, MASCOT_ERR_BAD_ARG, "k must be 64 or 128");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return fail(nullptr, MASCOT_ERR_NO_DEVICE, "no usable CUDA device; libmascot has no CPU path");
    }
    CU(nullptr, cudaSetDevice(device));
    float *dP = nullptr, *dQ = nullptr; mascot_rating* dT = nullptr;
    cudaError_t e = dev_alloc(&dP, (size_t)n_users * k, nullptr);
    if (e == cudaSuccess) e = dev_alloc(&dQ, (size_t)n_items * k, nullptr);
    if (e == cudaSuccess) e = dev_alloc(&dT, n_test, nullptr);
    if (e == cudaSuccess) e = copy_to_device(dP, P, sizeof(float) * (size_t)n_users * k, nullptr);
    if (e == cudaSuccess) e = copy_to_device(dQ, Q, sizeof(float) * (size_t)n_items * k, nullptr);
    if (e == cudaSuccess) e = copy_to_device(dT, test, sizeof(mascot_rating) * n_test, nullptr);
    Results sums((n_test + 511) / 512, nullptr);
    if (e == cudaSuccess) e = sums.status();
    if (e == cudaSuccess) e = launch_rmse_plain((int)k, dT, n_test, dP, dQ, n_users, n_items, sums.device(), sums.device_flag(), nullptr);
    if (e == cudaSuccess) e = sums.wait();
    dev_free(dP, nullptr); dev_free(dQ, nullptr); dev_free(dT, nullptr);
    CU(nullptr, e);
    if (sums.flag()) return fail(nullptr, MASCOT_ERR_BAD_ARG, "test rating with id out of range");
    *rmse = (double)reference_rmse_from_partials(sums, n_test);
    return MASCOT_OK;
}

}  // extern "C"
