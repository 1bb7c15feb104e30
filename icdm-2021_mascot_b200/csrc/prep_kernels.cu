// Set-up and conversion kernels: stream encoding (shuffle + id remap + precision bit), factor
// scatter/gather between the caller's fp32 row-major view and the permuted mixed-precision arenas,
// group promotion, and factor initialisation.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cub/block/block_radix_sort.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "engine.h"
#include "layout.cuh"

namespace mascot {

namespace {

struct NodeAos { float r; uint32_t u; uint32_t i; };

inline int grid_for(uint64_t n, int block) {
    uint64_t g = (n + block - 1) / block;
    const uint64_t cap = (uint64_t)sm_count() * 16;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

// Replaces the id remap matrix_reconst_gpu_triplet (preprocess_utils.h:28-36): stream position j takes source rating j (the
// kernels below: rating permute(j), in place of the host random_shuffle, mf_methods.cu:38-39), ids are mapped to sorted
// indices and tagged with the row's storage precision.
// An id outside [0, n_users) x [0, n_items) is never used as an index: the rating is replaced by a
// no-op record on row 0 (r = 0 would still train, so the host reports the raised flag as an error).
__device__ __forceinline__ NodeAos checked(NodeAos nd, uint32_t n_users, uint32_t n_items, uint32_t* err) {
    if (nd.u >= n_users || nd.i >= n_items) { atomicOr(err, 1u); nd.u = 0; nd.i = 0; nd.r = 0.f; }
    return nd;
}

__global__ void encode_kernel(const NodeAos* src, uint64_t n, const uint32_t* umap, const uint32_t* imap,
                              const uint8_t* uprec, const uint8_t* iprec, uint32_t n_users, uint32_t n_items, uint32_t* err,
                              float* r, uint32_t* u, uint32_t* i, uint32_t* src_out, uint32_t src_base) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const NodeAos nd = checked(src[j], n_users, n_items, err);
        uint32_t uu = umap ? umap[nd.u] : nd.u;
        uint32_t ii = imap ? imap[nd.i] : nd.i;
        uu |= row_flags_to_code(uprec[uu]);
        ii |= row_flags_to_code(iprec[ii]);
        r[j] = nd.r; u[j] = uu; i[j] = ii;
        if (src_out) src_out[j] = src_base + (uint32_t)j;
    }
}

// Locality-aware variant used when the stream is shuffled: after the seeded permutation the stream is
// cut into windows of kWindow consecutive positions and each window is stably sorted by item row.
// Ratings of a popular item then sit next to each other, and the update kernel keeps that item's
// row in registers for the whole run instead of reading and writing it once per rating - which is
// what bounds throughput on skewed data (every update of the most popular item otherwise goes
// through the same L2 lines).  Order inside a window carries no meaning for SGD; across windows the
// stream stays randomly ordered.  src_out records which source rating landed at each position.
//
// A block per window.  What it takes is the gathers and the passes of the sort: permuted positions are worked out once and
// are what is sorted, and the results leave in stripes (a thread's neighbours, one store after the other, touched every sector as
// many times).  A piece of 8.4M ratings: 0.572 -> 0.313 ms; 0.39 with 256 threads of sixteen records, 0.33 with the records kept in
// shared memory meanwhile instead of read twice, 0.34 with five bits a pass.
constexpr int kSortThreads = 512;
constexpr int kSortItemsPerThread = 8;
constexpr int kWindow = kSortThreads * kSortItemsPerThread;

__global__ void __launch_bounds__(kSortThreads) encode_sorted_kernel(
        const NodeAos* src, uint64_t n, Permutation perm, const uint32_t* umap, const uint32_t* imap,
        const uint8_t* uprec, const uint8_t* iprec, uint32_t n_users, uint32_t n_items, uint32_t* err, int key_bits,
        float* r, uint32_t* u, uint32_t* i, uint32_t* src_out, uint32_t src_base) {
    typedef cub::BlockRadixSort<uint32_t, kSortThreads, kSortItemsPerThread, uint32_t> Sort;
    __shared__ typename Sort::TempStorage temp;
    const uint64_t base = (uint64_t)blockIdx.x * kWindow;
    uint32_t keys[kSortItemsPerThread], vals[kSortItemsPerThread];       // item row, source position
#pragma unroll
    for (int t = 0; t < kSortItemsPerThread; t++) {
        const uint64_t pos = base + threadIdx.x * kSortItemsPerThread + t;
        vals[t] = pos < n ? permute(perm, (uint32_t)pos) : 0u;
    }
#pragma unroll
    for (int t = 0; t < kSortItemsPerThread; t++) {
        uint32_t it = src[vals[t]].i;
        if (it >= n_items) it = 0;                                  // reported when the record is read below
        const uint32_t row = imap ? imap[it] : it;
        keys[t] = base + threadIdx.x * kSortItemsPerThread + t < n ? row : 0xffffffffu >> (32 - key_bits);      // padding sorts last
    }
    Sort(temp).SortBlockedToStriped(keys, vals, 0, key_bits);
#pragma unroll
    for (int t = 0; t < kSortItemsPerThread; t++) {
        const uint64_t out = base + t * kSortThreads + threadIdx.x;
        if (out < n) {
            const NodeAos nd = checked(src[vals[t]], n_users, n_items, err);
            uint32_t uu = umap ? umap[nd.u] : nd.u;
            uint32_t ii = (imap ? imap[nd.i] : nd.i);        // equals keys[t] unless the record was replaced
            uu |= row_flags_to_code(uprec[uu]);
            ii |= row_flags_to_code(iprec[ii]);
            r[out] = nd.r; u[out] = uu; i[out] = ii;
            if (src_out) src_out[out] = src_base + vals[t];
        }
    }
}

__global__ void recode_kernel(uint32_t* ids, uint64_t n, const uint8_t* prec_row) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t id = ids[j] & kIdMask;
        ids[j] = id | row_flags_to_code(prec_row[id]);
    }
}

// cpyparams2grouped_params_for_comparison_indexing (model_init.cu:30-83): caller row e goes to
// arena row row_map[e]; here both arenas are filled so a later promotion is a plain widening.
template <int K>
__global__ void scatter_kernel(const float* src, uint32_t rows, const uint32_t* row_map, int through_half,
                               __half* dst16, float* dst32) {
    const uint64_t total = (uint64_t)rows * K;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t e = (uint32_t)(t / K);
        const int d = (int)(t % K);
        const uint32_t row = row_map ? row_map[e] : e;
        const int ph = phys_of_logical(K, d);
        const float v = src[t];
        const __half h = __float2half_rn(v);
        if (dst16) dst16[(size_t)row * K + ph] = h;
        if (dst32) dst32[(size_t)row * K + f32_pos_of_phys(K, ph)] = through_half ? __half2float(h) : v;
    }
}

// Output row e is the arena row row_map[e] (caller's id order) or, without a map, the arena row of
// sorted index e (sorted-index order).
template <int K>
__global__ void gather_kernel(const __half* a16, const float* a32, const uint8_t* prec_row, uint32_t rows,
                              const uint32_t* row_map, RowLayout layout, float* dst) {
    const uint64_t total = (uint64_t)rows * K;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t e = (uint32_t)(t / K);
        const int d = (int)(t % K);
        const uint32_t row = row_map ? row_map[e] : arena_row(layout, e);
        const int ph = phys_of_logical(K, d);
        dst[t] = (prec_row[row] & kRowPrec) ? a32[(size_t)row * K + f32_pos_of_phys(K, ph)] : __half2float(a16[(size_t)row * K + ph]);
    }
}

// mem_cpy_fp162fp32 (precision_switching.h:1-6) without the re-allocation around it: widens the rows of
// the sorted indices [begin, end) - one group - wherever the layout put them, and marks them fp32.
template <int K>
__global__ void promote_kernel(const __half* a16, float* a32, uint8_t* row_flags, RowLayout layout, uint32_t begin, uint32_t end) {
    const uint64_t total = (uint64_t)(end - begin) * K;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t row = arena_row(layout, begin + (uint32_t)(t / K));
        const int ph = (int)(t % K);
        a32[(size_t)row * K + f32_pos_of_phys(K, ph)] = __half2float(a16[(size_t)row * K + ph]);
        if (ph == 0) row_flags[row] |= kRowPrec;
    }
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// ---- reproducible double arithmetic for the factor initialisation -------------------------------
// The library logarithm and cosine are accurate to a unit in the last place but not correctly rounded,
// so a host program cannot reproduce their results bit for bit.  The two functions below use only
// single IEEE-754 operations (add, multiply, divide - written as intrinsics so that nothing is fused)
// in a fixed order; the same sequence on a host gives the same bits.
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }

// ln(x) for a normal x in (0, 1]: x = m * 2^e with m in (sqrt(1/2), sqrt(2)], s = (m-1)/(m+1),
// ln(m) = 2s * (1 + z/3 + z^2/5 + ... + z^10/21), z = s^2 <= 0.0295 (truncation below 1e-17).
__device__ double exact_log(double x) {
    const long long bits = __double_as_longlong(x);
    int e = (int)((bits >> 52) & 0x7ff) - 1023;
    double m = __longlong_as_double((bits & 0xfffffffffffffLL) | 0x3ff0000000000000LL);
    if (m > 1.4142135623730951) { m = rmul(m, 0.5); e += 1; }
    const double f = radd(m, -1.0);
    const double s = __ddiv_rn(f, radd(2.0, f));
    const double z = rmul(s, s);
    double p = 1.0 / 21.0;
    p = radd(rmul(p, z), 1.0 / 19.0); p = radd(rmul(p, z), 1.0 / 17.0); p = radd(rmul(p, z), 1.0 / 15.0);
    p = radd(rmul(p, z), 1.0 / 13.0); p = radd(rmul(p, z), 1.0 / 11.0); p = radd(rmul(p, z), 1.0 / 9.0);
    p = radd(rmul(p, z), 1.0 / 7.0); p = radd(rmul(p, z), 1.0 / 5.0); p = radd(rmul(p, z), 1.0 / 3.0);
    p = radd(rmul(p, z), 1.0);
    return radd(rmul((double)e, 0.6931471805599453), rmul(rmul(2.0, s), p));
}

// cos(pi * y) for y in [0, 2], y a multiple of 2^-52: y = q/2 + r with |r| <= 1/4 (exact), then the
// Taylor series of cos or sin of t = pi*r (|t| <= 0.786, truncation below 1e-17).
__device__ double exact_cospi(double y) {
    const int q = (int)floor(radd(rmul(y, 2.0), 0.5));
    const double r = radd(y, -rmul((double)q, 0.5));
    const double t = rmul(r, 3.141592653589793), t2 = rmul(t, t);
    double c = 1.0 / 20922789888000.0;                       // 1/16!
    c = radd(rmul(c, t2), -1.0 / 87178291200.0); c = radd(rmul(c, t2), 1.0 / 479001600.0);
    c = radd(rmul(c, t2), -1.0 / 3628800.0); c = radd(rmul(c, t2), 1.0 / 40320.0);
    c = radd(rmul(c, t2), -1.0 / 720.0); c = radd(rmul(c, t2), 1.0 / 24.0);
    c = radd(rmul(c, t2), -0.5); c = radd(rmul(c, t2), 1.0);
    double sn = 1.0 / 355687428096000.0;                     // 1/17!
    sn = radd(rmul(sn, t2), -1.0 / 1307674368000.0); sn = radd(rmul(sn, t2), 1.0 / 6227020800.0);
    sn = radd(rmul(sn, t2), -1.0 / 39916800.0); sn = radd(rmul(sn, t2), 1.0 / 362880.0);
    sn = radd(rmul(sn, t2), -1.0 / 5040.0); sn = radd(rmul(sn, t2), 1.0 / 120.0);
    sn = radd(rmul(sn, t2), -1.0 / 6.0); sn = radd(rmul(sn, t2), 1.0);
    sn = rmul(sn, t);
    switch (q & 3) { case 0: return c; case 1: return -sn; case 2: return -c; default: return sn; }
}

// N(0, 0.01^2) like init_rand_feature_single (model_init.cu:19-28), from a counter-based generator:
// element t of stream `sid` depends only on (seed, sid, t) - two splitmix64 draws, Box-Muller with the
// reproducible logarithm and cosine above, one rounding to float.  A host program that follows the
// same steps gets the same factors bit for bit.
__global__ void init_normal_kernel(float* dst, uint64_t count, uint64_t seed, uint64_t sid) {
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t z = splitmix64(splitmix64(seed ^ (sid * 0xd1342543de82ef95ull)) + t);
        const double u1 = rmul((double)((z >> 11) + 1), 1.0 / 9007199254740992.0);    // (0, 1]
        const uint64_t z2 = splitmix64(z);
        const double u2 = rmul((double)(z2 >> 11), 1.0 / 9007199254740992.0);         // [0, 1)
        const double radius = __dsqrt_rn(rmul(-2.0, exact_log(u1)));
        dst[t] = (float)rmul(rmul(radius, exact_cospi(rmul(2.0, u2))), 0.01);
    }
}

}  // namespace

cudaError_t launch_encode_stream(const void* d_src_aos, uint64_t n, bool shuffle, uint64_t seed,
                                 const uint32_t* user_map, const uint32_t* item_map,
                                 const uint8_t* uprec_row, const uint8_t* iprec_row, uint32_t n_users, uint32_t n_items,
                                 uint32_t item_rows, uint32_t* err_flag,
                                 float* r, uint32_t* u, uint32_t* i, uint32_t* src_out, uint32_t src_base,
                                 cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const NodeAos* src = static_cast<const NodeAos*>(d_src_aos);
    if (shuffle) {
        int key_bits = 1;
        while (key_bits < 31 && (1ull << key_bits) < (uint64_t)item_rows + 1) key_bits++;
        encode_sorted_kernel<<<(unsigned)((n + kWindow - 1) / kWindow), kSortThreads, 0, st>>>(src, n, make_permutation(n, seed), user_map, item_map, uprec_row, iprec_row,
                                                             n_users, n_items, err_flag, key_bits, r, u, i, src_out, src_base);
    } else {
        encode_kernel<<<grid_for(n, 256), 256, 0, st>>>(src, n, user_map, item_map, uprec_row, iprec_row,
                                                         n_users, n_items, err_flag, r, u, i, src_out, src_base);
    }
    return cudaGetLastError();
}

cudaError_t launch_recode(uint32_t* ids, uint64_t n, const uint8_t* prec_row, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    recode_kernel<<<grid_for(n, 256), 256, 0, st>>>(ids, n, prec_row);
    return cudaGetLastError();
}

// ---- re-ordering of the coded stream: item-sorted run windows, precision classes --------------------
// Item-sorted run windows: one stable radix sort by the key  (segment << window_bits | window) << item_bits | item row, with
// window = position >> run_window_log2 and the item's arena row.  A run of equal items is then as long as the item's share of
// such a window, not of the 4096 positions the encode kernel sorts, and a worker reads and writes the item's row once per run.
struct StreamKey {
    int run_window_log2;     // log2 of the window length
    int window_bits, item_bits;
};
__device__ __forceinline__ int segment_of(uint64_t j, const uint64_t* seg_off, int nseg) {      // the last segment whose offset is <= j
    int lo = 0, hi = nseg - 1;
    while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (seg_off[mid] <= j) lo = mid; else hi = mid - 1; }
    return lo;
}
// Key: 32 bits where they hold the key (stream_sort_key_bytes), else 64.
template <class Key>
__global__ void stream_key_kernel(const uint32_t* i, uint64_t n, const uint64_t* seg_off, int nseg, StreamKey sk, Key* key, uint32_t* idx) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = (((uint64_t)segment_of(j, seg_off, nseg) << sk.window_bits) | (j >> sk.run_window_log2)) << sk.item_bits | (i[j] & kIdMask);
        key[j] = (Key)k;
        idx[j] = (uint32_t)j;
    }
}
__global__ void stream_gather_kernel(const uint32_t* perm, uint64_t n, const float* r, const uint32_t* u, const uint32_t* i,
                                     const uint32_t* src, float* r2, uint32_t* u2, uint32_t* i2, uint32_t* src2) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = perm[j];
        r2[j] = r[s]; u2[j] = u[s]; i2[j] = i[s];
        if (src) src2[j] = src[s];
    }
}

static StreamKey make_stream_key(uint64_t n, int run_window_log2, uint32_t item_rows) {
    StreamKey sk{run_window_log2, 0, 0};
    while (((n - 1) >> run_window_log2) >> sk.window_bits) sk.window_bits++;
    while (sk.item_bits < 30 && (item_rows - 1u) >> sk.item_bits) sk.item_bits++;
    if (sk.item_bits == 0) sk.item_bits = 1;
    return sk;
}

size_t stream_sort_temp_bytes(uint64_t n, int seg_bits, int run_window_log2, uint32_t item_rows) {
    size_t bytes = 0;
    const StreamKey sk = make_stream_key(n, run_window_log2, item_rows);
    const int bits = seg_bits + sk.window_bits + sk.item_bits;
    if (bits <= 32) cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const uint32_t*)nullptr, (uint32_t*)nullptr, (const uint32_t*)nullptr, (uint32_t*)nullptr, n, 0, bits);
    else cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const uint64_t*)nullptr, (uint64_t*)nullptr, (const uint32_t*)nullptr, (uint32_t*)nullptr, n, 0, bits);
    return bytes;
}

size_t stream_sort_key_bytes(uint64_t n, int seg_bits, int run_window_log2, uint32_t item_rows) {
    const StreamKey sk = make_stream_key(n, run_window_log2, item_rows);
    return seg_bits + sk.window_bits + sk.item_bits <= 32 ? 4 : 8;
}

template <class Key>
static cudaError_t stream_sort(const float* r, const uint32_t* u, const uint32_t* i, const uint32_t* src, uint64_t n, const uint64_t* d_seg_off, int nseg,
                               int bits, const StreamKey& sk, Key* key_a, Key* key_b, uint32_t* idx_a, uint32_t* idx_b, void* temp, size_t temp_bytes,
                               float* r2, uint32_t* u2, uint32_t* i2, uint32_t* src2, cudaStream_t st) {
    const int g = grid_for(n, 256);
    stream_key_kernel<Key><<<g, 256, 0, st>>>(i, n, d_seg_off, nseg, sk, key_a, idx_a);
    cudaError_t e = cub::DeviceRadixSort::SortPairs(temp, temp_bytes, key_a, key_b, idx_a, idx_b, n, 0, bits, st);
    if (e != cudaSuccess) return e;
    stream_gather_kernel<<<g, 256, 0, st>>>(idx_b, n, r, u, i, src, r2, u2, i2, src2);
    return cudaGetLastError();
}

cudaError_t launch_stream_sort(const float* r, const uint32_t* u, const uint32_t* i, const uint32_t* src, uint64_t n,
                               const uint64_t* d_seg_off, int nseg, int seg_bits, int run_window_log2, uint32_t item_rows,
                               void* key_a, void* key_b, uint32_t* idx_a, uint32_t* idx_b, void* temp, size_t temp_bytes,
                               float* r2, uint32_t* u2, uint32_t* i2, uint32_t* src2, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const StreamKey sk = make_stream_key(n, run_window_log2, item_rows);
    const int bits = seg_bits + sk.window_bits + sk.item_bits;
    if (bits <= 32)
        return stream_sort(r, u, i, src, n, d_seg_off, nseg, bits, sk, static_cast<uint32_t*>(key_a), static_cast<uint32_t*>(key_b), idx_a, idx_b, temp, temp_bytes,
                           r2, u2, i2, src2, st);
    return stream_sort(r, u, i, src, n, d_seg_off, nseg, bits, sk, static_cast<uint64_t*>(key_a), static_cast<uint64_t*>(key_b), idx_a, idx_b, temp, temp_bytes,
                       r2, u2, i2, src2, st);
}

// Partition by precision class.  Inside a class the ratings keep the order in which they are, so after promotions one after the
// other a class is sorted by the groups that came into it.  Classes in the order in which the stream was coded would be faster to train (ms
// per epoch: 8M ratings, all 100 + 100 groups promoted one by one, 4.1 and 1.32; 63M, the upper 40 of them, 9.2 and 7.0), but not
// to the same model: runs of equal items are longer there (63M: 6.6 ratings against 1.9), an item row is written back with a plain
// store once per run, and the test RMSE is higher (0.5193 and 0.5184 at 8M, 0.57333 and 0.57262 at 40M, four epochs).
//
// Tiles of kTile positions, none of which crosses a segment: the classes of each tile are counted, and one sum over (segment, class,
// tile) says where each class of each tile begins.  A tile is then ordered in shared memory and moved with coalesced writes.  A promotion
// among 63M ratings takes 1.0 ms; 1.9 with a radix sort of keys and indices and a gather after it.
constexpr int kTile = 4096, kTileWarps = 8;
struct Tiles { const uint64_t* seg_off; const uint32_t* first; int nseg; };      // first[s]: number of tiles before segment s
struct Tile { uint64_t begin; int count; uint32_t slot, stride; };               // its counter of class c is number slot + c * stride
__device__ __forceinline__ Tile tile_of(const Tiles& T, uint32_t t) {
    int lo = 0, hi = T.nseg - 1;                                                   // the last segment that begins at or before tile t
    while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (T.first[mid] <= t) lo = mid; else hi = mid - 1; }
    const uint32_t in = t - T.first[lo], tiles = T.first[lo + 1] - T.first[lo];
    const uint64_t begin = T.seg_off[lo] + (uint64_t)in * kTile, left = T.seg_off[lo + 1] - begin;
    return Tile{begin, (int)(left < kTile ? left : kTile), 4 * T.first[lo] + in, tiles};
}
__device__ __forceinline__ int class_of(uint32_t u, uint32_t i) { return (u & kPrecBit ? 2 : 0) | (i & kPrecBit ? 1 : 0); }
__global__ void __launch_bounds__(32 * kTileWarps) class_count_kernel(const uint32_t* u, const uint32_t* i, Tiles T, uint32_t* counts) {
    __shared__ uint32_t sum[4];
    if (threadIdx.x < 4) sum[threadIdx.x] = 0;
    __syncthreads();
    const Tile t = tile_of(T, blockIdx.x);
    uint32_t mine[4] = {0, 0, 0, 0};
    for (int e = threadIdx.x; e < t.count; e += 32 * kTileWarps) {
        const int k = class_of(u[t.begin + e], i[t.begin + e]);
#pragma unroll
        for (int c = 0; c < 4; c++) mine[c] += k == c;
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint32_t s = __reduce_add_sync(0xffffffffu, mine[c]);
        if ((threadIdx.x & 31) == 0) atomicAdd(sum + c, s);
    }
    __syncthreads();
    if (threadIdx.x < 4) counts[t.slot + threadIdx.x * t.stride] = sum[threadIdx.x];
}
__global__ void __launch_bounds__(32 * kTileWarps) class_move_kernel(Tiles T, const uint32_t* start, const float* r, const uint32_t* u, const uint32_t* i,
                                                                     const uint32_t* src, float* r2, uint32_t* u2, uint32_t* i2, uint32_t* src2) {
    constexpr int kRounds = kTile / (32 * kTileWarps);
    __shared__ uint16_t order[kTile];                       // positions of the tile, class by class
    __shared__ uint32_t held[kTileWarps][4], begin[5];      // ratings per warp and class; where a class begins in `order`
    const Tile t = tile_of(T, blockIdx.x);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e0 = warp * 32 * kRounds + lane;
    const unsigned below = (1u << lane) - 1u;
    uint32_t rank[kRounds], n[4] = {0, 0, 0, 0};           // class in the upper half
#pragma unroll
    for (int q = 0; q < kRounds; q++) {
        const int e = e0 + 32 * q, k = e < t.count ? class_of(u[t.begin + e], i[t.begin + e]) : 4;
        rank[q] = 4u << 16;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const unsigned who = __ballot_sync(0xffffffffu, k == c);
            if (k == c) rank[q] = (uint32_t)c << 16 | (n[c] + __popc(who & below));
            n[c] += __popc(who);
        }
    }
    if (lane == 0) { held[warp][0] = n[0]; held[warp][1] = n[1]; held[warp][2] = n[2]; held[warp][3] = n[3]; }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t at = 0;
        for (int c = 0; c < 4; c++) {
            begin[c] = at;
            for (int w = 0; w < kTileWarps; w++) { const uint32_t h = held[w][c]; held[w][c] = at; at += h; }
        }
        begin[4] = at;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kRounds; q++) if (rank[q] >> 16 < 4) order[held[warp][rank[q] >> 16] + (rank[q] & 0xffffu)] = (uint16_t)(e0 + 32 * q);
    __syncthreads();
    // four ratings of a thread at a time, or the chain order -> rating -> store is all it does
    constexpr int kBatch = 4;
#pragma unroll 1
    for (int o0 = threadIdx.x; o0 < t.count; o0 += kBatch * 32 * kTileWarps) {
        uint64_t from[kBatch];
        uint32_t vu[kBatch], vi[kBatch], vs[kBatch];
        float vr[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; b++) from[b] = t.begin + order[min(o0 + b * 32 * kTileWarps, t.count - 1)];
#pragma unroll
        for (int b = 0; b < kBatch; b++) { vr[b] = r[from[b]]; vu[b] = u[from[b]]; vi[b] = i[from[b]]; vs[b] = src ? src[from[b]] : 0u; }
#pragma unroll
        for (int b = 0; b < kBatch; b++) {
            const int o = o0 + b * 32 * kTileWarps;
            if (o >= t.count) break;
            const int c = (o >= (int)begin[1]) + (o >= (int)begin[2]) + (o >= (int)begin[3]);
            const uint32_t to = start[t.slot + c * t.stride] + (uint32_t)(o - (int)begin[c]);
            r2[to] = vr[b]; u2[to] = vu[b]; i2[to] = vi[b];
            if (src) src2[to] = vs[b];
        }
    }
}
// first[4 s + c]: where class c of segment s begins
__global__ void class_first_kernel(const uint32_t* start, Tiles T, uint32_t* first) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < 4u * (uint32_t)T.nseg; k += gridDim.x * blockDim.x) {
        const uint32_t s = k / 4, tiles = T.first[s + 1] - T.first[s];
        first[k] = tiles ? start[4 * T.first[s] + (k & 3) * tiles] : (uint32_t)T.seg_off[s];
    }
}

uint32_t class_tiles(const uint64_t* seg_off, int nseg, uint32_t* first) {
    uint32_t tiles = 0;
    for (int s = 0; s < nseg; s++) { first[s] = tiles; tiles += (uint32_t)((seg_off[s + 1] - seg_off[s] + kTile - 1) / kTile); }
    first[nseg] = tiles;
    return tiles;
}

size_t class_partition_temp_bytes(uint32_t tiles) {
    size_t bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, bytes, (const uint32_t*)nullptr, (uint32_t*)nullptr, (uint64_t)4 * tiles);
    return bytes;
}

cudaError_t launch_class_partition(const float* r, const uint32_t* u, const uint32_t* i, const uint32_t* src, uint64_t n,
                                   const uint64_t* d_seg_off, const uint32_t* d_first_tile, int nseg, uint32_t tiles,
                                   uint32_t* counts, uint32_t* starts, void* temp, size_t temp_bytes, uint32_t* d_first,
                                   float* r2, uint32_t* u2, uint32_t* i2, uint32_t* src2, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const Tiles T{d_seg_off, d_first_tile, nseg};
    class_count_kernel<<<tiles, 32 * kTileWarps, 0, st>>>(u, i, T, counts);
    const cudaError_t e = cub::DeviceScan::ExclusiveSum(temp, temp_bytes, counts, starts, (uint64_t)4 * tiles, st);
    if (e != cudaSuccess) return e;
    class_move_kernel<<<tiles, 32 * kTileWarps, 0, st>>>(T, starts, r, u, i, src, r2, u2, i2, src2);
    class_first_kernel<<<grid_for(4 * (uint64_t)nseg, 256), 256, 0, st>>>(starts, T, d_first);
    return cudaGetLastError();
}

// ---- the coded stream in one sort -----------------------------------------------------------------
// encode_sorted_kernel's windows of kWindow positions only matter for what is not sorted any further.  Where run windows
// follow - whose boundaries fall on multiples of kWindow - a stable sort of the permuted SOURCE positions by (segment, run
// window, item row) gives the same order in one go: the block sort, the second pass over the coded arrays and the
// copies back fall away, and the key fits 32 bits.
__global__ void source_key_kernel(const NodeAos* src, const uint32_t* items, uint64_t n, const uint64_t* seg_off, int nseg, uint64_t seed, Permutation first, const uint32_t* imap, uint32_t n_items,
                                  StreamKey sk, uint32_t* key, uint32_t* val) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const int lo = segment_of(j, seg_off, nseg);
        const uint64_t off = seg_off[lo], seg_seed = seed + 0x9e3779b97f4a7c15ull * (uint64_t)lo;
        const uint32_t s = (uint32_t)off + permute(nseg == 1 ? first : make_permutation(seg_off[lo + 1] - off, seg_seed), (uint32_t)(j - off));
        uint32_t it = items ? items[s] : src[s].i;
        if (it >= n_items) it = 0;                    // reported when the record is read below
        key[j] = (((uint32_t)lo << sk.window_bits | (uint32_t)(j >> sk.run_window_log2)) << sk.item_bits) | (imap ? imap[it] : it);
        val[j] = s;
    }
}
__global__ void source_gather_kernel(const uint32_t* val, uint64_t n, const NodeAos* src, const uint32_t* umap, const uint32_t* imap,
                                     const uint8_t* uprec, const uint8_t* iprec, uint32_t n_users, uint32_t n_items, uint32_t* err,
                                     float* r, uint32_t* u, uint32_t* i, uint32_t* src_out) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = val[j];
        const NodeAos nd = checked(src[s], n_users, n_items, err);
        uint32_t uu = umap ? umap[nd.u] : nd.u, ii = imap ? imap[nd.i] : nd.i;
        uu |= row_flags_to_code(uprec[uu]);
        ii |= row_flags_to_code(iprec[ii]);
        r[j] = nd.r; u[j] = uu; i[j] = ii; src_out[j] = s;
    }
}

static int source_key_bits(uint64_t n, int nseg, int run_window_log2, uint32_t item_rows, StreamKey* sk) {
    *sk = make_stream_key(n, run_window_log2, item_rows);
    int seg_bits = 0;
    while ((1ll << seg_bits) < nseg) seg_bits++;
    return seg_bits + sk->window_bits + sk->item_bits;
}

size_t source_sort_bytes(uint64_t n, const uint64_t* seg_off, int nseg, int run_window_log2, uint32_t item_rows) {
    StreamKey sk;
    if (n == 0 || run_window_log2 <= 0 || source_key_bits(n, nseg, run_window_log2, item_rows, &sk) > 32) return 0;
    for (int s = 0; s < nseg; s++) if (seg_off[s] % kWindow) return 0;
    size_t temp = 0;
    cub::DoubleBuffer<uint32_t> keys(nullptr, nullptr), vals(nullptr, nullptr);
    cub::DeviceRadixSort::SortPairs(nullptr, temp, keys, vals, n, 0, 32);
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    return 4 * up(4 * n) + up(8 * (size_t)(nseg + 1)) + up(temp);
}

// The last of the four buffers is not written before the keys, which are made from the item ids, are there.
uint32_t* source_sort_items(void* space, uint64_t n) { return reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(space) + 3 * ((4 * n + 255) / 256 * 256)); }

cudaError_t launch_source_sort(const void* d_src_aos, uint64_t n, const uint64_t* seg_off, int nseg, uint64_t seed, int run_window_log2, uint32_t item_rows,
                               const uint32_t* user_map, const uint32_t* item_map, const uint8_t* uprec_row, const uint8_t* iprec_row,
                               uint32_t n_users, uint32_t n_items, uint32_t* err_flag, void* space, const uint32_t* items, float* r, uint32_t* u, uint32_t* i,
                               uint32_t* src_out, cudaStream_t st) {
    StreamKey sk;
    const int bits = source_key_bits(n, nseg, run_window_log2, item_rows, &sk);
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    unsigned char* base = static_cast<unsigned char*>(space);
    uint32_t* buf[4];
    for (uint32_t*& b : buf) { b = reinterpret_cast<uint32_t*>(base); base += up(4 * n); }
    uint64_t* d_seg = reinterpret_cast<uint64_t*>(base); base += up(8 * (size_t)(nseg + 1));
    cudaError_t e = cudaMemcpyAsync(d_seg, seg_off, sizeof(uint64_t) * (nseg + 1), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const NodeAos* src = static_cast<const NodeAos*>(d_src_aos);
    const int g = grid_for(n, 256);
    source_key_kernel<<<g, 256, 0, st>>>(src, items, n, d_seg, nseg, seed, make_permutation(n, seed), item_map, n_items, sk, buf[0], buf[1]);
    cub::DoubleBuffer<uint32_t> keys(buf[0], buf[2]), vals(buf[1], buf[3]);
    size_t temp = 0;
    e = cub::DeviceRadixSort::SortPairs(nullptr, temp, keys, vals, n, 0, bits, st);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(base, temp, keys, vals, n, 0, bits, st);
    if (e != cudaSuccess) return e;
    source_gather_kernel<<<g, 256, 0, st>>>(vals.Current(), n, src, user_map, item_map, uprec_row, iprec_row, n_users, n_items, err_flag, r, u, i, src_out);
    return cudaGetLastError();
}

cudaError_t launch_scatter_factors(int K, const float* src, uint32_t rows, const uint32_t* row_map,
                                   bool round_through_half, __half* dst16, float* dst32, cudaStream_t st) {
    if (rows == 0) return cudaSuccess;
    const int g = grid_for((uint64_t)rows * K, 256);
    if (K == 128) scatter_kernel<128><<<g, 256, 0, st>>>(src, rows, row_map, round_through_half ? 1 : 0, dst16, dst32);
    else if (K == 64) scatter_kernel<64><<<g, 256, 0, st>>>(src, rows, row_map, round_through_half ? 1 : 0, dst16, dst32);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_gather_factors(int K, Arena a, const uint8_t* prec_row, uint32_t rows,
                                  const uint32_t* row_map, const RowLayout& layout, float* dst, cudaStream_t st) {
    if (rows == 0) return cudaSuccess;
    const int g = grid_for((uint64_t)rows * K, 256);
    if (K == 128) gather_kernel<128><<<g, 256, 0, st>>>(a.f16, a.f32, prec_row, rows, row_map, layout, dst);
    else if (K == 64) gather_kernel<64><<<g, 256, 0, st>>>(a.f16, a.f32, prec_row, rows, row_map, layout, dst);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_promote_rows(int K, Arena a, uint8_t* row_flags, const RowLayout& layout, uint32_t sorted_begin, uint32_t sorted_end,
                                cudaStream_t st) {
    if (sorted_end <= sorted_begin) return cudaSuccess;
    const int g = grid_for((uint64_t)(sorted_end - sorted_begin) * K, 256);
    if (K == 128) promote_kernel<128><<<g, 256, 0, st>>>(a.f16, a.f32, row_flags, layout, sorted_begin, sorted_end);
    else if (K == 64) promote_kernel<64><<<g, 256, 0, st>>>(a.f16, a.f32, row_flags, layout, sorted_begin, sorted_end);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_init_normal(float* dst, uint64_t count, uint64_t seed, uint64_t stream_id, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    init_normal_kernel<<<grid_for(count, 256), 256, 0, st>>>(dst, count, seed, stream_id);
    return cudaGetLastError();
}

}  // namespace mascot
