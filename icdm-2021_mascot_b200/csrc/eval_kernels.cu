// Test-RMSE kernels.
//
// The reduction is the reference's, so the result is reproducible bit for bit: per rating an fp32
// dot product (per-lane left-to-right product chain, then the 16-8-4-2-1 lane tree), the squared
// error in fp32, a 512-entry pairwise tree per block of 512 consecutive test ratings
// (get_test_rmse_coalesced_k128/k64, rmse.h:26-166), and a sequential float sum of the block
// partials on the host (rmse.h:183-188).  Unlike the reference there is no device->host->device
// round trip of the factors (mf_methods.cu:248-313, rmse.h:170-171): the kernel reads the
// mixed-precision arenas in place.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>

#include "../../include/mascot.h"
#include "engine.h"
#include "layout.cuh"

namespace mascot {

namespace {

constexpr int kRmseBlock = 512;    // ratings per block partial (BLOCK_SIZE in rmse.h:3)

// tmp[j] += tmp[j+s] for s = 256 .. 1  (rmse.h:85-91 and warpReduce, rmse.h:5-24), by the first eight warps: two levels
// through shared memory, the rest in the registers of one warp (a xor butterfly adds the same pairs).
__device__ __forceinline__ void block_tree_512(float* tmp, float* out) {
    const int t = threadIdx.x;
    __syncthreads();
    if (t < 256) tmp[t] = __fadd_rn(tmp[t], tmp[t + 256]);
    __syncthreads();
    if (t < 32) {
        const float a = __fadd_rn(__fadd_rn(tmp[t], tmp[t + 128]), __fadd_rn(tmp[t + 64], tmp[t + 192]));
        const float b = __fadd_rn(__fadd_rn(tmp[t + 32], tmp[t + 160]), __fadd_rn(tmp[t + 96], tmp[t + 224]));
        float v = __fadd_rn(a, b);
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, d));
        if (t == 0) *out = v;
    }
}

// What bounds an evaluation is the latency of two dependent loads (ids, then rows) and the rows' traffic.  The ids of a
// block come in with one coalesced load, so that all row loads of a lane can be in flight together; each team
// takes kBatch ratings at once and reduces them together: the first steps of the lane tree exchange half of the
// ratings instead of adding all of them in every lane, which adds the same pairs with a third of the shuffles.
struct BlockIds {
    float r[kRmseBlock];
    uint32_t u[kRmseBlock], i[kRmseBlock];
};

// A lane's eight consecutive physical elements of a row as fp32 (positions: see layout.cuh).
struct Row8 { uint4 a, b; };
template <int K>
__device__ __forceinline__ Row8 fetch8(const Arena& A, uint32_t code, int tl) {
    const uint32_t row = code & kIdMask;
    Row8 v;
    if (code & kPrecBit) {
        const uint4* p = reinterpret_cast<const uint4*>(A.f32 + (size_t)row * K) + tl;        // two half-rows (layout.cuh)
        v.a = __ldcg(p); v.b = __ldcg(p + K / 8);
    } else {
        v.a = __ldcg(reinterpret_cast<const uint4*>(A.f16 + (size_t)row * K) + tl);
    }
    return v;
}
__device__ __forceinline__ void widen8(const Row8& v, uint32_t code, float* x) {
    if (code & kPrecBit) {
        x[0] = __uint_as_float(v.a.x); x[1] = __uint_as_float(v.a.y); x[2] = __uint_as_float(v.a.z); x[3] = __uint_as_float(v.a.w);
        x[4] = __uint_as_float(v.b.x); x[5] = __uint_as_float(v.b.y); x[6] = __uint_as_float(v.b.z); x[7] = __uint_as_float(v.b.w);
    } else {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.a.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.a.y));
        const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&v.a.z)), d = __half22float2(*reinterpret_cast<const __half2*>(&v.a.w));
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y; x[4] = c.x; x[5] = c.y; x[6] = d.x; x[7] = d.y;
    }
}

// Sums four values over a team of T lanes, xor steps T/2 .. 1; lane with index t ends with the sum of value
// 2 * (t & T/2 set) + (t & T/4 set).
template <int T>
__device__ __forceinline__ float team_sum4(const float (&v)[4], int t) {
    const bool up = t & (T / 2), up2 = t & (T / 4);
    const float s0 = __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], T / 2), s1 = __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], T / 2);
    const float w0 = __fadd_rn(up ? v[2] : v[0], s0), w1 = __fadd_rn(up ? v[3] : v[1], s1);
    float x = __fadd_rn(up2 ? w1 : w0, __shfl_xor_sync(0xffffffffu, up2 ? w0 : w1, T / 4));
#pragma unroll
    for (int d = T / 8; d >= 1; d >>= 1) x = __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, d));
    return x;
}

template <int K>
__global__ void __launch_bounds__(512) rmse_kernel(const Stream t, const Arena P, const Arena Q, float* block_err) {
    constexpr int T = K / 8;                      // lanes per rating, eight elements each
    constexpr int kTeams = 512 / T;
    __shared__ float tmp[kRmseBlock];
    __shared__ BlockIds ids;
    const int tl = threadIdx.x % T, team = threadIdx.x / T;
    const uint64_t base = (uint64_t)blockIdx.x * kRmseBlock;
    const int left = (int)min((uint64_t)kRmseBlock, t.n - base);
    {   // positions past the end repeat the last rating; their error counts as zero below
        const uint64_t at = base + min((int)threadIdx.x, left - 1);
        ids.r[threadIdx.x] = __ldg(t.r + at); ids.u[threadIdx.x] = __ldg(t.u + at); ids.i[threadIdx.x] = __ldg(t.i + at);
    }
    __syncthreads();
    for (int j = team; j < kRmseBlock; j += 4 * kTeams) {      // ratings j, j + kTeams, j + 2 kTeams, j + 3 kTeams
        Row8 rp[4], rq[4];
        uint32_t uc[4], ic[4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            uc[b] = ids.u[j + b * kTeams]; ic[b] = ids.i[j + b * kTeams];
            rp[b] = fetch8<K>(P, uc[b], tl);
            rq[b] = fetch8<K>(Q, ic[b], tl);
        }
        float part[4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            float p[8], q[8];
            widen8(rp[b], uc[b], p);
            widen8(rq[b], ic[b], q);
            // positions 0 2 4 6 hold e0..e3, positions 1 3 5 7 hold e4..e7
            if (K == 128) {
                // two reference lanes (m, m+16): product chain over four elements each (rmse.h:75),
                // their sum is the tree's 16 step
                float c[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float acc = __fmaf_rn(p[h], q[h], __fmul_rn(p[2 + h], q[2 + h]));
                    acc = __fmaf_rn(p[4 + h], q[4 + h], acc);
                    c[h] = __fmaf_rn(p[6 + h], q[6 + h], acc);
                }
                part[b] = __fadd_rn(c[0], c[1]);
            } else {
                // four reference lanes (m, m+16, m+8, m+24) with two elements each: 16 step, then 8 step
                const float f0 = __fmaf_rn(p[0], q[0], __fmul_rn(p[2], q[2]));
                const float f1 = __fmaf_rn(p[4], q[4], __fmul_rn(p[6], q[6]));
                const float f2 = __fmaf_rn(p[1], q[1], __fmul_rn(p[3], q[3]));
                const float f3 = __fmaf_rn(p[5], q[5], __fmul_rn(p[7], q[7]));
                part[b] = __fadd_rn(__fadd_rn(f0, f1), __fadd_rn(f2, f3));
            }
        }
        const float pred = team_sum4<T>(part, tl);
        if ((tl & (T / 4 - 1)) == 0) {
            const int at = j + (2 * ((tl & (T / 2)) != 0) + ((tl & (T / 4)) != 0)) * kTeams;
            const float e = __fsub_rn(ids.r[at], pred);
            tmp[at] = at < left ? __fmul_rn(e, e) : 0.f;
        }
    }
    block_tree_512(tmp, block_err + blockIdx.x);
}

struct NodeAos { float r; uint32_t u; uint32_t i; };

// Plain fp32 rows in the reference's own element order: reference lane l adds elements l, l+32, ... of a row.  Eight
// lanes take a rating; lane t loads the 16 bytes of reference lanes 4t..4t+3 in each of the K/32 slots, so that a row
// comes in whole 128-byte lines, and the steps 16, 8, 4 of the lane tree go across the eight lanes, 2 and 1 between
// what they end up with: six shuffles for the four ratings of a warp.
// The matrices may start at any float; rows off 16-byte boundaries are read float by float.
template <bool ALIGNED> __device__ __forceinline__ float4 load4(const float* p) {
    if (ALIGNED) return __ldg(reinterpret_cast<const float4*>(p));
    return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}
template <int K, bool ALIGNED>
__global__ void __launch_bounds__(512) rmse_plain_kernel(const NodeAos* t, uint64_t n, const float* P, const float* Q, uint32_t n_users, uint32_t n_items,
                                                         float* block_err, uint32_t* bad) {
    constexpr int T = 8, kSlots = K / 32, kTeams = 512 / T, kBatch = K == 128 ? 2 : 4;
    __shared__ float tmp[kRmseBlock];
    __shared__ BlockIds ids;
    const int tl = threadIdx.x % T, team = threadIdx.x / T;
    const uint64_t base = (uint64_t)blockIdx.x * kRmseBlock;
    const int left = (int)min((uint64_t)kRmseBlock, n - base);
    {
        const NodeAos* const nd = t + base + min((int)threadIdx.x, left - 1);
        uint32_t u = __ldg(&nd->u), i = __ldg(&nd->i);
        if (bad && (u >= n_users || i >= n_items)) { *bad = 1u; u = 0; i = 0; }      // never used as an index
        ids.r[threadIdx.x] = __ldg(&nd->r); ids.u[threadIdx.x] = u; ids.i[threadIdx.x] = i;
    }
    __syncthreads();
    for (int j0 = team; j0 < kRmseBlock; j0 += kBatch * kTeams) {
        float4 p[kBatch][kSlots], q[kBatch][kSlots];
#pragma unroll
        for (int b = 0; b < kBatch; b++) {
            const float* rp = P + (size_t)ids.u[j0 + b * kTeams] * K + 4 * tl;
            const float* rq = Q + (size_t)ids.i[j0 + b * kTeams] * K + 4 * tl;
#pragma unroll
            for (int s = 0; s < kSlots; s++) { p[b][s] = load4<ALIGNED>(rp + 32 * s); q[b][s] = load4<ALIGNED>(rq + 32 * s); }
        }
#pragma unroll
        for (int b = 0; b < kBatch; b++) {
            auto chain = [&](auto of) {
                float acc = __fmaf_rn(of(p[b][0]), of(q[b][0]), __fmul_rn(of(p[b][1]), of(q[b][1])));
#pragma unroll
                for (int s = 2; s < kSlots; s++) acc = __fmaf_rn(of(p[b][s]), of(q[b][s]), acc);
                return acc;
            };
            const float v[4] = {chain([](const float4& x) { return x.x; }), chain([](const float4& x) { return x.y; }),
                                chain([](const float4& x) { return x.z; }), chain([](const float4& x) { return x.w; })};
            float x = team_sum4<T>(v, tl);                       // lane: reference lanes 4t + (2 up + up2), steps 16 8 4
            x = __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, T / 2));      // step 2: values 0 + 2, 1 + 3
            x = __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, T / 4));      // step 1
            if (tl == 0) {
                const int at = j0 + b * kTeams;
                const float e = __fsub_rn(ids.r[at], x);
                tmp[at] = at < left ? __fmul_rn(e, e) : 0.f;
            }
        }
    }
    block_tree_512(tmp, block_err + blockIdx.x);
}

}  // namespace

cudaError_t launch_rmse(int K, const Stream& t, Arena P, Arena Q, float* block_err, cudaStream_t st) {
    if (t.n == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((t.n + kRmseBlock - 1) / kRmseBlock);
    if (K == 128) rmse_kernel<128><<<blocks, 512, 0, st>>>(t, P, Q, block_err);
    else if (K == 64) rmse_kernel<64><<<blocks, 512, 0, st>>>(t, P, Q, block_err);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_rmse_plain(int K, const void* d_test_aos, uint64_t n, const float* P, const float* Q,
                              uint32_t n_users, uint32_t n_items, float* block_err, uint32_t* bad, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((n + kRmseBlock - 1) / kRmseBlock);
    const NodeAos* t = static_cast<const NodeAos*>(d_test_aos);
    const bool aligned = ((reinterpret_cast<uintptr_t>(P) | reinterpret_cast<uintptr_t>(Q)) & 15) == 0;
    if (K == 128 && aligned) rmse_plain_kernel<128, true><<<blocks, 512, 0, st>>>(t, n, P, Q, n_users, n_items, block_err, bad);
    else if (K == 128) rmse_plain_kernel<128, false><<<blocks, 512, 0, st>>>(t, n, P, Q, n_users, n_items, block_err, bad);
    else if (K == 64 && aligned) rmse_plain_kernel<64, true><<<blocks, 512, 0, st>>>(t, n, P, Q, n_users, n_items, block_err, bad);
    else if (K == 64) rmse_plain_kernel<64, false><<<blocks, 512, 0, st>>>(t, n, P, Q, n_users, n_items, block_err, bad);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

}  // namespace mascot

// ---------------------------------------------------------------------------------------------
// Evaluation without any allocation.
//
// Some callers must not allocate device memory at call time: an evaluation hook that runs between
// training steps of a host program which has handed the whole GPU to its own memory pool (a
// cudaMalloc there can fail or fragment the pool), a serving loop that cannot afford the implicit
// device-wide synchronisation of cudaMalloc/cudaFree, or a process working inside a memory budget
// that was fixed at start-up.  For them the per-block partial sums live in the fixed array below
// instead of a cudaMalloc'ed buffer.  Every GPU that loads this library holds the array (256 KiB)
// until the process exits.
// ---------------------------------------------------------------------------------------------
namespace mascot {
namespace {

constexpr uint64_t kStaticMaxBlocks = 1u << 16;                       // 65,536 partials = 256 KiB
constexpr uint64_t kStaticMaxRatings = kStaticMaxBlocks * kRmseBlock; // 33,554,432 test ratings
constexpr int kMaxDevices = 64;

static __device__ __align__(256) float g_static_block_err[kStaticMaxBlocks];

// In host code the name above is only a stand-in for the symbol, not an address a kernel can use:
// the device address is looked up once per device (with that device current) and cached here.
float* g_static_block_err_addr[kMaxDevices] = {nullptr};
float g_static_host_partials[kStaticMaxBlocks];

}  // namespace
}  // namespace mascot

extern "C" int mascot_rmse_device_noalloc(const float* d_P, const float* d_Q, uint32_t k, const mascot_rating* d_test,
                                          uint64_t n_test, double* rmse) {
    using namespace mascot;
    char msg[256];
    if (!d_P || !d_Q || !d_test || !rmse || !n_test) { set_global_error("null pointer or empty test set"); return MASCOT_ERR_BAD_ARG; }
    if (k != 64 && k != 128) { set_global_error("k must be 64 or 128"); return MASCOT_ERR_BAD_ARG; }
    if (n_test > kStaticMaxRatings) {
        snprintf(msg, sizeof msg, "mascot_rmse_device_noalloc handles at most %llu test ratings per call (got %llu); "
                 "use mascot_rmse_device for larger sets", (unsigned long long)kStaticMaxRatings, (unsigned long long)n_test);
        set_global_error(msg);
        return MASCOT_ERR_BAD_ARG;
    }
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        set_global_error("no current CUDA device (or device ordinal beyond 63)");
        return MASCOT_ERR_NO_DEVICE;
    }
    if (!g_static_block_err_addr[dev]) {
        // first call on this device: resolve the symbol's device address
        float* addr = nullptr;
        e = cudaGetSymbolAddress(reinterpret_cast<void**>(&addr), g_static_block_err);
        if (e != cudaSuccess || !addr) {
            snprintf(msg, sizeof msg, "cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            set_global_error(msg);
            return MASCOT_ERR_CUDA;
        }
        g_static_block_err_addr[dev] = addr;
    }
    float* d_err = g_static_block_err_addr[dev];
    const size_t blocks = (size_t)((n_test + kRmseBlock - 1) / kRmseBlock);
    // every one of the `blocks` partials is overwritten by its block, so nothing has to be cleared
    e = launch_rmse_plain((int)k, d_test, n_test, d_P, d_Q, 0, 0, d_err, nullptr, nullptr);
    if (e == cudaSuccess) e = cudaMemcpy(g_static_host_partials, d_err, sizeof(float) * blocks, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        snprintf(msg, sizeof msg, "evaluation failed: %s", cudaGetErrorString(e));
        set_global_error(msg);
        return MASCOT_ERR_CUDA;
    }
    float sum = 0;                                   // same float accumulation order as mascot_rmse_device
    for (size_t b = 0; b < blocks; b++) sum += g_static_host_partials[b];
    *rmse = (double)(float)std::sqrt(sum / (double)n_test);
    return MASCOT_OK;
}
