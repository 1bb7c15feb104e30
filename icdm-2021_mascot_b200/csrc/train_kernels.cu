// Per-rating SGD update kernels for sm_100a.
//
// WORKERS.  The reference runs `-wg` warps, each applying one rating at a time; the number of such
// sequential workers decides how many updates of a popular row are lost to races, i.e. how fast the
// model converges per epoch.  This engine keeps that meaning of `-wg` - a worker is a group of
// K/8 lanes (16 for k=128, 8 for k=64; two or four workers per warp), or of K/4 lanes where there are few of them
// (launch_one), that applies its ratings strictly one after the other - and gets its speed from making each worker fast
// instead of adding workers:
//   * every lane holds eight consecutive physical elements of a row (one 128-bit access for
//     binary16 storage, two for fp32), or four of them (one access);
//   * the workers of a warp go through their ratings in step, with whole-warp shuffles, and the loop has no branch
//     that they could take differently: what only some of them do (a new item row, a dropped write-back) is
//     predicated, chunks are fetched and tickets drawn without branches, and a worker that has run out of ratings goes
//     on with empty records.  Per-worker branches cost a warp barrier in front of every shuffle and split the update
//     into pieces that cannot be scheduled into each other: 131 warp instructions per step of all workers of a warp
//     before, 91 now (K/8 lanes a worker, binary16 rows).
//   * what the ratings to come need (records, row copies, the vote on item rows) is done between the dependent shuffles
//     of the dot product instead of in front of it: 8M ratings 1.39 -> 1.295 ms per epoch, fp32 rows 1.70 -> 1.52;
//   * the rating records of a chunk (one rating per lane) are loaded one chunk ahead, tagged
//     (repeated user, start of an item run, repeated item, dropped write-back) and put into shared memory, from where
//     the worker reads one rating with a single 128-bit broadcast load;
//   * rows travel global -> shared memory by cp.async into small per-worker rings, user rows five
//     ratings ahead, item rows three; copy groups complete in order, so the wait for the
//     row of rating j leaves the younger copies in flight (register loads cannot do that: the wait
//     for an old load also waits for every younger load on the same scoreboard);
//   * the row of an item that repeats (the stream is item-sorted inside shuffle windows) stays in
//     registers for the whole run and is written back once;
//   * chunks are handed out in runs of up to K ratings (eight chunks, or four of K/4 lanes) through one atomic ticket per run; the
//     runs shrink to single chunks near the end of the stream, so that all workers finish together.
//   * user rows are written back as vector reductions of their change whenever several workers run,
//     so racing updates of one user add up instead of overwriting each other (add_row_delta).
// The item lead is short on purpose.  Between the request of an item row and its write-back (a plain
// store, once per run) every update another worker makes to that row is lost, so the loss grows with
// (workers x lead time).  The leads are counted in ratings, and a rating takes 0.2 us where it took 0.35 when the leads
// were three and one: the same time, and the same RMSE (0.5169 after one epoch, 0.5180 after six on the k=64
// configuration either way).  With leads of three and two the 8M-rating configuration took 1.65 ms per epoch where it
// took 1.39 with five and three, the k=64 one 1.97 against 1.65; user leads of six and seven gave nothing more.
//
// WHAT BOUNDS IT (one B200, k=128).  Sets with few workers per SM (8M ratings: two warps per scheduler, a worker each): the chain of
// one update - dot product, its sum over the lanes, update - and the 77 instructions around it, 2.42 -> 1.18 ms per epoch (340 cycles a
// rating: 1.5 cycles an instruction wait for results of fixed latency, 0.6 for shared memory and shuffles, 0.5 for L2).  The
// same with fp32 rows 1.24 ms (1.52 with K/8 lanes a worker), and with 278 instructions for 4M ratings of AFP 3.37 (5.69).  Full SMs
// (100M ratings, 7.17 -> 5.50 ms): the traffic between SMs and L2.  The launches that fill the GPU all move 9.9 to 10.2
// TB/s of row reads, stores and reductions (reads alone: 16 to 17.7), whatever else they do: 100M and 126M ratings with
// binary16 rows (541 and 621 bytes an update), 63M with fp32 rows on both sides (SGD, 1,230 bytes; the fp32 class of a
// promoted set, 1,580), with 71 down to 35 % of the issue slots busy and 16 to 28 warps per SM.  Nothing but random rows read with
// cp.async and reduced runs at 17.4e9 binary16 or 9.0e9 fp32 rows/s (20 MB of rows; 16.8 and 8.4 with 127 MB), a reduction
// alone at 24.5e9 and 12.0e9: the 100M-rating set, 18.1e9 updates/s, is there.
//
// ELEMENT ORDER.  layout.cuh stores rows permuted so that lane m of a worker holds the elements of
// reference lanes m and m+16 (k=128) or m, m+16, m+8, m+24 (k=64).  With pair products
// f_j = fma(a_2j, b_2j, a_2j+1 * b_2j+1) the lane partial (f_0 + f_1) + (f_2 + f_3) and a xor
// butterfly over the worker's lanes add exactly the pairs that the reference's per-lane sum and
// shfl_down 16-8-4-2-1 tree add, so results are bit-identical to the reference kernels:
//   all binary16      mascot/mascot_sgd_kernel.h:188-278     binary16 user / fp32 item  :279-342
//   fp32 / binary16   mascot/mascot_sgd_kernel.h:343-407     all fp32                   :408-443
//   (sgd/sgd_kernel.h:35-76 compiles to the same operations as the all-fp32 case)
//   MPT               mpt/mpt_sgd_kernel.h:38-91              fp16 storage (-v 7)  sgd/sgd_kernel.h:110-161
//   MuPPET            muppet/muppet_sgd_kernel.h:121-285      AFP                  afp/afp_sgd_kernel.h:194-371
//   whole-model switching (-v 8)  sgd/sgd_kernel.h:205-326 (binary16 phase = the all-binary16 case above
//   with MuPPET's form of the statistics; fp32 phase = the fp32 trainer)
// including the fused multiply-adds the compiled reference executes.  Every operation is written
// with a rounding-mode intrinsic so that ptxas cannot contract or re-associate anything further.
//
// Bit 31 of a stream id says which arena (binary16 or fp32) the row lives in, which replaces the
// reference's per-rating group search (mascot_sgd_kernel.h:104-180).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "engine.h"
#include "launch_cache.h"
#include "layout.cuh"
#include "scale_bits.h"

namespace mascot {

namespace {

constexpr uint32_t kNoRow = 0xffffffffu;     // never a valid stream id

// MuPPET's trainer is three kernels: passes of 8 bits (KIND_MUPPET), of 12 to 16 bits (this one), and the fp32 trainer's at 32
constexpr int kMuppetHalf = 100;
template <int KIND> constexpr bool kMuppet = KIND == KIND_MUPPET || KIND == kMuppetHalf;

template <int N> struct Vh { __half2 v[N / 2]; };      // a lane's values, physical order
template <int N> struct Vf { float x[N]; };
typedef Vh<8> V8h;
typedef Vf<8> V8f;

// How the rows of one side are stored in a launch.  Known on the host, so the common cases carry no
// per-rating precision test, no unused registers and no oversized ring slots.  The mixed-precision
// trainer keeps its stream partitioned by (user precision, item precision), and every part runs the
// instantiation made for it; ROWS_DYN (precision read from bit 31 of the id, per rating) remains for
// the deterministic single-worker mode, which must follow the stream in its original order.
// ROWS_HALFQ, ROWS_F32Q: a lane holds four elements of a row instead of eight, so that a worker has K/4 lanes.  Lane m and lane
// m + K/8 of a worker share the eight elements that lane m of the wider form would hold: the first has (e0, e4, e1, e5),
// the second (e2, e6, e3, e7) (layout.cuh).  Of an fp32 row lane l thus holds the 16 bytes at 16 l.
enum RowMode { ROWS_HALF = 0, ROWS_F32 = 1, ROWS_DYN = 2, ROWS_HALFQ = 3, ROWS_F32Q = 4 };
template <int MODE> constexpr int kElems = MODE == ROWS_HALFQ || MODE == ROWS_F32Q ? 4 : 8;      // per lane
template <int MODE> constexpr bool kHalfRows = MODE == ROWS_HALF || MODE == ROWS_HALFQ;
template <int MODE> constexpr bool kTwoParts = MODE == ROWS_F32 || MODE == ROWS_DYN;             // a second access for (some) rows
// where a lane's part of a row begins, in bytes
template <int K, int MODE> __device__ __forceinline__ int lane_at(int m) {
    return MODE == ROWS_HALFQ ? 16 * (m & (K / 8 - 1)) + (m & (K / 8) ? 8 : 0) : 16 * m;
}

// A lane's slice of a row as fetched: 16 bytes for binary16 storage, 32 bytes for fp32 storage, half of that with four elements.
template <int MODE> struct Raw { uint4 a, b; };
template <> struct Raw<ROWS_HALF> { uint4 a; };
template <> struct Raw<ROWS_F32Q> { uint4 a; };
template <> struct Raw<ROWS_HALFQ> { uint2 a; };

__device__ __forceinline__ V8h v8h_of(const uint4& a) {
    V8h h;
    h.v[0] = *reinterpret_cast<const __half2*>(&a.x); h.v[1] = *reinterpret_cast<const __half2*>(&a.y);
    h.v[2] = *reinterpret_cast<const __half2*>(&a.z); h.v[3] = *reinterpret_cast<const __half2*>(&a.w);
    return h;
}
__device__ __forceinline__ V8f v8f_of(const uint4& a, const uint4& b) {
    V8f f;
    f.x[0] = __uint_as_float(a.x); f.x[1] = __uint_as_float(a.y); f.x[2] = __uint_as_float(a.z); f.x[3] = __uint_as_float(a.w);
    f.x[4] = __uint_as_float(b.x); f.x[5] = __uint_as_float(b.y); f.x[6] = __uint_as_float(b.z); f.x[7] = __uint_as_float(b.w);
    return f;
}
template <int MODE> __device__ __forceinline__ Vh<kElems<MODE>> as_vh(const Raw<MODE>& r) {
    if constexpr (kElems<MODE> == 8) return v8h_of(r.a);
    else {                                            // binary16 rows never occur in ROWS_F32Q
        Vh<4> h;
        h.v[0] = *reinterpret_cast<const __half2*>(&r.a.x); h.v[1] = *reinterpret_cast<const __half2*>(&r.a.y);
        return h;
    }
}
template <int MODE> __device__ __forceinline__ Vf<kElems<MODE>> as_vf(const Raw<MODE>& r) {
    if constexpr (MODE == ROWS_HALFQ) return Vf<4>{{0.f, 0.f, 0.f, 0.f}};      // fp32 rows never occur here
    else if constexpr (MODE == ROWS_F32Q) return Vf<4>{{__uint_as_float(r.a.x), __uint_as_float(r.a.y), __uint_as_float(r.a.z), __uint_as_float(r.a.w)}};
    else if constexpr (MODE != ROWS_HALF) return v8f_of(r.a, r.b);
    else return v8f_of(r.a, r.a);                     // fp32 rows never occur in ROWS_HALF
}

template <int MODE> __device__ __forceinline__ void put(Raw<MODE>& r, const Vh<kElems<MODE>>& h) {
    r.a.x = *reinterpret_cast<const unsigned*>(&h.v[0]); r.a.y = *reinterpret_cast<const unsigned*>(&h.v[1]);
    if constexpr (kElems<MODE> == 8) { r.a.z = *reinterpret_cast<const unsigned*>(&h.v[2]); r.a.w = *reinterpret_cast<const unsigned*>(&h.v[3]); }
}
template <int MODE> __device__ __forceinline__ void put(Raw<MODE>& r, const Vf<kElems<MODE>>& f) {
    if constexpr (!kHalfRows<MODE>) {
        r.a = make_uint4(__float_as_uint(f.x[0]), __float_as_uint(f.x[1]), __float_as_uint(f.x[2]), __float_as_uint(f.x[3]));
        if constexpr (kTwoParts<MODE>) r.b = make_uint4(__float_as_uint(f.x[4]), __float_as_uint(f.x[5]), __float_as_uint(f.x[6]), __float_as_uint(f.x[7]));
    }
}

template <int N> __device__ __forceinline__ Vf<N> widen(const Vh<N>& h) {
    Vf<N> f;
#pragma unroll
    for (int s = 0; s < N / 2; s++) { const float2 t = __half22float2(h.v[s]); f.x[2 * s] = t.x; f.x[2 * s + 1] = t.y; }
    return f;
}
template <int N> __device__ __forceinline__ Vh<N> narrow(const Vf<N>& f) {
    Vh<N> h;
#pragma unroll
    for (int s = 0; s < N / 2; s++) h.v[s] = __halves2half2(__float2half_rn(f.x[2 * s]), __float2half_rn(f.x[2 * s + 1]));
    return h;
}

// Is the row behind this stream id stored in fp32?
template <int MODE> __device__ __forceinline__ bool is_f32(uint32_t code) {
    return MODE == ROWS_F32 || MODE == ROWS_F32Q || (MODE == ROWS_DYN && (code & kPrecBit));
}

// The rows of one side as a lane sees them: addresses of its slice of row 0 in the two arenas.  (One multiply-add
// makes the address of a row; the second half of an fp32 row is 2 K bytes further on.)
template <int K, int MODE> struct Rows {
    const unsigned char* b16;
    const unsigned char* b32;
    __device__ __forceinline__ Rows(const Arena& A, int m)
        : b16(reinterpret_cast<const unsigned char*>(A.f16) + lane_at<K, MODE>(m)), b32(reinterpret_cast<const unsigned char*>(A.f32) + lane_at<K, MODE>(m)) {}
    __device__ __forceinline__ const unsigned char* at(uint32_t code) const {
        if constexpr (kHalfRows<MODE>) return b16 + (uint64_t)code * (2u * K);
        else if constexpr (MODE == ROWS_F32 || MODE == ROWS_F32Q) return b32 + (uint64_t)code * (4u * K);
        else return (code & kPrecBit) ? b32 + (uint64_t)(code & kIdMask) * (4u * K) : b16 + (uint64_t)(code & kIdMask) * (2u * K);
    }
};

// `go` for the second half of a row: fp32 rows only
template <int MODE> __device__ __forceinline__ unsigned second_half(unsigned go, uint32_t code) {
    return MODE == ROWS_DYN ? ((code & kPrecBit) ? go : 0u) : go;
}

// Predicated accesses to a lane's 16 bytes (8 of ROWS_HALFQ): the code around them stays free of branches, which two or four workers of
// a warp would take one after the other.
template <int OFF> __device__ __forceinline__ void ldg_if(unsigned go, uint4& v, const unsigned char* p) {
    asm volatile("{ .reg .pred g; setp.ne.u32 g, %4, 0; @g ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%5 + %6]; }" : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
                 : "r"(go), "l"(p), "n"(OFF) : "memory");
}
template <int OFF> __device__ __forceinline__ void stg_if(unsigned go, const unsigned char* p, const uint4& v) {
    asm volatile("{ .reg .pred g; setp.ne.u32 g, %4, 0; @g st.global.cg.v4.u32 [%5 + %6], {%0, %1, %2, %3}; }" ::"r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w),
                 "r"(go), "l"(p), "n"(OFF) : "memory");
}
template <int OFF> __device__ __forceinline__ void ldg_if(unsigned go, uint2& v, const unsigned char* p) {
    asm volatile("{ .reg .pred g; setp.ne.u32 g, %2, 0; @g ld.global.cg.v2.u32 {%0, %1}, [%3 + %4]; }" : "+r"(v.x), "+r"(v.y) : "r"(go), "l"(p), "n"(OFF) : "memory");
}
template <int OFF> __device__ __forceinline__ void stg_if(unsigned go, const unsigned char* p, const uint2& v) {
    asm volatile("{ .reg .pred g; setp.ne.u32 g, %2, 0; @g st.global.cg.v2.u32 [%3 + %4], {%0, %1}; }" ::"r"(v.x), "r"(v.y), "r"(go), "l"(p), "n"(OFF) : "memory");
}
template <int OFF> __device__ __forceinline__ void lds_if(unsigned go, uint2& v, unsigned addr) {
    asm volatile("{ .reg .pred g; setp.ne.u32 g, %2, 0; @g ld.shared.v2.u32 {%0, %1}, [%3 + %4]; }" : "+r"(v.x), "+r"(v.y) : "r"(go), "r"(addr), "n"(OFF) : "memory");
}
template <int OFF> __device__ __forceinline__ void lds_if(unsigned go, uint4& v, unsigned addr) {
    asm volatile("{ .reg .pred g; setp.ne.u32 g, %4, 0; @g ld.shared.v4.u32 {%0, %1, %2, %3}, [%5 + %6]; }" : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
                 : "r"(go), "r"(addr), "n"(OFF) : "memory");
}

// Row slice of a lane, L2 only (rows are shared between SMs and never reused from L1).
template <int K, int MODE>
__device__ __forceinline__ void ld_row_if(unsigned go, Raw<MODE>& r, const Rows<K, MODE>& A, uint32_t code) {
    const unsigned char* p = A.at(code);
    ldg_if<0>(go, r.a, p);
    if constexpr (kTwoParts<MODE>) ldg_if<2 * K>(second_half<MODE>(go, code), r.b, p);
}
template <int K, int MODE>
__device__ __forceinline__ void st_row_if(unsigned go, const Rows<K, MODE>& A, uint32_t code, const Raw<MODE>& r) {
    const unsigned char* p = A.at(code);
    stg_if<0>(go, p, r.a);
    if constexpr (kTwoParts<MODE>) stg_if<2 * K>(second_half<MODE>(go, code), p, r.b);
}

// Adds (now - before) to a row, unless `skip`, instead of storing `now`: with several workers on the same row at the
// same time a plain store erases what the others wrote since this worker read the row, a reduction keeps it.  When
// nobody else touched the row the result equals `now` (the difference of two nearby values is exact).  128-bit
// vector reductions, fire and forget, predicated rather than branched around: the update stays one straight piece
// of code, in which the scheduler can fill the latency of the dot product.
template <int OFF> __device__ __forceinline__ void red_f32x4(const unsigned char* p, unsigned skip, float x, float y, float z, float w) {
    asm volatile("{ .reg .pred s; setp.ne.u32 s, %5, 0; @!s red.global.add.v4.f32 [%0 + %6], {%1, %2, %3, %4}; }" ::"l"(p), "f"(x), "f"(y), "f"(z),
                 "f"(w), "r"(skip), "n"(OFF) : "memory");
}
template <int K, int MODE>
__device__ __forceinline__ void add_row_delta(const Rows<K, MODE>& A, uint32_t code, unsigned skip, const Raw<MODE>& now, const Raw<MODE>& before) {
    const unsigned char* p = A.at(code);
    if (is_f32<MODE>(code)) {
        if constexpr (!kHalfRows<MODE>) {
            constexpr int N = kElems<MODE>;
            const Vf<N> n = as_vf(now), o = as_vf(before);
            const float2 minus = make_float2(-1.f, -1.f);      // n - o as fma(-1, o, n): the same single rounding, two lanes at once
            float2 d[N / 2];
#pragma unroll
            for (int j = 0; j < N / 2; j++) d[j] = __ffma2_rn(minus, make_float2(o.x[2 * j], o.x[2 * j + 1]), make_float2(n.x[2 * j], n.x[2 * j + 1]));
            red_f32x4<0>(p, skip, d[0].x, d[0].y, d[1].x, d[1].y);
            if constexpr (kTwoParts<MODE>) red_f32x4<2 * K>(p, skip, d[2].x, d[2].y, d[3].x, d[3].y);
        }
    } else if constexpr (MODE == ROWS_HALFQ) {
        const Vh<4> n = as_vh(now), o = as_vh(before);
        unsigned d[2];
#pragma unroll
        for (int t = 0; t < 2; t++) { const __half2 x = __hsub2(n.v[t], o.v[t]); d[t] = *reinterpret_cast<const unsigned*>(&x); }
        asm volatile("{ .reg .pred s; setp.ne.u32 s, %3, 0; @!s red.global.add.noftz.v2.f16x2 [%0], {%1, %2}; }" ::"l"(p), "r"(d[0]), "r"(d[1]), "r"(skip) : "memory");
    } else if constexpr (MODE != ROWS_F32Q) {
        const V8h n = v8h_of(now.a), o = v8h_of(before.a);
        unsigned d[4];
#pragma unroll
        for (int t = 0; t < 4; t++) { const __half2 x = __hsub2(n.v[t], o.v[t]); d[t] = *reinterpret_cast<const unsigned*>(&x); }
        asm volatile("{ .reg .pred s; setp.ne.u32 s, %5, 0; @!s red.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4}; }" ::"l"(p), "r"(d[0]), "r"(d[1]),
                     "r"(d[2]), "r"(d[3]), "r"(skip) : "memory");
    }
}

// ---- lane partials -------------------------------------------------------------------------
// A lane's elements e0..e7 sit at positions 0 2 4 6 1 3 5 7 (layout.cuh), i.e. as the binary16 pairs
// (e0,e4) (e1,e5) (e2,e6) (e3,e7).  Lane partial: (f_0 + f_1) + (f_2 + f_3) with
// f_j = fma(e_2j, e'_2j, e_2j+1 * e'_2j+1).
// fp32 arithmetic runs on the packed two-lane instructions of sm_100 (fma / mul / add .f32x2): each lane
// is rounded on its own, exactly like the scalar instruction, and a row slice needs half as many issue
// slots - which is what bounds this kernel.
template <int N> __device__ __forceinline__ float2 pr(const Vf<N>& v, int j) { return make_float2(v.x[2 * j], v.x[2 * j + 1]); }
template <int N> __device__ __forceinline__ void set_pr(Vf<N>& v, int j, float2 t) { v.x[2 * j] = t.x; v.x[2 * j + 1] = t.y; }

__device__ __forceinline__ float pair_partial(const V8f& a, const V8f& b) {
    // (f0, f2) = (a0 b0 + a2 b2, a1 b1 + a3 b3), (f1, f3) likewise from positions 4..7
    const float2 f02 = __ffma2_rn(pr(a, 0), pr(b, 0), __fmul2_rn(pr(a, 1), pr(b, 1)));
    const float2 f13 = __ffma2_rn(pr(a, 2), pr(b, 2), __fmul2_rn(pr(a, 3), pr(b, 3)));
    const float2 t = __fadd2_rn(f02, f13);                                     // (f0+f1, f2+f3)
    return __fadd_rn(t.x, t.y);
}
// binary16: both halves of the result hold the lane partial, so the butterfly below and the error need no unpacking.
__device__ __forceinline__ __half2 pair_partial(const V8h& p, const V8h& q) {
    const __half2 f02 = __hfma2(p.v[0], q.v[0], __hmul2_rn(p.v[1], q.v[1]));   // (f_0, f_2)
    const __half2 f13 = __hfma2(p.v[2], q.v[2], __hmul2_rn(p.v[3], q.v[3]));   // (f_1, f_3)
    const __half2 t = __hadd2_rn(f02, f13);                                     // (f_0+f_1, f_2+f_3)
    return __hadd2_rn(__low2half2(t), __high2half2(t));
}
// k=128 only: the left-to-right product chain of a reference lane over its four elements,
// fma(a3,b3, fma(a2,b2, fma(a0,b0, a1*b1))), for the two reference lanes this lane holds
// (fp16-storage trainer sgd/sgd_kernel.h:124, RMSE rmse.h:75).
__device__ __forceinline__ float chain_partial_k128(const V8f& a, const V8f& b) {
    float c[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {          // h = 0: e0..e3 at positions 0 2 4 6;  h = 1: e4..e7 at 1 3 5 7
        float acc = __fmaf_rn(a.x[h], b.x[h], __fmul_rn(a.x[2 + h], b.x[2 + h]));
        acc = __fmaf_rn(a.x[4 + h], b.x[4 + h], acc);
        c[h] = __fmaf_rn(a.x[6 + h], b.x[6 + h], acc);
    }
    return __fadd_rn(c[0], c[1]);
}

// Sum over a worker's lanes.  Three or four dependent shuffles of some 25 cycles each: `mid(i)` is called while shuffle i
// is under way, for work that does not need the sum.
struct Nothing { __device__ __forceinline__ void operator()(int) const {} };
template <int TS, class Mid = Nothing>
__device__ __forceinline__ float worker_sum(float x, unsigned wmask, Mid mid = Mid()) {
#pragma unroll
    for (int d = TS / 2, i = 0; d >= 1; d >>= 1, i++) {
        const float o = __shfl_xor_sync(wmask, x, d);
        mid(i);
        x = __fadd_rn(x, o);
    }
    return x;
}
template <int TS, class Mid = Nothing>
__device__ __forceinline__ __half2 worker_sum(__half2 x, unsigned wmask, Mid mid = Mid()) {
#pragma unroll
    for (int d = TS / 2, i = 0; d >= 1; d >>= 1, i++) {
        const unsigned o = __shfl_xor_sync(wmask, *reinterpret_cast<const unsigned*>(&x), d);
        mid(i);
        x = __hadd2_rn(x, *reinterpret_cast<const __half2*>(&o));
    }
    return x;
}

// Dot product of two rows over a worker's lanes.  With four elements a lane, the two lanes that make up a lane of the wider
// form have (f_0, f_2) and (f_1, f_3): both get the other's pair, and the lane partial and its butterfly follow as above.
template <int TS, class Mid = Nothing>
__device__ __forceinline__ float worker_dot(const V8f& a, const V8f& b, unsigned wmask, Mid mid = Mid()) { return worker_sum<TS>(pair_partial(a, b), wmask, mid); }
template <int TS, class Mid = Nothing>
__device__ __forceinline__ __half2 worker_dot(const V8h& a, const V8h& b, unsigned wmask, Mid mid = Mid()) { return worker_sum<TS>(pair_partial(a, b), wmask, mid); }
template <class Mid> struct After {           // the steps of `mid` from the second on
    Mid mid;
    __device__ __forceinline__ void operator()(int i) const { mid(i + 1); }
};
template <int TS, class Mid = Nothing>
__device__ __forceinline__ float worker_dot(const Vf<4>& a, const Vf<4>& b, unsigned wmask, Mid mid = Mid()) {
    const float2 f = __ffma2_rn(pr(a, 0), pr(b, 0), __fmul2_rn(pr(a, 1), pr(b, 1)));
    const float2 o = make_float2(__shfl_xor_sync(wmask, f.x, TS / 2), __shfl_xor_sync(wmask, f.y, TS / 2));
    mid(0);
    const float2 t = __fadd2_rn(f, o);
    return worker_sum<TS / 2>(__fadd_rn(t.x, t.y), wmask, After<Mid>{mid});
}
template <int TS, class Mid = Nothing>
__device__ __forceinline__ __half2 worker_dot(const Vh<4>& a, const Vh<4>& b, unsigned wmask, Mid mid = Mid()) {
    const __half2 f = __hfma2(a.v[0], b.v[0], __hmul2_rn(a.v[1], b.v[1]));
    const unsigned o = __shfl_xor_sync(wmask, *reinterpret_cast<const unsigned*>(&f), TS / 2);
    mid(0);
    const __half2 t = __hadd2_rn(f, *reinterpret_cast<const __half2*>(&o));
    return worker_sum<TS / 2>(__hadd2_rn(__low2half2(t), __high2half2(t)), wmask, After<Mid>{mid});
}

// The same sum through shared memory: every lane puts its partial down and reads all of them, and adds them up in the order of
// the butterfly - half of the shuffles' latency at as many instructions.  slot: room for the worker's partials, 2 or 4
// bytes each; steps take two of them in turn, so that one warp barrier a step keeps what is read from what is written next.
__device__ __forceinline__ uint4 lds128(unsigned addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
template <int P, class Mid>
__device__ __forceinline__ __half2 tree_sum(__half2 x, unsigned slot, Mid mid) {      // x: the partial in both halves
    static_assert(P == 16 || P == 8, "partials of a worker");
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(slot + 2 * (threadIdx.x & (P - 1))), "h"(__half_as_ushort(__low2half(x))) : "memory");
    __syncwarp();
    mid(0);
    auto h2 = [](uint32_t w) { return *reinterpret_cast<const __half2*>(&w); };
    const uint4 a = lds128(slot);
    __half2 c;
    if constexpr (P == 16) {
        const uint4 b = lds128(slot + 16);
        mid(1); mid(2);
        const __half2 s0 = __hadd2_rn(h2(a.x), h2(b.x)), s1 = __hadd2_rn(h2(a.y), h2(b.y)), s2 = __hadd2_rn(h2(a.z), h2(b.z)), s3 = __hadd2_rn(h2(a.w), h2(b.w));
        c = __hadd2_rn(__hadd2_rn(s0, s2), __hadd2_rn(s1, s3));
    } else {
        mid(1); mid(2);
        c = __hadd2_rn(__hadd2_rn(h2(a.x), h2(a.z)), __hadd2_rn(h2(a.y), h2(a.w)));
    }
    return __hadd2_rn(__low2half2(c), __high2half2(c));
}
template <int P, class Mid>
__device__ __forceinline__ float tree_sum(float x, unsigned slot, Mid mid, bool who = true) {      // who: lanes that have a partial
    if (who) asm volatile("st.shared.f32 [%0], %1;" ::"r"(slot + 4 * (threadIdx.x & (P - 1))), "f"(x) : "memory");
    __syncwarp();
    mid(0);
    auto f2 = [](uint32_t lo, uint32_t hi) { return make_float2(__uint_as_float(lo), __uint_as_float(hi)); };
    const uint4 a = lds128(slot), b = lds128(slot + 16);
    float2 s0, s1;                                     // sums of the partials 0 1 and 2 3 modulo 4
    if constexpr (P == 16) {
        const uint4 c = lds128(slot + 32), d = lds128(slot + 48);
        mid(1); mid(2);
        s0 = __fadd2_rn(__fadd2_rn(f2(a.x, a.y), f2(c.x, c.y)), __fadd2_rn(f2(b.x, b.y), f2(d.x, d.y)));
        s1 = __fadd2_rn(__fadd2_rn(f2(a.z, a.w), f2(c.z, c.w)), __fadd2_rn(f2(b.z, b.w), f2(d.z, d.w)));
    } else {
        mid(1); mid(2);
        s0 = __fadd2_rn(f2(a.x, a.y), f2(b.x, b.y));
        s1 = __fadd2_rn(f2(a.z, a.w), f2(b.z, b.w));
    }
    const float2 s = __fadd2_rn(s0, s1);
    return __fadd_rn(s.x, s.y);
}
// The same for pairs of binary16 sums; who: lanes that have a partial
template <int P> __device__ __forceinline__ __half2 tree_sum2(__half2 x, bool who, unsigned slot) {
    if (who) asm volatile("st.shared.u32 [%0], %1;" ::"r"(slot + 4 * (threadIdx.x & (P - 1))), "r"(*reinterpret_cast<const unsigned*>(&x)) : "memory");
    __syncwarp();
    auto h2 = [](uint32_t w) { return *reinterpret_cast<const __half2*>(&w); };
    uint4 v[P / 4];
#pragma unroll
    for (int j = 0; j < P / 4; j++) v[j] = lds128(slot + 16 * j);
    __half2 s[4];                                      // sums of the partials 0, 1, 2, 3 modulo 4
    if constexpr (P == 16) {
        s[0] = __hadd2_rn(__hadd2_rn(h2(v[0].x), h2(v[2].x)), __hadd2_rn(h2(v[1].x), h2(v[3].x)));
        s[1] = __hadd2_rn(__hadd2_rn(h2(v[0].y), h2(v[2].y)), __hadd2_rn(h2(v[1].y), h2(v[3].y)));
        s[2] = __hadd2_rn(__hadd2_rn(h2(v[0].z), h2(v[2].z)), __hadd2_rn(h2(v[1].z), h2(v[3].z)));
        s[3] = __hadd2_rn(__hadd2_rn(h2(v[0].w), h2(v[2].w)), __hadd2_rn(h2(v[1].w), h2(v[3].w)));
    } else {
        s[0] = __hadd2_rn(h2(v[0].x), h2(v[1].x)); s[1] = __hadd2_rn(h2(v[0].y), h2(v[1].y));
        s[2] = __hadd2_rn(h2(v[0].z), h2(v[1].z)); s[3] = __hadd2_rn(h2(v[0].w), h2(v[1].w));
    }
    return __hadd2_rn(__hadd2_rn(s[0], s[2]), __hadd2_rn(s[1], s[3]));
}
// Dot product with that sum
template <int K, class Mid> __device__ __forceinline__ float tree_dot(const Vf<4>& a, const Vf<4>& b, unsigned slot, Mid mid) {
    const float2 f = __ffma2_rn(pr(a, 0), pr(b, 0), __fmul2_rn(pr(a, 1), pr(b, 1)));
    const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, f.x, K / 8), __shfl_xor_sync(0xffffffffu, f.y, K / 8));
    const float2 t = __fadd2_rn(f, o);
    return tree_sum<K / 8>(__fadd_rn(t.x, t.y), slot, mid);
}
template <int K, class Mid> __device__ __forceinline__ __half2 tree_dot(const Vh<4>& a, const Vh<4>& b, unsigned slot, Mid mid) {
    const __half2 f = __hfma2(a.v[0], b.v[0], __hmul2_rn(a.v[1], b.v[1]));
    const unsigned o = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<const unsigned*>(&f), K / 8);
    const __half2 t = __hadd2_rn(f, *reinterpret_cast<const __half2*>(&o));
    return tree_sum<K / 8>(__hadd2_rn(__low2half2(t), __high2half2(t)), slot, mid);
}

// The chain over four lanes' worth of elements where a lane has two of each: the lanes with e0, e1 begin, those with e2, e3 go on,
// and put down what is added up.
template <int K, class Mid>
__device__ __forceinline__ float tree_chain_k128(const Vf<4>& a, const Vf<4>& b, unsigned slot, Mid mid) {
    float c[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const float begun = __shfl_xor_sync(0xffffffffu, __fmaf_rn(a.x[h], b.x[h], __fmul_rn(a.x[2 + h], b.x[2 + h])), K / 8);
        c[h] = __fmaf_rn(a.x[2 + h], b.x[2 + h], __fmaf_rn(a.x[h], b.x[h], begun));
    }
    return tree_sum<K / 8>(__fadd_rn(c[0], c[1]), slot, mid, threadIdx.x & (K / 8));
}

// t = fma(e, y, -(lam*x)) and x' = fma(lr, t, x), element-wise
template <int N> __device__ __forceinline__ Vf<N> grad(float e, const Vf<N>& y, float lam, const Vf<N>& x) {
    Vf<N> g;
    const float2 e2 = make_float2(e, e), nlam2 = make_float2(-lam, -lam);      // (-lam) * x == -(lam * x), bit for bit
#pragma unroll
    for (int j = 0; j < N / 2; j++) set_pr(g, j, __ffma2_rn(e2, pr(y, j), __fmul2_rn(nlam2, pr(x, j))));
    return g;
}
template <int N> __device__ __forceinline__ Vh<N> grad(__half2 e, const Vh<N>& y, __half2 nlam, const Vh<N>& x) {
    Vh<N> g;
#pragma unroll
    for (int s = 0; s < N / 2; s++) g.v[s] = __hfma2(e, y.v[s], __hmul2_rn(nlam, x.v[s]));     // (-lam) * x == -(lam * x), bit for bit
    return g;
}
template <int N> __device__ __forceinline__ Vf<N> step(float lr, const Vf<N>& g, const Vf<N>& x) {
    Vf<N> o;
    const float2 lr2 = make_float2(lr, lr);
#pragma unroll
    for (int j = 0; j < N / 2; j++) set_pr(o, j, __ffma2_rn(lr2, pr(g, j), pr(x, j)));
    return o;
}
template <int N> __device__ __forceinline__ Vh<N> step(__half2 lr, const Vh<N>& g, const Vh<N>& x) {
    Vh<N> o;
#pragma unroll
    for (int s = 0; s < N / 2; s++) o.v[s] = __hfma2(lr, g.v[s], x.v[s]);
    return o;
}

// Minimum and sum of an integer over a worker's lanes, all workers of the warp at once: one warp-wide reduction per
// worker, to which the other workers' lanes give nothing.  They do not depend on one another, where a butterfly is
// a chain of shuffles.
template <int TS, class Op> __device__ __forceinline__ int worker_redux(int v, int nothing, Op op) {
    const int w = (threadIdx.x & 31) / TS;
    int mine = nothing;
#pragma unroll
    for (int i = 0; i < 32 / TS; i++) {
        const int r = op(w == i ? v : nothing);
        mine = w == i ? r : mine;
    }
    return mine;
}
template <int TS> __device__ __forceinline__ int worker_min(int v) { return worker_redux<TS>(v, 0x7fffffff, [](int x) { return __reduce_min_sync(0xffffffffu, x); }); }
template <int TS> __device__ __forceinline__ int worker_add(int v) { return worker_redux<TS>(v, 0, [](int x) { return __reduce_add_sync(0xffffffffu, x); }); }

struct Consts {
    float lr, lam;
    __half2 lr_h, nlam_h;         // mascot_sgd_kernel.h:79-80 (lambda negated)
    __half2 mpt_scale;            // mpt_sgd_kernel.h:15-16
    __half2 mpt_nlam;             // mf_methods.cu:764-765 (negated)
    float mpt_rev;
    int bits;                     // MuPPET: width of the forward and the backward pass
    int afp_epoch, afp_init_threshold;   // AFP: epoch index; ratings per worker / 10 (afp_sgd_kernel.h:143)
};

// Sampled statistics (mascot_sgd_kernel.h:240-277): per group the element-wise sum of the gradients
// and the sum of their squared norms.  They go to global memory as 128-bit fire-and-forget
// reductions.  The reference adds every rating's gradient with scalar atomics in no particular
// order; here the user side does the same per rating, while the item side - whose ratings arrive in
// runs of the same group, because shuffle windows are item-sorted - is summed in registers over a run
// of equal item groups and flushed once per run, which removes the contention on popular items.
template <int N> struct Sample {
    Vf<N> gp, gq;
    bool user, item;      // which sides of this rating contribute (binary16-stored rows only)
};

// ... unless `skip`
template <int N> __device__ __forceinline__ void red_add_if_not(unsigned skip, float* dst, const Vf<N>& g) {
    const unsigned char* const p = reinterpret_cast<const unsigned char*>(dst);
    red_f32x4<0>(p, skip, g.x[0], g.x[1], g.x[2], g.x[3]);
    if constexpr (N == 8) red_f32x4<16>(p, skip, g.x[4], g.x[5], g.x[6], g.x[7]);
}
__device__ __forceinline__ void red_add_if_not(unsigned skip, float* dst, float x) {
    asm volatile("{ .reg .pred s; setp.ne.u32 s, %2, 0; @!s red.global.add.f32 [%0], %1; }" ::"l"(dst), "f"(x), "r"(skip) : "memory");
}
template <int N> __device__ __forceinline__ void red_add(float* dst, const Vf<N>& g) {
    atomicAdd(reinterpret_cast<float4*>(dst), make_float4(g.x[0], g.x[1], g.x[2], g.x[3]));
    if constexpr (N == 8) atomicAdd(reinterpret_cast<float4*>(dst) + 1, make_float4(g.x[4], g.x[5], g.x[6], g.x[7]));
}

struct KernelArgs {
    Stream s;
    Arena P, Q;
    float lr, lam;
    SampleStats st;
    int bits;                     // MuPPET pass width
    int epoch;                    // AFP: epoch index
    int add_user_delta;           // user rows are written back as reductions of the change (concurrent launches)
    unsigned workers;             // concurrent sequential workers actually launched
    unsigned spread;              // AFP: log2 of how few of its workers a warp has, (32 / lanes of a worker) >> spread
    unsigned long long* next_chunk;   // work counter, zero at launch: chunks beyond the first two runs per
                                      // worker are handed out dynamically, so the launch never depends on
                                      // every block being resident at the same time
    unsigned long long* zero_counter; // another counter, which this launch resets for a later launch
    uint64_t whole;                   // host only: ratings of the epoch or segment that this launch is a part of
    unsigned hot_user_shift;          // one in 2^this of the updates of a marked user row is written back
};

// ---- MuPPET (muppet/muppet_sgd_kernel.h:7-48, 121-264; _k64.h) -------------------------------
// Power-of-two scale for a `bits`-wide fixed-point grid that covers [lo, hi]: the reference takes
// floor(log2(min(|qmax/hi|, |qmin/lo|))) with qmax = 2^(bits-1)-0.5, qmin = -2^(bits-1)-0.5, stores
// it in an unsigned index (negative -> 0) and scales by 2^index.
__device__ __noinline__ float muppet_scale_exact(float top, float bottom, float hi, float lo) {
    const float best = fminf(fabsf(__fdiv_rn(top, hi)), fabsf(__fdiv_rn(bottom, lo)));
    const float idx = floorf(log2f(best));
    if (!(idx > 0.f)) return 1.f;
    const int e = idx > 127.f ? 128 : (int)idx;
    return e >= 128 ? __int_as_float(0x7f800000) : __int_as_float((e + 127) << 23);
}
// The scale is a power of two and only floor(log2) of the smaller quotient decides it, which the bit patterns tell
// without a division: as integers, bits(a) - bits(b) has floor(log2(a / b)) above bit 23 for normal a, b > 0 (the
// difference of the exponents, less one when the mantissa of b is the larger).  Where the quotient is within 256 units of
// a power of two - once in ten thousand ratings - or an operand is zero or denormal, the formula itself decides, with its
// rounded divisions and logarithm.
__device__ __forceinline__ float muppet_scale(int bits, float hi, float lo) {
    const float val = (float)(1 << (bits - 1));
    const float top = __fadd_rn(__fsub_rn(val, 1.f), 0.5f), bottom = __fsub_rn(-val, 0.5f);
    const int d = min(__float_as_int(top) - (__float_as_int(hi) & 0x7fffffff), __float_as_int(-bottom) - (__float_as_int(lo) & 0x7fffffff));
    float s = __uint_as_float(scale_bits(d));
    if (((d + 256) & 0x007fffff) < 512 || d >= (120 << 23)) s = (hi == 0.f && lo == 0.f) ? 1.f : muppet_scale_exact(top, bottom, hi, lo);
    return s;
}
// The same over the lanes of a worker without knowing the extremes: the difference above is the smaller of two, and so is its
// minimum over any parts of the values, here the eight of a lane.  Values on one side of zero only are the exception.  If
// all are positive the result stands (the upper bound is the nearer one); if all are negative, the one with the
// smallest magnitude against the upper bound may decide, by as much as the bounds differ.  `scale_unsure` is wider by that.
__device__ __forceinline__ int2 scale_bounds(int bits) {
    const float val = (float)(1 << (bits - 1));
    return make_int2(__float_as_int(__fadd_rn(__fsub_rn(val, 1.f), 0.5f)), __float_as_int(-__fsub_rn(-val, 0.5f)));
}
__device__ __forceinline__ int scale_key(int2 bound, float hi, float lo) {
    return min(bound.x - max(__float_as_int(hi), 0), bound.y - max(__float_as_int(-lo), 0));
}
__device__ __forceinline__ float scale_of(int key) { return __uint_as_float(scale_bits(key)); }
// (From 2^60 on, the formula too: below that the reciprocal of a product of two scales is a normal number, and comes from the bits.)
__device__ __forceinline__ bool scale_unsure(int2 bound, int key) { return ((key + 256) & 0x007fffff) < 512 + bound.y - bound.x || key >= (60 << 23); }
__device__ __forceinline__ float near_rev(float s) { return __uint_as_float(rev_bits(__float_as_uint(s))); }
__device__ __forceinline__ float near_rev(float s, float t) { return __uint_as_float(rev_bits(__float_as_uint(s), __float_as_uint(t))); }
// roundf (halves away from zero) in three instructions: trunc(x + copysign(largest float below one half, x)).
// The sum is rounded to nearest-even, which is what makes it exact: x = n + f with f < 1/2 cannot reach n + 1,
// f >= 1/2 always does.  Equal to roundf for every one of the 2^32 float patterns (checked exhaustively on the
// host, tests/round_check.c); the library routine costs about three times as much.
__device__ __forceinline__ float round_away(float x) {
    const float h = __uint_as_float((__float_as_uint(x) & 0x80000000u) | 0x3effffffu);
    return truncf(__fadd_rn(x, h));
}
// 1 / s for a scale that is a power of two: the exponent mirrored around zero, exact while both s and 1 / s are
// normal numbers; anything else (2^127, infinity) takes the division.
__device__ __forceinline__ float pow2_rev(float s) {
    const uint32_t b = __float_as_uint(s);
    return (b >= 0x00800000u && b < 0x7f000000u && !(b & 0x007fffffu)) ? __uint_as_float(0x7f000000u - b) : __fdiv_rn(1.f, s);
}
__device__ __forceinline__ float fix_round(float v, float s, float s_rev) { return __fmul_rn(round_away(__fmul_rn(v, s)), s_rev); }
// The values of a lane times a power-of-two scale, rounded like round_away - with full-rate instructions, two
// values at a time, in place of truncations and conversions, which run at an eighth of that rate and were 64 of an
// update's instructions.  x s is exact, so adding 1.5 * 2^23 in one multiply-add rounds it to the nearest integer, and the
// two roundings differ at exact halves only: `odd` receives the largest distance from the integers, and a warp
// that meets one half (rare: it takes the bits of x below the grid to be 100...0) rounds again the long way.  Results are
// exact below 2^22, larger ones stay above 2^21, and zero is +0.
template <int N> __device__ __forceinline__ Vf<N> quantize_near(const Vf<N>& x, float s, float& odd) {
    Vf<N> o;
    float far[N / 2];
    const float2 s2 = make_float2(s, s), magic = make_float2(12582912.f, 12582912.f), minus = make_float2(-12582912.f, -12582912.f);
#pragma unroll
    for (int j = 0; j < N / 2; j++) {
        const float2 r = __fadd2_rn(__ffma2_rn(pr(x, j), s2, magic), minus);
        const float2 d = __ffma2_rn(pr(x, j), s2, make_float2(-r.x, -r.y));
        far[j] = fmaxf(fabsf(d.x), fabsf(d.y));
        set_pr(o, j, r);
    }
    odd = fmaxf(far[0], far[1]);
    if constexpr (N == 8) odd = fmaxf(odd, fmaxf(far[2], far[3]));
    return o;
}
// The same for two values that all lanes have
__device__ __forceinline__ float2 quantize_near(float2 x, float s, float& odd) {
    const float2 s2 = make_float2(s, s), magic = make_float2(12582912.f, 12582912.f), minus = make_float2(-12582912.f, -12582912.f);
    const float2 r = __fadd2_rn(__ffma2_rn(x, s2, magic), minus), d = __ffma2_rn(x, s2, make_float2(-r.x, -r.y));
    odd = fmaxf(fabsf(d.x), fabsf(d.y));
    return r;
}
template <int N> __device__ __forceinline__ Vf<N> quantize_away(const Vf<N>& x, float s) {
    Vf<N> o;
#pragma unroll
    for (int t = 0; t < N; t++) o.x[t] = __fadd_rn(round_away(__fmul_rn(x.x[t], s)), 0.f);
    return o;
}
// The int8 passes work on the integers as floats: products and sums of int8 values stay far below 2^24.
__device__ __forceinline__ float clamp8(float v) { return v == v ? fminf(fmaxf(v, -128.f), 127.f) : 0.f; }
template <int N> __device__ __forceinline__ Vf<N> clamp8(const Vf<N>& x) {
    Vf<N> o;
#pragma unroll
    for (int t = 0; t < N; t++) o.x[t] = clamp8(x.x[t]);
    return o;
}
__device__ __forceinline__ float quantize8(float v, float s) { return clamp8(round_away(__fmul_rn(v, s))); }
// A rounded row in binary16; what rounded to zero keeps its sign, as it does in fix_round
template <int N> __device__ __forceinline__ Vh<N> grid_half(const Vf<N>& r, const Vf<N>& x, float s_rev) {
    Vh<N> h;
    const float2 rev2 = make_float2(s_rev, s_rev);
    auto signed_as = [](float v, float like) { return __uint_as_float(__float_as_uint(v) | (__float_as_uint(like) & 0x80000000u)); };
#pragma unroll
    for (int t = 0; t < N / 2; t++)
        h.v[t] = __float22half2_rn(__fmul2_rn(make_float2(signed_as(r.x[2 * t], x.x[2 * t]), signed_as(r.x[2 * t + 1], x.x[2 * t + 1])), rev2));
    return h;
}
template <int N> __device__ __forceinline__ Vh<N> fix_round_half(const Vf<N>& x, float s, float s_rev) {
    Vh<N> h;
#pragma unroll
    for (int t = 0; t < N / 2; t++)
        h.v[t] = __floats2half2_rn(fix_round(x.x[2 * t], s, s_rev), fix_round(x.x[2 * t + 1], s, s_rev));
    return h;
}
// Both rounded rows on their grids; `big`: some value may reach 2^21 steps of its grid
template <int N>
__device__ __forceinline__ void to_grid(const Vf<N>& p, const Vf<N>& pi, float sp, float sp_rev, const Vf<N>& q, const Vf<N>& qi, float sq, float sq_rev, bool big,
                                        Vh<N>& ph, Vh<N>& qh) {
    if (__builtin_expect(big, 0)) { ph = fix_round_half(p, sp, sp_rev); qh = fix_round_half(q, sq, sq_rev); }
    else { ph = grid_half(pi, p, sp_rev); qh = grid_half(qi, q, sq_rev); }
}
template <int N> __device__ __forceinline__ float abs_max(const Vf<N>& x) {
    const float m = fmaxf(fmaxf(fabsf(x.x[0]), fabsf(x.x[1])), fmaxf(fabsf(x.x[2]), fabsf(x.x[3])));
    if constexpr (N == 4) return m;
    else return fmaxf(m, fmaxf(fmaxf(fabsf(x.x[4]), fabsf(x.x[5])), fmaxf(fabsf(x.x[6]), fabsf(x.x[7]))));
}
template <int TS> __device__ __forceinline__ float worker_max(float x, unsigned wmask) {
#pragma unroll
    for (int d = TS / 2; d >= 1; d >>= 1) x = fmaxf(x, __shfl_xor_sync(wmask, x, d));
    return x;
}
// Four maxima over a worker's lanes.  The first two steps halve what a lane holds instead of reducing all four
// everywhere: nine shuffles (k=128) in place of sixteen.
template <int TS> __device__ __forceinline__ void worker_max4(float (&a)[4], unsigned wmask) {
    const int m = threadIdx.x & (TS - 1);
    const bool up = m & (TS / 2), up2 = m & (TS / 4);
    float r0 = fmaxf(up ? a[2] : a[0], __shfl_xor_sync(wmask, up ? a[0] : a[2], TS / 2));
    const float r1 = fmaxf(up ? a[3] : a[1], __shfl_xor_sync(wmask, up ? a[1] : a[3], TS / 2));
    r0 = fmaxf(up2 ? r1 : r0, __shfl_xor_sync(wmask, up2 ? r0 : r1, TS / 4));
#pragma unroll
    for (int d = TS / 8; d >= 1; d >>= 1) r0 = fmaxf(r0, __shfl_xor_sync(wmask, r0, d));
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = __shfl_sync(wmask, r0, (i >> 1) * (TS / 2) + (i & 1) * (TS / 4), TS);
}
template <int N> __device__ __forceinline__ float max_of(const Vf<N>& x) {
    const float m = fmaxf(fmaxf(x.x[0], x.x[1]), fmaxf(x.x[2], x.x[3]));
    if constexpr (N == 4) return m;
    else return fmaxf(m, fmaxf(fmaxf(x.x[4], x.x[5]), fmaxf(x.x[6], x.x[7])));
}
template <int N> __device__ __forceinline__ float min_of(const Vf<N>& x) {
    const float m = fminf(fminf(x.x[0], x.x[1]), fminf(x.x[2], x.x[3]));
    if constexpr (N == 4) return m;
    else return fminf(m, fminf(fminf(x.x[4], x.x[5]), fminf(x.x[6], x.x[7])));
}
// Squared norm of both gradients the way the reference groups it: per reference lane
// (norm_p + norm_q), then the lane tree.  A lane here holds two (k=128) or four (k=64) reference lanes; with four elements a
// lane it holds half of each (k=128) or two of them (k=64), and muppet_norm_join adds what lane l ^ K/8 holds.
template <int K> __device__ __forceinline__ float4 muppet_norm_parts(const Vf<4>& gp, const Vf<4>& gq) {
    auto sq = [](const Vf<4>& g, int a, int b) { return __fmaf_rn(g.x[a], g.x[a], __fmul_rn(g.x[b], g.x[b])); };
    const float4 s = make_float4(sq(gp, 0, 2), sq(gp, 1, 3), sq(gq, 0, 2), sq(gq, 1, 3));
    return K == 128 ? s : make_float4(__fadd_rn(s.x, s.z), __fadd_rn(s.y, s.w), 0.f, 0.f);
}
template <int K> __device__ __forceinline__ float muppet_norm_join(const float4& s) {
    auto both = [](float v) { return __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, K / 8)); };
    if (K == 128) {
        const float a = both(s.x), b = both(s.y), c = both(s.z), d = both(s.w);
        return __fadd_rn(__fadd_rn(a, c), __fadd_rn(b, d));
    }
    const float a = both(s.x), b = both(s.y);
    return __fadd_rn(a, b);
}
template <int K>
__device__ __forceinline__ float muppet_norm_partial(const V8f& gp, const V8f& gq) {
    auto sq = [](const V8f& g, int a, int b) { return __fmaf_rn(g.x[a], g.x[a], __fmul_rn(g.x[b], g.x[b])); };
    if (K == 128) {
        const float la = __fadd_rn(__fadd_rn(sq(gp, 0, 2), sq(gp, 4, 6)), __fadd_rn(sq(gq, 0, 2), sq(gq, 4, 6)));
        const float lb = __fadd_rn(__fadd_rn(sq(gp, 1, 3), sq(gp, 5, 7)), __fadd_rn(sq(gq, 1, 3), sq(gq, 5, 7)));
        return __fadd_rn(la, lb);
    }
    const float l0 = __fadd_rn(sq(gp, 0, 2), sq(gq, 0, 2)), l1 = __fadd_rn(sq(gp, 4, 6), sq(gq, 4, 6));
    const float l2 = __fadd_rn(sq(gp, 1, 3), sq(gq, 1, 3)), l3 = __fadd_rn(sq(gp, 5, 7), sq(gq, 5, 7));
    return __fadd_rn(__fadd_rn(l0, l1), __fadd_rn(l2, l3));
}

// ---- passes shared by MuPPET and AFP ------------------------------------------------------------
// int8 forward pass: saturated fixed-point values, exact integer dot product, one division (by a power of two).
// pi, qi: rounded rows, clamped if need be; rev: 1 / (product of their scales).  A lane's sum stays below 2^18, the whole one below 2^22, so both pass
// between integer and float in the low bits of 1.5 * 2^23 + x.
template <int TS, int N>
__device__ __forceinline__ float forward_int8(const Vf<N>& pi, const Vf<N>& qi, float rev) {
    float2 a = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < N / 2; j++) a = __ffma2_rn(pr(pi, j), pr(qi, j), a);
    const int whole = worker_add<TS>(__float_as_int(__fadd_rn(__fadd_rn(a.x, a.y), 12582912.f)) - 0x4b400000);
    return __fmul_rn(__fsub_rn(__int_as_float(whole + 0x4b400000), 12582912.f), rev);
}
// binary16 forward pass on the fixed-point grid; the two halves of the reference's half2 accumulator
// go through the lane tree separately and meet at the end (muppet_sgd_kernel.h:170-194,
// afp_sgd_kernel.h:252-273)
template <int K>
__device__ __forceinline__ float forward_half(const V8h& ph, const V8h& qh, unsigned wmask, unsigned) {
    constexpr int TS = K / 8;
    __half2 xy;
    if (K == 128) {
        const __half2 xab = __hfma2(ph.v[0], qh.v[0], __hmul2_rn(ph.v[2], qh.v[2]));   // (x of lane m, x of lane m+16)
        const __half2 yab = __hfma2(ph.v[1], qh.v[1], __hmul2_rn(ph.v[3], qh.v[3]));
        xy = __hadd2_rn(__lows2half2(xab, yab), __highs2half2(xab, yab));              // tree step 16
    } else {
        const __half2 x = __hadd2_rn(__hmul2_rn(ph.v[0], qh.v[0]), __hmul2_rn(ph.v[2], qh.v[2]));   // step 16: (m)+(m+16), (m+8)+(m+24)
        const __half2 y = __hadd2_rn(__hmul2_rn(ph.v[1], qh.v[1]), __hmul2_rn(ph.v[3], qh.v[3]));
        xy = __hadd2_rn(__lows2half2(x, y), __highs2half2(x, y));                                   // step 8
    }
#pragma unroll
    for (int d = TS / 2; d >= 1; d >>= 1) {
        const unsigned o = __shfl_xor_sync(wmask, *reinterpret_cast<unsigned*>(&xy), d);
        xy = __hadd2_rn(xy, *reinterpret_cast<const __half2*>(&o));
    }
    return __half2float(__hadd_rn(__low2half(xy), __high2half(xy)));
}
// The same with four elements a lane.  K=128: the lanes with (e2, e6, e3, e7) hand their products to those that have the first
// terms of the sums.  K=64: both lanes add both products.
template <int K>
__device__ __forceinline__ float forward_half(const Vh<4>& ph, const Vh<4>& qh, unsigned wmask, unsigned slot) {
    auto other = [&](const __half2& v) {
        const unsigned o = __shfl_xor_sync(wmask, *reinterpret_cast<const unsigned*>(&v), K / 8);
        return *reinterpret_cast<const __half2*>(&o);
    };
    const __half2 m0 = __hmul2_rn(ph.v[0], qh.v[0]), m1 = __hmul2_rn(ph.v[1], qh.v[1]);
    const __half2 o0 = other(m0), o1 = other(m1);
    __half2 xab, yab;
    if (K == 128) { xab = __hfma2(ph.v[0], qh.v[0], o0); yab = __hfma2(ph.v[1], qh.v[1], o1); }
    else { xab = __hadd2_rn(m0, o0); yab = __hadd2_rn(m1, o1); }
    const __half2 xy = tree_sum2<K / 8>(__hadd2_rn(__lows2half2(xab, yab), __highs2half2(xab, yab)), !(threadIdx.x & (K / 8)), slot);
    return __half2float(__hadd_rn(__low2half(xy), __high2half(xy)));
}
// backward passes: g_p = q*e + p*(-lam), g_q = p*e + q*(-lam) in int8 or binary16 fixed point; e, l: error and -lam on the grid, rev: 1 / (sb sb)
template <int N> __device__ __forceinline__ void backward_int8(const Vf<N>& pi, const Vf<N>& qi, float e, float l, float rev, Vf<N>& gp, Vf<N>& gq) {
    const float2 rev2 = make_float2(rev, rev), e2 = make_float2(e, e), l2 = make_float2(l, l), zero = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < N / 2; j++) {      // + 0: the integer sum has no negative zero
        set_pr(gp, j, __ffma2_rn(__ffma2_rn(pr(qi, j), e2, __fmul2_rn(pr(pi, j), l2)), rev2, zero));
        set_pr(gq, j, __ffma2_rn(__ffma2_rn(pr(pi, j), e2, __fmul2_rn(pr(qi, j), l2)), rev2, zero));
    }
}
template <int N> __device__ __forceinline__ void backward_half(const Vh<N>& ph, const Vh<N>& qh, __half2 e2, __half2 l2, Vf<N>& gp, Vf<N>& gq) {
    Vh<N> gph, gqh;
#pragma unroll
    for (int t = 0; t < N / 2; t++) {
        gph.v[t] = __hadd2_rn(__hmul2_rn(qh.v[t], e2), __hmul2_rn(ph.v[t], l2));
        gqh.v[t] = __hadd2_rn(__hmul2_rn(ph.v[t], e2), __hmul2_rn(qh.v[t], l2));
    }
    gp = widen(gph); gq = widen(gqh);
}

// Do some of the values [lo, hi] times s round to something outside the int8 range?  (The scale is chosen so that
// hardly ever one does.)  An infinite scale (rows of nothing but tiny values) counts as outside.
__device__ __forceinline__ bool outside8(float hi, float lo, float s) { return !(__fmul_rn(hi, s) <= 127.25f && __fmul_rn(lo, s) >= -128.25f); }
__device__ __forceinline__ bool beyond_grid(float hi, float lo, float s) { return !(__fmul_rn(fmaxf(hi, -lo), s) < 2097152.f); }

// Where scale_unsure: the formula itself, from the extremes of the rows
template <int TS> __device__ __noinline__ float2 muppet_scales_exact(int bits, float phi, float plo, float qhi, float qlo) {
    float a[4] = {phi, -plo, qhi, -qlo};
    worker_max4<TS>(a, 0xffffffffu);
    return make_float2(muppet_scale(bits, a[0], -a[1]), muppet_scale(bits, a[2], -a[3]));
}
template <int TS> __device__ __noinline__ float muppet_back_scale_exact(int bits, float hi, float lo, float nlam, float ruv) {
    hi = worker_max<TS>(hi, 0xffffffffu);
    lo = -worker_max<TS>(-lo, 0xffffffffu);
    return muppet_scale(bits, fmaxf(hi, fmaxf(nlam, ruv)), fminf(lo, fminf(nlam, ruv)));
}
// The workers of a warp go through this together.  mid(0) .. mid(3): as in update_one, between the steps of one rating's
// chain: extremes -> scales -> rows on the grid -> dot product -> scale of the gradients -> rows on that grid.  With some
// hundred workers that chain is the epoch, so what shortens it counts: keys in place of four extremes, warp-wide
// integer reductions in place of shuffles, one vote a pass, the norm of the rating before on the side.  2M ratings, 592
// workers: 2.98 -> 2.25 ms per epoch.
// A pass has one vote: is there a scale that the keys leave open, an exact half, a value outside the int8 range (or at 2^21
// steps of its grid)?  The rows are rounded with the scale of the keys before that is known, and again where it is so.
// INT8: passes of 8 bits; else 12 to 16 bits on a binary16 grid.
template <int K, bool INT8, int N, class Mid>
__device__ __forceinline__ void muppet_update(const Consts& c, float r, Vf<N>& p, Vf<N>& q, Vf<N>& gp, Vf<N>& gq, unsigned slot, Mid mid) {
    constexpr int TS = K / N;
    constexpr unsigned kAll = 0xffffffffu;
    const int bits = INT8 ? 8 : c.bits;
    const float nlam = -c.lam;
    const int2 bound = scale_bounds(bits);
    const float phi = max_of(p), plo = min_of(p), qhi = max_of(q), qlo = min_of(q);
    mid(0);
    const int kp = worker_min<TS>(scale_key(bound, phi, plo)), kq = worker_min<TS>(scale_key(bound, qhi, qlo));
    mid(1);
    float sp = scale_of(kp), sq = scale_of(kq), odd_p, odd_q;
    Vf<N> pi = quantize_near(p, sp, odd_p), qi = quantize_near(q, sq, odd_q);
    auto outside = [](float hi, float lo, float s) { return INT8 ? outside8(hi, lo, s) : beyond_grid(hi, lo, s); };
    float sp_rev = near_rev(sp), sq_rev = near_rev(sq), both_rev = near_rev(sp, sq);
    bool big = false;
    if (__builtin_expect(__any_sync(kAll, scale_unsure(bound, kp) || scale_unsure(bound, kq) || outside(phi, plo, sp) || outside(qhi, qlo, sq)
                                          || !(fmaxf(odd_p, odd_q) < 0.5f)), 0)) {
        if (__any_sync(kAll, scale_unsure(bound, kp) || scale_unsure(bound, kq))) {
            const float2 s = muppet_scales_exact<TS>(bits, phi, plo, qhi, qlo);
            sp = s.x; sq = s.y;
            sp_rev = pow2_rev(sp); sq_rev = pow2_rev(sq); both_rev = pow2_rev(__fmul_rn(sp, sq));
        }
        pi = quantize_away(p, sp); qi = quantize_away(q, sq);
        if (INT8) { pi = clamp8(pi); qi = clamp8(qi); }
        else big = beyond_grid(phi, plo, sp) || beyond_grid(qhi, qlo, sq);
    }
    mid(2);
    Vh<N> ph, qh;
    float pred;
    if constexpr (INT8) pred = forward_int8<TS>(pi, qi, both_rev);
    else {
        to_grid(p, pi, sp, sp_rev, q, qi, sq, sq_rev, big, ph, qh);
        pred = forward_half<K>(ph, qh, kAll, slot);
    }
    mid(3);
    const float ruv = __fsub_rn(r, pred);
    const float ehi = fmaxf(nlam, ruv), elo = fminf(nlam, ruv), hi = fmaxf(fmaxf(phi, qhi), ehi), lo = fminf(fminf(plo, qlo), elo);
    const int kb = min(min(kp, kq), scale_key(bound, ehi, elo));
    float sb = scale_of(kb), odd_e;
    pi = quantize_near(p, sb, odd_p); qi = quantize_near(q, sb, odd_q);
    float2 el = quantize_near(make_float2(ruv, nlam), sb, odd_e);      // error and -lam on the grid
    float sb_rev = near_rev(sb), sb2_rev = near_rev(sb, sb);
    big = false;
    if (__builtin_expect(__any_sync(kAll, scale_unsure(bound, kb) || outside(hi, lo, sb) || !(fmaxf(odd_p, odd_q) < 0.5f) || !(odd_e < 0.5f)), 0)) {
        if (__any_sync(kAll, scale_unsure(bound, kb))) {
            sb = muppet_back_scale_exact<TS>(bits, hi, lo, nlam, ruv);
            sb_rev = pow2_rev(sb); sb2_rev = pow2_rev(__fmul_rn(sb, sb));
        }
        pi = quantize_away(p, sb); qi = quantize_away(q, sb);
        if (INT8) { pi = clamp8(pi); qi = clamp8(qi); }
        else big = beyond_grid(hi, lo, sb);
        el = make_float2(round_away(__fmul_rn(ruv, sb)), round_away(__fmul_rn(nlam, sb)));
        if (INT8) el = make_float2(clamp8(el.x), clamp8(el.y));
    }
    mid(4);
    if constexpr (INT8) backward_int8(pi, qi, el.x, el.y, sb2_rev, gp, gq);
    else {
        to_grid(p, pi, sb, sb_rev, q, qi, sb, sb_rev, big, ph, qh);
        // (a value that rounds to zero keeps its sign)
        backward_half(ph, qh, __half2half2(__float2half_rn(__fmul_rn(copysignf(el.x, ruv), sb_rev))), __half2half2(__float2half_rn(__fmul_rn(copysignf(el.y, nlam), sb_rev))),
                      gp, gq);
    }
    p = step(c.lr, gp, p); q = step(c.lr, gq, q);
}

// ---- AFP (afp/afp_sgd_kernel.h:1-125 helpers, 127-376 k=128; afp_sgd_kernel_k64.h) ----------------
// One side's quantization parameters and the rating count at which they are estimated next.  The
// reference keeps three of these per warp for a whole kernel launch; here per worker.
struct AfpSide { int n; float scale; float mov_avg; long long next; };
// Parameters change once in many ratings, so what follows from them is kept beside them.
struct AfpState {
    AfpSide user, item, back;
    unsigned cur;                             // ratings of this worker so far
    unsigned due;                             // ratings until one of the warp's workers estimates a parameter again
    bool forward16, forward8, back16, back8;  // passes that some worker of the warp needs
    float user_rev, item_rev, both_rev, back_rev, back2_rev, lam8;      // 1 / scales and products of two; -lam on the int8 grid
    __half2 lam16;                            // -lam on the binary16 grid
};

// log2 in double precision, rounded once to float: the CPU restatement computes it the same way, so
// both take identical re-estimation decisions (it runs only when parameters are re-estimated).
// The re-estimation helpers below are deliberately NOT inlined: they run once in many ratings, and inlined -
// six copies of the double-precision logarithm per update, times the unrolled ring - they made the AFP kernel
// so large that its warps waited 5 cycles per issued instruction for instruction fetches.
__device__ __noinline__ float log2_rounded(float x) { return (float)log2((double)x); }

// ceil((float)log2((double)x)) for x > 0 without the logarithm.  x = (1 + M / 2^23) * 2^E: log2(x) lies in
// [E, E + 1); rounded to float it is E itself when M = 0, or when the fraction is below half the spacing of the
// floats next to E on the side of E + 1 - the first few M only, the more the larger |E| - and otherwise a value in
// (E, E + 1], whose ceiling is E + 1.  Equal to the double-precision formula of the CPU restatement for every
// positive finite float (checked exhaustively on the host, tests/ceil_log2_check.c).  Zero gives a large negative
// number, as the logarithm would.
__device__ __forceinline__ int ceil_log2_rounded(float x) {
    const uint32_t bits = __float_as_uint(x) & 0x7fffffffu;
    if (bits == 0u) return -100000;
    int E = (int)(bits >> 23) - 127;
    uint32_t M = bits & 0x7fffffu;
    if ((bits >> 23) == 0u) {                      // denormal: normalise
        const int lz = __clz((int)M) - 9;
        E = -126 - (lz + 1);
        M = (M << (lz + 1)) & 0x7fffffu;
    }
    if (M == 0u) return E;
    uint32_t a = (uint32_t)(E < 0 ? -E : E);
    if (E < 0) a -= 1u;                            // the floats between E and E + 1 are smaller in magnitude than |E|
    if (E <= 0 && a == 0u) return E + 1;
    const int j = 31 - __clz((int)a);
    const uint32_t limit = j <= 1 ? 0u : (j == 2 ? 1u : (j == 3 ? 2u : (j == 4 ? 5u : (j == 5 ? 11u : (j == 6 ? 22u : 44u)))));
    return M <= limit ? E : E + 1;
}

// The eight elements of lane l mod K/8 of the wider form, from the two lanes that hold four of them each
template <int K> __device__ __forceinline__ const V8f& eight(const V8f& x) { return x; }
template <int K> __device__ __forceinline__ V8f eight(const Vf<4>& x) {
    const bool up = threadIdx.x & (K / 8);
    V8f o;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const float other = __shfl_xor_sync(0xffffffffu, x.x[t], K / 8);
        o.x[t] = up ? other : x.x[t];
        o.x[4 + t] = up ? x.x[t] : other;
    }
    return o;
}

// 2^|ceil(log2(range / (2^(bits-1) - 1)))| (afp_sgd_kernel.h:8-16, 112-118); exponent capped at 126
__device__ __forceinline__ float afp_scale(int bits, float range) {
    if (range == 0.f) return 1.f;
    const float top = bits == 8 ? 127.f : 32767.f;
    const int c = ceil_log2_rounded(__fdiv_rn(range, top));
    const int e = c < 0 ? -c : c;
    const int ei = e > 126 ? 126 : e;
    return __int_as_float((ei + 127) << 23);
}
// Sum of magnitudes of the values a reference lane adds, left to right, before and after 8-bit
// rounding; `G` reference lanes live in this lane, `N` values each, v[g][j].
template <int G, int N>
__device__ __forceinline__ void afp_lane_sums(const float (&v)[G][N], float scale, float rev, float& sum, float& sum_q) {
    float s[G], sq[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
        s[g] = fabsf(v[g][0]); sq[g] = fabsf(__fmul_rn(round_away(__fmul_rn(v[g][0], scale)), rev));
#pragma unroll
        for (int j = 1; j < N; j++) {
            s[g] = __fadd_rn(s[g], fabsf(v[g][j]));
            sq[g] = __fadd_rn(sq[g], fabsf(__fmul_rn(round_away(__fmul_rn(v[g][j], scale)), rev)));
        }
    }
    if (G == 2) { sum = __fadd_rn(s[0], s[1]); sum_q = __fadd_rn(sq[0], sq[1]); }
    else { sum = __fadd_rn(__fadd_rn(s[0], s[1]), __fadd_rn(s[2], s[3])); sum_q = __fadd_rn(__fadd_rn(sq[0], sq[1]), __fadd_rn(sq[2], sq[3])); }
}
// QEM / QEM_BP (afp_sgd_kernel.h:31-104): log2(1 + relative loss of the magnitude sum under 8 bits)
template <int K>
__device__ __noinline__ float afp_qem(V8f x, float max_val, unsigned wmask) {
    constexpr int TS = K / 8;
    const float scale = afp_scale(8, max_val), rev = __fdiv_rn(1.f, scale);
    float sum, sum_q;
    if (K == 128) {
        const float v[2][4] = {{x.x[0], x.x[2], x.x[4], x.x[6]}, {x.x[1], x.x[3], x.x[5], x.x[7]}};
        afp_lane_sums<2, 4>(v, scale, rev, sum, sum_q);
    } else {
        const float v[4][2] = {{x.x[0], x.x[2]}, {x.x[4], x.x[6]}, {x.x[1], x.x[3]}, {x.x[5], x.x[7]}};
        afp_lane_sums<4, 2>(v, scale, rev, sum, sum_q);
    }
    sum = worker_sum<TS>(sum, wmask); sum_q = worker_sum<TS>(sum_q, wmask);
    return log2_rounded(__fadd_rn(fabsf(__fdiv_rn(__fsub_rn(sum, sum_q), sum)), 1.f));
}
template <int K>
__device__ __noinline__ float afp_qem_back(V8f p, V8f q, float lam, float ruv, float max_val, unsigned wmask) {
    constexpr int TS = K / 8;
    const float scale = afp_scale(8, max_val), rev = __fdiv_rn(1.f, scale);
    float sum, sum_q;
    if (K == 128) {
        const float v[2][10] = {{p.x[0], p.x[2], p.x[4], p.x[6], q.x[0], q.x[2], q.x[4], q.x[6], lam, ruv},
                                {p.x[1], p.x[3], p.x[5], p.x[7], q.x[1], q.x[3], q.x[5], q.x[7], lam, ruv}};
        afp_lane_sums<2, 10>(v, scale, rev, sum, sum_q);
    } else {
        const float v[4][6] = {{p.x[0], p.x[2], q.x[0], q.x[2], lam, ruv}, {p.x[4], p.x[6], q.x[4], q.x[6], lam, ruv},
                               {p.x[1], p.x[3], q.x[1], q.x[3], lam, ruv}, {p.x[5], p.x[7], q.x[5], q.x[7], lam, ruv}};
        afp_lane_sums<4, 6>(v, scale, rev, sum, sum_q);
    }
    sum = worker_sum<TS>(sum, wmask); sum_q = worker_sum<TS>(sum_q, wmask);
    return log2_rounded(__fadd_rn(fabsf(__fdiv_rn(__fsub_rn(sum, sum_q), sum)), 1.f));
}
// QPA (afp_sgd_kernel.h:106-125) and the bookkeeping around each call (196-206)
__device__ __noinline__ AfpSide afp_requantize(AfpSide s, float diff, float range, long long cur, int epoch, int init_threshold) {
    const float threshold = 0.0005, alpha = 0.04, beta = 0.1, delta = 100, gamma = 2;
    if (cur == 0) s.mov_avg = range;
    const float prev = s.mov_avg;
    s.n = diff <= threshold ? 8 : 16;
    s.scale = afp_scale(s.n, range);
    s.mov_avg = __fmaf_rn(alpha, range, __fmul_rn(__fsub_rn(1.0f, alpha), prev));
    const float i1 = __fmul_rn(__fmul_rn(delta, diff), diff), i2 = fabsf(__fsub_rn(s.mov_avg, prev));
    int itv = __float2int_rz(__fsub_rn(__fdiv_rn(beta, fmaxf(i1, i2)), gamma));     // saturates; NaN -> 0
    if (epoch == 0 && cur < init_threshold) itv = 1;
    s.next += itv;
    return s;
}
// The workers of a warp go through this together: what one of them needs (a re-estimation, the int8 or the binary16
// pass) all of them compute, and each keeps the result if it is its own case.  active: is there a rating?
// What passes there are and when the next estimate is due only changes with an estimate, so a rating without one has two votes: is
// there an exact half, or a value outside the int8 range (2^21 steps of the grid)?
template <int K, int N>
__device__ __forceinline__ void afp_update(const Consts& c, AfpState& st, float r, bool active, Vf<N>& p, Vf<N>& q, unsigned slot) {
    constexpr int TS = K / N;
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned cur = st.cur;
    const bool estimate = st.due == 0;
    float pmax = 0.f, qmax = 0.f;
    if (__builtin_expect(estimate, 0)) {
        // ratings without a binary16 pass have no barrier of their own, and the pass may come back with an estimate: what was read from its
        // slot two ratings ago is kept from what is written to it next
        __syncwarp();
        const bool new_user = active && cur == st.user.next, new_item = active && cur == st.item.next;
        pmax = worker_max<TS>(abs_max(p), kAll);
        qmax = worker_max<TS>(abs_max(q), kAll);
        if (__any_sync(kAll, new_user)) {
            const AfpSide s = afp_requantize(st.user, afp_qem<K>(eight<K>(p), pmax, kAll), pmax, cur, c.afp_epoch, c.afp_init_threshold);
            if (new_user) st.user = s;
        }
        if (__any_sync(kAll, new_item)) {
            const AfpSide s = afp_requantize(st.item, afp_qem<K>(eight<K>(q), qmax, kAll), qmax, cur, c.afp_epoch, c.afp_init_threshold);
            if (new_item) st.item = s;
        }
        const bool mine8 = st.user.n == 8 && st.item.n == 8;
        st.forward16 = __any_sync(kAll, active && !mine8);
        st.forward8 = !st.forward16 || __any_sync(kAll, active && mine8);
        st.user_rev = pow2_rev(st.user.scale); st.item_rev = pow2_rev(st.item.scale);
        st.both_rev = pow2_rev(__fmul_rn(st.user.scale, st.item.scale));
    }
    // The formats are those of an earlier rating, so values may lie outside their range at any time.
    float pred = 0.f, odd_p, odd_q;
    Vf<N> pi = quantize_near(p, st.user.scale, odd_p), qi = quantize_near(q, st.item.scale, odd_q);
    Vh<N> ph, qh;
    bool big = false, clamp = false;
    auto check = [&](float sp, float sq, bool some8, float also, float odd_also) {
        float most = fmaxf(fmaxf(abs_max(pi), abs_max(qi)), fabsf(also));
        const bool again = __any_sync(kAll, !(fmaxf(odd_p, odd_q) < 0.5f) || !(odd_also < 0.5f) || !(most <= (some8 ? 127.f : 2097151.f)));
        if (__builtin_expect(again, 0)) {
            pi = quantize_away(p, sp); qi = quantize_away(q, sq);
            most = fmaxf(abs_max(pi), abs_max(qi));
            big = __any_sync(kAll, !(most < 2097152.f));
            clamp = __any_sync(kAll, !(most <= 127.f));
        }
        return again;
    };
    check(st.user.scale, st.item.scale, st.forward8, 0.f, 0.f);
    if (st.forward16) {
        to_grid(p, pi, st.user.scale, st.user_rev, q, qi, st.item.scale, st.item_rev, big, ph, qh);
        pred = forward_half<K>(ph, qh, kAll, slot);
    }
    if (st.forward8) {
        if (__builtin_expect(clamp, 0)) { pi = clamp8(pi); qi = clamp8(qi); }
        const float whole = forward_int8<TS>(pi, qi, st.both_rev);
        if (st.user.n == 8 && st.item.n == 8) pred = whole;
    }
    const float ruv = __fsub_rn(r, pred);
    if (__builtin_expect(estimate, 0)) {
        const bool new_back = active && cur == st.back.next;
        if (__any_sync(kAll, new_back)) {
            const float range = fmaxf(fmaxf(fmaxf(pmax, qmax), fabsf(c.lam)), fabsf(ruv));
            const AfpSide s = afp_requantize(st.back, afp_qem_back<K>(eight<K>(p), eight<K>(q), c.lam, ruv, range, kAll), range, cur, c.afp_epoch, c.afp_init_threshold);
            if (new_back) st.back = s;
        }
        const bool mine8 = st.back.n == 8;
        st.back16 = __any_sync(kAll, active && !mine8);
        st.back8 = !st.back16 || __any_sync(kAll, active && mine8);
        st.back_rev = pow2_rev(st.back.scale); st.back2_rev = pow2_rev(__fmul_rn(st.back.scale, st.back.scale));
        st.lam8 = quantize8(-c.lam, st.back.scale);
        st.lam16 = __half2half2(__float2half_rn(fix_round(-c.lam, st.back.scale, st.back_rev)));
        // an estimate whose time has passed never comes again
        auto wait = [&](long long next) { const long long d = next - cur - 1; return d < 0 || d > 0x7fffffff ? 0x7fffffff : (int)d; };
        st.due = (unsigned)__reduce_min_sync(kAll, min(min(wait(st.user.next), wait(st.item.next)), wait(st.back.next)));
    } else {
        st.due--;
    }
    pi = quantize_near(p, st.back.scale, odd_p); qi = quantize_near(q, st.back.scale, odd_q);
    float odd_e;
    float2 e = quantize_near(make_float2(ruv, ruv), st.back.scale, odd_e);      // the error on the two grids
    big = clamp = false;
    if (__builtin_expect(check(st.back.scale, st.back.scale, st.back8, e.x, odd_e), 0)) e = make_float2(quantize8(ruv, st.back.scale), round_away(__fmul_rn(ruv, st.back.scale)));
    Vf<N> gp, gq;
    if (st.back16) {
        to_grid(p, pi, st.back.scale, st.back_rev, q, qi, st.back.scale, st.back_rev, big, ph, qh);
        backward_half(ph, qh, __half2half2(__float2half_rn(__fmul_rn(copysignf(e.y, ruv), st.back_rev))), st.lam16, gp, gq);
    }
    if (st.back8) {
        if (__builtin_expect(clamp, 0)) { pi = clamp8(pi); qi = clamp8(qi); }
        Vf<N> wp, wq;
        backward_int8(pi, qi, e.x, st.lam8, st.back2_rev, wp, wq);
        if (!st.back16 || st.back.n == 8) { gp = wp; gq = wq; }
    }
    p = step(c.lr, gp, p); q = step(c.lr, gq, q);
    st.cur = cur + 1;
}

// Does a launch add its dot products up through shared memory?  It shortens the chain of a rating, which bounds the narrow form; the
// statistics use the steps of the shuffles.  A GPU full of K/8-lane workers has better uses for the shared memory (100M ratings 5.56 ->
// 5.81 ms per epoch).
template <int KIND, int UM, int IM, bool STATS> constexpr bool kTreeSum = !STATS && kElems<UM> == 4 && KIND != KIND_AFP && !kMuppet<KIND>;
// Does a launch work with binary16 ratings?  Its records then hold the converted value in both halves of a word.
template <int KIND, int UM, int IM> constexpr bool kHalfRating =
    KIND == KIND_MPT || ((KIND == KIND_MIXED || KIND == KIND_SWITCH) && kHalfRows<UM> && kHalfRows<IM>);
__device__ __forceinline__ __half2 half2_of(uint32_t w) { return *reinterpret_cast<const __half2*>(&w); }

// One update.  rw is the rating as its record holds it; p_raw / q_raw are the row slices in their storage precision,
// both replaced by the updated values.  The workers of a warp come here together, with `wmask` the whole warp - or,
// where they may take different branches (ROWS_DYN), each with the mask of its own lanes.  mid(0), mid(1), mid(2): what the
// worker has to do meanwhile, done under the shuffles of the dot product.
template <int K, int KIND, int UM, int IM, bool STATS, class Mid>
__device__ __forceinline__ void update_one(const Consts& c, uint32_t rw, uint32_t uc, uint32_t ic, Raw<UM>& p_raw, Raw<IM>& q_raw,
                                           Sample<kElems<UM>>& smp, AfpState& afp, bool active, unsigned wmask, unsigned slot, Mid mid) {
    constexpr int N = kElems<UM>, TS = K / N;
    static_assert(N == kElems<IM>, "both rows are spread over the worker's lanes the same way");
    constexpr bool kAhead = KIND == KIND_AFP || UM == ROWS_DYN || IM == ROWS_DYN;      // no single dot product to hide under
    constexpr bool kTree = kTreeSum<KIND, UM, IM, STATS>;
    if constexpr (kAhead) { mid(0); mid(1); mid(2); }
    if (STATS) { smp.user = false; smp.item = false; }
    if constexpr (KIND == KIND_MPT) {
        const Vf<N> p = as_vf(p_raw), q = as_vf(q_raw);
        const Vh<N> ph = narrow(p), qh = narrow(q);
        __half2 dot;
        if constexpr (kTree) dot = tree_dot<K>(ph, qh, slot, mid);
        else dot = worker_dot<TS>(ph, qh, wmask, mid);
        const __half2 e = __hmul2_rn(c.mpt_scale, __hsub2_rn(half2_of(rw), dot));
        const Vf<N> gp = widen(grad(e, qh, c.mpt_nlam, ph)), gq = widen(grad(e, ph, c.mpt_nlam, qh));
        Vf<N> po, qo;
        const float2 lr2 = make_float2(c.lr, c.lr), rev2 = make_float2(c.mpt_rev, c.mpt_rev);
#pragma unroll
        for (int j = 0; j < N / 2; j++) {
            set_pr(po, j, __ffma2_rn(lr2, __fmul2_rn(rev2, pr(gp, j)), pr(p, j)));
            set_pr(qo, j, __ffma2_rn(lr2, __fmul2_rn(rev2, pr(gq, j)), pr(q, j)));
        }
        put(p_raw, po); put(q_raw, qo);
    } else if constexpr (KIND == KIND_MUPPET || KIND == kMuppetHalf) {
        Vf<N> p = as_vf(p_raw), q = as_vf(q_raw);
        muppet_update<K, KIND == KIND_MUPPET>(c, __uint_as_float(rw), p, q, smp.gp, smp.gq, slot, mid);
        put(p_raw, p); put(q_raw, q);
        if (STATS) smp.user = true;
    } else if constexpr (KIND == KIND_AFP) {
        Vf<N> p = as_vf(p_raw), q = as_vf(q_raw);
        afp_update<K>(c, afp, __uint_as_float(rw), active, p, q, slot);
        put(p_raw, p); put(q_raw, q);
    } else if constexpr (KIND == KIND_MEMQUANT) {
        const Vf<N> p = widen(as_vh(p_raw)), q = widen(as_vh(q_raw));
        float dot;
        if constexpr (K == 128 && N == 4) dot = tree_chain_k128<K>(p, q, slot, mid);
        else if constexpr (K == 128) dot = worker_sum<TS>(chain_partial_k128(p, q), wmask, mid);
        else if constexpr (kTree) dot = tree_dot<K>(p, q, slot, mid);
        else dot = worker_dot<TS>(p, q, wmask, mid);
        const float e = __fsub_rn(__uint_as_float(rw), dot);
        put(p_raw, narrow(step(c.lr, grad(e, q, c.lam, p), p)));
        put(q_raw, narrow(step(c.lr, grad(e, p, c.lam, q), q)));
    } else {
        const bool uf = is_f32<UM>(uc), itf = is_f32<IM>(ic);
        auto both_half = [&]() {
            const Vh<N> p = as_vh(p_raw), q = as_vh(q_raw);
            __half2 dot;
            if constexpr (kTree) dot = tree_dot<K>(p, q, slot, mid);
            else if constexpr (kAhead) dot = worker_dot<TS>(p, q, wmask);
            else dot = worker_dot<TS>(p, q, wmask, mid);
            const __half2 e = __hsub2_rn(kHalfRating<KIND, UM, IM> ? half2_of(rw) : __float2half2_rn(__uint_as_float(rw)), dot);
            const Vh<N> gp = grad(e, q, c.nlam_h, p), gq = grad(e, p, c.nlam_h, q);
            put(p_raw, step(c.lr_h, gp, p));
            put(q_raw, step(c.lr_h, gq, q));
            if (STATS) { smp.gp = widen(gp); smp.gq = widen(gq); smp.user = true; smp.item = true; }
        };
        auto some_f32 = [&]() {
            const Vf<N> p = uf ? as_vf(p_raw) : widen(as_vh(p_raw));
            const Vf<N> q = itf ? as_vf(q_raw) : widen(as_vh(q_raw));
            float dot;
            if constexpr (kTree) dot = tree_dot<K>(p, q, slot, mid);
            else if constexpr (kAhead) dot = worker_dot<TS>(p, q, wmask);
            else dot = worker_dot<TS>(p, q, wmask, mid);
            const float e = __fsub_rn(__uint_as_float(rw), dot);
            const Vf<N> gp = grad(e, q, c.lam, p), gq = grad(e, p, c.lam, q);
            const Vf<N> po = step(c.lr, gp, p), qo = step(c.lr, gq, q);
            if (uf) put(p_raw, po); else put(p_raw, narrow(po));
            if (itf) put(q_raw, qo); else put(q_raw, narrow(qo));
            if (STATS) { smp.gp = gp; smp.gq = gq; smp.user = !uf; smp.item = !itf; }
        };
        if constexpr (kHalfRows<UM> && kHalfRows<IM>) both_half();
        else if constexpr (UM != ROWS_DYN && IM != ROWS_DYN) some_f32();
        else { if (!uf && !itf) both_half(); else some_f32(); }
    }
}

// ---- asynchronous row copies (global -> the worker's shared-memory rings) ----------------------
// Rows are fetched with cp.async, not with loads into registers: a register load ties the wait for
// an old row to every younger load that shares its scoreboard, which exposes one full memory
// latency per rating; copy groups complete in order, so waiting for the group of rating j leaves
// the copies of ratings j+1 .. j+D in flight.
// Shared memory is addressed by its 32-bit address.
template <int OFF> __device__ __forceinline__ void cp16(unsigned dst, const unsigned char* src) {
    asm volatile("cp.async.cg.shared.global [%0 + %2], [%1 + %2], 16;" ::"r"(dst), "l"(src), "n"(OFF) : "memory");
}
template <int OFF> __device__ __forceinline__ void cp16_if_row(uint32_t row, unsigned dst, const unsigned char* src) {
    asm volatile("{ .reg .pred g; setp.ne.u32 g, %2, 0xffffffff; @g cp.async.cg.shared.global [%0 + %3], [%1 + %3], 16; }" ::"r"(dst), "l"(src), "r"(row), "n"(OFF) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// Slot layout = row layout: the first 16 bytes of every lane, then (fp32 rows) the second 16 bytes of
// every lane (layout.cuh), so that neither the 128-bit shared-memory accesses of neighbouring lanes collide
// on a bank nor the global accesses of a worker touch partial sectors.  `slot` includes the lane's 16 m.
template <int K, int MODE>
__device__ __forceinline__ void cp_row_if(unsigned slot, const Rows<K, MODE>& A, uint32_t code) {      // kNoRow: nothing
    const unsigned char* g = A.at(code);
    // copies are of 16 bytes: of binary16 rows the first half of the lanes fetches what both halves hold
    if constexpr (MODE == ROWS_HALFQ) code = threadIdx.x & (K / 8) ? kNoRow : code;
    cp16_if_row<0>(code, slot, g);
    if constexpr (MODE == ROWS_F32) cp16_if_row<2 * K>(code, slot, g);
    if constexpr (MODE == ROWS_DYN) cp16_if_row<2 * K>((code & kPrecBit) ? code : kNoRow, slot, g);
}
template <int K, int MODE>
__device__ __forceinline__ void cp_row(unsigned slot, const Rows<K, MODE>& A, uint32_t code) {
    if constexpr (MODE == ROWS_HALFQ) { cp_row_if<K, MODE>(slot, A, code); return; }
    const unsigned char* g = A.at(code);
    cp16<0>(slot, g);
    if constexpr (MODE == ROWS_F32) cp16<2 * K>(slot, g);                                   // second half of the row
    if constexpr (MODE == ROWS_DYN) cp16_if_row<2 * K>((code & kPrecBit) ? 0u : kNoRow, slot, g);
}
template <int K, int MODE>
__device__ __forceinline__ Raw<MODE> lds_row(unsigned slot, uint32_t code) {
    Raw<MODE> r;
    if constexpr (MODE == ROWS_HALFQ) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.a.x), "=r"(r.a.y) : "r"(slot) : "memory");
    else r.a = lds128(slot);
    if constexpr (MODE == ROWS_F32) r.b = lds128(slot + 2 * K);
    if constexpr (MODE == ROWS_DYN) { if (is_f32<MODE>(code)) r.b = lds128(slot + 2 * K); }
    return r;
}

// One rating as the worker's lanes read it from shared memory (one 128-bit broadcast load): flags, item id, user id
// (both without the marks nobody reads any more), rating.
constexpr uint32_t F_UDUP = 1u;     // its user also occurs among the ratings whose update may not be in the copied row: read the row at use
constexpr uint32_t F_RS = 2u;       // its item differs from the item of the rating before it (a run starts)
constexpr uint32_t F_IDUP = 4u;     // run start whose item also occurs shortly before
constexpr uint32_t F_DROP = 8u;     // the user row is not written back (an update of a very popular user, or no rating at all)
constexpr uint32_t F_NONE = 16u;    // there is no rating at this position


// Shared memory of one worker: two chunks of records, what to request while each of them is processed (8 bytes: the
// user row of the rating D further on, the item row of the rating DI further on if a run starts there), then the user
// ring, then the item ring.  A ring
// slot is as large as the widest row its side can hold in this launch.
template <int K, int KIND, int UM, int IM, bool STATS, int NS, int NSI> struct WorkerSmem {
    static constexpr int TS = K / kElems<UM>;
    static constexpr int kURowBytes = K * (kHalfRows<UM> ? 2 : 4);
    static constexpr int kIRowBytes = K * (kHalfRows<IM> ? 2 : 4);
    static constexpr int kRecBytes = 2 * TS * 16 + 2 * TS * 8;
    // The records of the workers of a warp are shifted by 16 bytes from worker to worker: those read at the same time
    // then lie in different banks.  The rings stay at multiples of 128 bytes (off them, copies and loads of rows touch
    // a line more each: 5.9 instead of 5.5 ms per epoch of the 100M-rating set).
    // Behind the records of the narrow form follow two slots for the partials of a dot product (tree_sum): 64 bytes, which the shift
    // leaves of its 128 - or 128, and as much room more, for partials of four bytes at k=128.
    static constexpr bool kWideSlots = K == 128 && kElems<UM> == 4 && (!(kHalfRows<UM> && kHalfRows<IM>) || KIND == KIND_MEMQUANT);
    static constexpr int kSlotBytes = kWideSlots ? 64 : 32;
    static constexpr int kShift = kWideSlots ? 256 : 128;
    // With statistics: the groups of both rows of every record, looked up for a whole chunk at once.  (A lookup per
    // rating is a memory latency per rating: the sampled twentieth of an epoch took a seventh of its time.)
    static constexpr int kGroupBytes = STATS ? 2 * TS * 4 : 0;
    static constexpr int kBytes = kRecBytes + kShift + NS * kURowBytes + NSI * kIRowBytes + (kGroupBytes + 127) / 128 * 128;
};

// NS / NSI: slots of the user / item ring.  User rows are requested D ratings ahead, item rows DI ratings ahead; a
// user row is read from its slot one rating before its own, so a slot is free for the request of a rating D < NS ahead.
// The lead is kept as short as the memory latency allows: an item row that another worker updates between the
// request and the write-back loses that update, and the chance of that grows with the lead.
template <int K, int KIND, int UM, int IM, bool STATS, int NS, int NSI, int D, int DI>
__global__ void __launch_bounds__(256, (kHalfRows<UM> && kHalfRows<IM> && !STATS) ? 4 : ((UM == ROWS_DYN || STATS || KIND == KIND_AFP || kMuppet<KIND>) ? 2 : 3)) train_kernel(const KernelArgs a) {
    using SM = WorkerSmem<K, KIND, UM, IM, STATS, NS, NSI>;
    constexpr int TS = SM::TS;                     // lanes per worker = ratings per chunk
    constexpr int N = kElems<UM>;                  // elements per lane
    constexpr unsigned kSpan = K / TS;             // consecutive chunks handed out together: K ratings, the longest run of one ticket
    constexpr unsigned kAll = 0xffffffffu;
    static_assert(TS % NS == 0 && (NS & (NS - 1)) == 0 && (NSI & (NSI - 1)) == 0, "the rings must divide the chunk");
    static_assert(DI >= 1 && D >= 2 && DI <= D && D < NS && DI < NSI && NSI <= NS, "leads must fit the rings");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int m = lane % TS;
    const unsigned gmask = (0xffffffffu >> (32 - TS)) << (lane - m);      // the lanes of this worker
    const unsigned W = a.workers;
    // AFP's workers may be alone in their warps (launch_ns); the other lanes then keep them company without work.
    constexpr bool kSpread = KIND == KIND_AFP;
    const unsigned per_warp = (32 / TS) >> a.spread, sub = lane / TS;
    const unsigned worker = !kSpread ? (blockIdx.x * blockDim.x + threadIdx.x) / TS
                                     : sub < per_warp ? (blockIdx.x * blockDim.x + threadIdx.x) / 32 * per_warp + sub : W;
    // fewer than 2^32 ratings, so chunks are counted in 32 bits
    const unsigned nchunks = (unsigned)((a.s.n + TS - 1) / TS);

    unsigned char* const mine = smem_raw + (size_t)(threadIdx.x / TS) * SM::kBytes;
    uint4* const recs = reinterpret_cast<uint4*>(mine + 16 * (lane / TS));      // [2][TS]
    uint32_t* const reqs = reinterpret_cast<uint32_t*>(recs + 2 * TS);          // [2][TS][user, item]
    const unsigned s_rec = (unsigned)__cvta_generic_to_shared(recs);
    const unsigned s_req = s_rec + 2 * TS * 16;
    const unsigned slots = s_req + 2 * TS * 8;
    const unsigned rings = (unsigned)__cvta_generic_to_shared(mine) + SM::kRecBytes + SM::kShift;
    const unsigned uring = rings + lane_at<K, UM>(m);                            // [NS][kURowBytes]
    const unsigned iring = rings + NS * SM::kURowBytes + lane_at<K, IM>(m);      // [NSI][kIRowBytes]
    uint32_t* const groups = reinterpret_cast<uint32_t*>(mine + SM::kRecBytes + SM::kShift + NS * SM::kURowBytes + NSI * SM::kIRowBytes);
    constexpr bool kGroups = STATS && KIND == KIND_MIXED;
    const Rows<K, UM> P(a.P, m);
    const Rows<K, IM> Q(a.Q, m);

    Consts c;
    c.lr = a.lr; c.lam = a.lam;
    c.lr_h = __half2half2(__float2half_rn(a.lr));
    c.nlam_h = __half2half2(__float2half_rn(-a.lam));
    c.mpt_scale = __float2half2_rn(1000.0f);
    c.mpt_nlam = __half2half2(__float2half_rn(-__fmul_rn(a.lam, 1000.0f)));
    c.mpt_rev = __fdiv_rn(1.0f, 1000.0f);
    c.bits = a.bits;
    c.afp_epoch = a.epoch;
    c.afp_init_threshold = (int)((float)((a.s.n + W - 1) / W) / 10.0f);
    // only the mixed-precision mode reads the precision bit of an id
    constexpr uint32_t kKeep = (UM == ROWS_DYN || IM == ROWS_DYN) ? (kPrecBit | kIdMask) : kIdMask;

    // ---- which chunks this worker processes ----
    // Runs of consecutive chunks: first the static runs [worker*kSpan, +kSpan) and [(worker+W)*kSpan,
    // +kSpan), then runs handed out by the shared counter, which counts chunks beyond the static part.
    // A dynamic run is kSpan chunks long while plenty of work is left and shrinks to a single chunk as
    // the counter nears the end (its length is what is left, as seen at the previous ticket, divided by
    // about twice the number of workers), so that the workers finish within about one chunk of each other.  A
    // ticket is requested one run before it is needed and stays in lane 0 until then, so the launch
    // neither waits for the counter nor depends on all blocks being resident.  Lanes beyond the last worker keep
    // their warp company without chunks of their own.
    // The code from here to the end of the loop has no branch that the workers of a warp could take differently: what
    // only some lanes do is predicated.  (With divergent branches around, the compiler puts a warp barrier in front
    // of every shuffle and vote of the loop.)
    const unsigned static_chunks = 2 * W * kSpan;
    const unsigned dyn_chunks = nchunks > static_chunks ? nchunks - static_chunks : 0;
    const unsigned share_log2 = 32 - __clz(2 * W - 1);              // 2 W rounded up to a power of two
    auto run_length = [&](unsigned seen) -> unsigned {
        const unsigned g = (dyn_chunks > seen ? dyn_chunks - seen : 0) >> share_log2;
        return min(max(g, 1u), kSpan);
    };
    // lane 0 of a worker takes `len` chunks off the shared counter
    auto draw_ticket = [&](bool go, unsigned len) -> unsigned {
        unsigned long long t = 0;
        asm volatile("{ .reg .pred g; setp.ne.u32 g, %1, 0; @g atom.global.add.u64 %0, [%2], %3; }" : "+l"(t) : "r"((unsigned)(go && m == 0)), "l"(a.next_chunk),
                     "l"((unsigned long long)len) : "memory");
        return (unsigned)t;
    };
    const bool works = worker < W;
    unsigned run_cur = works ? worker * kSpan : nchunks, run_next = (worker + W) * kSpan;
    unsigned len_cur = kSpan, len_next = kSpan, kin = 0;
    unsigned tlen = run_length(0), ticket = draw_ticket(works, tlen);
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.zero_counter = 0ull;      // the counter of the launch after next
    auto next_chunk_id = [&]() -> unsigned {
        const bool left = run_cur < nchunks;
        const unsigned ci = left ? run_cur + kin : nchunks;
        const bool turn = left && ++kin == len_cur;
        const unsigned drawn = __shfl_sync(kAll, ticket, 0, TS), drawn_len = __shfl_sync(kAll, tlen, 0, TS);
        if (turn) {
            kin = 0;
            run_cur = run_next; len_cur = len_next;
            len_next = drawn_len;
            run_next = static_chunks + drawn;
            tlen = run_length(drawn);
        }
        const unsigned t = draw_ticket(turn, tlen);
        if (turn) ticket = t;
        return ci;
    };

    // ---- chunk pipeline: global loads (registers) -> flags -> records in shared memory -> use ----
    struct Loaded { float r; uint32_t u, i; int cnt; };
    auto fetch_chunk = [&](unsigned ci) {
        Loaded k;
        const uint64_t base = (uint64_t)ci * TS;
        k.cnt = ci < nchunks ? (int)min((uint64_t)TS, a.s.n - base) : 0;
        const bool in = m < k.cnt;
        const uint64_t at = in ? base + m : 0;         // any rating there is
        k.r = __ldg(a.s.r + at);
        k.u = __ldg(a.s.u + at);
        k.i = __ldg(a.s.i + at) & kKeep;
        if (!in) { k.u = kNoRow; k.i = kNoRow; }
        return k;
    };
    unsigned hot_seen = worker;             // counts the ratings of marked users this worker has met
    const unsigned hot_mask = (1u << a.hot_user_shift) - 1u;
    uint32_t prev_u = kNoRow, prev_i = kNoRow;        // lane m: rating m of the chunk before `inflight`
    Loaded inflight = fetch_chunk(next_chunk_id());
    // Turns `inflight` into records in buffer `b` and starts loading the chunk after it; returns its rating count.
    auto publish = [&](int b) -> int {
        __syncwarp();
        const bool valid = m < inflight.cnt;
        // A marked user (see the set-up): every 2^shift-th update of marked rows that this worker meets is written
        // back; the others are dropped.
        const bool hot = valid && (inflight.u & kHotBit) && a.add_user_delta;
        const unsigned hot_set = (__ballot_sync(kAll, hot) & gmask) >> (lane - m);
        const bool drop = hot && ((hot_seen + __popc(hot_set & ((2u << m) - 1u))) & hot_mask) != 0u;
        hot_seen += __popc(hot_set);
        const uint32_t u = valid ? inflight.u & kKeep : kNoRow, i = inflight.i;
        if constexpr (kGroups) groups[b * TS + m] = valid ? (uint32_t)__ldg(a.st.ugroup + (u & kIdMask)) | (uint32_t)__ldg(a.st.igroup + (i & kIdMask)) << 16 : 0u;
        bool udup = false, idup = false, rs = false;
#pragma unroll
        for (int d = 1; d <= (D > DI + 2 ? D + 1 : DI + 3); d++) {
            // the rating d places earlier: lane m-d of this chunk, or lane m-d+TS of the previous one;
            // the SOURCE lane knows which of its two values a reader d lanes further on wants
            const bool from_this = m < TS - d;
            if (d <= D + 1) udup |= __shfl_sync(kAll, from_this ? u : prev_u, (m - d) & (TS - 1), TS) == u;
            if (d <= DI + 3) {
                const bool same = __shfl_sync(kAll, from_this ? i : prev_i, (m - d) & (TS - 1), TS) == i;
                if (d == 1) rs = !same; else idup |= same;
            }
        }
        // The position after a worker's last rating starts a run of nothing, which writes the last item row back.
        const uint32_t f = valid ? (udup ? F_UDUP : 0u) | (rs ? F_RS : 0u) | ((rs && idup) ? F_IDUP : 0u) | (drop ? F_DROP : 0u)
                                 : F_NONE | F_DROP | ((!kSpread || works) && m == inflight.cnt ? F_RS : 0u);
        uint32_t rw = __float_as_uint(inflight.r);
        if constexpr (kHalfRating<KIND, UM, IM>) { const __half2 h = __float2half2_rn(inflight.r); rw = *reinterpret_cast<const uint32_t*>(&h); }
        recs[b * TS + m] = make_uint4(f, valid ? i : 0u, valid ? u : 0u, rw);
        const int pos = b * TS + m;
        reqs[2 * ((pos - D) & (2 * TS - 1))] = valid ? u : (kSpread ? kNoRow : 0u);
        reqs[2 * ((pos - DI) & (2 * TS - 1)) + 1] = (f & F_RS) ? (valid ? i : 0u) : kNoRow;
        prev_u = u; prev_i = i;
        const int cnt = inflight.cnt;
        inflight = fetch_chunk(next_chunk_id());
        __syncwarp();
        return cnt;
    };
    if constexpr (kSpread) {
        // lanes without work go through the updates with harmless rows, which take no slow path
        if (!works) for (int b = 16 * m; b < NS * SM::kURowBytes + NSI * SM::kIRowBytes; b += 16 * TS)
            *reinterpret_cast<float4*>(mine + SM::kRecBytes + SM::kShift + b) = make_float4(0.01f, 0.01f, 0.01f, 0.01f);
    }
    int cnt_cur = publish(0), cnt_next = publish(1);

    // item row of the current run
    uint32_t cur_ic = 0;
    unsigned have_item = 0;                          // F_RS while there is one
    Raw<IM> q = Raw<IM>();
    if constexpr (kSpread) {
        Vf<N> harmless;
#pragma unroll
        for (int t = 0; t < N; t++) harmless.x[t] = 0.01f;
        put(q, harmless);
    }

    // item-side statistics of the current run of equal item groups
    const int stat_at = N == 8 ? 8 * m : 8 * (m & (TS / 2 - 1)) + (m & (TS / 2) ? 4 : 0);      // the lane's first element in physical order
    Vf<N> gq_acc; float nq_acc = 0.f; uint32_t acc_group = kNoRow;
#pragma unroll
    for (int t = 0; t < N; t++) gq_acc.x[t] = 0.f;
    // this block's private set of accumulators (fewer workers per address, less serialisation)
    const size_t my_set = STATS ? (size_t)(blockIdx.x % (unsigned)a.st.copies) * a.st.copy_stride : 0;
    float* const gsum_p = a.st.gsum_p + my_set; float* const gsum_q = a.st.gsum_q + my_set;
    float* const nsum_p = a.st.nsum_p + my_set; float* const nsum_q = a.st.nsum_q + my_set;
    auto flush_item_stats = [&]() {
        if (acc_group != kNoRow) {
            red_add(gsum_q + (size_t)acc_group * K + stat_at, gq_acc);
            if (m == 0) atomicAdd(nsum_q + acc_group, nq_acc);
        }
    };
    // MuPPET, whole-model switching (muppet_sgd_kernel.h:266-285, sgd_kernel.h:266-285): the element-wise sum of both
    // gradients and the sum of their squared norms, one set for all groups, over the ratings of the worker.  The
    // norm of a rating goes through the worker's lanes during the next rating (`norm_step`), in the same order as at once.
    constexpr bool kWhole = STATS && (kMuppet<KIND> || KIND == KIND_SWITCH);
    float norm = 0.f;
    float4 norm_parts = make_float4(0.f, 0.f, 0.f, 0.f);      // with four elements a lane: what the first step joins
    // MASCOT, few workers: the same for the norms of both sides, each with the group it belongs to.  Nothing of it branches where the
    // workers of a warp could differ, and the two sums run under the next rating's dot product: a sampled rating took four times as long as
    // another one (check epoch of 8M ratings 1.353 -> 1.302 ms, k=64 20M 1.594 -> 1.531).  With K/8 lanes a worker the sums at once are
    // faster (20M 1.92 and 1.97, 40M 2.81 and 2.82; 100M equal: there the statistics are traffic).
    constexpr bool kDefer = kGroups && N == 4;
    constexpr bool kUserStats = kHalfRows<UM>, kItemStats = kHalfRows<IM>;
    float norm_q = 0.f;
    uint32_t late_groups = 0;
    bool late = false;                               // is there a rating before whose norms are to be added?
    auto late_step = [&](int part) {
        auto add = [&](float v) { return __fadd_rn(v, __shfl_xor_sync(kAll, v, (TS / 2) >> part)); };
        if (part == 0) {
            if (kUserStats) norm = __fadd_rn(add(norm_parts.x), add(norm_parts.y));
            if (kItemStats) norm_q = __fadd_rn(add(norm_parts.z), add(norm_parts.w));
        } else if ((TS / 2) >> part) {
            if (kUserStats) norm = add(norm);
            if (kItemStats) norm_q = add(norm_q);
        }
    };
    auto late_norms = [&]() {
        if (kUserStats) red_add_if_not(!late || m != 0, nsum_p + (late_groups & 0xffffu), norm);
        if (kItemStats && late) nq_acc = __fadd_rn(nq_acc, norm_q);
    };
    auto record_deferred = [&](const Sample<N>& smp, uint32_t both_groups, bool there) {
        late_norms();
        if (kUserStats) red_add_if_not(!there, gsum_p + (size_t)(both_groups & 0xffffu) * K + stat_at, smp.gp);
        if (kItemStats) {
            const uint32_t g = both_groups >> 16;
            const bool other = there && g != acc_group;
            if (__any_sync(kAll, other)) {
                const unsigned skip = !other || acc_group == kNoRow;
                const uint32_t to = skip ? 0u : acc_group;
                red_add_if_not(skip, gsum_q + (size_t)to * K + stat_at, gq_acc);
                red_add_if_not(skip || m != 0, nsum_q + to, nq_acc);
                if (other) {
                    acc_group = g; nq_acc = 0.f;
#pragma unroll
                    for (int t = 0; t < N; t++) gq_acc.x[t] = 0.f;
                }
            }
#pragma unroll
            for (int t = 0; t < N; t++) gq_acc.x[t] = there ? __fadd_rn(gq_acc.x[t], smp.gq.x[t]) : gq_acc.x[t];
        }
        late = there; late_groups = both_groups;
        float2 p2 = make_float2(0.f, 0.f), q2 = p2;
        if (kUserStats) p2 = __ffma2_rn(pr(smp.gp, 0), pr(smp.gp, 0), __fmul2_rn(pr(smp.gp, 1), pr(smp.gp, 1)));
        if (kItemStats) q2 = __ffma2_rn(pr(smp.gq, 0), pr(smp.gq, 0), __fmul2_rn(pr(smp.gq, 1), pr(smp.gq, 1)));
        norm_parts = make_float4(p2.x, p2.y, q2.x, q2.y);
    };
    auto norm_step = [&](int part) {
        if (kDefer) late_step(part);
        else if (kWhole && N == 4 && part == 0) norm = muppet_norm_join<K>(norm_parts);
        else if (kWhole && (TS / 2) >> part) norm = __fadd_rn(norm, __shfl_xor_sync(kAll, norm, (TS / 2) >> part));
    };
    auto record_whole = [&](const Sample<N>& smp, bool there) {
        nq_acc = __fadd_rn(nq_acc, norm);
        if constexpr (N == 4) norm_parts = there ? muppet_norm_parts<K>(smp.gp, smp.gq) : make_float4(0.f, 0.f, 0.f, 0.f);
        else norm = there ? muppet_norm_partial<K>(smp.gp, smp.gq) : 0.f;
        if (there) {
#pragma unroll
            for (int t = 0; t < N; t++) gq_acc.x[t] = __fadd_rn(gq_acc.x[t], __fadd_rn(smp.gp.x[t], smp.gq.x[t]));
        }
    };
    auto record = [&](const Sample<N>& smp, uint32_t both_groups) {
        if (smp.user) {
            const uint32_t g = both_groups & 0xffffu;
            const float n = worker_dot<TS>(smp.gp, smp.gp, gmask);
            red_add(gsum_p + (size_t)g * K + stat_at, smp.gp);
            if (m == 0) atomicAdd(nsum_p + g, n);
        }
        if (smp.item) {
            const uint32_t g = both_groups >> 16;
            const float n = worker_dot<TS>(smp.gq, smp.gq, gmask);
            if (g != acc_group) {
                flush_item_stats();
                acc_group = g; nq_acc = 0.f;
#pragma unroll
                for (int t = 0; t < N; t++) gq_acc.x[t] = 0.f;
            }
#pragma unroll
            for (int t = 0; t < N; t++) gq_acc.x[t] = __fadd_rn(gq_acc.x[t], smp.gq.x[t]);
            nq_acc = __fadd_rn(nq_acc, n);
        }
    };
    Sample<N> smp;
    AfpState afp;
    afp.user = AfpSide{8, 1.f, 0.f, 0}; afp.item = afp.user; afp.back = afp.user; afp.cur = 0; afp.due = 0;

    // requests the user row / the item row of a rating into ring slot `slot`
    auto request_user = [&](uint32_t uc, int slot) {
        if constexpr (kSpread) cp_row_if<K, UM>(uring + slot * SM::kURowBytes, P, uc);
        else cp_row<K, UM>(uring + slot * SM::kURowBytes, P, uc);
    };
    // A lane reads what it fetched itself - but of binary16 rows over K/4 lanes only one of two lanes fetches what both read, so there the lanes
    // meet between the wait and the read (and, once a rating, between a read and the request that uses the slot again).
    constexpr bool kMeet = UM == ROWS_HALFQ || IM == ROWS_HALFQ;
    auto request_item = [&](uint32_t ic, int slot) { cp_row_if<K, IM>(iring + slot * SM::kIRowBytes, Q, ic); };
    // Binary16 rows over K/4 lanes: copies are of 16 bytes, so the first half of the lanes fetches the user row and the second
    // half the item row, with one instruction.
    constexpr bool kOneRequest = UM == ROWS_HALFQ && IM == ROWS_HALFQ;
    const bool second = m & (TS / 2);
    const unsigned char* const one_base = reinterpret_cast<const unsigned char*>(second ? a.Q.f16 : a.P.f16) + 16 * (m & (TS / 2 - 1));
    const unsigned one_ring = rings + (second ? NS * SM::kURowBytes : 0) + 16 * (m & (TS / 2 - 1));
    auto request_one = [&](uint32_t uc, int uslot, uint32_t ic, int islot) {
        const uint32_t code = second ? ic : uc;
        cp16_if_row<0>(code, one_ring + (second ? islot * SM::kIRowBytes : uslot * SM::kURowBytes), one_base + (uint64_t)code * (2u * K));
    };
    // Copy groups complete in order, and every rating commits one: the item row of the rating DI ahead and the user
    // row of the rating D ahead.  Before rating j commits, the groups younger than the user row of rating j+1 are
    // D - 2, those younger than the item row of rating j are DI - 1: waiting for exactly that many to remain
    // pending leaves every younger copy in flight.
#pragma unroll
    for (int t = 0; t < D; t++) {
        if (t >= D - DI) request_item((recs[t - (D - DI)].x & F_RS) ? recs[t - (D - DI)].y : kNoRow, (t - (D - DI)) & (NSI - 1));
        request_user(kSpread && (recs[t].x & F_NONE) ? kNoRow : recs[t].z, t);
        cp_commit();
    }
    uint4 rec = recs[0];
    cp_wait<D - 1>();
    if constexpr (kMeet) __syncwarp();
    Raw<UM> p = lds_row<K, UM>(uring, rec.z);
    bool turn = __any_sync(kAll, rec.x & (F_RS | F_UDUP));      // does the coming rating of some worker need another item row?

    constexpr int kUnroll = (KIND == KIND_AFP || KIND == KIND_MUPPET) ? 1 : KIND == kMuppetHalf ? 2 : NS;
    int cb = 0;                                     // buffer of the chunk in use
    while (__any_sync(kAll, cnt_cur > 0)) {
#pragma unroll 1
        for (int jb = 0; jb < TS; jb += NS) {
            // this group of NS records and the next one (in the other buffer at the end of a chunk)
            const unsigned r0 = s_rec + 16 * (cb * TS + jb), r1 = s_rec + 16 * ((cb * TS + jb + NS) & (2 * TS - 1));
            const unsigned q0 = s_req + 8 * (cb * TS + jb);
            // The fixed-point updates are some hundred instructions long: one copy of them, or the warps wait for
            // instruction fetches (3.4 cycles per instruction with four copies of the AFP update).
#pragma unroll(kUnroll)
            for (int t = 0; t < NS; t++) {
                const uint32_t uc = rec.z, ic = rec.y, f = rec.x, rw = rec.w;
                if (turn) {
                    // a run of equal items ends for at least one of the warp's workers (or a row has to be read again)
                    cp_wait<DI - 1>();
                    if constexpr (kMeet) __syncwarp();
                    const unsigned start = f & F_RS;
                    st_row_if<K, IM>(start & have_item, Q, cur_ic, q);
                    const unsigned slot = iring + (t & (NSI - 1)) * SM::kIRowBytes;
                    lds_if<0>(start, q.a, slot);
                    if constexpr (kTwoParts<IM>) lds_if<2 * K>(second_half<IM>(start, ic), q.b, slot);
                    if (__any_sync(kAll, f & (F_IDUP | F_UDUP))) {
                        ld_row_if<K, IM>(f & F_IDUP, q, Q, ic);
                        ld_row_if<K, UM>(f & F_UDUP, p, P, uc);
                    }
                    if (start) { cur_ic = ic; have_item = (f & F_NONE) ? 0u : F_RS; }
                }
                // what the ratings to come need, into slots whose contents have been consumed
                Raw<UM> p_next;
                uint32_t req_u, req_i;
                auto meanwhile = [&](int part) {
                    norm_step(part);
                    if (part == 0) {
                        rec = lds128(t + 1 < NS ? r0 + 16 * (t + 1) : r1);
                        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(req_u), "=r"(req_i) : "r"(q0 + 8 * t) : "memory");
                    } else if (part == 1) {
                        cp_wait<D - 2>();
                        if constexpr (kMeet) __syncwarp();
                        p_next = lds_row<K, UM>(uring + ((t + 1) & (NS - 1)) * SM::kURowBytes, rec.z);
                    } else if (part == 2) {
                        if constexpr (kOneRequest) request_one(req_u, (t + D) & (NS - 1), req_i, (t + DI) & (NSI - 1));
                        else {
                            request_item(req_i, (t + DI) & (NSI - 1));
                            request_user(req_u, (t + D) & (NS - 1));
                        }
                        cp_commit();
                        turn = __any_sync(kAll, rec.x & (F_RS | F_UDUP));
                    }
                };
                const Raw<UM> p_before = p;
                constexpr bool kDyn = UM == ROWS_DYN || IM == ROWS_DYN;
                update_one<K, KIND, UM, IM, STATS>(c, rw, uc, ic, p, q, smp, afp, !(f & F_NONE), kDyn ? gmask : kAll, slots + (t & 1) * SM::kSlotBytes, meanwhile);
                if (a.add_user_delta) add_row_delta<K, UM>(P, uc, f & F_DROP, p, p_before);
                else st_row_if<K, UM>(~f & F_DROP, P, uc, p);
                if constexpr (kWhole) record_whole(smp, !(f & F_NONE));
                else if constexpr (kDefer) record_deferred(smp, groups[cb * TS + jb + t], !(f & F_NONE));
                else if (STATS) { if (!(f & F_NONE)) record(smp, kGroups ? groups[cb * TS + jb + t] : 0u); }
                p = p_next;
            }
        }
        cnt_cur = cnt_next;
        cnt_next = publish(cb);      // the chunk after next takes the buffer of the finished one
        cb ^= 1;
    }
    cp_wait<0>();
    st_row_if<K, IM>(have_item, Q, cur_ic, q);
    if (STATS) {
        if constexpr (kWhole) {
            // the norm of the last rating
            if constexpr (N == 4) nq_acc = __fadd_rn(nq_acc, worker_sum<TS / 2>(muppet_norm_join<K>(norm_parts), kAll));
            else nq_acc = __fadd_rn(nq_acc, worker_sum<TS>(norm, kAll));
            red_add(gsum_p + stat_at, gq_acc);
            if (m == 0) atomicAdd(nsum_p, nq_acc);
        }
        else {
            if constexpr (kDefer) {
#pragma unroll
                for (int part = 0; (TS / 2) >> part; part++) late_step(part);
                late_norms();
            }
            flush_item_stats();
        }
    }
}

__global__ void reduce_stats_kernel(float* sets, int copies, size_t stride, size_t n) {
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (size_t)gridDim.x * blockDim.x) {
        float acc = sets[j];
        for (int c = 1; c < copies; c++) acc = __fadd_rn(acc, sets[(size_t)c * stride + j]);
        sets[j] = acc;
    }
}

template <int K, int KIND, int UM, int IM, bool STATS, int NS, int NSI, int D, int DI>
cudaError_t launch_ns(KernelArgs a, unsigned warps_per_sm, unsigned workers, cudaStream_t st, LaunchShape* shape, bool dry) {
    constexpr int TS = K / kElems<UM>;
    constexpr int kPerWarp = 32 / TS;
    using SM = WorkerSmem<K, KIND, UM, IM, STATS, NS, NSI>;
    auto kern = train_kernel<K, KIND, UM, IM, STATS, NS, NSI, D, DI>;
    // the most dynamic shared memory a launch of this instantiation can ask for: a block of 8 warps
    constexpr size_t kSmemMax = (size_t)8 * kPerWarp * SM::kBytes;
    static LaunchCache cache;                    // one per instantiation; see launch_cache.h
    int grid, block;
    unsigned warps = (workers + kPerWarp - 1) / kPerWarp;
    // The workers of an AFP warp compute both passes whenever their formats differ, so few of them are spread over more
    // warps, up to two per scheduler (K/8 lanes, 4M ratings, 592 workers: 6.75 ms per epoch with two workers a warp, 5.78 with one).
    // For the other trainers a second warp on a scheduler costs more than it gives: MPT 1.81 ms spread out 2.21, MASCOT
    // 1.30 and 1.49, MuPPET 3.00 and 3.12.
    constexpr unsigned kSpreadWarps = KIND == KIND_AFP ? 8 : 0;
    unsigned spread = 0;
    if (warps > 8) {
        const unsigned even = (unsigned)sm_count() * warps_per_sm * kPerWarp;             // the workers of the launch
        while ((kPerWarp >> spread) > 1 && (warps_per_sm << (spread + 1)) <= kSpreadWarps) spread++;
        if (spread) { warps_per_sm <<= spread; warps = even / (kPerWarp >> spread); }
    }
    a.spread = spread;
    if (workers <= 1) a.add_user_delta = 0;      // a single worker has nobody to race with: plain stores
    unsigned blocks_per_sm = 1, warps_per_block = warps;
    if (warps > 8) {
        // the same number of warps on every SM, in blocks of at most 8 warps
        blocks_per_sm = (warps_per_sm + 7) / 8;
        warps_per_block = (warps_per_sm + blocks_per_sm - 1) / blocks_per_sm;
    }
    block = (int)(32 * warps_per_block);
    const size_t smem = (size_t)warps_per_block * kPerWarp * SM::kBytes;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int fit = 0;
    const int rc = cache.lookup(
        dev, block, smem, kSmemMax,
        [&](size_t bytes) { return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); },
        [&](int blk, size_t sm, int* f) { return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(f, kern, blk, sm); }, &fit);
    if (rc != 0) return (cudaError_t)rc;
    if (fit < 1) return cudaErrorLaunchOutOfResources;
    size_t smem_used = smem;
    if (warps > 8 && blocks_per_sm > (unsigned)fit && warps_per_block < 8) {
        // The SM cannot hold as many blocks as the even split asked for: blocks of the full eight warps may then put
        // more warps on it (27 warps wanted, fp32 rows on both sides: four blocks of seven, of which three fit = 21
        // warps; three blocks of eight = 24).
        int fit8 = 0;
        const size_t smem8 = (size_t)8 * kPerWarp * SM::kBytes;
        const int rc8 = cache.lookup(
            dev, 256, smem8, kSmemMax,
            [&](size_t bytes) { return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); },
            [&](int blk, size_t sm, int* f) { return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(f, kern, blk, sm); }, &fit8);
        if (rc8 != 0) return (cudaError_t)rc8;
        if (fit8 * 8 > fit * (int)warps_per_block) {
            warps_per_block = 8; block = 256; smem_used = smem8; fit = fit8;
            blocks_per_sm = (warps_per_sm + 7) / 8;
        }
    }
    if (warps <= 8) {
        // a single block (deterministic runs, tiny worker counts) uses exactly the requested workers
        grid = 1;
        a.workers = workers;
    } else {
        // no more blocks than the SM can hold at once (registers, shared memory)
        if (blocks_per_sm > (unsigned)fit) blocks_per_sm = (unsigned)fit;
        grid = (int)((unsigned)sm_count() * blocks_per_sm);
        a.workers = (unsigned)grid * warps_per_block * (kPerWarp >> spread);
    }
    if (!dry) kern<<<grid, block, smem_used, st>>>(a);      // a dry call stops here: the function is loaded and configured
    if (shape) { shape->grid = grid; shape->block = block; shape->smem = smem_used; shape->workers = a.workers; }
    return cudaGetLastError();
}

template <int K, int KIND, int UM, int IM, bool STATS>
cudaError_t launch_one(const KernelArgs& args, unsigned workers, cudaStream_t st, LaunchShape* shape, bool dry) {
    constexpr int TS = K / 8;
    constexpr int kPerWarp = 32 / TS;
    if (workers < 1) workers = 1;
    // more workers than can ever be resident at once (64 warps per SM) only add launch overhead
    const unsigned resident_cap = (unsigned)sm_count() * 64u * kPerWarp;
    if (workers > resident_cap) workers = resident_cap;
    const unsigned warps = (workers + kPerWarp - 1) / kPerWarp;
    const unsigned sms = (unsigned)sm_count();
    const unsigned per_sm = warps <= 8 ? warps : (warps + sms - 1) / sms;
    // User rows are requested five ratings ahead (ring of eight slots), item rows three (ring of four): about a microsecond
    // at 0.2 us a rating.  Three and two ahead cost the small configurations 5 to 20 % (8M ratings: 1.30 -> 1.57 ms per
    // epoch; four and two 1.40) and the 100M-rating one nothing; six and seven gain nothing.  The fixed-point updates
    // are three to four times as long, and for them three and two are enough.
    constexpr bool kFixedPoint = KIND == KIND_AFP || kMuppet<KIND>;
    constexpr int NS = kFixedPoint ? 4 : 8, D = kFixedPoint ? 3 : 5, DI = kFixedPoint ? 2 : 3;
    // A step of few warps is a chain of some ninety instructions.  With K/4 lanes a worker the warp has half of the row work
    // and one worker fewer to wait for: shorter steps, on twice as many warps - as long as the schedulers can take those.  ms per
    // epoch with K/8 and K/4 lanes, by warps of the narrow form per SM: AFP 4M ratings (4) 5.69 and 3.37, 12M (10) 8.94 and 5.17; MuPPET,
    // 8 bits, 2M (4) 2.25 and 1.13, 14M (12) 5.73 and 4.08; MPT 8M (8) 1.81 and 1.37, 18M (16) 2.38 and 2.16; SGD 8M (8) 1.52 and
    // 1.24, 16M (14) 2.08 and 1.92, k=64 0.8M (6) 0.132 and 0.100, 20M (10) 2.04 and 1.64; fp16 storage 8M 1.64 and 1.47, 16M (14) 2.13 and
    // 2.04; MASCOT k=64 8M (4) 1.44 and 1.19, 20M (10) 1.56 and 1.41, 30M (14) 1.73 and 1.66, 40 % promoted, 8M (8) 2.93 and 2.74, 16M (14) 3.80 and 3.81.  At 18 and
    // more the narrow form gives nothing more (SGD 20M 2.32 and 2.32) or loses (fp16 storage 20M 2.08 and 2.23).  Binary16 rows with
    // packed binary16 arithmetic have the shortest steps and stop gaining earlier: k=128, 2M (4) 0.637 and 0.531, 8M (8) 1.302 and
    // 1.184, 14M (12) 1.646 and 1.565, 16M (14) 1.659 and 1.671, 20M (18) 1.66 and 1.91.
    if constexpr (UM != ROWS_DYN) {
        constexpr int UQ = UM == ROWS_HALF ? ROWS_HALFQ : ROWS_F32Q, IQ = IM == ROWS_HALF ? ROWS_HALFQ : ROWS_F32Q;
        constexpr unsigned kMost = K == 128 && kHalfRating<KIND, UM, IM> && KIND != KIND_MPT && !STATS ? 12 : 16;      // warps per SM
        // Binary16 rows: steps of 0.16 to 0.2 us, a fifth shorter than those the leads were made for, so one rating more each - the same
        // time ahead (k=64, 20M 1.42 -> 1.395, 8M 1.191 -> 1.160; k=128, 2M 0.530 -> 0.517, 8M 1.182 -> 1.176).  Seven and five are slower
        // again, and MPT loses by it (1.370 and 1.383).
        constexpr bool kLonger = kHalfRows<UM> && kHalfRows<IM>;
        // (a single block has exactly the workers that were asked for: they have to fit it in this form, too)
        // Grids whose workers have few runs of K ratings each keep the wide form, in all launches of an epoch.  Workers that begin together hold
        // the same popular items and write them back together, and whose row stays hangs on how the steps fall together: the same from pass to
        // pass, another in the other form.  Over few runs that does not average out.  Distance of the factors after three trainings of 10
        // to 12 epochs to those of the wide form, in multiples of what two passes of one form differ by: fp32 SGD, 300,000 ratings, two runs
        // a worker 8.4; memory quantization, 1.45M, six runs 4.4; MPT, ten runs 3.4; from 16 runs on 1.3 to 2.4 for sets of the
        // benchmarks' density.  It costs a set of 0.8M ratings of fp32 SGD 0.100 -> 0.132 ms per epoch.  The fixed-point updates, whose
        // steps differ less between the forms: AFP 6 at one run, 3.4 at 2.6, 2.4 and less from 4 on.
        constexpr unsigned kRuns = kFixedPoint ? 4 : 16;
        const bool settled = args.whole >= (uint64_t)kRuns * K * (sms * per_sm * kPerWarp);
        if (2 * per_sm <= kMost && (warps > 8 ? settled : 2 * workers <= 8 * kPerWarp))
            return launch_ns<K, KIND, UQ, IQ, STATS, NS, kLonger ? 8 : 4, kLonger ? 6 : D, kLonger ? 4 : DI>(args, 2 * per_sm, workers, st, shape, dry);
    }
    // With fp32 rows the deep rings leave room for fewer warps than the registers do (k=128, both sides fp32: 16 per SM
    // against 24).  Where a launch of a mixed-precision class with an fp32 side asks for more workers than the deep rings hold and
    // rings of 4 + 2 slots hold more, it takes these, three ratings and one ahead, and has the workers, which wait for rows that others have
    // just written.  ms per epoch, deep rings for all classes and this rule: 40 % of the groups promoted, 40M ratings 7.12 and
    // 7.11, 63M 9.37 and 9.20, k=64 100M 13.93 and 12.96; 100M (a fifth) 10.38 and 9.99; all promoted, 63M 10.97 and 10.72.  The other
    // trainers do without (SGD 7.73 and 7.74 at 63M, 10.53 and 10.58 at 100M): they are bound by what the rows' traffic allows.
    constexpr bool kShortRings = KIND == KIND_MIXED && !STATS && UM != ROWS_DYN && (UM == ROWS_F32 || IM == ROWS_F32);
    if constexpr (kShortRings) {
        LaunchShape deep, shallow;
        cudaError_t e = launch_ns<K, KIND, UM, IM, STATS, NS, 4, D, DI>(args, per_sm, workers, st, &deep, true);
        if (e == cudaSuccess && deep.workers < workers) e = launch_ns<K, KIND, UM, IM, STATS, 4, 2, 3, 1>(args, per_sm, workers, st, &shallow, true);
        if (e != cudaSuccess) return e;
        if (shallow.workers > deep.workers) return launch_ns<K, KIND, UM, IM, STATS, 4, 2, 3, 1>(args, per_sm, workers, st, shape, dry);
    }
    return launch_ns<K, KIND, UM, IM, STATS, NS, 4, D, DI>(args, per_sm, workers, st, shape, dry);
}

template <int K, int KIND, int UM, int IM>
cudaError_t launch_st(const KernelArgs& a, bool stats, unsigned workers, cudaStream_t st, LaunchShape* sh, bool dry) {
    return stats ? launch_one<K, KIND, UM, IM, true>(a, workers, st, sh, dry) : launch_one<K, KIND, UM, IM, false>(a, workers, st, sh, dry);
}

template <int K>
cudaError_t launch_k(TrainKind kind, const KernelArgs& a, bool stats, RowClass cls, unsigned workers, cudaStream_t st, LaunchShape* sh, bool dry) {
    switch (kind) {
        case KIND_MIXED:
            switch (cls) {
                case ROWCLASS_HH: return launch_st<K, KIND_MIXED, ROWS_HALF, ROWS_HALF>(a, stats, workers, st, sh, dry);
                case ROWCLASS_HF: return launch_st<K, KIND_MIXED, ROWS_HALF, ROWS_F32>(a, stats, workers, st, sh, dry);
                case ROWCLASS_FH: return launch_st<K, KIND_MIXED, ROWS_F32, ROWS_HALF>(a, stats, workers, st, sh, dry);
                case ROWCLASS_FF: return launch_one<K, KIND_MIXED, ROWS_F32, ROWS_F32, false>(a, workers, st, sh, dry);      // fp32 groups are not sampled
                case ROWCLASS_ANY: return launch_st<K, KIND_MIXED, ROWS_DYN, ROWS_DYN>(a, stats, workers, st, sh, dry);
            }
            return cudaErrorInvalidValue;
        case KIND_FP32: return launch_one<K, KIND_FP32, ROWS_F32, ROWS_F32, false>(a, workers, st, sh, dry);
        case KIND_MPT: return launch_one<K, KIND_MPT, ROWS_F32, ROWS_F32, false>(a, workers, st, sh, dry);
        case KIND_MEMQUANT: return launch_one<K, KIND_MEMQUANT, ROWS_HALF, ROWS_HALF, false>(a, workers, st, sh, dry);
        case KIND_AFP: return launch_one<K, KIND_AFP, ROWS_F32, ROWS_F32, false>(a, workers, st, sh, dry);
        case KIND_SWITCH: return launch_st<K, KIND_SWITCH, ROWS_HALF, ROWS_HALF>(a, stats, workers, st, sh, dry);
        case KIND_MUPPET:
            // at 32 bits MuPPET is plain fp32 SGD and samples nothing (2M ratings: 0.81 ms per epoch in a kernel for all widths, 0.64 in this one)
            if (a.bits == 32) return launch_one<K, KIND_FP32, ROWS_F32, ROWS_F32, false>(a, workers, st, sh, dry);
            if (a.bits == 8) return launch_st<K, KIND_MUPPET, ROWS_F32, ROWS_F32>(a, stats, workers, st, sh, dry);
            return launch_st<K, kMuppetHalf, ROWS_F32, ROWS_F32>(a, stats, workers, st, sh, dry);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_reduce_stats(float* sets, int copies, size_t copy_stride, size_t floats_per_set, cudaStream_t st) {
    if (copies <= 1 || floats_per_set == 0) return cudaSuccess;
    const int grid = (int)((floats_per_set + 255) / 256);
    reduce_stats_kernel<<<grid, 256, 0, st>>>(sets, copies, copy_stride, floats_per_set);
    return cudaGetLastError();
}

int sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    int& v = sms[dev & 63];
    if (!v) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 1;
}

cudaError_t launch_train(int K, TrainKind kind, const Stream& s, Arena P, Arena Q, float lr, float lam,
                         const SampleStats* stats, RowClass row_class, unsigned workers, WorkCounters* counters,
                         int bits, int epoch, bool add_user_delta, unsigned hot_user_shift, uint64_t whole, cudaStream_t st, LaunchShape* shape) {
    KernelArgs a;
    a.hot_user_shift = hot_user_shift;
    a.whole = whole;
    a.add_user_delta = add_user_delta ? 1 : 0;
    a.s = s; a.P = P; a.Q = Q; a.lr = lr; a.lam = lam; a.workers = workers; a.bits = bits; a.epoch = epoch;
    if (stats) a.st = *stats;
    if (s.n == 0) { if (shape) *shape = LaunchShape(); return cudaSuccess; }
    if (!counters) {
        // dry call: loads the instantiation this launch would use and sets its shared-memory limit, launches nothing
        if (K == 128) return launch_k<128>(kind, a, stats != nullptr, row_class, workers, st, shape, true);
        if (K == 64) return launch_k<64>(kind, a, stats != nullptr, row_class, workers, st, shape, true);
        return cudaErrorInvalidValue;
    }
    // Launches of one engine run one after the other on its stream.  Launch number L hands out chunks
    // through counter L mod 4 and resets counter (L + 2) mod 4, which the launch after next will use and
    // which no launch in flight touches; all four start at zero.
    a.next_chunk = counters->d_slots + (counters->launches & 3);
    a.zero_counter = counters->d_slots + ((counters->launches + 2) & 3);
    counters->launches++;
    if (K == 128) return launch_k<128>(kind, a, stats != nullptr, row_class, workers, st, shape, false);
    if (K == 64) return launch_k<64>(kind, a, stats != nullptr, row_class, workers, st, shape, false);
    return cudaErrorInvalidValue;
}

}  // namespace mascot
