// hj_single.cu - the one-pass partition phase of radix joins whose build relation needs at most 2^11
// partitions.
//
// The number of radix bits a caller asks for (NUM_RADIX_BITS, 14 by default) fits build relations of
// 10^8 tuples. A build relation of 2^20 tuples would fall into 2^14 partitions of 64 tuples, and the
// two-pass pipeline then works on units of ~90 tuples, each a partial tile (2^20 x 2^22: 0.40 of 0.79 ms
// in pass 2). A partition join needs only that the build partitions fit shared memory, so this pipeline
// takes the lowest bits that bring them to kSingleTarget tuples on average and partitions in one pass:
//   single_count    CTA c reads a contiguous range of R and one of S: a histogram row of the digit per
//                   relation, and the ORs that decide the element layout
//   single_plan     per digit, the exclusive prefix of the rows (in place) and the totals; the CTA that
//                   finishes last turns the totals into partition starts, join items and large
//                   partitions
//   single_scatter  CTA c reads its ranges again, last tuple first (what the count read last is still in
//                   L2), takes each element's place from a shared-memory cursor per digit and stores it
// The partitions are those of `bits` low bits of the key or of mix_key, so the join kernels are the two-pass
// pipelines'.
//
// Elements: compact words ci_word (8 bytes) when the widths allow them, else tuples. First-match joins
// need the lowest input position among equal build keys; their build elements are 16 bytes, {ci_word,
// position} or {key, position}, so the order inside a partition does not matter and no pass is ordered.
#include <cstdio>

#include "hj_common.cuh"
#include "hj_internal.h"
#include "hj_partition.cuh"

namespace hj {

constexpr int kCountThreads = 1024;
constexpr int kPlaceThreads = 512;  // scatter: one CTA per SM
constexpr int kWordItems = 20, kTupleItems = kWordItems / 2;  // staged 8-byte / 16-byte elements per thread and tile
constexpr int kSingleDigitsPerThread = ((1 << kSingleMaxBits) + kPlaceThreads - 1) / kPlaceThreads;

// The contiguous range of n tuples that block c of G takes (a multiple of 8 tuples, one 128-byte line).
__device__ __forceinline__ void single_range(uint64_t n, uint32_t c, uint32_t G, uint64_t *lo, uint64_t *hi) {
    const uint64_t per = ((n + G - 1) / G + 7) & ~7ull;
    *lo = c * per < n ? c * per : n;
    *hi = *lo + per < n ? *lo + per : n;
}

// Shared memory of the scatter: a staged tile, and four words per digit.
constexpr size_t kSingleStage = (size_t)kPlaceThreads * kWordItems * 8;
inline size_t single_scatter_smem(int bits) { return kSingleStage + 128 + ((size_t)4 << bits) * 4; }

// Input tuple of the count: read again by the scatter, so its line keeps the normal L2 priority.
__device__ __forceinline__ tuple_v ld_twice(const tuple_v *p) {
    tuple_v v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

// ------------------------------------------------------------------------------------------------
// 1. Count. Bound by reading the relations (four 16-byte loads per thread in flight, 1024 threads per SM);
//    the shared-memory increments return nothing. With few partitions the warps spread over `copies`
//    histograms, since 32 lanes on a handful of counters serialise.
// ------------------------------------------------------------------------------------------------
// MIX (always in a wave): digits of mix_key.
template <bool MULTI, bool MIX>
__global__ void __launch_bounds__(kCountThreads, 1) single_count(SingleArgs a0, MultiRef mr) {
    extern __shared__ uint32_t sh[];  // [copies][P]
    __shared__ SingleArgs s_a;
    uint32_t blk = blockIdx.x, G = gridDim.x;
    if (MULTI) {
        const uint2 e = mr.map[blockIdx.x];
        multi_copy(&s_a, &mr.jobs[e.x].sa);
        blk = e.y;
        G = mr.jobs[e.x].grid;
        __syncthreads();
    }
    const SingleArgs &a = MULTI ? s_a : a0;
    const int tid = threadIdx.x;
    const uint32_t P = 1u << a.bits, mask = P - 1;
    uint32_t *mine = sh + (size_t)((uint32_t)(tid >> 5) % (uint32_t)a.copies) * P;
    __shared__ unsigned long long s_or[3];
    if (tid < 3) s_or[tid] = 0;
    // The kernels after this one find their counters (and the result) at zero.
    if (blk == 0 && tid < kNumCounters) a.counters[tid] = 0;
    if (blk == 0 && a.clear_acc && tid == 0) *a.acc = JoinAccum{};
    for (int rel = 0; rel < 2; rel++) {
        for (uint32_t j = tid; j < P * a.copies; j += kCountThreads) sh[j] = 0;
        __syncthreads();
        const tuple_v *in = rel ? a.S : a.R;
        uint64_t lo, hi;
        single_range(rel ? a.nS : a.nR, blk, G, &lo, &hi);
        unsigned long long kor = 0, ror = 0;
        constexpr int U = 4;
        uint64_t i = lo + tid;
        for (; i + (U - 1) * kCountThreads < hi; i += U * kCountThreads) {
            tuple_v t[U];
#pragma unroll
            for (int u = 0; u < U; u++) t[u] = ld_twice(in + i + u * kCountThreads);
#pragma unroll
            for (int u = 0; u < U; u++) {
                atomicAdd(&mine[(uint32_t)(MIX ? mix_key(t[u].x, a.bits) : t[u].x) & mask], 1u);
                kor |= t[u].x;
                ror |= t[u].y;
            }
        }
        for (; i < hi; i += kCountThreads) {
            const tuple_v t = ld_twice(in + i);
            atomicAdd(&mine[(uint32_t)(MIX ? mix_key(t.x, a.bits) : t.x) & mask], 1u);
            kor |= t.x;
            ror |= t.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            kor |= __shfl_xor_sync(0xffffffffu, kor, o);
            ror |= __shfl_xor_sync(0xffffffffu, ror, o);
        }
        if ((tid & 31) == 0) {
            if (rel == 0) {
                atomicOr(&s_or[0], kor);
                atomicOr(&s_or[1], ror);
            } else {
                atomicOr(&s_or[2], ror);
            }
        }
        __syncthreads();
        uint32_t *row = a.hist + ((size_t)rel * G + blk) * P;
        for (uint32_t j = tid; j < P; j += kCountThreads) {
            uint32_t n = 0;
            for (int c = 0; c < a.copies; c++) n += sh[(size_t)c * P + j];
            row[j] = n;
        }
        __syncthreads();
    }
    if (tid < 3) a.ors[(size_t)blk * 3 + tid] = s_or[tid];
}

// ------------------------------------------------------------------------------------------------
// 2. Prefixes and plan. A CTA takes 32 columns (digits of one relation; consecutive lanes read
//    consecutive digits of a row), its 32 warps share the rows. The CTA that finishes last plans.
// ------------------------------------------------------------------------------------------------
template <bool MULTI>
__global__ void __launch_bounds__(1024, 1) single_plan(SingleArgs a0, PlanArgs pa0, uint32_t G0, MultiRef mr) {
    __shared__ uint32_t part[32][33];
    __shared__ uint32_t tmp[32];
    __shared__ uint64_t s_run[2];
    __shared__ bool s_last;
    extern __shared__ uint32_t sm_tot[];  // [2][P]
    __shared__ SingleArgs s_a;
    __shared__ PlanArgs s_pa;
    uint32_t blk = blockIdx.x, nblk = gridDim.x, G = G0;
    if (MULTI) {
        const uint2 e = mr.map[blockIdx.x];
        multi_copy(&s_a, &mr.jobs[e.x].sa);
        multi_copy(&s_pa, &mr.jobs[e.x].pa);
        blk = e.y;
        nblk = mr.jobs[e.x].plan_blocks;
        G = mr.jobs[e.x].grid;
        __syncthreads();
    }
    const SingleArgs &a = MULTI ? s_a : a0;
    const PlanArgs &pa = MULTI ? s_pa : pa0;
    uint32_t *total = const_cast<uint32_t *>(pa.total);
    const uint32_t P = 1u << a.bits;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t col = blk * 32 + lane;
    const uint32_t rel = col >= P;
    if (col < 2 * P) {
        uint32_t *h = a.hist + (size_t)rel * G * P + (col - rel * P);
        const uint32_t per = (G + 31) / 32;
        const uint32_t r0 = min(G, w * per), r1 = min(G, r0 + per);
        uint32_t sum = 0;
#pragma unroll 8
        for (uint32_t r = r0; r < r1; r++) sum += h[(size_t)r * P];
        part[w][lane] = sum;
    }
    __syncthreads();
    if (w == 0 && col < 2 * P) {
        uint32_t run = 0;
#pragma unroll
        for (int q = 0; q < 32; q++) {
            const uint32_t x = part[q][lane];
            part[q][lane] = run;
            run += x;
        }
        total[col] = run;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&a.counters[kCtrTicket], 1u) == nblk - 1;
    if (col < 2 * P) {
        uint32_t *h = a.hist + (size_t)rel * G * P + (col - rel * P);
        const uint32_t per = (G + 31) / 32;
        const uint32_t r0 = min(G, w * per), r1 = min(G, r0 + per);
        uint32_t run = part[w][lane];
#pragma unroll 8
        for (uint32_t r = r0; r < r1; r++) {
            const uint32_t x = h[(size_t)r * P];
            h[(size_t)r * P] = run;
            run += x;
        }
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (uint32_t j = threadIdx.x; j < 2 * P; j += 1024) sm_tot[j] = __ldcg(&total[j]);
    // ORs of all CTAs -> the counters that ci_applies and compact_applies read.
    if (w < 3) {
        unsigned long long v = 0;
        for (uint32_t c = lane; c < G; c += 32) v |= a.ors[(size_t)c * 3 + w];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) reinterpret_cast<unsigned long long *>(a.counters + kCtrMaxKey)[w] = v;
    }
    __syncthreads();
    plan_body(pa, sm_tot, tmp, s_run);
}

// ------------------------------------------------------------------------------------------------
// 3. Scatter. Tiles of 10240 8-byte or 5120 16-byte elements: a thread takes 20 (10) elements, all their loads
//    in flight together and issued under the previous tile's write-out; their ranks within their digit come
//    from shared-memory atomics; a block scan over the digits gives each digit's start in the tile; the tile
//    is staged in digit order and written out, consecutive threads to consecutive places of a digit's run. A
//    CTA's elements of a digit go to its own consecutive places, so the next place of every digit is a
//    counter in shared memory. A staged element still tells its digit, so none is kept beside it.
//    One CTA per SM: every tile visits every page of the output, and those visits, not the length of the
//    runs, are what scattered stores cost (12.6 M words to 1024 partitions of 100 MB: 77 us stored in
//    place, 76 us scattered over 8 MB, 98 us over the 100 MB; 2 CTAs with half the tile: 125 us; 4 CTAs:
//    153 us; direct stores without staging: 36-65 G elements per second).
// ------------------------------------------------------------------------------------------------
enum SingleMode {
    kModeWord,      // staged {low 32 key bits, row id} (build keys below 2^31), written as a compact word
    kModeTuple,     // staged and written as a tuple
    kModeTupleWord, // staged as a tuple, written as a compact word
    kModePosWord,   // first-match builds: {compact word, position | digit << 32}, written as {word, position}
    kModePos,       // first-match builds, wide: {key, position}
};

// Staged and written element of a mode. bits: radix bits; mask = 2^bits - 1.
template <int MODE>
struct SingleElem {
    using Staged = tuple_v;
    using Out = tuple_v;
    static __device__ __forceinline__ tuple_v stage(const tuple_v &t, uint64_t i, int bits, uint32_t mask, bool z0) {
        if (MODE == kModePosWord)
            return make_ulonglong2(ci_word_z0(t.x, t.y, bits, z0), i | ((unsigned long long)((uint32_t)t.x & mask) << 32));
        return MODE == kModePos ? make_ulonglong2(t.x, i) : t;
    }
    static __device__ __forceinline__ uint32_t digit(const tuple_v &v, uint32_t mask) {
        return MODE == kModePosWord ? (uint32_t)(v.y >> 32) : (uint32_t)v.x & mask;
    }
    static __device__ __forceinline__ tuple_v out(const tuple_v &v, int) {
        return MODE == kModePosWord ? make_ulonglong2(v.x, v.y & 0xffffffffull) : v;
    }
};
template <>
struct SingleElem<kModeTupleWord> {
    using Staged = tuple_v;
    using Out = unsigned long long;
    static __device__ __forceinline__ tuple_v stage(const tuple_v &t, uint64_t, int, uint32_t, bool) { return t; }
    static __device__ __forceinline__ uint32_t digit(const tuple_v &v, uint32_t mask) { return (uint32_t)v.x & mask; }
    static __device__ __forceinline__ unsigned long long out(const tuple_v &v, int bits) { return ci_word(v.x, v.y, bits); }
};
template <>
struct SingleElem<kModeWord> {
    using Staged = uint2;  // x: row id, y: key (a probe key of 2^31 or more: its digit with bit 31 set)
    using Out = unsigned long long;
    static __device__ __forceinline__ uint2 stage(const tuple_v &t, uint64_t, int, uint32_t mask, bool) {
        const uint32_t lo = (uint32_t)t.x, hi = (uint32_t)(t.x >> 32);
        return make_uint2((uint32_t)t.y, (hi | (lo & 0x80000000u)) ? 0x80000000u | (lo & mask) : lo);
    }
    static __device__ __forceinline__ uint32_t digit(const uint2 &v, uint32_t mask) { return v.y & mask; }
    static __device__ __forceinline__ unsigned long long out(const uint2 &v, int bits) {
        const uint32_t h = (int)v.y < 0 ? 0xffffffffu : v.y >> bits;
        return ((unsigned long long)h << 32) | v.x;
    }
};

// Exclusive scan of one u32 per thread; tmp is reused only after two more barriers.
__device__ __forceinline__ uint32_t place_scan(uint32_t v, uint32_t *tmp) {
    const unsigned lane = lane_id(), w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) tmp[w] = x;
    __syncthreads();
    // Every warp adds up the totals of the warps before it.
    return __reduce_add_sync(0xffffffffu, lane < w ? tmp[lane] : 0u) + x - v;
}

// Place one relation's range. A function of its own per mode: inlined side by side the modes spilled. MIX: the key
// becomes mix_key when it is staged.
template <int MODE, bool MIX>
__device__ __noinline__ void single_scatter_rel(const SingleArgs &a, int rel, uint32_t blk, uint32_t G) {
    using Elem = SingleElem<MODE>;
    using E = typename Elem::Staged;
    using O = typename Elem::Out;
    constexpr int NT = kPlaceThreads, ITEMS = MODE == kModeWord ? kWordItems : kTupleItems;
    constexpr int D = kSingleDigitsPerThread;
    constexpr uint32_t T = NT * ITEMS;
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t tid = threadIdx.x;
    const int bits = a.bits;
    const uint32_t P = 1u << bits, mask = P - 1;
    E *stage = reinterpret_cast<E *>(smem);                                   // [T]
    uint32_t *scan_tmp = reinterpret_cast<uint32_t *>(smem + kSingleStage);   // [32]
    uint32_t *cnt = scan_tmp + 32;                                            // [P] elements of the tile
    uint32_t *tst = cnt + P;                                                  // [P] start in the tile
    uint32_t *gofs = tst + P;                                                 // [P] place - staged index
    uint32_t *place = gofs + P;                                               // [P] next place in the output
    const uint32_t n = (uint32_t)(rel ? a.nS : a.nR);
    O *out;
    if constexpr (sizeof(O) == 8)
        out = rel ? a.outS8 : a.outR8;
    else
        out = rel ? a.outS : a.outR;
    const bool z0 = a.z0 && rel == 0;
    uint64_t lo, hi;
    single_range(rel ? a.nS : a.nR, blk, G, &lo, &hi);
    const tuple_v *in = (rel ? a.S : a.R) + lo;
    const uint32_t len = (uint32_t)(hi - lo);
    if (len == 0) return;
    tuple_v t[ITEMS];
    uint32_t base = (len - 1) / T * T;
#pragma unroll
    for (int q = 0; q < ITEMS; q++) t[q] = base + q * NT + tid < len ? ld_stream(in + base + q * NT + tid) : make_ulonglong2(0, 0);
    {
        const uint32_t *pre = a.hist + ((size_t)rel * G + blk) * P;
        const uint64_t *start = a.start + (size_t)rel * (P + 1);
        for (uint32_t j = tid; j < P; j += NT) {
            place[j] = (uint32_t)start[j] + pre[j];
            cnt[j] = 0;
        }
    }
    __syncthreads();
    for (;;) {
        const uint32_t m = len - base < T ? len - base : T;
        E v[ITEMS];
        uint32_t rk[ITEMS / 2];  // ranks, two 16-bit ones per word
#pragma unroll
        for (int q = 0; q < ITEMS; q++) {
            if (MIX) t[q].x = mix_key(t[q].x, bits);
            v[q] = Elem::stage(t[q], lo + base + q * NT + tid, bits, mask, z0);
            uint32_t r = 0;
            if (q * NT + tid < m) r = atomicAdd(&cnt[Elem::digit(v[q], mask)], 1u);
            rk[q / 2] = (q & 1) ? rk[q / 2] | (r << 16) : r;
        }
        __syncthreads();
        {
            const uint32_t per = (P + NT - 1) / NT;  // this thread's digits: [tid * per, tid * per + per)
            uint32_t cq[D], sum = 0;
#pragma unroll
            for (int q = 0; q < D; q++) {
                cq[q] = q < per && tid * per + q < P ? cnt[tid * per + q] : 0u;
                sum += cq[q];
            }
            uint32_t ex = place_scan(sum, scan_tmp);
#pragma unroll
            for (int q = 0; q < D; q++) {
                if (q < per && tid * per + q < P) {
                    const uint32_t pl = place[tid * per + q];
                    cnt[tid * per + q] = 0;
                    tst[tid * per + q] = ex;
                    gofs[tid * per + q] = pl - ex;
                    place[tid * per + q] = pl + cq[q];
                    ex += cq[q];
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < ITEMS; q++)
            if (q * NT + tid < m)
                stage[tst[Elem::digit(v[q], mask)] + ((q & 1) ? rk[q / 2] >> 16 : rk[q / 2] & 0xffffu)] = v[q];
        const bool more = base != 0;
        if (more) {  // the next tile's loads pass under the write-out
            base -= T;
#pragma unroll
            for (int q = 0; q < ITEMS; q++) t[q] = ld_stream(in + base + q * NT + tid);
        }
        __syncthreads();
#pragma unroll 4
        for (uint32_t j = tid; j < m; j += NT) {
            const E e = stage[j];
            const uint32_t dst = gofs[Elem::digit(e, mask)] + j;
            if (dst < n)
                out[dst] = Elem::out(e, bits);
            else
                set_error(&a.counters[kCtrErr], kErrBounds);
        }
        if (!more) break;
    }
    __syncthreads();
}

template <bool MULTI, bool MIX>
__global__ void __launch_bounds__(kPlaceThreads, 1) single_scatter(SingleArgs a0, MultiRef mr) {
    __shared__ SingleArgs s_a;
    uint32_t blk = blockIdx.x, G = gridDim.x;
    if (MULTI) {
        const uint2 e = mr.map[blockIdx.x];
        multi_copy(&s_a, &mr.jobs[e.x].sa);
        blk = e.y;
        G = mr.jobs[e.x].grid;
        __syncthreads();
    }
    const SingleArgs &a = MULTI ? s_a : a0;
    const bool ci = a.ci_ok && ci_applies(a.counters, a.bits);
    const bool narrow = ci && *reinterpret_cast<const unsigned long long *>(a.counters + kCtrMaxKey) < (1ull << 31);
    // S, then R; one instantiation per mode serves both.
    for (int rel = 1; rel >= 0; rel--) {
        if (rel == 0 && a.lp) {
            if (ci)
                single_scatter_rel<kModePosWord, MIX>(a, rel, blk, G);
            else
                single_scatter_rel<kModePos, MIX>(a, rel, blk, G);
        } else if (narrow) {
            single_scatter_rel<kModeWord, MIX>(a, rel, blk, G);
        } else if (ci) {
            single_scatter_rel<kModeTupleWord, MIX>(a, rel, blk, G);
        } else {
            single_scatter_rel<kModeTuple, MIX>(a, rel, blk, G);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
// Histograms per CTA of the count (32 KB of them) for 2^bits digits.
constexpr size_t kCountSmem = 32768;
static int single_copies(int bits) {
    const uint32_t n = (uint32_t)(kCountSmem / 4) >> bits;
    return n < 1 ? 1 : n < 32 ? (int)n : 32;
}

uint32_t single_grid(size_t nR, size_t nS, int num_sms) {
    const uint64_t sms = (uint64_t)(num_sms > 0 ? num_sms : 148);
    const uint64_t want = ((uint64_t)nR + nS + 4095) / 4096;
    return (uint32_t)(want < 1 ? 1 : want < sms ? want : sms);
}

#define HJ_CU(call)                                                                   \
    do {                                                                              \
        cudaError_t e_ = (call);                                                      \
        if (e_ != cudaSuccess) {                                                      \
            fprintf(stderr, "hjscm: %s failed: %s\n", #call, cudaGetErrorString(e_)); \
            return HJ_E_DEVICE;                                                       \
        }                                                                             \
    } while (0)

int single_prepare_device() {
    const int most = (int)single_scatter_smem(kSingleMaxBits);
    HJ_CU(cudaFuncSetAttribute(single_scatter<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    HJ_CU(cudaFuncSetAttribute(single_scatter<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    HJ_CU(cudaFuncSetAttribute(single_scatter<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    return HJ_OK;
}

void single_args(const RadixGeom &g, bool lp, bool skip0, bool ci_ok, const ulonglong2 *R, size_t nR,
                 const ulonglong2 *S, size_t nS, const PhjScratch &s, JoinAccum *acc, bool clear_acc, bool agg_ok,
                 SingleArgs *out, PlanArgs *pout) {
    const uint32_t P = 1u << g.bits;
    SingleArgs &a = *out;
    a = SingleArgs{};
    a.R = R;
    a.S = S;
    a.nR = nR;
    a.nS = nS;
    a.bits = g.bits;
    a.copies = single_copies(g.bits);
    a.hist = s.chunk_hist;
    a.ors = s.ors;
    a.start = s.start;
    a.counters = s.counters;
    a.acc = acc;
    a.clear_acc = clear_acc ? 1 : 0;
    a.ci_ok = ci_ok ? 1 : 0;
    a.lp = lp ? 1 : 0;
    a.z0 = skip0 ? 1 : 0;
    a.outR = s.tmp1;
    a.outS = s.tmp1 + nR;
    a.outR8 = reinterpret_cast<unsigned long long *>(s.tmp1);
    a.outS8 = single_probe_words(s, nR, lp);
    PlanArgs &pa = *pout;
    pa = PlanArgs{};
    pa.bits = g.bits;
    pa.passes = 1;
    pa.b1 = g.bits;
    pa.F1 = (int)P;
    pa.F2 = 1;
    pa.nR = nR;
    pa.nS = nS;
    pa.total = s.total;
    pa.start = s.start;
    pa.counters = s.counters;
    pa.items = reinterpret_cast<JoinItem *>(s.items);
    pa.max_items = s.max_items;
    pa.large = reinterpret_cast<LargePart *>(s.large);
    pa.max_large = s.max_large;
    pa.large_table_words = s.large_table_words;
    pa.small_cap = lp ? kFirstCap : kSmemCap;
    pa.agg_ok = agg_ok ? 1 : 0;
}

int single_partition_enqueue(const RadixGeom &g, bool lp, bool skip0, bool ci_ok, const ulonglong2 *R, size_t nR,
                             const ulonglong2 *S, size_t nS, const PhjScratch &s, JoinAccum *acc, bool clear_acc,
                             cudaStream_t st, bool agg_ok, cudaEvent_t *ph, uint32_t *launches) {
    const uint32_t P = 1u << g.bits, G = s.cR;
    SingleArgs a;
    PlanArgs pa;
    single_args(g, lp, skip0, ci_ok, R, nR, S, nS, s, acc, clear_acc, agg_ok, &a, &pa);
    const MultiRef none = {};
    if (g.mix)
        single_count<false, true><<<G, kCountThreads, (size_t)a.copies * P * 4, st>>>(a, none);
    else
        single_count<false, false><<<G, kCountThreads, (size_t)a.copies * P * 4, st>>>(a, none);
    if (ph) HJ_CU(record_event(ph[1], st));
    single_plan<false><<<(2 * P + 31) / 32, 1024, (size_t)2 * P * 4, st>>>(a, pa, G, none);
    if (ph) HJ_CU(record_event(ph[2], st));
    if (g.mix)
        single_scatter<false, true><<<G, kPlaceThreads, single_scatter_smem(g.bits), st>>>(a, none);
    else
        single_scatter<false, false><<<G, kPlaceThreads, single_scatter_smem(g.bits), st>>>(a, none);
    HJ_CU(cudaGetLastError());
    if (ph) {
        HJ_CU(record_event(ph[3], st));
        HJ_CU(record_event(ph[4], st));
    }
    *launches += 3;
    return HJ_OK;
}

int multi_partition_launch(const MultiJob *jobs, const uint2 *part_map, unsigned part_blocks, const uint2 *plan_map,
                           unsigned plan_blocks, int max_bits, cudaStream_t st, uint32_t *launches) {
    const SingleArgs none_a = {};
    const PlanArgs none_p = {};
    const MultiRef part = {jobs, part_map}, plan = {jobs, plan_map};
    single_count<true, true><<<part_blocks, kCountThreads, kCountSmem, st>>>(none_a, part);
    single_plan<true><<<plan_blocks, 1024, (size_t)8 << max_bits, st>>>(none_a, none_p, 0, plan);
    single_scatter<true, true><<<part_blocks, kPlaceThreads, single_scatter_smem(max_bits), st>>>(none_a, part);
    HJ_CU(cudaGetLastError());
    *launches += 3;
    return HJ_OK;
}

}  // namespace hj
