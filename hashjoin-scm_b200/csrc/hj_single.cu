// hj_single.cu - the one-pass partition phase of radix joins whose build relation needs at most 2^12
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
// The partitions are those of `bits` low key bits, so the join kernels are the two-pass pipelines'.
//
// Elements: compact words ci_word (8 bytes) when the widths allow them, else tuples. First-match joins
// need the lowest input position among equal build keys; their build elements are 16 bytes, {ci_word,
// position} or {key, position}, so the order inside a partition does not matter and no pass is ordered.
#include <cstdio>

#include "hj_common.cuh"
#include "hj_internal.h"
#include "hj_partition.cuh"

namespace hj {

constexpr int kCountThreads = 1024, kSingleThreads = 512;
// Scatter: one CTA per SM, 512 threads that place tuples and one warp that loads them.
constexpr int kScatThreads = kSingleThreads + 32;
constexpr int kRingChunk = 1024, kRingChunks = 4;  // input ring: chunks of 1024 tuples (16 KB)
constexpr int kTileChunks = 12;                    // a tile of words: 12 chunks; of 16-byte elements: 6
constexpr int kSingleWordItems = kTileChunks * kRingChunk / kSingleThreads, kSingleTupleItems = kSingleWordItems / 2;
constexpr int kSingleDigitsPerThread = ((1 << kSingleMaxBits) + kSingleThreads - 1) / kSingleThreads;

// CTA c's contiguous range of n tuples (a multiple of 8 tuples, one 128-byte line).
__device__ __forceinline__ void single_range(uint64_t n, uint64_t *lo, uint64_t *hi) {
    const uint64_t per = ((n + gridDim.x - 1) / gridDim.x + 7) & ~7ull;
    *lo = blockIdx.x * per < n ? blockIdx.x * per : n;
    *hi = *lo + per < n ? *lo + per : n;
}

// Shared memory of the scatter: a staged tile with its digits, and four words per digit.
constexpr size_t kSingleStage = (size_t)kSingleThreads * kSingleWordItems * 8;
static_assert(kSingleStage == (size_t)kSingleThreads * kSingleTupleItems * 16, "one staging area for both layouts");
inline size_t single_scatter_smem(int bits) {
    return (size_t)kRingChunks * kRingChunk * 16 + kSingleStage + (size_t)kSingleThreads * kSingleWordItems * 2 +
           ((size_t)4 << bits) * 4;
}

// Input tuple of the count: read again by the scatter, so its line keeps the normal L2 priority.
__device__ __forceinline__ tuple_v ld_twice(const tuple_v *p) {
    tuple_v v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

struct SingleArgs {
    const tuple_v *R, *S;
    uint64_t nR, nS;
    int bits;                // P = 2^bits partitions
    int copies;              // count: histograms per CTA (its warps spread over them)
    uint32_t *hist;          // [2][G][P]: rows of R, rows of S; exclusive prefixes after single_plan
    unsigned long long *ors; // [G][3]: ORs of build keys, build row ids, probe row ids
    const uint64_t *start;   // [2][P + 1]
    uint32_t *counters;
    int ci_ok;               // compact words allowed
    int lp;                  // first match: build elements carry their input position
    int z0;                  // build key 0 never matches
    tuple_v *outR, *outS;    // tuples
    unsigned long long *outR8, *outS8;  // compact words
};

// ------------------------------------------------------------------------------------------------
// 1. Count. Bound by reading the relations (four 16-byte loads per thread in flight, 1024 threads per SM);
//    the shared-memory increments return nothing. With few partitions the warps spread over `copies`
//    histograms, since 32 lanes on a handful of counters serialise.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kCountThreads, 1) single_count(SingleArgs a) {
    extern __shared__ uint32_t sh[];  // [copies][P]
    const int tid = threadIdx.x;
    const uint32_t P = 1u << a.bits, mask = P - 1;
    uint32_t *mine = sh + (size_t)((uint32_t)(tid >> 5) % (uint32_t)a.copies) * P;
    __shared__ unsigned long long s_or[3];
    if (tid < 3) s_or[tid] = 0;
    for (int rel = 0; rel < 2; rel++) {
        for (uint32_t j = tid; j < P * a.copies; j += kCountThreads) sh[j] = 0;
        __syncthreads();
        const tuple_v *in = rel ? a.S : a.R;
        uint64_t lo, hi;
        single_range(rel ? a.nS : a.nR, &lo, &hi);
        unsigned long long kor = 0, ror = 0;
        constexpr int U = 4;
        uint64_t i = lo + tid;
        for (; i + (U - 1) * kCountThreads < hi; i += U * kCountThreads) {
            tuple_v t[U];
#pragma unroll
            for (int u = 0; u < U; u++) t[u] = ld_twice(in + i + u * kCountThreads);
#pragma unroll
            for (int u = 0; u < U; u++) {
                atomicAdd(&mine[(uint32_t)t[u].x & mask], 1u);
                kor |= t[u].x;
                ror |= t[u].y;
            }
        }
        for (; i < hi; i += kCountThreads) {
            const tuple_v t = ld_twice(in + i);
            atomicAdd(&mine[(uint32_t)t.x & mask], 1u);
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
        uint32_t *row = a.hist + ((size_t)rel * gridDim.x + blockIdx.x) * P;
        for (uint32_t j = tid; j < P; j += kCountThreads) {
            uint32_t n = 0;
            for (int c = 0; c < a.copies; c++) n += sh[(size_t)c * P + j];
            row[j] = n;
        }
        __syncthreads();
    }
    if (tid < 3) a.ors[(size_t)blockIdx.x * 3 + tid] = s_or[tid];
}

// ------------------------------------------------------------------------------------------------
// 2. Prefixes and plan. A CTA takes 32 columns (digits of one relation; consecutive lanes read
//    consecutive digits of a row), its 32 warps share the rows. The CTA that finishes last plans.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024, 1) single_plan(SingleArgs a, uint32_t G, uint32_t *total, PlanArgs pa) {
    __shared__ uint32_t part[32][33];
    __shared__ uint32_t tmp[32];
    __shared__ uint64_t s_run[2];
    __shared__ bool s_last;
    extern __shared__ uint32_t sm_tot[];  // [2][P]
    const uint32_t P = 1u << a.bits;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t col = blockIdx.x * 32 + lane;
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
    if (threadIdx.x == 0) s_last = atomicAdd(&a.counters[kCtrTicket], 1u) == gridDim.x - 1;
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
// 3. Scatter. One CTA per SM with the largest tile that fits (12288 words or 6144 16-byte elements): what a
//    run of a digit costs in L2 does not depend on its length (about 35 G runs per second here, whatever
//    the tile), so the runs N * P / tile have to be few. A producer warp keeps a ring of bulk copies in
//    flight through all phases of a tile; per tile the 512 placing threads take the elements' ranks within
//    their digit from shared-memory atomics, a block scan over the digits gives each digit's start in the
//    tile, and the tile is staged in digit order and written out, consecutive threads to consecutive places
//    of a digit's run. A CTA's elements of a digit go to its own consecutive places, so the next place of
//    every digit is a counter in shared memory.
// ------------------------------------------------------------------------------------------------
// KIND 0: tuples, 1: compact words, 2: {word or key, position} of first-match builds.
template <int KIND>
struct SingleElem {
    using type = tuple_v;
};
template <>
struct SingleElem<1> {
    using type = unsigned long long;
};

template <int KIND>
__device__ __forceinline__ typename SingleElem<KIND>::type single_elem(const tuple_v &t, uint64_t i, bool ci, int bits,
                                                                       bool z0) {
    if constexpr (KIND == 0)
        return t;
    else if constexpr (KIND == 1)
        return ci_word_z0(t.x, t.y, bits, z0);
    else
        return make_ulonglong2(ci ? ci_word_z0(t.x, t.y, bits, z0) : t.x, i);
}

// Barrier of the placing threads (the producer warp takes no part).
__device__ __forceinline__ void place_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kSingleThreads) : "memory"); }

// Exclusive scan of one u32 per placing thread.
__device__ __forceinline__ uint32_t place_scan(uint32_t v, uint32_t *tmp) {
    const unsigned lane = lane_id(), w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) tmp[w] = x;
    place_sync();
    uint32_t before = 0;  // every warp sums the totals of the warps before it
    uint32_t tot = lane < (unsigned)(kSingleThreads / 32) ? tmp[lane] : 0u;
    before = __reduce_add_sync(0xffffffffu, lane < w ? tot : 0u);
    return before + x - v;
}

struct SingleShared {
    unsigned long long full[kRingChunks], empty[kRingChunks];
    uint32_t scan_tmp[32];
    uint32_t stop;  // a placing thread's bounded wait expired (written before a barrier of theirs only)
};

// The order in which a CTA reads its ranges: S before R, each from its last tile to its first, a tile's
// chunks in order. Producer and placing threads walk it alike.
template <class F>
__device__ __forceinline__ bool single_walk(uint32_t len, uint32_t tile, F &&f) {
    for (uint32_t k = (len + tile - 1) / tile; k > 0; k--)
        if (!f((k - 1) * tile, len - (k - 1) * tile < tile ? len - (k - 1) * tile : tile)) return false;
    return true;
}

__device__ __forceinline__ void single_produce(const SingleArgs &a, uint32_t tile_r, uint32_t tile_s, tuple_v *ring,
                                               SingleShared &sh) {
    uint32_t c = 0;  // chunks issued
    bool ok = true;
    for (int rel = 1; rel >= 0 && ok; rel--) {
        uint64_t lo, hi;
        single_range(rel ? a.nS : a.nR, &lo, &hi);
        const tuple_v *in = (rel ? a.S : a.R) + lo;
        ok = single_walk((uint32_t)(hi - lo), rel ? tile_s : tile_r, [&](uint32_t base, uint32_t m) {
            for (uint32_t o = 0; o < m; o += kRingChunk, c++) {
                const uint32_t slot = c % kRingChunks;
                if (c >= kRingChunks && !mbar_wait(smem_addr(&sh.empty[slot]), (c / kRingChunks - 1) & 1u)) return false;
                if (*reinterpret_cast<volatile uint32_t *>(&sh.stop)) return false;
                const uint32_t cnt = m - o < (uint32_t)kRingChunk ? m - o : (uint32_t)kRingChunk;
                tma_load_1d(ring + (size_t)slot * kRingChunk, in + base + o, cnt * 16u, smem_addr(&sh.full[slot]));
            }
            return true;
        });
    }
    if (!ok) set_error(&a.counters[kCtrErr], kErrSpinLimit);
    // Let what is in flight land (bounded) before the CTA may give up its shared memory.
    for (uint32_t q = c > (uint32_t)kRingChunks ? c - kRingChunks : 0u; q < c; q++)
        mbar_wait(smem_addr(&sh.full[q % kRingChunks]), (q / kRingChunks) & 1u);
}

// Place one relation's range; c counts the ring chunks taken so far. False: a wait expired.
template <int KIND>
__device__ __forceinline__ bool single_scatter_rel(const SingleArgs &a, bool ci, int rel, unsigned char *smem,
                                                   SingleShared &sh, uint32_t &c) {
    using E = typename SingleElem<KIND>::type;
    constexpr int NT = kSingleThreads, ITEMS = KIND == 1 ? kSingleWordItems : kSingleTupleItems;
    constexpr int PC = kRingChunk / NT;  // tuples of a chunk per thread
    constexpr uint32_t T = NT * ITEMS;
    constexpr int D = kSingleDigitsPerThread;
    const int tid = threadIdx.x;
    const uint32_t P = 1u << a.bits, mask = P - 1;
    unsigned int *err = &a.counters[kCtrErr];
    const tuple_v *ring = reinterpret_cast<const tuple_v *>(smem);                     // [kRingChunks][kRingChunk]
    E *stage = reinterpret_cast<E *>(smem + (size_t)kRingChunks * kRingChunk * 16);    // [T]
    uint16_t *dig = reinterpret_cast<uint16_t *>(smem + (size_t)kRingChunks * kRingChunk * 16 + kSingleStage);  // [T]
    uint32_t *cnt = reinterpret_cast<uint32_t *>(dig + NT * kSingleWordItems);         // [P] elements of the tile
    uint32_t *tst = cnt + P;                                                           // [P] start in the tile
    uint32_t *gofs = tst + P;                                                          // [P] place - staged index
    uint32_t *place = gofs + P;                                                        // [P] next place in the output
    const uint64_t n = rel ? a.nS : a.nR;
    const uint32_t *pre = a.hist + ((size_t)rel * gridDim.x + blockIdx.x) * P;
    const uint64_t *start = a.start + (size_t)rel * (P + 1);
    const uint32_t per = (P + NT - 1) / NT;  // this thread's digits in the scan: [tid * per, tid * per + per)
    for (uint32_t j = tid; j < P; j += NT) {
        place[j] = (uint32_t)start[j] + pre[j];
        cnt[j] = 0;
    }
    E *out;
    if constexpr (KIND == 1)
        out = rel ? a.outS8 : a.outR8;
    else
        out = rel ? a.outS : a.outR;
    const bool z0 = a.z0 && rel == 0;
    uint64_t lo, hi;
    single_range(n, &lo, &hi);
    place_sync();
    return single_walk((uint32_t)(hi - lo), T, [&](uint32_t base, uint32_t m) {
        E v[ITEMS];
        uint32_t dr[ITEMS];  // digit << 16 | rank
#pragma unroll
        for (int ch = 0; ch < ITEMS / PC; ch++) {
            if ((uint32_t)(ch * kRingChunk) < m) {
                const uint32_t slot = c % kRingChunks;
                if (!mbar_wait(smem_addr(&sh.full[slot]), (c / kRingChunks) & 1u)) {
                    set_error(err, kErrSpinLimit);
                    *reinterpret_cast<volatile uint32_t *>(&sh.stop) = 1u;
                }
                tuple_v t[PC];
#pragma unroll
                for (int u = 0; u < PC; u++) t[u] = ring[(size_t)slot * kRingChunk + u * NT + tid];
                __syncwarp();
                if ((tid & 31) == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&sh.empty[slot])) : "memory");
                c++;
#pragma unroll
                for (int u = 0; u < PC; u++) {
                    const uint32_t i = ch * kRingChunk + u * NT + tid;
                    const uint32_t d = (uint32_t)t[u].x & mask;
                    v[ch * PC + u] = single_elem<KIND>(t[u], lo + base + i, ci, a.bits, z0);
                    dr[ch * PC + u] = i < m ? (d << 16) | atomicAdd(&cnt[d], 1u) : 0xffffffffu;
                }
            } else {
#pragma unroll
                for (int u = 0; u < PC; u++) dr[ch * PC + u] = 0xffffffffu;
            }
        }
        place_sync();
        if (*reinterpret_cast<volatile uint32_t *>(&sh.stop)) return false;  // the same for every thread
        uint32_t cq[D], sum = 0;
#pragma unroll
        for (int q = 0; q < D; q++) {
            cq[q] = q < per && tid * per + q < P ? cnt[tid * per + q] : 0u;
            sum += cq[q];
        }
        uint32_t ex = place_scan(sum, sh.scan_tmp);
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
        place_sync();
#pragma unroll
        for (int q = 0; q < ITEMS; q++) {
            if (dr[q] == 0xffffffffu) continue;
            const uint32_t d = dr[q] >> 16, p = tst[d] + (dr[q] & 0xffffu);
            stage[p] = v[q];
            dig[p] = (uint16_t)d;
        }
        place_sync();
#pragma unroll 4
        for (uint32_t j = tid; j < m; j += NT) {
            const uint32_t dst = gofs[dig[j]] + j;
            if (dst < n)
                out[dst] = stage[j];
            else
                set_error(err, kErrBounds);
        }
        return true;
    });
}

__global__ void __launch_bounds__(kScatThreads, 1) single_scatter(SingleArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ SingleShared sh;
    const bool ci = a.ci_ok && ci_applies(a.counters, a.bits);
    if (threadIdx.x == 0) {
        for (int q = 0; q < kRingChunks; q++) {
            mbar_init(smem_addr(&sh.full[q]), 1);
            mbar_init(smem_addr(&sh.empty[q]), kSingleThreads / 32);
        }
        sh.stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    constexpr uint32_t kWordTile = kSingleThreads * kSingleWordItems, kTupleTile = kSingleThreads * kSingleTupleItems;
    if (threadIdx.x >= kSingleThreads) {
        if (threadIdx.x == kSingleThreads)
            single_produce(a, ci && !a.lp ? kWordTile : kTupleTile, ci ? kWordTile : kTupleTile,
                           reinterpret_cast<tuple_v *>(smem), sh);
        return;
    }
    uint32_t c = 0;
    bool ok;
    if (ci)
        ok = single_scatter_rel<1>(a, true, 1, smem, sh, c);
    else
        ok = single_scatter_rel<0>(a, false, 1, smem, sh, c);
    if (!ok) return;
    place_sync();
    if (a.lp)
        single_scatter_rel<2>(a, ci, 0, smem, sh, c);
    else if (ci)
        single_scatter_rel<1>(a, true, 0, smem, sh, c);
    else
        single_scatter_rel<0>(a, false, 0, smem, sh, c);
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
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
    HJ_CU(cudaFuncSetAttribute(single_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)single_scatter_smem(kSingleMaxBits)));
    return HJ_OK;
}

int single_partition_enqueue(const RadixGeom &g, bool lp, bool skip0, bool ci_ok, const ulonglong2 *R, size_t nR,
                             const ulonglong2 *S, size_t nS, const PhjScratch &s, cudaStream_t st, bool agg_ok,
                             cudaEvent_t *ph, uint32_t *launches) {
    const uint32_t P = 1u << g.bits;
    SingleArgs a;
    a.R = R;
    a.S = S;
    a.nR = nR;
    a.nS = nS;
    a.bits = g.bits;
    a.copies = P >= 8192 ? 1 : (int)(8192u / P < 32u ? 8192u / P : 32u);
    a.hist = s.chunk_hist;
    a.ors = s.ors;
    a.start = s.start;
    a.counters = s.counters;
    a.ci_ok = ci_ok ? 1 : 0;
    a.lp = lp ? 1 : 0;
    a.z0 = skip0 ? 1 : 0;
    a.outR = s.tmp1;
    a.outS = s.tmp1 + nR;
    a.outR8 = reinterpret_cast<unsigned long long *>(s.tmp1);
    a.outS8 = single_probe_words(s, nR, lp);
    const uint32_t G = s.cR;
    PlanArgs pa;
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
    single_count<<<G, kCountThreads, (size_t)a.copies * P * 4, st>>>(a);
    if (ph) HJ_CU(record_event(ph[1], st));
    single_plan<<<(2 * P + 31) / 32, 1024, (size_t)2 * P * 4, st>>>(a, G, s.total, pa);
    if (ph) HJ_CU(record_event(ph[2], st));
    single_scatter<<<G, kScatThreads, single_scatter_smem(g.bits), st>>>(a);
    HJ_CU(cudaGetLastError());
    if (ph) {
        HJ_CU(record_event(ph[3], st));
        HJ_CU(record_event(ph[4], st));
    }
    *launches += 3;
    return HJ_OK;
}

}  // namespace hj
