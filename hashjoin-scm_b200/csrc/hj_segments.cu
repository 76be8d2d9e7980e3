// hj_segments.cu - pass 1 of the two-pass radix pipeline's segment mode (hj_partition.cu has the rest of it). A
// translation unit of its own: its two dozen kernel forms are loaded when a join first runs it.
#include <cstdio>

#include "hj_common.cuh"
#include "hj_internal.h"
#include "hj_partition.cuh"

namespace hj {

// ------------------------------------------------------------------------------------------------
// Segment mode, pass 1: partition into chains of segments, counting the histograms on the way.
//
// The exact-offset pipeline reads both relations once for histograms before pass 1 may write. For
// the joins that count every match, the order of tuples within a partition does not matter, and
// pass 1 can write without knowing offsets: every (CTA, relation, pass-1 digit) owns a chain of
// kTile-tuple segments, taken from a global counter (in slabs of kSegSlab per CTA), filled in order
// and linked through seg_next. Since a tile holds at most kTile tuples of one digit, a tile's run of
// a digit ends the current segment at most once. The same CTA counts the joint histogram of the low
// `bits` key bits of its tuples in 16-bit counters (two per word), and adds them to its row of hist
// when the relation ends. No counter overflows: `since` bounds every counter (a tile adds at most its
// size), and before a tile could take the bound past 65535 the CTA moves every counter above
// kSegSpillAt into its row and sets the bound to the largest counter left. That gives pass 2 its exact
// offsets: pass 2 takes (CTA, digit) chains as its units and writes the final partitions as in the
// exact-offset pipeline.
// ------------------------------------------------------------------------------------------------
constexpr uint32_t kSegNone = 0xffffffffu;
constexpr uint32_t kSegSpillAt = 8192;
constexpr uint32_t kSegEndItems = 0x40000000;  // more than the work items of any relation (2^32 / kTile each)

struct SegArgs {
    const tuple_v *R, *S;
    uint64_t nR, nS;
    int bits, F1;              // joint bins 2^bits; pass-1 digit = key & (F1 - 1)
    int b1;                    // log2(F1)
    int w8_first;              // a pass that wrote 8-byte words ran first: run only if w8_fits fails
    uint32_t it_tiles;         // tiles per work item
    uint32_t tilesR, tilesS;   // tiles of each relation
    uint32_t itemsR, items;    // items of R (first), all items
    tuple_v *out;              // segment storage: segment i holds tuples [i*kTile, (i+1)*kTile)
    uint32_t max_segs;
    uint32_t *seg_head;        // [2*grid][F1]
    uint32_t *seg_next;        // [max_segs]
    uint32_t *hist;            // [2*grid][2^bits]: row c = R tuples of CTA c, row grid + c = its S tuples
    uint32_t *counters;        // kCtrItem1 (items), kCtrSegAlloc, kCtrErr, kCtrMaxKey/kCtrMaxRid
    int test_stall;            // test hook: CTA 0 withholds its first tile load (its wait must expire)
};

struct SegSlot {
    const tuple_v *in;
    uint32_t cnt;              // tuples in the tile (0: no more tiles)
    int rel;
};

// Where a digit's run of the staged tile goes: staged index j < split to base + j - kTile (the rest of the
// current segment), j >= split to base2 + j - kTile (the new segment). 40-bit bases, biased so that they are
// not negative, in one 16-byte load; kSegNowhere fails the bounds check of the store.
constexpr unsigned long long kSegNowhere = (1ull << 40) - 1;
struct __align__(16) SegRun {
    uint32_t base_lo, base2_lo, split_hi, pad;  // split_hi: split | base >> 32 << 16 | base2 >> 32 << 24
};
__device__ __forceinline__ SegRun seg_run(unsigned long long base, unsigned long long base2, uint32_t split) {
    SegRun r;
    r.base_lo = (uint32_t)base;
    r.base2_lo = (uint32_t)base2;
    r.split_hi = split | (uint32_t)(base >> 32) << 16 | (uint32_t)(base2 >> 32) << 24;
    r.pad = 0;
    return r;
}
__device__ __forceinline__ unsigned long long seg_dst(const SegRun *run, uint32_t j) {
    const uint4 r = *reinterpret_cast<const uint4 *>(run);
    const bool first = j < (r.z & 0xffffu);
    const unsigned long long base =
        ((unsigned long long)(first ? (r.z >> 16) & 0xffu : r.z >> 24) << 32) | (first ? r.x : r.y);
    return base + j - kTile;
}

// Thread 0: the next tile of this CTA's current work item, claiming items as needed. STATIC_R: the build
// relation's items [r_next, r_end) belong to this CTA and come first, in order; the probe relation's
// items are claimed from the counter.
template <bool STATIC_R>
__device__ __forceinline__ SegSlot seg_next_tile(const SegArgs &a, uint32_t &item, uint32_t &t_next,
                                                 uint32_t &t_end, uint32_t &r_next, uint32_t r_end) {
    SegSlot s;
    while (item == ~0u || t_next >= t_end) {
        if (STATIC_R && r_next < r_end && !*reinterpret_cast<volatile uint32_t *>(&a.counters[kCtrSegWide]))
            item = r_next++;
        else
            item = atomicAdd(&a.counters[kCtrItem1], 1u) + (STATIC_R ? a.itemsR : 0u);
        if (item >= a.items) {
            item = ~0u;
            s.in = nullptr;
            s.cnt = 0;
            s.rel = 0;
            return s;
        }
        const bool rel = item >= a.itemsR;
        const uint32_t k = rel ? item - a.itemsR : item;
        const uint32_t nt = rel ? a.tilesS : a.tilesR;
        t_next = k * a.it_tiles;
        t_end = t_next + a.it_tiles < nt ? t_next + a.it_tiles : nt;
    }
    const bool rel = item >= a.itemsR;
    const uint64_t n = rel ? a.nS : a.nR;
    const uint64_t lo = (uint64_t)t_next * kTile;
    s.in = (rel ? a.S : a.R) + lo;
    s.cnt = (uint32_t)(n - lo < (uint64_t)kTile ? n - lo : (uint64_t)kTile);
    s.rel = rel ? 1 : 0;
    t_next++;
    return s;
}

// Add the CTA's 16-bit counter pairs to its histogram row (reductions: no round trip) and clear them.
// All threads; the caller synchronises before and after.
__device__ __forceinline__ void seg_flush(uint32_t *jh, uint32_t *row, int nbins) {
    for (int w = threadIdx.x; w < (nbins >> 1); w += blockDim.x) {
        const uint32_t v = jh[w];
        if (!v) continue;
        jh[w] = 0;
        if (v & 0xffffu) atomicAdd(&row[2 * w], v & 0xffffu);
        if (v >> 16) atomicAdd(&row[2 * w + 1], v >> 16);
    }
}

// K = ceil(F1 / 32): pass-1 digits per lane of warp 0, which keeps their segment state in registers.
// W8: store 8-byte words (w8_word) in segments of 2 * kTile words (the same 32 KB); the launch that stores
// tuples after it runs only when the widths did not allow words (w8_first).
// STABLE_R (first-match joins): every build-relation chain keeps input order. CTA c takes the build
// relation's items [c * itemsR / G, (c + 1) * itemsR / G) in order before any probe item, and ranks
// their tiles stably (warp-ordered ballots, as the stable scatter does), so pass 2, which writes each
// digit's chains in CTA order and each chain in order, leaves every final build partition in input
// order. Probe tiles keep the atomic rank: their order inside a partition changes no result.
// Build key 0 of first-match joins needs nothing here: its word (high part 0) reaches key 0's final
// partition, whose joins skip it (JoinItem::part0); a select per word cost pass 1 3%.
// MIX: partition by mix_key, and store it in place of the key.
template <int THREADS, int ITEMS, int K, bool W8 = false, bool STABLE_R = false, bool MIX = false>
__global__ void __launch_bounds__(THREADS, kSegCtasPerSm) seg_pass1_kernel(SegArgs a) {
    constexpr int T = THREADS * ITEMS;
    static_assert(T == kTile, "a tile fills one segment of tuples");
    constexpr uint32_t SEGW = W8 ? 2 * T : T;  // elements per segment
    if (!W8 && a.w8_first && w8_fits(a.counters, a.b1)) return;
    unsigned long long *out8 = reinterpret_cast<unsigned long long *>(a.out);
    static_assert(K >= 1 && K <= 8, "at most 256 pass-1 digits");
    extern __shared__ __align__(128) unsigned char smem[];
    tuple_v *inbuf = reinterpret_cast<tuple_v *>(smem);              // [2][T]
    SegRun *runs = reinterpret_cast<SegRun *>(inbuf + 2 * T);          // [256] where each digit's run goes
    uint32_t *thist = reinterpret_cast<uint32_t *>(runs + 256);        // [256] tile histogram
    uint32_t *tdstart = thist + 256;                                   // [256] digit start in the staged tile
    uint32_t *jh = tdstart + 256;                                      // [2^bits / 2] counter pairs
    uint16_t *whist = reinterpret_cast<uint16_t *>(jh + (1 << a.bits) / 2);  // STABLE_R: [warps][F1]
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ SegSlot slots[2];
    __shared__ uint32_t s_item, s_tnext, s_tend, s_rnext, s_rend;  // thread 0's item iterator

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int F = a.F1;
    const uint32_t dmask = (uint32_t)F - 1u;
    const int nbins = 1 << a.bits;
    const uint64_t bmask = (uint64_t)nbins - 1;
    const uint32_t G = gridDim.x, c = blockIdx.x;
    unsigned int *err = &a.counters[kCtrErr];
    const uint32_t bar0 = smem_addr(&bars[0]);
    const uint64_t cap = (uint64_t)a.max_segs * SEGW;

    for (int j = tid; j < 256; j += THREADS) thist[j] = 0;
    for (int j = tid; j < (nbins >> 1); j += THREADS) jh[j] = 0;
    // Warp 0, lane l: current segment and fill of digits l*K .. l*K + K - 1.
    uint32_t scur[K], sfill[K];
#pragma unroll
    for (int j = 0; j < K; j++) {
        scur[j] = kSegNone;
        sfill[j] = 0;
    }
    // This CTA's rows of hist start at zero; counters are added to them.
    for (int j = tid; j < 2 * nbins; j += THREADS)
        a.hist[((size_t)(j >= nbins ? G : 0) + c) * nbins + (j >= nbins ? j - nbins : j)] = 0;
    uint32_t slab_lo = 0, slab_rem = 0;  // thread 0 (lane 0 of warp 0): ids left in this CTA's slab
    if (tid == 0) {
        s_item = ~0u;
        s_tnext = s_tend = 0;
        s_rnext = (uint32_t)((uint64_t)c * a.itemsR / G);
        s_rend = (uint32_t)((uint64_t)(c + 1) * a.itemsR / G);
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        uint32_t item = s_item, tn = s_tnext, te = s_tend, rn = s_rnext;
        const SegSlot s0 = seg_next_tile<STABLE_R>(a, item, tn, te, rn, s_rend);
        s_item = item;
        s_tnext = tn;
        s_tend = te;
        s_rnext = rn;
        slots[0] = s0;
        if (s0.cnt && !(a.test_stall && blockIdx.x == 0)) tma_load_1d(inbuf, s0.in, s0.cnt * 16u, bar0);
    }
    __syncthreads();

    int phase_rel = 0;           // relation whose tuples the counters and segment state hold
    uint32_t since = 0;          // upper bound of every counter (uniform)
    // ORs of the high 32 bits of build keys, build row ids and probe row ids: every width test
    // (w8_fits, ci_applies, compact_applies) compares with a power of two of 2^32 or more.
    uint32_t kor = 0, ror = 0, rors = 0;
    __shared__ uint32_t s_max[THREADS / 32];

    for (uint32_t k = 0;; k++) {
        const uint32_t cur = k & 1u;
        const SegSlot sl = slots[cur];
        if (sl.cnt == 0) break;
        tuple_v *buf = inbuf + (size_t)cur * T;
        // R tiles come before S tiles in every CTA's sequence: on the first S tile, R's counters go
        // to their row and the segment state starts over.
        if (sl.rel != phase_rel) {
            seg_flush(jh, a.hist + ((size_t)phase_rel * G + c) * nbins, nbins);
#pragma unroll
            for (int j = 0; j < K; j++) {
                scur[j] = kSegNone;
                sfill[j] = 0;
            }
            phase_rel = sl.rel;
            since = 0;
            __syncthreads();
        }
        const uint32_t cnt = sl.cnt;
        if (since + cnt > 65535u) {
            // Move the large counters to the row; the largest one kept is the new bound.
            uint32_t *hrow = a.hist + ((size_t)phase_rel * G + c) * nbins;
            uint32_t mx = 0;
            for (int q = tid; q < (nbins >> 1); q += THREADS) {
                const uint32_t v0 = jh[q];
                uint32_t lo = v0 & 0xffffu, hi = v0 >> 16;
                if (lo > kSegSpillAt) {
                    atomicAdd(&hrow[2 * q], lo);
                    lo = 0;
                }
                if (hi > kSegSpillAt) {
                    atomicAdd(&hrow[2 * q + 1], hi);
                    hi = 0;
                }
                if (v0 != (lo | (hi << 16))) jh[q] = lo | (hi << 16);
                mx = max(mx, max(lo, hi));
            }
            mx = __reduce_max_sync(0xffffffffu, mx);
            if (lane == 0) s_max[w] = mx;
            __syncthreads();
            since = 0;
#pragma unroll
            for (int q = 0; q < THREADS / 32; q++) since = max(since, s_max[q]);
            __syncthreads();
        }
        since += cnt;
        const bool ok = mbar_wait(bar0 + 8u * cur, (k >> 1) & 1u);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                set_error(err, kErrSpinLimit);
                // Let this buffer's copy land first (bounded), unless the stall hook withheld it (CTA 0's
                // first tile); nothing else is in flight (the next tile's copy is issued below).
                if (!(a.test_stall && blockIdx.x == 0 && k == 0)) mbar_wait(bar0 + 8u * cur, (k >> 1) & 1u);
            }
            break;
        }
        // Prefetch the next tile into the other buffer: every thread has passed the barrier above, so
        // the previous tile's staging and write-out, the last accesses to that buffer, are done.
        if (tid == 0) {
            uint32_t item = s_item, tn = s_tnext, te = s_tend, rn = s_rnext;
            const SegSlot sn = seg_next_tile<STABLE_R>(a, item, tn, te, rn, s_rend);
            s_item = item;
            s_tnext = tn;
            s_tend = te;
            s_rnext = rn;
            slots[cur ^ 1u] = sn;
            if (sn.cnt) tma_load_1d(inbuf + (size_t)(cur ^ 1u) * T, sn.in, sn.cnt * 16u, bar0 + 8u * (cur ^ 1u));
        }

        tuple_v v[ITEMS];
        uint32_t rk[ITEMS];
        const bool st = STABLE_R && sl.rel == 0;  // uniform: this tile takes the stable rank
        uint32_t xo = 0, yo = 0, lo = 0;
        if (cnt == (uint32_t)T) {
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                v[i] = buf[w * 32 * ITEMS + i * 32 + lane];
                if (MIX) v[i].x = mix_key(v[i].x, a.bits);
                const uint32_t d = (uint32_t)v[i].x & dmask;
                if (!st) rk[i] = atomicAdd(&thist[d], 1u);
                const uint32_t bin = (uint32_t)(v[i].x & bmask);
                atomicAdd(&jh[bin >> 1], 1u << ((bin & 1u) << 4));
                xo |= (uint32_t)(v[i].x >> 32);
                yo |= (uint32_t)(v[i].y >> 32);
                lo |= (uint32_t)v[i].x;
            }
        } else {
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const uint32_t idx = (uint32_t)(w * 32 * ITEMS + i * 32 + lane);
                if (idx < cnt) {
                    v[i] = buf[idx];
                    if (MIX) v[i].x = mix_key(v[i].x, a.bits);
                    const uint32_t d = (uint32_t)v[i].x & dmask;
                    if (!st) rk[i] = atomicAdd(&thist[d], 1u);
                    const uint32_t bin = (uint32_t)(v[i].x & bmask);
                    atomicAdd(&jh[bin >> 1], 1u << ((bin & 1u) << 4));
                    xo |= (uint32_t)(v[i].x >> 32);
                    yo |= (uint32_t)(v[i].y >> 32);
                    lo |= (uint32_t)v[i].x;
                }
            }
        }
        if (sl.rel == 0) {
            kor |= xo;
            ror |= yo;
        } else {
            rors |= yo;
        }
        // A value too wide for words: the tuple pass will have to run, so end this one. The claims of every
        // CTA run past the last item from now on (a relation of 63-bit keys costs a tile per CTA here, not
        // a whole pass).
        if (W8 && (yo || (sl.rel == 0 && (xo >> (a.b1 - 1)))) &&
            !*reinterpret_cast<volatile uint32_t *>(&a.counters[kCtrSegWide]) &&
            atomicExch(&a.counters[kCtrSegWide], 1u) == 0)
            atomicAdd(&a.counters[kCtrItem1], kSegEndItems);
        if (STABLE_R && st) {
            // Stable rank within the warp: items in order, lanes in order; the lanes holding one digit
            // are found with one ballot per digit bit (plus the bit that marks padding lanes).
            uint16_t *wh = whist + w * F;
            for (int j = lane; j < F; j += 32) wh[j] = 0;
            __syncwarp();
            const unsigned ltmask = lanemask_lt();
            // Digit bits: K = F1 / 32 for K >= 2 gives log2(F1) exactly; K = 1 covers F1 <= 32 with 5
            // bits (the unused high bits are zero in every lane). A partial tile's padding lanes carry
            // digit F1, one bit more.
            constexpr int NB = K == 1 ? 5 : K == 2 ? 6 : K == 4 ? 7 : 8;
            const bool fullt = cnt == (uint32_t)T;
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const uint32_t idx = (uint32_t)(w * 32 * ITEMS + i * 32 + lane);
                const uint32_t d = idx < cnt ? (uint32_t)v[i].x & dmask : (uint32_t)F;
                const unsigned peers = fullt ? digit_peers<NB>(d) : digit_peers<NB + 1>(d);
                const bool valid = d < (uint32_t)F;
                uint32_t pre = 0;
                if (valid) pre = wh[d];
                rk[i] = pre + __popc(peers & ltmask);
                __syncwarp();
                if (valid && (peers & ltmask) == 0) wh[d] = (uint16_t)(pre + __popc(peers));
                __syncwarp();
            }
            __syncthreads();
            // Tile count per digit, and each warp's start within the digit's run.
            if (tid < F) {
                uint32_t h = 0;
                for (int q = 0; q < THREADS / 32; q++) {
                    const uint32_t n = whist[q * F + tid];
                    whist[q * F + tid] = (uint16_t)h;
                    h += n;
                }
                thist[tid] = h;
            }
        }
        // Words: a tile whose keys are below 2^31 and row ids below 2^32 is staged as 8-byte {row id, key}, half
        // the shared-memory traffic of a tuple; the word is made from it when it is written.
        bool narrow = false;
        if (W8)
            narrow = !__syncthreads_or((xo | yo | (lo >> 31)) != 0);
        else
            __syncthreads();
        // Warp 0, step 1: digit starts in the staged tile, and which digits' runs need a new segment
        // (a run that does not fit the rest of its current segment). Lane l owns digits [l*K, l*K + K).
        uint32_t hv[K];      // warp 0: tile count of each owned digit
        uint32_t exl = 0;    // warp 0: tuples (low 16 bits) and new segments (high 16 bits) before lane l
        uint32_t ntot = 0;   // warp 0: new segments of the tile
        if (w == 0) {
            const int d0 = lane * K;
            uint32_t packed = 0;
#pragma unroll
            for (int j = 0; j < K; j++) {
                hv[j] = d0 + j < F ? thist[d0 + j] : 0u;
                const bool nw = hv[j] && (scur[j] == kSegNone || sfill[j] + hv[j] > SEGW);
                packed += hv[j] + (nw ? 0x10000u : 0u);
            }
            uint32_t incl = packed;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            ntot = __shfl_sync(0xffffffffu, incl, 31) >> 16;
            exl = incl - packed;
            uint32_t ex = exl & 0xffffu;
#pragma unroll
            for (int j = 0; j < K; j++) {
                const int d = d0 + j;
                if (d < F) {
                    thist[d] = 0;
                    tdstart[d] = ex;
                    ex += hv[j];
                }
            }
        }
        __syncthreads();
        // Stage the tile sorted by digit, in place.
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t idx = (uint32_t)(w * 32 * ITEMS + i * 32 + lane);
            if (idx < cnt) {
                const uint32_t d = (uint32_t)v[i].x & dmask;
                const uint32_t p = tdstart[d] + (STABLE_R && st ? (uint32_t)whist[w * F + d] : 0u) + rk[i];
                if (W8 && narrow)
                    reinterpret_cast<uint2 *>(buf)[p] = make_uint2((uint32_t)v[i].y, (uint32_t)v[i].x);
                else
                    buf[p] = v[i];
            }
        }
        // Warp 0, step 2 (while the other warps stage): where each digit's run goes, the rest of its
        // current segment, then (when that fills) a new segment.
        if (w == 0) {
            const int d0 = lane * K;
            // New segment ids: first what is left of the slab, then a fresh slab.
            uint32_t old_lo = 0, old_rem = 0, nb = 0;
            if (ntot) {
                if (lane == 0) {
                    old_lo = slab_lo;
                    old_rem = slab_rem;
                    if (ntot <= slab_rem) {
                        slab_lo += ntot;
                        slab_rem -= ntot;
                    } else {
                        const uint32_t deficit = ntot - slab_rem;
                        const uint32_t take = deficit > kSegSlab ? deficit : kSegSlab;
                        nb = atomicAdd(&a.counters[kCtrSegAlloc], take);
                        slab_lo = nb + deficit;
                        slab_rem = take - deficit;
                    }
                }
                old_lo = __shfl_sync(0xffffffffu, old_lo, 0);
                old_rem = __shfl_sync(0xffffffffu, old_rem, 0);
                nb = __shfl_sync(0xffffffffu, nb, 0);
            }
            uint32_t ex = exl & 0xffffu, e = exl >> 16;
#pragma unroll
            for (int j = 0; j < K; j++) {
                const int d = d0 + j;
                if (d < F) {
                    const uint32_t h = hv[j];
                    if (h) {
                        const uint32_t sc = scur[j], fill = sfill[j];
                        unsigned long long b1 = kSegNowhere, b2 = kSegNowhere;
                        uint32_t split = ex + h;
                        if (sc != kSegNone && fill + h <= SEGW) {
                            b1 = b2 = (unsigned long long)sc * SEGW + fill + kTile - ex;
                            sfill[j] = fill + h;
                        } else {
                            const uint32_t id = e < old_rem ? old_lo + e : nb + (e - old_rem);
                            e++;
                            if (id < a.max_segs) {
                                if (sc == kSegNone) {
                                    // The whole run starts the chain.
                                    a.seg_head[((size_t)phase_rel * G + c) * F + d] = id;
                                    b1 = b2 = (unsigned long long)id * SEGW + kTile - ex;
                                    sfill[j] = h;
                                } else {
                                    // The run fills the current segment, then goes on in segment
                                    // id: staged index ex + (SEGW - fill) lands at id * SEGW.
                                    a.seg_next[sc] = id;
                                    b1 = (unsigned long long)sc * SEGW + fill + kTile - ex;
                                    b2 = (unsigned long long)id * SEGW + kTile - ex - (SEGW - fill);
                                    split = ex + (SEGW - fill);
                                    sfill[j] = h - (SEGW - fill);
                                }
                                scur[j] = id;
                            } else {
                                // Cannot happen with the storage phj_carve reserves; the run's
                                // stores fail their bounds check and report it.
                                set_error(err, kErrCapacity);
                                scur[j] = kSegNone;
                                sfill[j] = 0;
                            }
                        }
                        runs[d] = seg_run(b1, b2, split);
                    }
                    ex += h;
                }
            }
        }
        __syncthreads();
        // Write each digit run: consecutive threads write consecutive 16-byte tuples (8-byte words).
        // A destination outside the segment storage (negative included) fails the unsigned bound check.
        if (W8 && narrow) {
            const uint2 *nbuf = reinterpret_cast<const uint2 *>(buf);
            auto word = [&](const uint2 &x) { return ((unsigned long long)(x.y >> a.b1) << 32) | x.x; };
            if (cnt == (uint32_t)T) {
                uint2 t[ITEMS];
                unsigned long long dst[ITEMS];
#pragma unroll
                for (int i = 0; i < ITEMS; i++) t[i] = nbuf[tid + i * THREADS];
#pragma unroll
                for (int i = 0; i < ITEMS; i++) dst[i] = seg_dst(&runs[t[i].y & dmask], (uint32_t)(tid + i * THREADS));
#pragma unroll
                for (int i = 0; i < ITEMS; i++) {
                    if (dst[i] < cap)
                        st_stream8(out8 + dst[i], word(t[i]));
                    else
                        set_error(err, kErrBounds);
                }
            } else {
                for (uint32_t j = tid; j < cnt; j += THREADS) {
                    const uint2 t = nbuf[j];
                    const unsigned long long dst = seg_dst(&runs[t.y & dmask], j);
                    if (dst < cap)
                        st_stream8(out8 + dst, word(t));
                    else
                        set_error(err, kErrBounds);
                }
            }
        } else if (cnt == (uint32_t)T) {
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                tuple_v t[ITEMS / 2];
                unsigned long long dst[ITEMS / 2];
#pragma unroll
                for (int i = 0; i < ITEMS / 2; i++) t[i] = buf[tid + (hh * ITEMS / 2 + i) * THREADS];
#pragma unroll
                for (int i = 0; i < ITEMS / 2; i++)
                    dst[i] = seg_dst(&runs[(uint32_t)t[i].x & dmask], (uint32_t)(tid + (hh * ITEMS / 2 + i) * THREADS));
#pragma unroll
                for (int i = 0; i < ITEMS / 2; i++) {
                    if (dst[i] < cap) {
                        if (W8)
                            st_stream8(out8 + dst[i], w8_word(t[i].x, t[i].y, a.b1));
                        else
                            st_stream(a.out + dst[i], t[i]);
                    } else {
                        set_error(err, kErrBounds);
                    }
                }
            }
        } else {
            for (uint32_t j = tid; j < cnt; j += THREADS) {
                const tuple_v t = buf[j];
                const unsigned long long dst = seg_dst(&runs[(uint32_t)t.x & dmask], j);
                if (dst < cap) {
                    if (W8)
                        st_stream8(out8 + dst, w8_word(t.x, t.y, a.b1));
                    else
                        st_stream(a.out + dst, t);
                } else {
                    set_error(err, kErrBounds);
                }
            }
        }
        // No barrier here: the next tile's wait barrier orders this write-out before the next prefetch
        // into this buffer and before the next tile's planning rewrites runs and tdstart.
    }
    // The counters of the relation in progress go to their row (the other row is complete).
    __syncthreads();
    seg_flush(jh, a.hist + ((size_t)phase_rel * G + c) * nbins, nbins);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        kor |= __shfl_xor_sync(0xffffffffu, kor, o);
        ror |= __shfl_xor_sync(0xffffffffu, ror, o);
        rors |= __shfl_xor_sync(0xffffffffu, rors, o);
    }
    if (lane == 0 && (kor | ror | rors)) {
        unsigned long long *mx = reinterpret_cast<unsigned long long *>(a.counters + kCtrMaxKey);
        if (kor) atomicOr(mx, (unsigned long long)kor << 32);
        if (ror) atomicOr(mx + 1, (unsigned long long)ror << 32);
        if (rors) atomicOr(mx + 2, (unsigned long long)rors << 32);
    }
}

// After a pass 1 that wrote 8-byte words: if the widths did not allow them, pass 1 runs again with
// tuples, from fresh item and segment counters (its own CTAs zero their histogram rows).
__global__ void seg_reset_if_wide(uint32_t *counters, int b1) {
    if (threadIdx.x == 0 && !w8_fits(counters, b1)) {
        counters[kCtrItem1] = 0;
        counters[kCtrSegAlloc] = 0;
        counters[kCtrSegWide] = 0;
    }
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
#define HJ_CU(call)                                                                   \
    do {                                                                              \
        cudaError_t e_ = (call);                                                      \
        if (e_ != cudaSuccess) {                                                      \
            fprintf(stderr, "hjscm: %s failed: %s\n", #call, cudaGetErrorString(e_)); \
            return HJ_E_DEVICE;                                                       \
        }                                                                             \
    } while (0)

// Dynamic shared memory of seg_pass1_kernel: two tile buffers, per-digit state, 2^bits 16-bit counters,
// and for the stable build-relation rank one 16-bit counter per (warp, digit).
static size_t seg_smem_bytes(int bits, bool stable) {
    // tile buffers, runs[256], thist[256], tdstart[256], counter pairs, whist
    return (size_t)2 * kTile * 16 + 256 * sizeof(SegRun) + 256 * 4 * 2 + ((size_t)1 << bits) * 2 +
           (stable ? (size_t)(kScatterThreads / 32) * 256 * 2 : 0);
}

// Segment mode's pass 1, by the key's digits or by mix_key.
template <bool MIX>
static int seg_prepare_form() {
#define HJ_SEG_ATTR(KK, W, ST)                                                                             \
    HJ_CU(cudaFuncSetAttribute(seg_pass1_kernel<kScatterThreads, kScatterItems, KK, W, ST, MIX>,             \
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)seg_smem_bytes(kSegMaxBits, ST)))
#define HJ_SEG_ATTR4(KK)         \
    HJ_SEG_ATTR(KK, false, false); \
    HJ_SEG_ATTR(KK, true, false);  \
    HJ_SEG_ATTR(KK, false, true);  \
    HJ_SEG_ATTR(KK, true, true)
    HJ_SEG_ATTR4(1);
    HJ_SEG_ATTR4(2);
    HJ_SEG_ATTR4(4);
    if constexpr (!MIX) {
        HJ_SEG_ATTR4(8);
    }
#undef HJ_SEG_ATTR4
#undef HJ_SEG_ATTR
    return HJ_OK;
}

int seg_prepare_device(bool mix) { return mix ? seg_prepare_form<true>() : seg_prepare_form<false>(); }

int seg_pass1_enqueue(const RadixGeom &g, const ulonglong2 *R, size_t nR, const ulonglong2 *S, size_t nS,
                      const PhjScratch &s, bool words_too, bool stable, bool stall, cudaStream_t st, uint32_t *launches) {
    const int F1 = g.F1;
    SegArgs ga;
    ga.R = R;
    ga.S = S;
    ga.nR = nR;
    ga.nS = nS;
    ga.bits = g.bits;
    ga.F1 = F1;
    ga.it_tiles = s.it_tiles;
    ga.tilesR = ceil_div_u64(nR, kTile);
    ga.tilesS = ceil_div_u64(nS, kTile);
    ga.itemsR = (ga.tilesR + s.it_tiles - 1) / s.it_tiles;
    ga.items = ga.itemsR + (ga.tilesS + s.it_tiles - 1) / s.it_tiles;
    ga.out = s.tmp1;
    ga.max_segs = s.max_segs;
    ga.seg_head = s.seg_head;
    ga.seg_next = s.seg_next;
    ga.hist = s.chunk_hist;
    ga.counters = s.counters;
    ga.test_stall = stall ? 1 : 0;
    ga.b1 = g.b1;
    ga.w8_first = 0;
    // Ordered first-match joins keep every build partition in input order (the stable build-relation form).
    const size_t sm = seg_smem_bytes(g.bits, stable);
    auto launch_pass1 = [&](bool words) {
#define HJ_SEG_LAUNCH_W(KK, W, MX)                                                                                   \
    if (stable)                                                                                                      \
        seg_pass1_kernel<kScatterThreads, kScatterItems, KK, W, true, MX><<<s.seg_grid, kScatterThreads, sm, st>>>(ga); \
    else                                                                                                             \
        seg_pass1_kernel<kScatterThreads, kScatterItems, KK, W, false, MX><<<s.seg_grid, kScatterThreads, sm, st>>>(ga)
#define HJ_SEG_LAUNCH(KK, MX)           \
    if (words) {                        \
        HJ_SEG_LAUNCH_W(KK, true, MX);  \
    } else {                            \
        HJ_SEG_LAUNCH_W(KK, false, MX); \
    }
        if (g.mix) {  // at most 7 bits in pass 1
            if (F1 <= 32) {
                HJ_SEG_LAUNCH(1, true);
            } else if (F1 <= 64) {
                HJ_SEG_LAUNCH(2, true);
            } else {
                HJ_SEG_LAUNCH(4, true);
            }
        } else if (F1 <= 32) {
            HJ_SEG_LAUNCH(1, false);
        } else if (F1 <= 64) {
            HJ_SEG_LAUNCH(2, false);
        } else if (F1 <= 128) {
            HJ_SEG_LAUNCH(4, false);
        } else {
            HJ_SEG_LAUNCH(8, false);
        }
#undef HJ_SEG_LAUNCH
#undef HJ_SEG_LAUNCH_W
    };
    if (words_too) {
        // Pass 1 in 8-byte words; if the widths turn out not to allow them, the counters are reset and
        // pass 1 runs again with tuples (that launch returns at once otherwise).
        launch_pass1(true);
        seg_reset_if_wide<<<1, 32, 0, st>>>(s.counters, g.b1);
        ga.w8_first = 1;
        ga.test_stall = 0;
        *launches += 2;
    }
    launch_pass1(false);
    HJ_CU(cudaGetLastError());
    *launches += 1;
    return HJ_OK;
}

}  // namespace hj
