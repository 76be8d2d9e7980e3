// hj_partition.cu - radix-partitioned join (phj_radix_bc / phj_radix_lp) on sm_100a.
//
// Reference algorithm (src/algo/phj.c):
//   pass 1  parallel_radix_partition / _optimized (phj.c:147-215, 257-360): per-thread histogram of
//           digit (key & (F1-1)), cross-thread prefix, stable scatter into padded partitions through
//           software write-combining buffers.
//   pass 2  serial_radix_partition -> radix_cluster (phj.c:366-491): each pass-1 partition re-clustered
//           on (key >> b1) & (F2-1), again stable; a join task per non-empty (R_p, S_p) pair.
//   join    bc_join (phj.c:496-571): bucket[next_pow_2(|R_p|)] + next[|R_p|] chains, every equal key
//           counted; lp_join (phj.c:574-680): open addressing, the probe stops at the first equal key,
//           which is the first R tuple of the partition in input order.
//
// B200 pipeline (one stream, no host round trip). Each relation is cut into equal chunks (about three
// per SM) and each chunk into ~32 sub-chunks; a chunk plays the role of one reference thread's
// contiguous input slice.
//   hist_chunk_kernel  one read of R and S: per chunk, the joint histogram of the low B key bits (the
//                      pass-1 digit and the pass-2 digit together) in shared memory; per sub-chunk (one
//                      warp each) the histogram of the pass-1 digit
//   colscan_kernel     per bin, exclusive prefix over the chunks of a relation (the reference's
//                      cross-thread output_offset sums, phj.c:188-200, for both passes at once)
//   plan_kernel        final partition starts, join work items, large partitions
//   units_kernel       per (chunk, pass-1 partition): its size and its start in the pass-1 output; per
//                      sub-chunk its start within that
//   scatter_kernel     per pass: persistent CTAs take work items (pass 1: sub-chunks; pass 2: (chunk,
//                      pass-1 partition) units) whose per-digit output offsets are known in advance;
//                      each 2048-tuple tile arrives by a TMA bulk copy (the next one is in flight while
//                      the current one is processed), is ranked per digit (one shared-memory atomic per
//                      tuple; stably with bit ballots for the lp joins, whose result depends on input
//                      order), staged in shared memory sorted by digit and written back as coalesced
//                      16-byte streaming stores per digit run (the shared-memory analogue of the
//                      reference's SWWCB + non-temporal flush). No inter-CTA waiting.
//   join_words         compact final partitions (8-byte words): persistent CTAs take (partition, S chunk)
//                      items; an open-addressing table of the words in shared memory
//   join_compact       tuples whose keys (after the radix shift) and row ids fit 32 bits, and ordered
//                      first-match joins over words: words with u16 bucket heads and chains
//   join_small         the general case: R_p arrives in shared memory by one TMA bulk copy, 16-byte
//                      entries, u16 head/next chains
//   join_first*        first-match joins of the one-pass pipeline, by input position
//   join_large_*       partitions whose R side exceeds shared memory: chains in global memory
// The join kernels have a materialising variant (MAT) for the ptr_* joins: one (r.row_id, s.row_id)
// pair per match instead of the sums.
//
// Build relations that few partitions cover go through one pass instead (hj_single.cu), those of at most
// kSmallMaxBuild tuples through one kernel (hj_small.cu); the join kernels here serve both pipelines.
//
// Segment mode (two passes, <= 14 bits, from 2^26 tuples): no histogram
// pass. seg_pass1_kernel (hj_segments.cu) writes pass 1 into per-(CTA, relation, digit) chains of tile-sized segments
// and counts each CTA's joint histogram itself; colscan/plan/units then treat the pass-1 CTAs as the
// chunks, and pass 2 (scatter_kernel) walks the chains as its units.
#include <atomic>
#include <cstdio>

#include "hj_common.cuh"
#include "hj_internal.h"
#include "hj_partition.cuh"

namespace hj {

// Count the tuples [lo, hi) of `in`, read by one warp (four 512-byte loads in flight), into the joint
// histogram and into the warp's histogram of the pass-1 digit, ORing together all row ids and (BUILD)
// all keys: their widths decide whether the compact join table and the compact final partitions apply
// (a value fits k bits iff the OR of all values does).
template <bool BUILD, bool MIX>
__device__ __forceinline__ void hist_range_warp(const tuple_v *__restrict__ in, uint64_t lo, uint64_t hi,
                                                uint32_t *sh_hist, uint32_t *wsub, uint64_t mask, uint32_t m1,
                                                int bits, unsigned long long &kor, unsigned long long &ror) {
    uint64_t i = lo + (threadIdx.x & 31u);
    for (; i + 96 < hi; i += 128) {
        tuple_v t0 = ld_stream(in + i), t1 = ld_stream(in + i + 32);
        tuple_v t2 = ld_stream(in + i + 64), t3 = ld_stream(in + i + 96);
        if (MIX) {
            t0.x = mix_key(t0.x, bits);
            t1.x = mix_key(t1.x, bits);
            t2.x = mix_key(t2.x, bits);
            t3.x = mix_key(t3.x, bits);
        }
        atomicAdd(&sh_hist[t0.x & mask], 1u);
        atomicAdd(&sh_hist[t1.x & mask], 1u);
        atomicAdd(&sh_hist[t2.x & mask], 1u);
        atomicAdd(&sh_hist[t3.x & mask], 1u);
        atomicAdd(&wsub[(uint32_t)t0.x & m1], 1u);
        atomicAdd(&wsub[(uint32_t)t1.x & m1], 1u);
        atomicAdd(&wsub[(uint32_t)t2.x & m1], 1u);
        atomicAdd(&wsub[(uint32_t)t3.x & m1], 1u);
        if (BUILD) kor |= t0.x | t1.x | t2.x | t3.x;
        ror |= t0.y | t1.y | t2.y | t3.y;
    }
    for (; i < hi; i += 32) {
        tuple_v t = ld_stream(in + i);
        if (MIX) t.x = mix_key(t.x, bits);
        atomicAdd(&sh_hist[t.x & mask], 1u);
        atomicAdd(&wsub[(uint32_t)t.x & m1], 1u);
        if (BUILD) kor |= t.x;
        ror |= t.y;
    }
}

// ------------------------------------------------------------------------------------------------
// 1. Per-chunk joint histogram of the low `bits` key bits, and per sub-chunk the histogram of the
//    pass-1 digit (the low log2(F1) bits). One CTA per chunk; each warp takes whole sub-chunks, so a
//    sub-chunk's digit histogram is complete after a warp barrier and no CTA barrier interrupts the
//    stream of loads. Every bin is written.
// ------------------------------------------------------------------------------------------------
template <bool MIX>
__global__ void __launch_bounds__(512) hist_chunk_kernel(const tuple_v *__restrict__ R, size_t nR,
                                                         const tuple_v *__restrict__ S, size_t nS, int bits,
                                                         int F1, ChunkGeom cg, uint32_t *__restrict__ chunk_hist,
                                                         uint32_t *__restrict__ subhist,
                                                         uint32_t *__restrict__ maxima) {
    extern __shared__ uint32_t sh_hist[];
    const int nbins = 1 << bits;
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u, nw = blockDim.x >> 5;
    uint32_t *wsub = sh_hist + nbins + (size_t)w * F1;  // [warps][F1] per-warp pass-1 digit histogram
    const uint64_t mask = (uint64_t)nbins - 1;
    const uint32_t m1 = (uint32_t)F1 - 1u;
    const uint32_t c = blockIdx.x;
    const int rel = c < cg.cR ? 0 : 1;
    const uint64_t lc = rel ? c - cg.cR : c;
    const tuple_v *in = rel ? S : R;
    const uint64_t n = rel ? nS : nR;
    for (int v = threadIdx.x; v < nbins + (int)nw * F1; v += blockDim.x) sh_hist[v] = 0;
    __syncthreads();
    const uint64_t clo = lc * cg.chunk;
    const uint64_t chi = clo + cg.chunk < n ? clo + cg.chunk : n;
    unsigned long long kor = 0, ror = 0;
    for (uint32_t j = w; j < cg.spc; j += nw) {
        const uint64_t lo = clo + (uint64_t)j * cg.sub < chi ? clo + (uint64_t)j * cg.sub : chi;
        const uint64_t hi = lo + cg.sub < chi ? lo + cg.sub : chi;
        if (rel == 0)
            hist_range_warp<true, MIX>(in, lo, hi, sh_hist, wsub, mask, m1, bits, kor, ror);
        else
            hist_range_warp<false, MIX>(in, lo, hi, sh_hist, wsub, mask, m1, bits, kor, ror);
        __syncwarp();
        uint32_t *so = subhist + ((size_t)c * cg.spc + j) * F1;
        for (int v = lane; v < F1; v += 32) {
            so[v] = wsub[v];
            wsub[v] = 0;
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        kor |= __shfl_xor_sync(0xffffffffu, kor, o);
        ror |= __shfl_xor_sync(0xffffffffu, ror, o);
    }
    if (lane == 0) {
        unsigned long long *mx = reinterpret_cast<unsigned long long *>(maxima);
        if (rel == 0) {
            if (kor) atomicOr(mx, kor);
            if (ror) atomicOr(mx + 1, ror);
        } else if (ror) {
            atomicOr(mx + 2, ror);
        }
    }
    __syncthreads();
    uint32_t *out = chunk_hist + (size_t)c * nbins;
    for (int v = threadIdx.x; v < nbins; v += blockDim.x) out[v] = sh_hist[v];
}

// ------------------------------------------------------------------------------------------------
// 2. Per bin, exclusive prefix over the chunks of its relation, and the relation totals. Four
//    consecutive lanes share one bin and split its chunks into four ranges: each lane sums its range,
//    the four sums are scanned with shuffles, then each lane writes the prefixes of its range.
// ------------------------------------------------------------------------------------------------
__global__ void colscan_kernel(const uint32_t *__restrict__ chunk_hist, uint32_t *__restrict__ prefix,
                               uint32_t *__restrict__ total, int nbins, ChunkGeom cg) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t col = g >> 2, seg = g & 3u;
    const bool active = col < 2u * (uint32_t)nbins;
    const int rel = active && col >= (uint32_t)nbins;
    const uint32_t v = active ? (rel ? col - nbins : col) : 0u;
    const uint32_t c0 = rel ? cg.cR : 0, c1 = rel ? cg.cR + cg.cS : cg.cR;
    const uint32_t per = (c1 - c0 + 3) / 4;
    const uint32_t r0 = c0 + seg * per < c1 ? c0 + seg * per : c1;
    const uint32_t r1 = r0 + per < c1 ? r0 + per : c1;
    uint32_t sum = 0;
    if (active) {
        uint32_t c = r0;
        for (; c + 8 <= r1; c += 8) {
            uint32_t x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = chunk_hist[(size_t)(c + u) * nbins + v];
#pragma unroll
            for (int u = 0; u < 8; u++) sum += x[u];
        }
        for (; c < r1; c++) sum += chunk_hist[(size_t)c * nbins + v];
    }
    // Exclusive scan of the four range sums (lanes 4k..4k+3 of the warp).
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o, 4);
        if (seg >= (uint32_t)o) incl += y;
    }
    const uint32_t colsum = __shfl_sync(0xffffffffu, incl, 3, 4);
    if (!active) return;
    uint32_t run = incl - sum;
    uint32_t c = r0;
    for (; c + 8 <= r1; c += 8) {
        uint32_t x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = chunk_hist[(size_t)(c + u) * nbins + v];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            prefix[(size_t)(c + u) * nbins + v] = run;
            run += x[u];
        }
    }
    for (; c < r1; c++) {
        const uint32_t x = chunk_hist[(size_t)c * nbins + v];
        prefix[(size_t)c * nbins + v] = run;
        run += x;
    }
    if (seg == 3) total[(size_t)rel * nbins + v] = colsum;
}

// ------------------------------------------------------------------------------------------------
// 3. Plan: final partition starts (in (pass-1 digit, pass-2 digit) order), join work items, large
//    partitions. One CTA of 1024 threads.
// ------------------------------------------------------------------------------------------------
// Dynamic shared memory: the relation totals ([2][2^B] u32) when they fit (B <= 14), so that the
// per-partition loops below read shared memory instead of waiting on one global load after another.
constexpr int kPlanStageBits = 14;

__global__ void __launch_bounds__(1024, 1) plan_kernel(PlanArgs a) {
    extern __shared__ uint32_t sm_tot[];
    __shared__ uint32_t tmp[32];
    __shared__ uint64_t s_run[2];
    const int tid = threadIdx.x;
    const int nparts = 1 << a.bits;
    const uint32_t *tot_all = a.total;
    if (a.bits <= kPlanStageBits) {
#pragma unroll 8
        for (int i = tid; i < 2 * nparts; i += 1024) sm_tot[i] = a.total[i];
        __syncthreads();
        tot_all = sm_tot;
    }
    plan_body(a, tot_all, tmp, s_run);
}

// ------------------------------------------------------------------------------------------------
// 4. Units: for every chunk c and pass-1 digit d1, the number of the chunk's tuples with that digit
//    and where they start in the pass-1 output: start[d1 * F2] + sum over d2 of prefix[c][(d1, d2)].
//    The sub-chunk histograms of the chunk become, in place, each sub-chunk's start within (c, d1).
// ------------------------------------------------------------------------------------------------
__global__ void units_kernel(const uint32_t *__restrict__ chunk_hist, const uint32_t *__restrict__ prefix,
                             const uint64_t *__restrict__ start, int bits, int b1, int F1, int F2,
                             ChunkGeom cg, uint64_t *__restrict__ unit_off, uint32_t *__restrict__ unit_cnt,
                             uint32_t *__restrict__ subhist, uint32_t *__restrict__ err) {
    // One CTA per chunk, one thread per pass-1 digit; for a fixed pass-2 digit the threads read
    // consecutive bins.
    const uint32_t c = blockIdx.x;
    const uint32_t d1 = threadIdx.x;
    if (d1 >= (uint32_t)F1) return;
    const int rel = c < cg.cR ? 0 : 1;
    const int nbins = 1 << bits;
    const uint32_t *h = chunk_hist + (size_t)c * nbins;
    const uint32_t *p = prefix + (size_t)c * nbins;
    uint64_t cnt = 0, pre = 0;
    int d2 = 0;
    for (; d2 + 8 <= F2; d2 += 8) {
        uint32_t x[8], y[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint32_t v = d1 | ((uint32_t)(d2 + u) << b1);
            x[u] = h[v];
            y[u] = p[v];
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            cnt += x[u];
            pre += y[u];
        }
    }
    for (; d2 < F2; d2++) {
        const uint32_t v = d1 | ((uint32_t)d2 << b1);
        cnt += h[v];
        pre += p[v];
    }
    const uint32_t wid = c * (uint32_t)F1 + d1;
    unit_cnt[wid] = (uint32_t)cnt;
    unit_off[wid] = start[(size_t)rel * (nbins + 1) + (size_t)d1 * F2] + pre;
    uint32_t *sh = subhist + (size_t)c * cg.spc * F1 + d1;
    uint32_t run = 0;
    uint32_t j = 0;
    for (; j + 8 <= cg.spc; j += 8) {
        uint32_t x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = sh[(size_t)(j + u) * F1];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            sh[(size_t)(j + u) * F1] = run;
            run += x[u];
        }
    }
    for (; j < cg.spc; j++) {
        const uint32_t x = sh[(size_t)j * F1];
        sh[(size_t)j * F1] = run;
        run += x;
    }
    if (cg.spc && run != (uint32_t)cnt) set_error(err, kErrCapacity);
}

// ------------------------------------------------------------------------------------------------
// 5. Stable scatter of one pass, from precomputed per-item digit offsets.
// ------------------------------------------------------------------------------------------------
struct ScatterArgs {
    int pass;        // 0: by the pass-1 digit, per chunk; 1: by the pass-2 digit, per (chunk, d1) unit
    int F, shift;    // digit of this pass: (key >> shift) & (F - 1)
    int logF;        // log2(F)
    int bits, b1, F1, F2;
    ChunkGeom cg;
    const tuple_v *inR, *inS;   // pass input (pass 0: the relations; pass 1: the pass-1 output)
    tuple_v *outR, *outS;       // pass output
    uint64_t nR, nS;
    const uint32_t *prefix;     // [chunk][2^B]
    const uint64_t *start;      // [2][2^B + 1]
    const uint64_t *unit_off;   // [chunk][F1]
    const uint32_t *unit_cnt;   // [chunk][F1]
    const uint32_t *subpre;     // [chunk][spc][F1] start of (sub-chunk, d1) within (chunk, d1)
    // Segment mode, pass 2: unit (chunk, d1) is a chain of kTile-tuple segments in inR (the pass-1
    // output of both relations): seg_head[unit], then seg_next[segment]; all but the last are full.
    const uint32_t *seg_head;   // nullptr: units are contiguous ranges (unit_off)
    const uint32_t *seg_next;
    uint32_t max_segs;
    int test_stall;             // test hook: CTA 0 withholds its first tile load (its wait must expire)
    uint32_t *counters;
    int ctr_item;
    // Work items of this launch: [item_base, item_end) of the pass's items (R's first, then S's), claimed
    // through counters[ctr_item]; item_end 0 = all of them.
    uint32_t item_base, item_end;
    // Last pass of a join that may read compact final partitions: when ci_applies holds, the output is
    // 8-byte words (ci_word) at outR8 / outS8 instead of tuples at outR / outS.
    int ci_out;
    int ci_z0;                  // build key 0 never matches: its compact words take ci_word_z0's high part
    unsigned long long *outR8, *outS8;
    // After a pass 1 that may have written 8-byte words: 1 = this launch reads words (runs when w8_fits
    // holds), 2 = this launch reads tuples (runs when it does not); 0 = no such pass 1.
    int w8;
    // Exact-offset pipeline: pass 1 stores 8-byte words (w8_word) at outR8 / outS8 when w8_fits holds,
    // and the word launch of pass 2 reads its units from inR8 / inS8 (word offsets, which may be odd:
    // such a tile's copy starts one word early and the tile skips it).
    int w8_out;
    const unsigned long long *inR8, *inS8;
};

// A tile claimed for processing: its source, length, output region and owning work item.
struct TileSlot {
    const tuple_v *in;
    tuple_v *out;
    uint64_t out_len;
    uint32_t item;   // work item (valid flag: item != ~0u)
    uint32_t cnt;    // tuples in this tile
    uint32_t first;  // first tile of its item: the item's digit offsets must be loaded
    uint32_t pad;    // elements before the tile's first in its copy (a word tile at an odd offset)
};

// Thread-0 state of the work-item iterator.
struct ItemIter {
    uint32_t item = ~0u;
    const tuple_v *in = nullptr;
    tuple_v *out = nullptr;
    uint64_t len = 0, out_len = 0, done = 0;
    uint32_t seg = 0;   // segment mode: segment of the next tile
};

// The next work item, claimed one item ahead (thread 0 only): its id comes from the counter while the
// current item is processed, and the loads of its description are issued one call later, so that
// neither the atomic nor the loads stall the CTA at the switch.
struct ItemAhead {
    uint32_t item;   // claimed id (stage >= 1)
    uint32_t stage;  // 0: nothing claimed, 1: claimed, 2: description loaded
    uint64_t len, off;
    uint32_t seg;
};

// The n-th claim's work item. Pass 2 takes the units by pass-1 digit, every chunk's unit of one digit before
// the next digit, so that the CTAs of the moment write one digit's stretch of the output (pass 2 of 2^26 x 2^28
// Zipf keys: 1790 -> 1735 us, of 2^27 x 2^29 uniform keys: 3015 -> 2990 us).
__device__ __forceinline__ uint32_t item_at(const ScatterArgs &a, uint32_t n, uint32_t nitems) {
    if (a.pass == 0 || n >= nitems) return n;
    const uint32_t cR = a.cg.cR, r_items = cR * (uint32_t)a.F1;
    if (n < r_items) return (n % cR) * (uint32_t)a.F1 + n / cR;
    const uint32_t m = n - r_items, cS = a.cg.cS;
    return r_items + (m % cS) * (uint32_t)a.F1 + m / cS;
}

// Issue the loads that describe `ah.item` (pass 2 units; pass-1 sub-chunks need none).
__device__ __forceinline__ void item_fetch(const ScatterArgs &a, ItemAhead &ah, uint32_t nitems) {
    ah.stage = 2;
    if (a.pass == 0 || ah.item >= nitems) return;
    ah.len = a.unit_cnt[ah.item];
    if (a.seg_head)
        ah.seg = a.seg_head[ah.item];  // read even for an empty unit (then unused): no dependent load
    else
        ah.off = a.unit_off[ah.item];
}

__device__ __forceinline__ void item_decode(const ScatterArgs &a, uint32_t item, const ItemAhead &ah, ItemIter &it) {
    const ChunkGeom &cg = a.cg;
    it.item = item;
    it.done = 0;
    if (a.pass == 0) {
        // Pass 1 work item: sub-chunk j of chunk c.
        const uint32_t c = item / cg.spc, j = item % cg.spc;
        const int rel = c < cg.cR ? 0 : 1;
        const uint64_t lc = rel ? c - cg.cR : c;
        const uint64_t n = rel ? a.nS : a.nR;
        const uint64_t clo = lc * cg.chunk;
        const uint64_t chi = clo + cg.chunk < n ? clo + cg.chunk : n;
        const uint64_t lo = clo + (uint64_t)j * cg.sub;
        it.len = lo < chi ? (chi - lo < cg.sub ? chi - lo : cg.sub) : 0;
        it.in = (rel ? a.inS : a.inR) + lo;
        it.out = rel ? a.outS : a.outR;
        it.out_len = n;
    } else {
        const uint32_t c = item / a.F1;
        const int rel = c < cg.cR ? 0 : 1;
        it.len = ah.len;
        if (a.seg_head) {
            it.in = a.inR;
            it.seg = ah.seg;
        } else if (a.w8 == 1) {
            it.in = reinterpret_cast<const tuple_v *>((rel ? a.inS8 : a.inR8) + ah.off);
        } else {
            it.in = (rel ? a.inS : a.inR) + ah.off;
        }
        it.out = rel ? a.outS : a.outR;
        it.out_len = rel ? a.nS : a.nR;
    }
}

// Claim the next tile (thread 0 only): continue the current item or take new items until one has
// tuples. Returns a slot with item == ~0u when the work is exhausted. Segment mode: `pend` carries
// seg_next of the tile returned last, loaded then so that its latency passes while that tile is
// processed.
template <int T, bool WIN = false>
__device__ __forceinline__ TileSlot next_tile(const ScatterArgs &a, ItemIter &it, uint32_t nitems,
                                              uint32_t &pend, ItemAhead &ah) {
    TileSlot s;
    if (a.seg_head && it.item != ~0u && it.done > 0 && it.done < it.len) it.seg = pend;
    if (ah.stage == 1) item_fetch(a, ah, nitems);
    for (;;) {
        while (it.item == ~0u || it.done >= it.len) {
            if (ah.stage == 0) {
                ah.item = item_at(a, a.item_base + atomicAdd(&a.counters[a.ctr_item], 1u), nitems);
                ah.stage = 1;
            }
            if (ah.stage == 1) item_fetch(a, ah, nitems);
            const ItemAhead cur = ah;
            ah.stage = 0;
            if (cur.item >= nitems) {
                s.item = ~0u;
                s.in = nullptr;
                s.out = nullptr;
                s.out_len = 0;
                s.cnt = 0;
                s.first = 0;
                s.pad = 0;
                it.item = ~0u;
                it.len = 0;
                it.done = 0;
                return s;
            }
            // Pass 2: claim the following item now; its id and description are needed only when this
            // one is done. (Pass-1 items are long, and an item held back per CTA lengthens the tail
            // by more than the claim costs.)
            if (a.pass != 0) {
                ah.item = item_at(a, a.item_base + atomicAdd(&a.counters[a.ctr_item], 1u), nitems);
                ah.stage = 1;
            }
            item_decode(a, cur.item, cur, it);
        }
        if (!a.seg_head) break;
        if (it.len == 0 || it.seg < a.max_segs) break;
        // A chain that leaves the segment storage (pass 1 stopped early): drop the rest of the unit.
        set_error(&a.counters[kCtrErr], kErrCapacity);
        it.done = it.len;
    }
    s.item = it.item;
    // A segment is kTile tuples (32 KB) in either layout; T counts the launch's elements per tile.
    s.pad = 0;
    if (WIN && !a.seg_head) {
        // Words at an odd offset: copy from one word earlier (bulk copies start on 16 bytes).
        const unsigned long long *p = reinterpret_cast<const unsigned long long *>(it.in) + it.done;
        s.pad = (reinterpret_cast<uintptr_t>(p) & 8u) ? 1u : 0u;
        s.in = reinterpret_cast<const tuple_v *>(p - s.pad);
    } else {
        s.in = a.seg_head ? it.in + (uint64_t)it.seg * kTile : it.in + it.done;
    }
    s.out = it.out;
    s.out_len = it.out_len;
    s.cnt = (uint32_t)(it.len - it.done < (uint64_t)T ? it.len - it.done : (uint64_t)T);
    s.first = it.done == 0;
    it.done += s.cnt;
    if (a.seg_head && it.done < it.len) pend = a.seg_next[it.seg];
    return s;
}

// STABLE: tuples of equal digit keep their input order (needed for the build side of joins that report
// the first match in input order). Otherwise the rank of a tuple within its digit is taken with one
// shared-memory atomic, in whatever order the warps reach it: the partitions hold the same tuples,
// and the joins that count every match do not depend on their order.
// NBUF = 2: the next tile streams into a second buffer while this one is processed; NBUF = 1: one
// buffer per CTA, the CTAs of an SM overlap each other's loads instead.
// Store one element of the last pass: a tuple, its compact final word (ci), or - from an 8-byte word of
// a segment-mode pass 1, which holds key >> b1 - the final word with key >> bits.
__device__ __forceinline__ void store_elem(const tuple_v &t, tuple_v *out, unsigned long long *out8, long long dst,
                                           bool ci, int bits, int, bool z0, bool w8o, int b1) {
    if (w8o)
        st_stream8(out8 + dst, w8_word_z0(t.x, t.y, b1, z0));
    else if (ci)
        st_stream8(out8 + dst, ci_word_z0(t.x, t.y, bits, z0));
    else
        st_stream(out + dst, t);
}
__device__ __forceinline__ void store_elem(unsigned long long w, tuple_v *, unsigned long long *out8, long long dst,
                                           bool, int, int b2, bool z0, bool, int) {
    // A pass-1 high part with bit 31 set is a probe key beyond every build key, or (z0) a build key 0.
    const unsigned long long h1 = w >> 32;
    const unsigned long long h = h1 < 0x80000000ull ? h1 >> b2 : (z0 ? 0x80000000ull : 0xffffffffull);
    st_stream8(out8 + dst, (h << 32) | (w & 0xffffffffull));
}

// Elements of a tile: 16-byte tuples, or (WIN) the 8-byte words of a segment-mode pass 1 (w8_word).
template <bool WIN>
struct ScatterElem {
    using type = tuple_v;
};
template <>
struct ScatterElem<true> {
    using type = unsigned long long;
};

// Bytes a tile's bulk copy moves: a bulk copy's size must be a multiple of 16, so a word tile with an odd
// count also copies the next word of its segment (segments hold 4096 words, so an odd count is at most
// 4095 and the extra word stays inside the segment; it lands in an unused buffer slot).
template <typename E>
__device__ __forceinline__ uint32_t tile_copy_bytes(uint32_t cnt) {
    return sizeof(E) == 16 ? cnt * 16u : ((cnt + 1u) & ~1u) * (uint32_t)sizeof(E);
}

// The same for a digit width known only at run time (at most 9 bits; uniform across the warp).
__device__ __forceinline__ unsigned digit_peers_n(uint32_t d, int nbits) {
    switch (nbits) {
        case 6: return digit_peers<6>(d);
        case 7: return digit_peers<7>(d);
        case 8: return digit_peers<8>(d);
        default: break;
    }
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; b++) {
        if (b < nbits) {
            const unsigned bit = (d >> b) & 1u;
            const unsigned bal = __ballot_sync(0xffffffffu, bit);
            peers &= bal ^ (bit - 1u);
        }
    }
    return peers;
}

// The pass that reads the relations takes mix_key for the key; words only occur later.
__device__ __forceinline__ void elem_mix(tuple_v &v, int bits) { v.x = mix_key(v.x, bits); }
__device__ __forceinline__ void elem_mix(unsigned long long &, int) {}

// Digit of an element in this pass: (key >> shift) & mask; a word holds key >> b1, which is pass 2's shift.
__device__ __forceinline__ uint32_t elem_digit(const tuple_v &v, int shift, uint64_t dmask) {
    return (uint32_t)((v.x >> shift) & dmask);
}
__device__ __forceinline__ uint32_t elem_digit(unsigned long long v, int, uint64_t dmask) {
    return (uint32_t)((v >> 32) & dmask);
}

// MIX (pass 0 only): partition by mix_key, and store it in place of the key; pass 1 then finds it in its input.
template <int THREADS, int ITEMS, bool STABLE, int NBUF, int MINB, bool WIN = false, bool MIX = false>
__global__ void __launch_bounds__(THREADS, MINB) scatter_kernel(ScatterArgs a) {
    using E = typename ScatterElem<WIN>::type;
    constexpr int T = THREADS * ITEMS;
    // Where the prefetch of the next tile is issued: after this tile's wait barrier (atomic ranks, two
    // buffers; measured faster: one barrier less per tile), or at the top of the iteration (stable
    // ranks: measured faster there, as the rank's ballots keep warp 0 busy after the barrier).
    constexpr bool LATE = NBUF == 2 && !STABLE;
    constexpr int NW = THREADS / 32;
    // Buffer stride: word tiles keep two spare words for a copy that starts one word early (and is
    // rounded up to whole 16-byte units).
    constexpr int ST = T + (WIN ? 2 : 0);
    extern __shared__ __align__(128) unsigned char smem[];
    E *inbuf = reinterpret_cast<E *>(smem);                               // [NBUF][ST]
    long long *gbase = reinterpret_cast<long long *>(inbuf + NBUF * ST);  // [256]
    long long *running = gbase + 256;                                   // [256]
    uint32_t *tdstart = reinterpret_cast<uint32_t *>(running + 256);    // [256]
    uint16_t *whist = reinterpret_cast<uint16_t *>(tdstart + 256);      // STABLE: [NW][F]
    uint32_t *thist = reinterpret_cast<uint32_t *>(tdstart + 256);      // !STABLE: [F] tile histogram
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ uint32_t scan_tmp[32];
    __shared__ TileSlot slots[2];

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int F = a.F;
    const uint64_t dmask = (uint64_t)F - 1;
    const uint32_t nchunks = a.cg.cR + a.cg.cS;
    const uint32_t nitems =
        a.item_end ? a.item_end : (a.pass == 0 ? nchunks * a.cg.spc : nchunks * (uint32_t)a.F1);
    unsigned int *err = &a.counters[kCtrErr];
    const unsigned ltmask = lanemask_lt();
    const uint32_t bar0 = smem_addr(&bars[0]);
    const int nbins = 1 << a.bits;
    const bool ci = a.ci_out && ci_applies(a.counters, a.bits);
    const bool w8o = a.w8_out && w8_fits(a.counters, a.b1);  // pass 1 of the exact pipeline stores words
    const int b2 = a.bits - a.b1;
    if (a.w8 && (a.w8 == 1) != w8_fits(a.counters, a.b1)) return;  // the other layout's launch runs
    __shared__ ItemIter it;  // used by thread 0 only
    uint32_t pend = 0;       // thread 0: next segment of the chain (segment mode)
    ItemAhead ah;            // thread 0: the item claimed ahead
    ah.item = 0;
    ah.stage = 0;
    ah.len = ah.off = 0;
    ah.seg = 0;

    if (!STABLE)
        for (int j = tid; j < 256; j += THREADS) thist[j] = 0;
    if (tid == 0) {
        it = ItemIter();
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (NBUF == 2) {
            const TileSlot s0 = next_tile<T, WIN>(a, it, nitems, pend, ah);
            slots[0] = s0;
            if (s0.item != ~0u && !(a.test_stall && blockIdx.x == 0))
                tma_load_1d(inbuf, s0.in, tile_copy_bytes<E>(s0.cnt + s0.pad), bar0);
        }
    }
    __syncthreads();

    for (uint32_t k = 0;; k++) {
        const uint32_t cur = NBUF == 2 ? (k & 1u) : 0u;
        if (NBUF == 1) {
            // One buffer: load this tile now (the barrier that ended the previous iteration ordered
            // every read of the buffer before this copy).
            if (tid == 0) {
                const TileSlot sn = next_tile<T, WIN>(a, it, nitems, pend, ah);
                slots[0] = sn;
                if (sn.item != ~0u && !(a.test_stall && blockIdx.x == 0 && k == 0))
                    tma_load_1d(inbuf, sn.in, tile_copy_bytes<E>(sn.cnt + sn.pad), bar0);
            }
            __syncthreads();
        }
        const TileSlot sl = slots[cur];
        if (sl.item == ~0u) break;
        E *buf = inbuf + (size_t)cur * ST + sl.pad;
        // Stable ranks: prefetch the next tile into the other buffer now; the barrier that ended the
        // previous iteration ordered every access to it before this copy.
        if (NBUF == 2 && !LATE && tid == 0) {
            const TileSlot sn = next_tile<T, WIN>(a, it, nitems, pend, ah);
            slots[cur ^ 1u] = sn;
            if (sn.item != ~0u)
                tma_load_1d(inbuf + (size_t)(cur ^ 1u) * ST, sn.in, tile_copy_bytes<E>(sn.cnt + sn.pad),
                            bar0 + 8u * (cur ^ 1u));
        }
        // First tile of a work item: load the item's per-digit output offsets.
        if (sl.first && tid < F) {
            long long off;
            if (a.pass == 0) {
                const uint32_t c = sl.item / a.cg.spc;
                off = (long long)(a.unit_off[(size_t)c * a.F1 + tid] + a.subpre[(size_t)sl.item * a.F1 + tid]);
            } else {
                const uint32_t c = sl.item / a.F1, d1 = sl.item % a.F1;
                const int rel = c < a.cg.cR ? 0 : 1;
                const uint32_t v = d1 | ((uint32_t)tid << a.b1);
                off = (long long)(a.start[(size_t)rel * (nbins + 1) + (size_t)d1 * a.F2 + tid] +
                                  a.prefix[(size_t)c * nbins + v]);
            }
            running[tid] = off;
        }
        const uint32_t cnt = sl.cnt;
        const uint32_t par = NBUF == 2 ? ((k >> 1) & 1u) : (k & 1u);
        const bool ok = mbar_wait(bar0 + 8u * cur, par);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                set_error(err, kErrSpinLimit);
                // Before leaving, let every copy this CTA issued land (bounded waits as well): no copy
                // may write into shared memory the CTA no longer owns. The load into this buffer was
                // issued unless the stall hook withheld it (CTA 0's first tile); a prefetch into the
                // other buffer is in flight only with stable ranks (issued above) if it has a tile.
                if (!(a.test_stall && blockIdx.x == 0 && k == 0)) mbar_wait(bar0 + 8u * cur, par);
                if (NBUF == 2 && !LATE && slots[cur ^ 1u].item != ~0u)
                    mbar_wait(bar0 + 8u * (cur ^ 1u), ((k + 1) >> 1) & 1u);
            }
            break;
        }
        // Atomic ranks: prefetch the next tile into the other buffer now. Every thread has passed the
        // barrier above, so the previous tile's staging and write-out, the last accesses to that
        // buffer, are done, and no barrier has to end the iteration.
        if (NBUF == 2 && LATE && tid == 0) {
            const TileSlot sn = next_tile<T, WIN>(a, it, nitems, pend, ah);
            slots[cur ^ 1u] = sn;
            if (sn.item != ~0u)
                tma_load_1d(inbuf + (size_t)(cur ^ 1u) * ST, sn.in, tile_copy_bytes<E>(sn.cnt + sn.pad),
                            bar0 + 8u * (cur ^ 1u));
        }

        // Elements of this tile: warp w owns [w*32*ITEMS, (w+1)*32*ITEMS), one row of 32 per item.
        E v[ITEMS];
        uint32_t d[ITEMS];
        const bool full = cnt == (uint32_t)T;
        if (full) {
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                v[i] = buf[w * 32 * ITEMS + i * 32 + lane];
                if (MIX) elem_mix(v[i], a.bits);
                d[i] = elem_digit(v[i], a.shift, dmask);
            }
        } else {
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const uint32_t idx = (uint32_t)(w * 32 * ITEMS + i * 32 + lane);
                if (idx < cnt) {
                    v[i] = buf[idx];
                    if (MIX) elem_mix(v[i], a.bits);
                    d[i] = elem_digit(v[i], a.shift, dmask);
                } else {
                    v[i] = E{};
                    d[i] = (uint32_t)F;
                }
            }
        }
        uint32_t rk[ITEMS];
        if constexpr (STABLE) {
            uint16_t *wh = whist + w * F;
            for (int j = lane; j < F; j += 32) wh[j] = 0;
            __syncwarp();
            // Stable rank within the warp: items in order, lanes in order. The lanes holding the same
            // digit are found with one ballot per digit bit (plus the bit that marks padding lanes of
            // a partial tile), which is cheaper here than match.any.
            const int nbits = a.logF + (cnt < (uint32_t)T ? 1 : 0);
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                // A row of padding only (a partial tile): nothing to rank (uniform across the warp).
                if ((uint32_t)(w * 32 * ITEMS + i * 32) >= cnt) {
                    rk[i] = 0;
                    continue;
                }
                const unsigned peers = digit_peers_n(d[i], nbits);
                const bool valid = d[i] < (uint32_t)F;
                uint32_t pre = 0;
                if (valid) pre = wh[d[i]];
                rk[i] = pre + __popc(peers & ltmask);
                __syncwarp();
                if (valid && (peers & ltmask) == 0) wh[d[i]] = (uint16_t)(pre + __popc(peers));
                __syncwarp();
            }
            __syncthreads();
            // Tile histogram per digit and exclusive prefix over warps.
            uint32_t h = 0;
            if (tid < F) {
                for (int q = 0; q < NW; q++) {
                    const uint32_t c = whist[q * F + tid];
                    whist[q * F + tid] = (uint16_t)h;
                    h += c;
                }
            }
            const uint32_t ex = block_excl_scan_u32(tid < F ? h : 0u, scan_tmp, nullptr);
            if (tid < F) {
                tdstart[tid] = ex;
                gbase[tid] = running[tid] - (long long)ex;
                running[tid] += h;
            }
        } else {
#pragma unroll
            for (int i = 0; i < ITEMS; i++)
                if (d[i] < (uint32_t)F) rk[i] = atomicAdd(&thist[d[i]], 1u);
            __syncthreads();
            // Warp 0 scans the tile histogram: lane l owns digits [l*K, l*K + K).
            if (w == 0) {
                const int K = (F + 31) >> 5;
                const int d0 = lane * K;
                uint32_t hv[8];
                uint32_t sum = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    hv[j] = (j < K && d0 + j < F) ? thist[d0 + j] : 0u;
                    sum += hv[j];
                }
                uint32_t incl = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                uint32_t ex = incl - sum;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (j < K && d0 + j < F) {
                        const int dd = d0 + j;
                        thist[dd] = 0;
                        tdstart[dd] = ex;
                        const long long r0 = running[dd];
                        gbase[dd] = r0 - (long long)ex;
                        running[dd] = r0 + hv[j];
                        ex += hv[j];
                    }
                }
            }
        }
        __syncthreads();
        // Stage the tile sorted by digit, in place (the digit is recomputed: fewer live registers).
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t idx = (uint32_t)(w * 32 * ITEMS + i * 32 + lane);
            if (full || idx < cnt) {
                const uint32_t di = elem_digit(v[i], a.shift, dmask);
                const uint32_t pos = tdstart[di] + (STABLE ? whist[w * F + di] : 0u) + rk[i];
                buf[pos] = v[i];
            }
        }
        __syncthreads();
        // Write each digit run: consecutive threads write consecutive 16-byte tuples (8-byte words for
        // compact final partitions). Full tiles load their staged tuples in two halves so that the stores
        // issue back to back.
        // A destination outside the output (negative included) fails the unsigned bound check. Build
        // key-0 words exist only for first-match joins (ci_z0), in the launches of the build relation.
        unsigned long long *out8 = sl.out == a.outS ? a.outS8 : a.outR8;
        const bool z0 = a.ci_z0 && sl.out == a.outR;
        if (full) {
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                E t[ITEMS / 2];
                long long dst[ITEMS / 2];
#pragma unroll
                for (int i = 0; i < ITEMS / 2; i++) t[i] = buf[tid + (hh * ITEMS / 2 + i) * THREADS];
#pragma unroll
                for (int i = 0; i < ITEMS / 2; i++)
                    dst[i] = gbase[elem_digit(t[i], a.shift, dmask)] + (long long)(tid + (hh * ITEMS / 2 + i) * THREADS);
#pragma unroll
                for (int i = 0; i < ITEMS / 2; i++) {
                    if ((uint64_t)dst[i] < sl.out_len)
                        store_elem(t[i], sl.out, out8, dst[i], ci, a.bits, b2, z0, w8o, a.b1);
                    else
                        set_error(err, kErrBounds);
                }
            }
        } else
        for (uint32_t j = tid; j < cnt; j += THREADS) {
            const E t = buf[j];
            const long long dst = gbase[elem_digit(t, a.shift, dmask)] + (long long)j;
            if ((uint64_t)dst < sl.out_len)
                store_elem(t, sl.out, out8, dst, ci, a.bits, b2, z0, w8o, a.b1);
            else
                set_error(err, kErrBounds);
        }
        // The next copy into this buffer (at the top of the next iteration with one buffer or stable
        // ranks) must wait for this write-out; otherwise the next tile's wait barrier orders them.
        if (!LATE) __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------
// 4. Partition join in shared memory.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return smem_addr(p); }

// 16-bit exchange on a shared-memory halfword through a 32-bit CAS on its word (lock-free: every
// failed CAS means another thread's CAS succeeded).
__device__ __forceinline__ uint32_t atomic_exch_u16(uint16_t *addr, uint32_t val) {
    uint32_t *word = reinterpret_cast<uint32_t *>(reinterpret_cast<uintptr_t>(addr) & ~(uintptr_t)3);
    const uint32_t shift = (uint32_t)(reinterpret_cast<uintptr_t>(addr) & 2) * 8;
    uint32_t old = *reinterpret_cast<volatile uint32_t *>(word), assumed;
    do {
        assumed = old;
        const uint32_t nw = (assumed & ~(0xffffu << shift)) | (val << shift);
        old = atomicCAS(word, assumed, nw);
    } while (old != assumed);
    return (assumed >> shift) & 0xffffu;
}

// A tuple of a final partition: the stored tuple, or for compact partitions {key >> bits, row id}.
// Joins compare x for equality and hash x >> shift with shift = bits (tuples) or 0 (compact words).
__device__ __forceinline__ tuple_v ld_fin(const tuple_v *p16, const unsigned long long *p8, uint64_t i, bool ci) {
    if (ci) {
        const unsigned long long w = ld_stream8(p8 + i);
        return make_ulonglong2(w >> 32, w & 0xffffffffull);
    }
    return ld_stream(p16 + i);
}

__device__ __forceinline__ tuple_v fin_r(const JoinArgs &a, bool ci, uint64_t i) {
    if (a.lp_pos) {  // y: the input position
        const tuple_v t = a.finR[i];
        return make_ulonglong2(ci ? t.x >> 32 : t.x, t.y);
    }
    if (ci) {
        const unsigned long long w = a.finR8[i];
        return make_ulonglong2(w >> 32, w & 0xffffffffull);
    }
    return a.finR[i];
}

// Chain head among 2^nb_log (1..14) in shared memory of a key's bits above the B lowest (the radix bits): the next
// nb_log bits, changed by a hash of those above (as mix_key), since a partition's keys may share those bits too. Runs
// of keys keep a head each, as without the hash (a hash of all bits cost dense keys in 16-byte tuples 3.5%). Four
// dependent instructions: a probe waits for them.
__device__ __forceinline__ uint32_t head_of(unsigned long long key, int B, uint32_t nb_log) {
    const uint32_t lo = (uint32_t)key, hi = (uint32_t)(key >> 32);
    const uint32_t f = ((lo >> (B + nb_log)) * 0x9e3779b1u + hi * 0x85ebca6bu) >> (32 - nb_log);
    return (__funnelshift_r(lo, hi, B) ^ f) & ((1u << nb_log) - 1u);
}
// log2 of the number of heads for nr build tuples: the next power of two, times two if `twice`, at least 2.
__device__ __forceinline__ uint32_t heads_log(uint32_t nr, bool twice, uint32_t max_log) {
    return min(max_log, max(1u, (nr <= 1 ? 0u : 32u - __clz(nr - 1)) + (twice ? 1u : 0u)));
}

constexpr int kHeadMax = 16384;  // next_pow_2(kSmemCap)
constexpr size_t kJoinSmem = (size_t)kSmemCap * 16 + kHeadMax * 2 + (size_t)kSmemCap * 2;

// The compact table applies when every build key, shifted right by the radix bits, and every build
// row id fit in 32 bits (OR of all of them gathered by the histogram pass).
__device__ __forceinline__ bool compact_applies(const JoinArgs &a) {
    const unsigned long long *mx = reinterpret_cast<const unsigned long long *>(a.counters + kCtrMaxKey);
    return (mx[0] >> a.bits) < (1ull << 32) && mx[1] < (1ull << 32);
}

constexpr size_t kCompactSmem = (size_t)kCompactCap * (4 + 4 + 2 + 2);

// First-match joins: record (acc->dup_flag) that some probe tuple of this block matched two or more
// build tuples. Only then does the first match depend on the order inside a build partition; a join
// whose partition passes ranked the build relation without keeping its input order is then run again
// with ordered passes. Called by every thread of the block.
__device__ __forceinline__ void flag_multi(bool multi, unsigned int *flag) {
    if (__syncthreads_or(multi) && threadIdx.x == 0) atomicOr(flag, 1u);
}

// Partition join with 4-byte keys (key >> bits) and 4-byte row ids in shared memory, packed into one
// 8-byte word per build tuple (key-high << 32 | row id: one load per visited node): 96 KiB per CTA,
// two CTAs per SM, so one CTA's build overlaps the other's probe. Same results as join_small_kernel;
// within a partition the low `bits` key bits are equal, so comparing key >> bits is comparing keys.
// MAT: write one (r.row_id, s.row_id) pair per match (the ptr_* joins) instead of summing; the probe
// then runs in block-wide rounds (count, reserve output slots, walk again and write). LP: first match
// (the lowest build position) per probe tuple.
template <bool MAT, bool CI = false, bool LP = false>
__global__ void __launch_bounds__(kCompactThreads, 2) join_compact_kernel(JoinArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned long long *rw = reinterpret_cast<unsigned long long *>(smem);  // [kCompactCap]
    uint16_t *head = reinterpret_cast<uint16_t *>(rw + kCompactCap);         // [kCompactCap]
    uint16_t *nxt = head + kCompactCap;                                      // [kCompactCap]
    __shared__ unsigned long long red[64];
    __shared__ uint32_t s_item;
    __shared__ uint32_t scan_tmp[32];
    __shared__ unsigned long long s_base;
    if (!compact_applies(a)) return;
    const int tid = threadIdx.x;
    unsigned int *err = &a.counters[kCtrErr];
    const uint32_t nA = a.counters[kCtrNItemsA];
    // Compiled once per partition layout; only the launch matching the device's choice runs.
    if (CI != (a.ci && ci_applies(a.counters, a.bits))) return;
    constexpr bool ci = CI;
    const int B = ci ? 0 : a.bits;  // shift from a stored x to the key's bits above the radix bits
    constexpr bool lp = LP;
    const bool skip0 = a.skip0 != 0;
    unsigned long long cnt = 0, sum = 0;
    bool multi = false;  // first-match joins: a probe tuple matched two build tuples
    for (;;) {
        if (tid == 0) s_item = atomicAdd(&a.counters[kCtrItemA], 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= nA) break;
        const JoinItem item = a.items[it];
        const uint32_t nr = item.r_len;
        const uint32_t nb_log = heads_log(nr, false, 13);
        uint32_t *head32 = reinterpret_cast<uint32_t *>(head);
        for (uint32_t q = tid; q < (1u << nb_log) / 2; q += kCompactThreads) head32[q] = 0;
        __syncthreads();
        // Load and chain the build side; lp_join skips key 0, which reads as an empty slot there (in
        // compact final partitions such a key's words have a high part that no probe word has).
        const tuple_v *R = a.finR + item.r_begin;
        const unsigned long long *R8 = a.finR8 + item.r_begin;
        for (uint32_t i0 = tid; i0 < nr; i0 += 4 * kCompactThreads) {
            tuple_v t[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t i = i0 + u * kCompactThreads;
                t[u] = i < nr ? ld_fin(R, R8, i, ci) : make_ulonglong2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t i = i0 + u * kCompactThreads;
                if (i >= nr) continue;
                rw[i] = ((t[u].x >> B) << 32) | (t[u].y & 0xffffffffull);
                if (skip0 && t[u].x == 0 && (!ci || item.part0)) continue;
                nxt[i] = (uint16_t)atomic_exch_u16(&head[head_of(t[u].x >> B, 0, nb_log)], i + 1);
            }
        }
        __syncthreads();
        const tuple_v *S = a.finS + item.s_begin;
        const unsigned long long *S8 = a.finS8 + item.s_begin;
        const uint32_t ns = item.s_len;
        if constexpr (MAT) {
            constexpr int U = 4;  // probe tuples per thread and round: loads in flight, fewer rounds
            for (uint32_t base = 0; base < ns; base += U * kCompactThreads) {
                tuple_v sv[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t j = base + u * kCompactThreads + tid;
                    sv[u] = j < ns ? ld_stream(S + j) : make_ulonglong2(0, 0);
                }
                uint32_t mm[U], best[U], m = 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    mm[u] = best[u] = 0;
                    if (base + u * kCompactThreads + tid >= ns) continue;
                    const uint64_t khi = sv[u].x >> B;
                    uint32_t e = head[head_of(khi, 0, nb_log)], steps = 0;
                    while (e) {
                        if ((rw[e - 1] >> 32) == khi) {
                            if (!lp) mm[u]++;
                            else if (best[u] == 0 || e < best[u]) best[u] = e;
                        }
                        e = nxt[e - 1];
                        if (++steps > nr) {
                            set_error(err, kErrProbeLimit);
                            break;
                        }
                    }
                    if (lp) mm[u] = best[u] ? 1u : 0u;
                    m += mm[u];
                }
                unsigned long long o = mat_reserve(m, scan_tmp, &s_base, &a.acc->pairs);
                cnt += m;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (!mm[u]) continue;
                    if (lp) {
                        mat_put(a.mat, o++, rw[best[u] - 1] & 0xffffffffull, sv[u].y, err);
                        continue;
                    }
                    const uint64_t khi = sv[u].x >> B;
                    uint32_t e = head[head_of(khi, 0, nb_log)], steps = 0;
                    while (e && steps++ <= nr) {
                        const unsigned long long w = rw[e - 1];
                        if ((w >> 32) == khi) mat_put(a.mat, o++, w & 0xffffffffull, sv[u].y, err);
                        e = nxt[e - 1];
                    }
                }
            }
        } else
        // Eight probe tuples per thread in flight (four left the DRAM queue short: 2.01 -> 1.92 ms
        // for the headline join phase).
        for (uint32_t j0 = tid; j0 < ns; j0 += 8 * kCompactThreads) {
            tuple_v sv[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint32_t j = j0 + u * kCompactThreads;
                sv[u] = j < ns ? ld_fin(S, S8, j, ci) : make_ulonglong2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const uint32_t j = j0 + u * kCompactThreads;
                if (j >= ns) continue;
                const uint64_t khi = sv[u].x >> B;
                uint32_t e = head[head_of(khi, 0, nb_log)];
                uint32_t best = 0, steps = 0, nm = 0;
                while (e) {
                    const unsigned long long w = rw[e - 1];
                    if ((w >> 32) == khi) {
                        if (lp) {
                            if (best == 0 || e < best) best = e;
                            nm++;
                        } else {
                            cnt++;
                            sum += (w & 0xffffffffull) + sv[u].y;
                        }
                    }
                    e = nxt[e - 1];
                    if (++steps > nr) {
                        set_error(err, kErrProbeLimit);
                        break;
                    }
                }
                if (lp && best) {
                    cnt++;
                    sum += (rw[best - 1] & 0xffffffffull) + sv[u].y;
                    multi |= nm > 1;
                }
            }
        }
        __syncthreads();
    }
    block_sum2_to(cnt, sum, red, &a.acc->matched, &a.acc->checksum);
    if (LP && !MAT) flag_multi(multi, &a.acc->dup_flag);
}

// End of the one-pass pipeline's partition join, called by every thread of every CTA after it has added its
// sums to *a.acc. With host_out, the CTA that finishes last writes the join's result there (pinned host
// memory), so that nothing has to be copied or launched after the join unless there are large partitions.
__device__ __forceinline__ void join_finish(const JoinArgs &a, bool ci) {
    if (!a.host_out || threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&a.counters[kCtrTicketJoin], 1u) != gridDim.x - 1) return;
    __threadfence();
    const volatile JoinAccum *acc = a.acc;
    JoinAccum r = {};
    r.matched = acc->matched;
    r.checksum = acc->checksum;
    r.error = acc->error | *reinterpret_cast<const volatile uint32_t *>(&a.counters[kCtrErr]);
    r.dup_flag = acc->dup_flag;
    r.large_parts = a.counters[kCtrNLarge];
    r.large_build = ld_u64_pair(&a.counters[kCtrLargeR]);
    if (a.ci && ci_applies(a.counters, a.flag_bits)) r.flags = HJ_RES_COMPACT_PARTITIONS;
    *a.host_out = r;
    // Large partitions add to the result after this: start them from zero.
    a.acc->matched = a.acc->checksum = 0;
    a.acc->dup_flag = a.acc->error = 0;
}

// Large-partition steps 0 (clear) and 1 (build) of a wave's job, by the blocks of its partition joins, which come as
// two launches (one per element layout): the first clears, the second builds, multi_large probes.
__device__ __noinline__ void multi_large_step(const JoinArgs &a, int step, uint32_t blk, uint32_t nblk);

// Partition join over compact words in an open-addressing table of the words themselves (every match
// counted): two CTAs of 512 threads per SM with 13312 slots each. A probe is one 8-byte shared load when its
// key sits in its first slot and the build saw no key twice, where a chain costs a head, a word and a link.
// Slots come from the high product of a multiplicative hash, so the table takes any size: twice the build
// partition (less for the largest, 10240 tuples). A thread walks for four probe words per round (8: 1240 us for
// 2^27 x 2^29 tuples, 4: 1200, 2: 1378: more overlaps more loads, less lets the warps drift apart).
// Equal keys sit in a row; a build that walks more than
// kOaMaxSteps slots (a key repeated often) is done again with chains in the same memory.
constexpr uint32_t kOaSlots = 13312, kOaMaxSteps = 64, kOaHeads = 2048;
constexpr size_t kOaSmem = (size_t)kOaSlots * 8;
static_assert(kOaSmem >= (size_t)kSmemCap * 10 + kOaHeads * 2, "the chains fit the same memory");

__device__ __forceinline__ uint32_t oa_hash(uint32_t hi) { return hi * 0x9e3779b1u; }

// Matches of probe word s in an open-addressing table of build words.
__device__ __forceinline__ uint32_t oa_matches(const unsigned long long *slots, uint32_t nslots, unsigned long long s) {
    const uint32_t hi = (uint32_t)(s >> 32);
    uint32_t h = __umulhi(oa_hash(hi), nslots), m = 0;
    for (uint32_t steps = 0; steps < nslots; steps++) {
        const unsigned long long e = slots[h];
        if (e == ~0ull) break;
        m += (uint32_t)(e >> 32) == hi;
        if (++h == nslots) h = 0;
    }
    return m;
}

// The first build word that matches, or ~0.
__device__ __forceinline__ unsigned long long oa_find(const unsigned long long *slots, uint32_t nslots,
                                                      unsigned long long s) {
    const uint32_t hi = (uint32_t)(s >> 32);
    uint32_t h = __umulhi(oa_hash(hi), nslots);
    for (uint32_t steps = 0; steps < nslots; steps++) {
        const unsigned long long e = slots[h];
        if (e == ~0ull || (uint32_t)(e >> 32) == hi) return e;
        if (++h == nslots) h = 0;
    }
    return ~0ull;
}

// One round of a materialising probe with at most one match per probe tuple: the matches' pairs (row ids of
// build word e[u] and probe word s[u]; e[u] = ~0: none) go to consecutive output slots per warp and u.
struct MatRound {
    uint32_t count[32], at[32];  // a warp's pairs of the round, its start among them
    unsigned long long base;     // the round's first output slot
};

template <int U, int NT>
__device__ __forceinline__ void mat_write_round(MatRound &r, const unsigned long long (&e)[U],
                                                const unsigned long long (&s)[U], const MatOut &out,
                                                unsigned long long *cursor, unsigned int *err) {
    const unsigned lane = lane_id(), w = threadIdx.x >> 5;
    unsigned masks[U], total = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
        masks[u] = __ballot_sync(0xffffffffu, e[u] != ~0ull);
        total += __popc(masks[u]);
    }
    if (lane == 0) r.count[w] = total;
    __syncthreads();
    if (w == 0) {
        const uint32_t x = lane < (unsigned)(NT / 32) ? r.count[lane] : 0u;
        uint32_t incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (unsigned)o) incl += y;
        }
        r.at[lane] = incl - x;
        if (lane == 31) r.base = incl ? atomicAdd(cursor, (unsigned long long)incl) : 0ull;
    }
    __syncthreads();
    unsigned long long o = r.base + r.at[w];
#pragma unroll
    for (int u = 0; u < U; u++) {
        if (e[u] != ~0ull)
            mat_put(out, o + __popc(masks[u] & lanemask_lt()), e[u] & 0xffffffffull, s[u] & 0xffffffffull, err);
        o += __popc(masks[u]);
    }
}

// MAT: one pair per match. Without repeated build keys a probe has at most one match, and the block reserves
// output for a round of eight probes per thread by ballots, so a warp writes consecutive pairs.
// LP: the unordered run of a first-match join: one match per probe tuple, whichever comes first; a probe tuple
// with a second one sets acc->dup_flag, and the join runs again in order. Build key 0 never matches (skip0).
template <bool MULTI, bool MAT = false, bool LP = false>
__global__ void __launch_bounds__(kCompactThreads, 2) join_words_kernel(JoinArgs a0, MultiRef mr) {
    __shared__ JoinArgs s_a;
    if (MULTI) {
        const uint2 e = mr.map[blockIdx.x];
        multi_copy(&s_a, &mr.jobs[e.x].ja);
        __syncthreads();
        multi_large_step(s_a, 0, e.y, mr.jobs[e.x].join_blocks);
    }
    const JoinArgs &a = MULTI ? s_a : a0;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned long long *slots = reinterpret_cast<unsigned long long *>(smem);
    __shared__ unsigned long long red[64];
    __shared__ uint32_t s_item, s_flags;  // s_flags: 1 a key occurs twice, 2 a walk was too long
    __shared__ MatRound mat_round;
    __shared__ uint32_t scan_tmp[32];
    __shared__ unsigned long long s_base;
    if (!(a.ci && ci_applies(a.counters, a.bits))) return;
    const int tid = threadIdx.x;
    constexpr int NT = kCompactThreads, UR = 4, U = 4;
    constexpr unsigned long long kNone = ~0ull;  // no build word has this high part
    unsigned int *err = &a.counters[kCtrErr];
    const uint32_t nitems = a.counters[kCtrNItems];
    unsigned long long cnt = 0, sum = 0;
    bool multi = false;
    for (;;) {
        if (tid == 0) {
            s_item = atomicAdd(&a.counters[kCtrItemA], 1u);
            s_flags = 0;
        }
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= nitems) break;
        const JoinItem item = a.items[it];
        const uint32_t nr = item.r_len, ns = item.s_len;
        const unsigned long long *R8 = a.finR8 + item.r_begin, *S8 = a.finS8 + item.s_begin;
        const uint32_t nslots = min(kOaSlots, (2 * nr + 511u) & ~511u);
        unsigned long long r[UR], s[U];
#pragma unroll
        for (int u = 0; u < UR; u++) r[u] = tid + u * NT < nr ? ld_stream8(R8 + tid + u * NT) : kNone;
        for (uint32_t q = tid; q < nslots / 2; q += NT) reinterpret_cast<ulonglong2 *>(slots)[q] = make_ulonglong2(kNone, kNone);
        __syncthreads();
        uint32_t fl = 0;
        for (uint32_t i0 = tid; i0 < nr; i0 += UR * NT) {
            unsigned long long nx[UR];
#pragma unroll
            for (int u = 0; u < UR; u++) {
                const uint32_t i = i0 + (UR + u) * NT;
                nx[u] = i < nr ? ld_stream8(R8 + i) : kNone;
            }
#pragma unroll
            for (int u = 0; u < UR; u++) {
                if (r[u] == kNone) continue;
                const uint32_t hi = (uint32_t)(r[u] >> 32);
                if (LP && a.skip0 && item.part0 && hi == 0) continue;
                uint32_t h = __umulhi(oa_hash(hi), nslots);
                for (uint32_t steps = 0;;) {
                    const unsigned long long cur = atomicCAS(&slots[h], kNone, r[u]);
                    if (cur == kNone) break;
                    if ((uint32_t)(cur >> 32) == hi) fl |= 1u;
                    if (++h == nslots) h = 0;
                    if (++steps >= kOaMaxSteps) {
                        fl |= 2u;
                        break;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < UR; u++) r[u] = nx[u];
        }
#pragma unroll
        for (int u = 0; u < U; u++) s[u] = tid + u * NT < ns ? ld_stream8(S8 + tid + u * NT) : kNone;
        if (fl) atomicOr(&s_flags, fl);
        __syncthreads();
        const bool dups = s_flags != 0;
        if (s_flags & 2u) {
            // Chains: words, links by position, bucket heads.
            uint16_t *nxt = reinterpret_cast<uint16_t *>(slots + kSmemCap), *head = nxt + kSmemCap;
            uint32_t *head32 = reinterpret_cast<uint32_t *>(head);
            for (uint32_t q = tid; q < kOaHeads / 2; q += NT) head32[q] = 0;
            __syncthreads();
            for (uint32_t i = tid; i < nr; i += NT) {
                const unsigned long long w = R8[i];
                slots[i] = w;
                if (LP && a.skip0 && item.part0 && (w >> 32) == 0) continue;
                nxt[i] = (uint16_t)atomic_exch_u16(&head[oa_hash((uint32_t)(w >> 32)) >> 21], i + 1);
            }
            __syncthreads();
            if constexpr (MAT) {
                // Count, reserve, walk again and write.
                for (uint32_t base = 0; base < ns; base += NT) {
                    const uint32_t j = base + tid;
                    const unsigned long long w = j < ns ? ld_stream8(S8 + j) : kNone;
                    const uint32_t hi = (uint32_t)(w >> 32), e0 = j < ns ? head[oa_hash(hi) >> 21] : 0u;
                    uint32_t m = 0, steps = 0;
                    for (uint32_t e = e0; e && steps++ < nr; e = nxt[e - 1]) m += (uint32_t)(slots[e - 1] >> 32) == hi;
                    unsigned long long o = mat_reserve(m, scan_tmp, &s_base, &a.acc->pairs);
                    cnt += m;
                    steps = 0;
                    for (uint32_t e = e0; e && steps++ < nr; e = nxt[e - 1])
                        if ((uint32_t)(slots[e - 1] >> 32) == hi)
                            mat_put(a.mat, o++, slots[e - 1] & 0xffffffffull, w & 0xffffffffull, err);
                }
                __syncthreads();
                continue;
            }
            for (uint32_t j = tid; j < ns; j += NT) {
                const unsigned long long w = ld_stream8(S8 + j);
                const uint32_t hi = (uint32_t)(w >> 32);
                uint32_t steps = 0;
                bool found = false;
                for (uint32_t e = head[oa_hash(hi) >> 21]; e; e = nxt[e - 1]) {
                    const unsigned long long b = slots[e - 1];
                    if ((uint32_t)(b >> 32) == hi) {
                        if (LP && found) {
                            multi = true;
                            break;
                        }
                        found = true;
                        cnt++;
                        sum += (b & 0xffffffffull) + (w & 0xffffffffull);
                    }
                    if (++steps > nr) {
                        set_error(err, kErrProbeLimit);
                        break;
                    }
                }
            }
            __syncthreads();
            continue;
        }
        if constexpr (MAT) {
            for (uint32_t base = 0; base < ns; base += U * NT) {  // the same rounds for every thread
                unsigned long long nx[U], e[U];
                uint32_t m = 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t j = base + tid + (U + u) * NT;
                    nx[u] = j < ns ? ld_stream8(S8 + j) : kNone;
                }
                if (dups) {
#pragma unroll
                    for (int u = 0; u < U; u++) m += oa_matches(slots, nslots, s[u]);
                    unsigned long long o = mat_reserve(m, scan_tmp, &s_base, &a.acc->pairs);
                    cnt += m;
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const uint32_t hi = (uint32_t)(s[u] >> 32);
                        uint32_t h = __umulhi(oa_hash(hi), nslots);
                        for (uint32_t steps = 0; steps < nslots && slots[h] != kNone; steps++) {
                            if ((uint32_t)(slots[h] >> 32) == hi)
                                mat_put(a.mat, o++, slots[h] & 0xffffffffull, s[u] & 0xffffffffull, err);
                            if (++h == nslots) h = 0;
                        }
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < U; u++) e[u] = oa_find(slots, nslots, s[u]);
                    mat_write_round<U, NT>(mat_round, e, s, a.mat, &a.acc->pairs, err);
#pragma unroll
                    for (int u = 0; u < U; u++) cnt += e[u] != kNone;
                }
#pragma unroll
                for (int u = 0; u < U; u++) s[u] = nx[u];
            }
        } else
        for (uint32_t j0 = tid; j0 < ns; j0 += U * NT) {
            unsigned long long nx[U], e[U];
            uint32_t h[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t j = j0 + (U + u) * NT;
                nx[u] = j < ns ? ld_stream8(S8 + j) : kNone;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                h[u] = __umulhi(oa_hash((uint32_t)(s[u] >> 32)), nslots);
                e[u] = slots[h[u]];
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t hi = (uint32_t)(s[u] >> 32);
                // A word past the end (kNone), as a probe key beyond every build key, matches nothing.
                bool found = false;
                for (uint32_t steps = 0; e[u] != kNone;) {
                    if ((uint32_t)(e[u] >> 32) == hi) {
                        if (LP && found) {
                            multi = true;
                            break;
                        }
                        found = true;
                        cnt++;
                        sum += (e[u] & 0xffffffffull) + (s[u] & 0xffffffffull);
                        if (!dups) break;
                    }
                    if (++h[u] == nslots) h[u] = 0;
                    if (++steps >= nslots) {
                        set_error(err, kErrProbeLimit);
                        break;
                    }
                    e[u] = slots[h[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) s[u] = nx[u];
        }
        __syncthreads();
    }
    block_sum2_to(cnt, sum, red, &a.acc->matched, &a.acc->checksum);
    if (LP) flag_multi(multi, &a.acc->dup_flag);
    join_finish(a, true);
}

// First-match join over {compact word, position} elements in an open-addressing table: a slot holds (key
// high part << 32 | position), equal keys share a slot and lower its position, and the row ids of the winners
// stand beside the slots. Equal keys never lengthen a walk. A bitmap marks the slots that two build tuples
// share: a probe that matches one sets acc->dup_flag (see flag_multi). One CTA of 1024 threads per SM, 194 KB;
// a thread keeps its build tuples in registers from the insert to the row-id store. Probes in rounds of four
// (8: 280 us for 2^24 x 2^26 tuples, 4: 244, 2: 264).
constexpr uint32_t kFwSlots = 16384;
constexpr size_t kFwSmem = (size_t)kFwSlots * 12 + kFwSlots / 8;

template <bool MULTI, bool MAT = false>
__global__ void __launch_bounds__(kJoinThreads, 1) join_first_words_kernel(JoinArgs a0, MultiRef mr) {
    __shared__ JoinArgs s_a;
    if (MULTI) {
        const uint2 e = mr.map[blockIdx.x];
        multi_copy(&s_a, &mr.jobs[e.x].ja);
        __syncthreads();
        multi_large_step(s_a, 0, e.y, mr.jobs[e.x].join_blocks);
    }
    const JoinArgs &a = MULTI ? s_a : a0;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned long long *slots = reinterpret_cast<unsigned long long *>(smem);  // [kFwSlots]
    uint32_t *rid = reinterpret_cast<uint32_t *>(slots + kFwSlots);             // [kFwSlots]
    uint32_t *dup = rid + kFwSlots;                                             // [kFwSlots / 32]
    __shared__ unsigned long long red[64];
    __shared__ uint32_t s_item, s_dups;
    __shared__ MatRound mat_round;
    if (!(a.ci && ci_applies(a.counters, a.bits))) return;
    const uint32_t tid = threadIdx.x;
    constexpr int NT = kJoinThreads, UR = kFirstCap / NT, U = 4;
    static_assert(UR * NT == kFirstCap, "a thread's build tuples");
    constexpr unsigned long long kNone = ~0ull;  // no build element has this high part
    unsigned int *err = &a.counters[kCtrErr];
    const uint32_t nitems = a.counters[kCtrNItems];
    unsigned long long cnt = 0, sum = 0;
    bool multi = false;
    for (;;) {
        if (tid == 0) {
            s_item = atomicAdd(&a.counters[kCtrItemA], 1u);
            s_dups = 0;
        }
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= nitems) break;
        const JoinItem item = a.items[it];
        const uint32_t nr = item.r_len, ns = item.s_len;
        const tuple_v *R = a.finR + item.r_begin;
        const unsigned long long *S8 = a.finS8 + item.s_begin;
        const uint32_t nslots = min(kFwSlots, (2 * nr + 511u) & ~511u);
        tuple_v r[UR];
#pragma unroll
        for (int u = 0; u < UR; u++)
            r[u] = tid + u * NT < nr ? ld_stream(R + tid + u * NT) : make_ulonglong2(kNone, 0);
        for (uint32_t q = tid; q < nslots / 2; q += NT) reinterpret_cast<ulonglong2 *>(slots)[q] = make_ulonglong2(kNone, kNone);
        for (uint32_t q = tid; q < nslots / 32; q += NT) dup[q] = 0;
        __syncthreads();
        uint32_t at[UR];
        bool any_dup = false;
#pragma unroll
        for (int u = 0; u < UR; u++) {
            at[u] = ~0u;
            if (r[u].x == kNone) continue;
            const uint32_t hi = (uint32_t)(r[u].x >> 32);
            const unsigned long long v = ((unsigned long long)hi << 32) | (uint32_t)r[u].y;
            uint32_t h = __umulhi(oa_hash(hi), nslots);
            for (uint32_t steps = 0;;) {
                const unsigned long long cur = atomicCAS(&slots[h], kNone, v);
                if (cur == kNone) break;
                if ((uint32_t)(cur >> 32) == hi) {
                    atomicMin(&slots[h], v);
                    atomicOr(&dup[h >> 5], 1u << (h & 31));
                    any_dup = true;
                    break;
                }
                if (++h == nslots) h = 0;
                if (++steps >= nslots) {
                    set_error(err, kErrProbeLimit);
                    break;
                }
            }
            at[u] = h;
        }
        unsigned long long s[U];
#pragma unroll
        for (int u = 0; u < U; u++) s[u] = tid + u * NT < ns ? ld_stream8(S8 + tid + u * NT) : kNone;
        if (any_dup) s_dups = 1u;
        __syncthreads();
        // The tuple whose position won its slot stores its row id there.
#pragma unroll
        for (int u = 0; u < UR; u++)
            if (at[u] != ~0u && (uint32_t)slots[at[u]] == (uint32_t)r[u].y) rid[at[u]] = (uint32_t)r[u].x;
        const bool dups = s_dups != 0;
        __syncthreads();
        if constexpr (MAT) {
            for (uint32_t base = 0; base < ns; base += U * NT) {  // the same rounds for every thread
                unsigned long long nx[U], e[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t j = base + tid + (U + u) * NT;
                    nx[u] = j < ns ? ld_stream8(S8 + j) : kNone;
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t hi = (uint32_t)(s[u] >> 32);
                    uint32_t h = __umulhi(oa_hash(hi), nslots);
                    e[u] = kNone;
                    for (uint32_t steps = 0; steps < nslots && slots[h] != kNone; steps++) {
                        if ((uint32_t)(slots[h] >> 32) == hi) {
                            e[u] = rid[h];
                            break;
                        }
                        if (++h == nslots) h = 0;
                    }
                }
                mat_write_round<U, NT>(mat_round, e, s, a.mat, &a.acc->pairs, err);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    cnt += e[u] != kNone;
                    s[u] = nx[u];
                }
            }
        } else
        for (uint32_t j0 = tid; j0 < ns; j0 += U * NT) {
            unsigned long long nx[U], e[U];
            uint32_t h[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t j = j0 + (U + u) * NT;
                nx[u] = j < ns ? ld_stream8(S8 + j) : kNone;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                h[u] = __umulhi(oa_hash((uint32_t)(s[u] >> 32)), nslots);
                e[u] = slots[h[u]];
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t hi = (uint32_t)(s[u] >> 32);
                for (uint32_t steps = 0; e[u] != kNone;) {
                    if ((uint32_t)(e[u] >> 32) == hi) {
                        cnt++;
                        sum += (unsigned long long)rid[h[u]] + (s[u] & 0xffffffffull);
                        if (dups) multi |= (dup[h[u] >> 5] >> (h[u] & 31)) & 1u;
                        break;
                    }
                    if (++h[u] == nslots) h[u] = 0;
                    if (++steps >= nslots) {
                        set_error(err, kErrProbeLimit);
                        break;
                    }
                    e[u] = slots[h[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) s[u] = nx[u];
        }
        __syncthreads();
    }
    block_sum2_to(cnt, sum, red, &a.acc->matched, &a.acc->checksum);
    if (!MAT) flag_multi(multi, &a.acc->dup_flag);
    join_finish(a, true);
}

// First-match join of the one-pass pipeline over {key, position} elements (wide). The match with the lowest
// position wins, so the partition may hold them in any order. Key, position and row id in
// separate arrays (20 bytes per build tuple, 16-bit bucket heads and chains: 215 KB, one CTA per SM);
// a build tuple's row id is gathered from the build relation once. A build tuple that loses a head to its own key
// lowers that node's position instead of becoming a node, and flags the partition, which happens where a key is
// repeated a few dozen times; first_merge then leaves one node per key, with its first position and row id, and a
// bit that there were more. Fewer duplicates are walked. (2^22 x 2^24 tuples of mixed 63-bit keys, 4 / 1000 a key:
// 615 / 18300 us with every duplicate walked, 601 / 632 now; 2^21 x 2^22 with one key 1000 times and half of the
// probes on it: 7680 and 200 us, the global table 2040. Distinct keys, 3e6 x 9e6: 147 and 151 us for this join; a
// look at the head's key before each insert 163, at the whole chain 170, walks measured in the probe 165.) One
// probe tuple per round, the next one under way (3e6 x 12e6 sparse keys: 166 us; four unrolled: 175).
constexpr uint32_t kFirstHeadsLog = 13, kFirstHeads = 1u << kFirstHeadsLog;
constexpr size_t kFirstSmem = (size_t)kFirstCap * (8 + 8 + 4 + 2) + kFirstHeads * 2 + kFirstCap / 8;
constexpr uint32_t kFirstMerged = 0x8000;  // nxt of a tuple merged into a node: this bit, and the node's index + 1
static_assert(kFirstCap < kFirstMerged && kFirstCap % 32 == 0, "an index and the bit fit a link");

struct FirstTable {  // the table of join_first_kernel
    unsigned long long *kx, *rid;
    uint32_t *pos, *dup;
    uint16_t *head, *nxt;
    uint32_t nr, nb_log;
    bool skip0;
};

// One node per key: the others of a chain leave it, and the node takes the first position among them and its row id. A
// thread per head; all threads of the block, before a probe walks.
__device__ __noinline__ void first_merge(const FirstTable &t) {
    unsigned long long *kx = t.kx, *rid = t.rid;
    uint32_t *pos = t.pos, *dup = t.dup;
    uint16_t *head = t.head, *nxt = t.nxt;
    const uint32_t nr = t.nr, nb_log = t.nb_log, tid = threadIdx.x;
    const bool skip0 = t.skip0;
    // Row ids of the tuples whose position won, and duplicate bits; then what is left of one key in a
    // chain (nodes that were not next to each other).
    for (uint32_t i = tid; i < nr; i += kJoinThreads) {
        const uint32_t e = nxt[i];
        if (!(e & kFirstMerged) || (skip0 && kx[i] == 0)) continue;
        const uint32_t r = (e & (kFirstMerged - 1)) - 1;
        if (pos[r] == pos[i]) rid[r] = rid[i];
        atomicOr(&dup[r >> 5], 1u << (r & 31));
    }
    __syncthreads();
    for (uint32_t q = tid; q < 1u << nb_log; q += kJoinThreads) {
        for (uint32_t r = head[q]; r; r = nxt[r - 1]) {
            // Take the nodes behind r with its key out of the chain.
            const unsigned long long k = kx[r - 1];
            uint32_t prev = r, first = r, fp = pos[r - 1];
            bool gap = false, any = false;  // any: bits of the nodes taken out pass to r
            for (uint32_t e = nxt[r - 1], next; e; e = next) {
                const uint32_t p = pos[e - 1];
                next = nxt[e - 1];
                if (kx[e - 1] == k) {
                    gap = any = true;
                    if (p < fp) {
                        fp = p;
                        first = e;
                    }
                } else {
                    if (gap) nxt[prev - 1] = (uint16_t)e;
                    gap = false;
                    prev = e;
                }
            }
            if (gap) nxt[prev - 1] = 0;
            if (any) {
                pos[r - 1] = fp;
                rid[r - 1] = rid[first - 1];
                atomicOr(&dup[(r - 1) >> 5], 1u << ((r - 1) & 31));
            }
        }
    }
    __syncthreads();
}

template <bool MAT, bool MULTI = false>
__global__ void __launch_bounds__(kJoinThreads, 1) join_first_kernel(JoinArgs a0, MultiRef mr) {
    __shared__ JoinArgs s_a;
    if (MULTI) {
        const uint2 e = mr.map[blockIdx.x];
        multi_copy(&s_a, &mr.jobs[e.x].ja);
        __syncthreads();
        multi_large_step(s_a, 1, e.y, mr.jobs[e.x].join_blocks);
    }
    const JoinArgs &a = MULTI ? s_a : a0;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned long long *kx = reinterpret_cast<unsigned long long *>(smem);  // [kFirstCap] keys
    unsigned long long *rid = kx + kFirstCap;                              // [kFirstCap]
    uint32_t *pos = reinterpret_cast<uint32_t *>(rid + kFirstCap);         // [kFirstCap]
    uint16_t *head = reinterpret_cast<uint16_t *>(pos + kFirstCap);        // [kFirstHeads]
    uint16_t *nxt = head + kFirstHeads;                                    // [kFirstCap]
    uint32_t *dup = reinterpret_cast<uint32_t *>(nxt + kFirstCap);         // [kFirstCap / 32]
    __shared__ unsigned long long red[64];
    __shared__ uint32_t s_item, s_dups;
    __shared__ uint32_t scan_tmp[32];
    __shared__ unsigned long long s_base;
    const int tid = threadIdx.x;
    unsigned int *err = &a.counters[kCtrErr];
    const uint32_t nitems = a.counters[kCtrNItems];
    if (a.ci && ci_applies(a.counters, a.bits)) return;  // join_first_words_kernel
    const int B = a.bits;
    const bool skip0 = a.skip0 != 0;
    unsigned long long cnt = 0, sum = 0;
    bool multi = false;
    constexpr int U = 4, UP = MAT ? 4 : 1;  // build and probe tuples per thread and round
    for (;;) {
        if (tid == 0) {
            s_item = atomicAdd(&a.counters[kCtrItemA], 1u);
            s_dups = 0;
        }
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= nitems) break;
        const JoinItem item = a.items[it];
        const uint32_t nr = item.r_len;
        const uint32_t nb_log = heads_log(nr, false, kFirstHeadsLog);
        uint32_t *head32 = reinterpret_cast<uint32_t *>(head);
        for (uint32_t q = tid; q < (1u << nb_log) / 2; q += kJoinThreads) head32[q] = 0;
        for (uint32_t q = tid; q < (nr + 31) / 32; q += kJoinThreads) dup[q] = 0;
        __syncthreads();
        const tuple_v *R = a.finR + item.r_begin, *S = a.finS + item.s_begin;
        const uint32_t ns = item.s_len;
        tuple_v sv[UP];  // the thread's next probe tuples, under way during the build and the walks before them
#pragma unroll
        for (int u = 0; u < UP; u++) sv[u] = tid + u * kJoinThreads < ns ? ld_stream(S + tid + u * kJoinThreads) : make_ulonglong2(0, 0);
        bool twice = false;
        for (uint32_t i0 = tid; i0 < nr; i0 += U * kJoinThreads) {
            tuple_v t[U];
            unsigned long long y[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t i = i0 + u * kJoinThreads;
                t[u] = i < nr ? ld_stream(R + i) : make_ulonglong2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const bool live = i0 + u * kJoinThreads < nr && t[u].y < a.nR;
                y[u] = live ? a.relR[t[u].y].y : 0ull;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t i = i0 + u * kJoinThreads;
                if (i >= nr) continue;
                kx[i] = t[u].x;
                rid[i] = y[u];
                pos[i] = (uint32_t)t[u].y;
            }
            __threadfence_block();  // before these become heads: a thread that loses a head reads its key
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t i = i0 + u * kJoinThreads;
                const unsigned long long k = t[u].x;
                if (i >= nr || (skip0 && k == 0)) continue;
                const uint32_t h = head_of(k, B, nb_log), shift = (h & 1) * 16;
                uint32_t *word = head32 + (h >> 1);
                uint32_t old = *reinterpret_cast<volatile uint32_t *>(word), e;
                for (;;) {  // lock-free: a failed CAS means another thread's succeeded
                    e = (old >> shift) & 0xffffu;
                    const uint32_t seen = atomicCAS(word, old, (old & ~(0xffffu << shift)) | ((i + 1) << shift));
                    if (seen == old) break;
                    __threadfence_block();
                    old = seen;
                    e = (seen >> shift) & 0xffffu;
                    if (e && *reinterpret_cast<volatile unsigned long long *>(&kx[e - 1]) == k) {
                        atomicMin(&pos[e - 1], (uint32_t)t[u].y);
                        e |= kFirstMerged;
                        twice = true;
                        break;
                    }
                }
                nxt[i] = (uint16_t)e;
            }
        }
        if (twice) s_dups = 1u;
        __syncthreads();
        const bool merged = s_dups != 0;
        if (merged) {
            const FirstTable table = {kx, rid, pos, dup, head, nxt, nr, nb_log, skip0};
            first_merge(table);
        }
        for (uint32_t base = 0; base < ns; base += UP * kJoinThreads) {
            tuple_v nx[UP];
            uint32_t best[UP], m = 0;
#pragma unroll
            for (int u = 0; u < UP; u++) {
                const uint32_t j = base + (UP + u) * kJoinThreads + tid;
                nx[u] = j < ns ? ld_stream(S + j) : make_ulonglong2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < UP; u++) {
                best[u] = 0;
                if (base + u * kJoinThreads + tid >= ns) continue;
                uint32_t e = head[head_of(sv[u].x, B, nb_log)], steps = 0, nm = 0, bp = 0;
                while (e) {
                    if (kx[e - 1] == sv[u].x) {
                        const uint32_t p = pos[e - 1];
                        if (nm++ == 0 || p < bp) {
                            best[u] = e;
                            bp = p;
                        }
                    }
                    e = nxt[e - 1];
                    if (++steps > nr) {
                        set_error(err, kErrProbeLimit);
                        break;
                    }
                }
                if (!best[u]) continue;
                m++;
                if (!MAT) sum += rid[best[u] - 1] + sv[u].y;
                multi |= nm > 1;
                if (merged) multi |= (dup[(best[u] - 1) >> 5] >> ((best[u] - 1) & 31)) & 1u;
            }
            cnt += m;
            if constexpr (MAT) {
                unsigned long long o = mat_reserve(m, scan_tmp, &s_base, &a.acc->pairs);
#pragma unroll
                for (int u = 0; u < UP; u++)
                    if (best[u]) mat_put(a.mat, o++, rid[best[u] - 1], sv[u].y, err);
            }
#pragma unroll
            for (int u = 0; u < UP; u++) sv[u] = nx[u];
        }
        __syncthreads();
    }
    block_sum2_to(cnt, sum, red, &a.acc->matched, &a.acc->checksum);
    if (!MAT) flag_multi(multi, &a.acc->dup_flag);
    join_finish(a, false);
}

// Partition join over 16-byte tuples (CI: over the words of compact partitions), every match, or with lp the
// first by partition order: the build partition in shared memory, chained by 16-bit links from up to 16384
// heads (two per tuple: a warp waits for its longest chain), one CTA of 1024 threads per SM. Bound by those
// waits, not by bytes: one probe tuple per thread and round, the next one under way, measured 1530 us for
// 2^26 x 2^28 sparse keys (one head per tuple and four unrolled walks: 2061 us; one head, one walk: 1744; two
// heads, three walks: 1781). A table of tagged 4-byte slots in place of the chains took 3060 us, its longest walks being longer.
template <bool MAT, bool CI = false, bool MULTI = false>
__global__ void __launch_bounds__(kJoinThreads, 1) join_small_kernel(JoinArgs a0, MultiRef mr) {
    __shared__ JoinArgs s_a;
    if (MULTI) {
        const uint2 e = mr.map[blockIdx.x];
        multi_copy(&s_a, &mr.jobs[e.x].ja);
        __syncthreads();
        multi_large_step(s_a, 1, e.y, mr.jobs[e.x].join_blocks);
    }
    const JoinArgs &a = MULTI ? s_a : a0;
    extern __shared__ __align__(128) unsigned char smem[];
    tuple_v *rt = reinterpret_cast<tuple_v *>(smem);                      // [kSmemCap]
    uint16_t *head = reinterpret_cast<uint16_t *>(rt + kSmemCap);         // [kHeadMax]
    uint16_t *nxt = head + kHeadMax;                                       // [kSmemCap]
    __shared__ __align__(8) unsigned long long bar_storage;
    __shared__ unsigned long long red[64];
    __shared__ uint32_t s_item;
    __shared__ uint32_t scan_tmp[32];
    __shared__ unsigned long long s_base;
    const int tid = threadIdx.x;
    const uint32_t bar = smem_u32(&bar_storage);
    unsigned int *err = &a.counters[kCtrErr];
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const uint32_t nitems = a.counters[kCtrNItems];
    // Compiled once per partition layout; only the launch matching the device's choice runs.
    if (CI != (a.ci && ci_applies(a.counters, a.bits))) return;
    constexpr bool ci = CI;
    const int B = ci ? 0 : a.bits;  // shift from a stored x to the key's bits above the radix bits
    const bool lp = a.lp != 0;
    const bool skip0 = a.skip0 != 0;
    // Items [0, nA) went to the compact kernel if the build side's keys and row ids fit it.
    const uint32_t first_item = !a.all_items && compact_applies(a) ? a.counters[kCtrNItemsA] : 0u;
    constexpr int U = MAT ? 4 : 1;  // probe tuples per thread and round
    unsigned long long cnt = 0, sum = 0;
    uint32_t phase = 0;
    bool ok = true, multi = false;
    for (;;) {
        if (tid == 0) s_item = first_item + atomicAdd(&a.counters[kCtrItem], 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= nitems) break;
        const JoinItem item = a.items[it];
        const uint32_t nr = item.r_len;
        const uint32_t nb_log = heads_log(nr, true, 14);  // up to kHeadMax
        if (!ci && tid == 0) {
            // Order earlier generic-proxy accesses to rt before the async-proxy writes.
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            const uint32_t bytes = nr * 16u;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                         : "memory");
            const char *src = reinterpret_cast<const char *>(a.finR + item.r_begin);
            const uint32_t dst = smem_u32(rt);
            for (uint32_t off = 0; off < bytes; off += 32768u) {
                const uint32_t sz = bytes - off < 32768u ? bytes - off : 32768u;
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        dst + off),
                    "l"(src + off), "r"(sz), "r"(bar)
                    : "memory");
            }
        }
        const tuple_v *S = a.finS + item.s_begin;
        const uint32_t ns = item.s_len;
        tuple_v s[U];  // the thread's next probe tuples, under way during the build and the walks before them
        if (!MAT) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t j = tid + u * kJoinThreads;
                s[u] = j < ns ? ld_fin(S, a.finS8 + item.s_begin, j, ci) : make_ulonglong2(0, 0);
            }
        }
        uint32_t *head32 = reinterpret_cast<uint32_t *>(head);
        for (uint32_t q = tid; q < (1u << nb_log) / 2; q += kJoinThreads) head32[q] = 0;
        if (ci) {
            // Compact final partitions: expand the build side's words into {key >> bits, row id}.
            for (uint32_t i = tid; i < nr; i += kJoinThreads)
                rt[i] = ld_fin(a.finR + item.r_begin, a.finR8 + item.r_begin, i, true);
        } else {
            if (!mbar_wait(bar, phase)) {
                set_error(err, kErrSpinLimit);
                ok = false;
            }
            // An expired wait: let the R-tile copy land (bounded) before the CTA leaves its shared memory.
            if (!ok && tid == 0) mbar_wait(bar, phase);
            phase ^= 1u;
        }
        if (__syncthreads_or(!ok)) break;
        // Build: chain every R tuple (lp_join skips key 0, which reads as an empty slot there).
        for (uint32_t i = tid; i < nr; i += kJoinThreads) {
            const uint64_t k = rt[i].x;
            if (skip0 && k == 0 && (!ci || item.part0)) continue;
            const uint32_t h = head_of(k, B, nb_log);
            nxt[i] = (uint16_t)atomic_exch_u16(&head[h], i + 1);
        }
        __syncthreads();
        // Probe.
        if constexpr (MAT) {
            for (uint32_t base = 0; base < ns; base += U * kJoinThreads) {
                tuple_v sv[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t j = base + u * kJoinThreads + tid;
                    sv[u] = j < ns ? ld_stream(S + j) : make_ulonglong2(0, 0);
                }
                uint32_t mm[U], best[U], m = 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    mm[u] = best[u] = 0;
                    if (base + u * kJoinThreads + tid >= ns) continue;
                    const uint64_t k = sv[u].x;
                    uint32_t e = head[head_of(k, B, nb_log)], steps = 0;
                    while (e) {
                        if (rt[e - 1].x == k) {
                            if (!lp) mm[u]++;
                            else if (best[u] == 0 || e < best[u]) best[u] = e;
                        }
                        e = nxt[e - 1];
                        if (++steps > nr) {
                            set_error(err, kErrProbeLimit);
                            break;
                        }
                    }
                    if (lp) mm[u] = best[u] ? 1u : 0u;
                    m += mm[u];
                }
                unsigned long long o = mat_reserve(m, scan_tmp, &s_base, &a.acc->pairs);
                cnt += m;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (!mm[u]) continue;
                    if (lp) {
                        mat_put(a.mat, o++, rt[best[u] - 1].y, sv[u].y, err);
                        continue;
                    }
                    const uint64_t k = sv[u].x;
                    uint32_t e = head[head_of(k, B, nb_log)], steps = 0;
                    while (e && steps++ <= nr) {
                        if (rt[e - 1].x == k) mat_put(a.mat, o++, rt[e - 1].y, sv[u].y, err);
                        e = nxt[e - 1];
                    }
                }
            }
        } else
        for (uint32_t j0 = tid; j0 < ns; j0 += U * kJoinThreads) {
            tuple_v nx[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t j = j0 + (U + u) * kJoinThreads;
                nx[u] = j < ns ? ld_fin(S, a.finS8 + item.s_begin, j, ci) : make_ulonglong2(0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t j = j0 + u * kJoinThreads;
                if (j >= ns) continue;
                const uint64_t k = s[u].x;
                uint32_t e = head[head_of(k, B, nb_log)];
                uint32_t best = 0, nm = 0;
                uint32_t steps = 0;
                while (e) {
                    const tuple_v r = rt[e - 1];
                    if (r.x == k) {
                        if (lp) {
                            if (best == 0 || e < best) best = e;
                            nm++;
                        } else {
                            cnt++;
                            sum += r.y + s[u].y;
                        }
                    }
                    e = nxt[e - 1];
                    if (++steps > nr) {
                        set_error(err, kErrProbeLimit);
                        break;
                    }
                }
                if (lp && best) {
                    cnt++;
                    sum += rt[best - 1].y + s[u].y;
                    multi |= nm > 1;
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) s[u] = nx[u];
        }
        __syncthreads();
    }
    block_sum2_to(cnt, sum, red, &a.acc->matched, &a.acc->checksum);
    if (!MAT) flag_multi(multi, &a.acc->dup_flag);
    join_finish(a, ci);
}

// Large partitions: chained tables in global memory, one flattened index space for all of them. A bucket is the low
// bits of the key above the radix bits, changed by a hash of the bits above those (as mix_key): the keys of a
// large partition often share more low bits than the radix bits (ids in the high half of the key) and would make
// one chain of all, while runs of them keep neighbouring buckets (2^26 x 2^28 multiples of 4, 24.2 ms; 26.2 with a
// full hash).
__device__ __forceinline__ uint64_t large_bucket(uint64_t high, uint32_t nb_log) {
    if (!nb_log) return 0;
    return (high ^ (((high >> nb_log) * 0x9e3779b97f4a7c15ull) >> (64 - nb_log))) & ((1ull << nb_log) - 1);
}

__device__ __forceinline__ int find_large(const LargePart *L, int nl, uint64_t g, bool by_r) {
    int lo = 0, hi = nl;  // largest l with flat[l] <= g
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        const uint64_t f = by_r ? L[mid].r_flat : L[mid].s_flat;
        if (f <= g) lo = mid; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void large_clear(const JoinArgs &a, uint32_t blk, uint32_t nblk) {
    const uint64_t words = ld_u64_pair(&a.counters[kCtrLargeWords]);
    for (uint64_t i = blk * (uint64_t)blockDim.x + threadIdx.x; i < words;
         i += (uint64_t)nblk * blockDim.x)
        a.large_table[i] = 0;
}

// Key-aggregated table of one large partition (see large_words_agg): one chain node per distinct build
// key, holding the count of its build tuples, the wrapping sum of their row ids and the smallest
// position among them (as the maximum of ~position). A probe then costs one lookup however many build
// tuples share its key, where a chain of every build tuple costs a walk over all of them (a hot build
// key makes that quadratic).
struct LargeAgg {
    unsigned long long *sum;
    uint32_t *head, *next, *cnt, *negpos;
};

__device__ __forceinline__ LargeAgg large_agg(uint32_t *table, const LargePart &L) {
    LargeAgg t;
    uint32_t *base = table + L.table_off;
    t.sum = reinterpret_cast<unsigned long long *>(base);
    t.head = base + 2 * L.r_len;
    t.next = t.head + (1ull << L.nb_log);
    t.cnt = t.next + L.r_len;
    t.negpos = t.cnt + L.r_len;
    return t;
}

__device__ __forceinline__ uint32_t ld_volatile_u32(const uint32_t *p) {
    return *reinterpret_cast<const volatile uint32_t *>(p);
}

// The node (index + 1) of key k in bucket h, inserting build tuple i as its node when the key is absent.
// Lock-free: a node is published by a CAS on the bucket head after its next link is written; a failed
// CAS means another insert succeeded, and only the nodes it added (above the old head) are re-checked.
// Returns 0 (and sets the error word) if the walk exceeds the partition's size.
__device__ __forceinline__ uint32_t large_agg_find_or_insert(const LargeAgg &t, const JoinArgs &a, bool ci,
                                                             uint64_t r_begin, uint64_t r_len, uint64_t h,
                                                             uint64_t k, uint32_t i, uint32_t *err) {
    uint32_t stop = 0;
    uint32_t e = ld_volatile_u32(&t.head[h]);
    uint64_t steps = 0;
    for (;;) {
        for (uint32_t x = e; x && x != stop; x = ld_volatile_u32(&t.next[x - 1])) {
            if (fin_r(a, ci, r_begin + x - 1).x == k) return x;
            if (++steps > r_len) {
                set_error(err, kErrProbeLimit);
                return 0;
            }
        }
        *reinterpret_cast<volatile uint32_t *>(&t.next[i]) = e;
        __threadfence();
        const uint32_t old = atomicCAS(&t.head[h], e, i + 1);
        if (old == e) return i + 1;
        stop = e;
        e = old;
        if (++steps > r_len) {
            set_error(err, kErrProbeLimit);
            return 0;
        }
    }
}

__device__ __forceinline__ void large_build(const JoinArgs &a, uint32_t blk, uint32_t nblk) {
    const int nl = (int)a.counters[kCtrNLarge];
    const uint64_t total = ld_u64_pair(&a.counters[kCtrLargeR]);
    const bool ci = a.ci && ci_applies(a.counters, a.bits);
    const int bshift = ci ? 0 : a.bits;
    if (a.counters[kCtrLargeAgg]) {
        // Warp-uniform rounds: lanes holding equal keys of one partition combine their count, row-id sum
        // and smallest position first, so a hot key costs one update per warp.
        const unsigned lane = threadIdx.x & 31;
        for (uint64_t g0 = blk * (uint64_t)blockDim.x + (threadIdx.x & ~31u); g0 < total;
             g0 += (uint64_t)nblk * blockDim.x) {
            const uint64_t g = g0 + lane;
            bool act = g < total;
            int l = 0;
            uint64_t i = 0;
            tuple_v r = make_ulonglong2(0, 0);
            if (act) {
                l = find_large(a.large, nl, g, true);
                i = g - a.large[l].r_flat;
                r = fin_r(a, ci, a.large[l].r_begin + i);
                act = !(a.skip0 && r.x == 0 && (!ci || a.large[l].part0));
            }
            const unsigned act_mask = __ballot_sync(0xffffffffu, act);
            if (!act) continue;
            // Group lanes by key and partition: a compact word holds only key >> bits, which keys of two
            // partitions can share (full keys of different partitions differ in their low bits anyway).
            const unsigned long long gkey = ci ? (r.x | ((unsigned long long)(unsigned)l << 32)) : r.x;
            const unsigned peers = __match_any_sync(act_mask, gkey);
            // Row-id sum of the group in three pieces of at most 24 bits (32 addends cannot overflow them).
            const unsigned s0 = __reduce_add_sync(peers, (unsigned)(r.y & 0xffffffu));
            const unsigned s1 = __reduce_add_sync(peers, (unsigned)((r.y >> 24) & 0xffffffu));
            const unsigned s2 = __reduce_add_sync(peers, (unsigned)(r.y >> 48));
            const unsigned minpos = __reduce_min_sync(peers, a.lp_pos ? (unsigned)r.y : (unsigned)i);
            if ((int)lane != __ffs(peers) - 1) continue;
            const LargePart &L = a.large[l];
            const LargeAgg t = large_agg(a.large_table, L);
            const uint64_t h = large_bucket(r.x >> bshift, L.nb_log);
            const uint32_t node = large_agg_find_or_insert(t, a, ci, L.r_begin, L.r_len, h, r.x, (uint32_t)i,
                                                           &a.counters[kCtrErr]);
            if (!node) continue;
            atomicAdd(&t.cnt[node - 1], (uint32_t)__popc(peers));
            atomicAdd(&t.sum[node - 1], (unsigned long long)s0 + ((unsigned long long)s1 << 24) +
                                            ((unsigned long long)s2 << 48));
            atomicMax(&t.negpos[node - 1], ~minpos);
        }
        return;
    }
    for (uint64_t g = blk * (uint64_t)blockDim.x + threadIdx.x; g < total;
         g += (uint64_t)nblk * blockDim.x) {
        const int l = find_large(a.large, nl, g, true);
        const LargePart &L = a.large[l];
        const uint64_t i = g - L.r_flat;
        const uint64_t k = fin_r(a, ci, L.r_begin + i).x;
        if (a.skip0 && k == 0 && (!ci || L.part0)) continue;
        uint32_t *head = a.large_table + L.table_off;
        uint32_t *nxt = head + (1ull << L.nb_log);
        const uint64_t h = large_bucket(k >> bshift, L.nb_log);
        nxt[i] = atomicExch(&head[h], (uint32_t)(i + 1));
    }
}

template <bool MAT>
__device__ __forceinline__ void large_probe(const JoinArgs &a, uint32_t blk, uint32_t nblk) {
    __shared__ unsigned long long red[64];
    __shared__ uint32_t scan_tmp[32];
    __shared__ unsigned long long s_base;
    const int nl = (int)a.counters[kCtrNLarge];
    const uint64_t total = ld_u64_pair(&a.counters[kCtrLargeS]);
    unsigned long long cnt = 0, sum = 0;
    bool multi = false;  // first-match joins: a probe tuple matched two build tuples
    const bool ci = a.ci && ci_applies(a.counters, a.bits);
    const int bshift = ci ? 0 : a.bits;
    if constexpr (MAT) {
        unsigned int *err = &a.counters[kCtrErr];
        // Block-uniform rounds over the flattened probe tuples of all large partitions.
        for (uint64_t g0 = blk * (uint64_t)blockDim.x; g0 < total; g0 += (uint64_t)nblk * blockDim.x) {
            const uint64_t g = g0 + threadIdx.x;
            uint32_t m = 0, best = 0, e0 = 0;
            tuple_v s = make_ulonglong2(0, 0);
            const LargePart *Lp = nullptr;
            if (g < total) {
                Lp = &a.large[find_large(a.large, nl, g, false)];
                s = ld_fin(a.finS, a.finS8, Lp->s_begin + (g - Lp->s_flat), ci);
                const uint32_t *head = a.large_table + Lp->table_off;
                const uint32_t *nxt = head + (1ull << Lp->nb_log);
                unsigned long long best_y = 0;
                e0 = head[large_bucket(s.x >> bshift, Lp->nb_log)];
                uint64_t steps = 0;
                for (uint32_t e = e0; e;) {
                    const tuple_v r = fin_r(a, ci, Lp->r_begin + e - 1);
                    if (r.x == s.x) {
                        if (!a.lp) {
                            m++;
                        } else if (best == 0 || (a.lp_pos ? r.y < best_y : e < best)) {
                            best = e;
                            best_y = r.y;
                        }
                    }
                    e = nxt[e - 1];
                    if (++steps > Lp->r_len) {
                        set_error(err, kErrProbeLimit);
                        break;
                    }
                }
                if (a.lp) m = best ? 1u : 0u;
            }
            unsigned long long o = mat_reserve(m, scan_tmp, &s_base, &a.acc->pairs);
            cnt += m;
            if (m) {
                const uint32_t *nxt = a.large_table + Lp->table_off + (1ull << Lp->nb_log);
                if (a.lp) {
                    const unsigned long long y = fin_r(a, ci, Lp->r_begin + best - 1).y;
                    mat_put(a.mat, o, !a.lp_pos ? y : y < a.nR ? a.relR[y].y : 0ull, s.y, err);
                } else {
                    uint64_t steps = 0;
                    for (uint32_t e = e0; e && steps++ <= Lp->r_len; e = nxt[e - 1]) {
                        const tuple_v r = fin_r(a, ci, Lp->r_begin + e - 1);
                        if (r.x == s.x) mat_put(a.mat, o++, r.y, s.y, err);
                    }
                }
            }
        }
    } else if (a.counters[kCtrLargeAgg]) {
        for (uint64_t g = blk * (uint64_t)blockDim.x + threadIdx.x; g < total;
             g += (uint64_t)nblk * blockDim.x) {
            const int l = find_large(a.large, nl, g, false);
            const LargePart &L = a.large[l];
            const tuple_v s = ld_fin(a.finS, a.finS8, L.s_begin + (g - L.s_flat), ci);
            const LargeAgg t = large_agg(a.large_table, L);
            uint32_t e = t.head[large_bucket(s.x >> bshift, L.nb_log)];
            uint64_t steps = 0;
            while (e && fin_r(a, ci, L.r_begin + e - 1).x != s.x) {
                e = t.next[e - 1];
                if (++steps > L.r_len) {
                    set_error(&a.counters[kCtrErr], kErrProbeLimit);
                    e = 0;
                }
            }
            if (!e) continue;
            if (a.lp) {
                const uint32_t first = ~t.negpos[e - 1];
                multi |= t.cnt[e - 1] > 1;
                if (first < (a.lp_pos ? a.nR : L.r_len)) {
                    cnt++;
                    sum += (a.lp_pos ? a.relR[first].y : fin_r(a, ci, L.r_begin + first).y) + s.y;
                } else {
                    set_error(&a.counters[kCtrErr], kErrBounds);
                }
            } else {
                const unsigned long long c = t.cnt[e - 1];
                cnt += c;
                sum += t.sum[e - 1] + c * s.y;
            }
        }
    } else
    for (uint64_t g = blk * (uint64_t)blockDim.x + threadIdx.x; g < total;
         g += (uint64_t)nblk * blockDim.x) {
        const int l = find_large(a.large, nl, g, false);
        const LargePart &L = a.large[l];
        const tuple_v s = ld_fin(a.finS, a.finS8, L.s_begin + (g - L.s_flat), ci);
        const uint32_t *head = a.large_table + L.table_off;
        const uint32_t *nxt = head + (1ull << L.nb_log);
        uint32_t e = head[large_bucket(s.x >> bshift, L.nb_log)];
        uint32_t best = 0, nm = 0;
        unsigned long long best_y = 0;  // the match's row id, or its input position (lp_pos)
        uint64_t steps = 0;
        while (e) {
            const tuple_v r = fin_r(a, ci, L.r_begin + e - 1);
            if (r.x == s.x) {
                if (a.lp) {
                    if (best == 0 || (a.lp_pos ? r.y < best_y : e < best)) {
                        best = e;
                        best_y = r.y;
                    }
                    nm++;
                } else {
                    cnt++;
                    sum += r.y + s.y;
                }
            }
            e = nxt[e - 1];
            if (++steps > L.r_len) {
                set_error(&a.counters[kCtrErr], kErrProbeLimit);
                break;
            }
        }
        if (a.lp && best) {
            cnt++;
            sum += (!a.lp_pos ? best_y : best_y < a.nR ? a.relR[best_y].y : 0ull) + s.y;
            multi |= nm > 1;
        }
    }
    block_sum2_to(cnt, sum, red, &a.acc->matched, &a.acc->checksum);
    if (!MAT) flag_multi(multi, &a.acc->dup_flag);
    if (blk == 0 && threadIdx.x == 0) {
        if (nl) atomicAdd(&a.acc->large_parts, (unsigned long long)nl);
        if (!MAT && a.ci && ci_applies(a.counters, a.flag_bits))
            atomicOr(&a.acc->flags, (unsigned long long)HJ_RES_COMPACT_PARTITIONS);
        if (a.w8_b1 >= 0 && w8_fits(a.counters, a.w8_b1))
            atomicOr(&a.acc->flags, (unsigned long long)HJ_RES_WORD_PASS1);
    }
}

__global__ void join_large_clear(JoinArgs a) { large_clear(a, blockIdx.x, gridDim.x); }
__global__ void join_large_build(JoinArgs a) { large_build(a, blockIdx.x, gridDim.x); }
template <bool MAT>
__global__ void join_large_probe(JoinArgs a) {
    large_probe<MAT>(a, blockIdx.x, gridDim.x);
}

__device__ __noinline__ void multi_large_step(const JoinArgs &a, int step, uint32_t blk, uint32_t nblk) {
    if (!a.counters[kCtrNLarge]) return;
    if (step == 0)
        large_clear(a, blk, nblk);
    else
        large_build(a, blk, nblk);
    __syncthreads();
}

// The last large-partition step of a wave of joins, the probe, over a map of (job, block) as its other steps: a block
// of a job without large partitions returns at once. (With one block per job for all three steps a batch of four
// 2^21 x 2^23 joins whose partitions were all large took 98.7 ms, one with a hot build key in each 10.3.) It also
// hands over the error word.
__global__ void __launch_bounds__(kMultiLargeThreads) multi_large(MultiRef mr) {
    const uint2 e = mr.map[blockIdx.x];
    const MultiJob &job = mr.jobs[e.x];
    const bool any = job.ja.counters[kCtrNLarge] != 0;
    if (!any && e.y != 0) return;
    __shared__ JoinArgs a;
    multi_copy(&a, &job.ja);
    __syncthreads();
    if (any) {
        large_probe<false>(a, e.y, job.large_blocks);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const uint32_t err = *reinterpret_cast<const volatile uint32_t *>(&a.counters[kCtrErr]);
        if (err) atomicOr(&a.acc->error, err);
    }
}

__global__ void copy_error(const uint32_t *counters, JoinAccum *acc) {
    if (threadIdx.x == 0 && counters[kCtrErr]) atomicOr(&acc->error, counters[kCtrErr]);
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
int radix_geom(int bits, int passes, RadixGeom *g, int b1_req) {
    if (bits < 1 || bits > 15) return HJ_E_INVAL;
    if (passes != 1 && passes != 2) return HJ_E_INVAL;
    // Partition contents do not depend on how the bits are split across passes; a single pass runs
    // as one physical pass only while its fanout fits the shared-memory staging (<= 256 digits).
    int P = passes;
    if (P == 1 && bits > 8) P = 2;
    if (P == 2 && bits < 2) P = 1;
    g->bits = bits;
    g->req_bits = bits;
    g->single = false;
    g->mix = false;
    g->passes = P;
    int b1 = bits / 2;
    if (b1_req > 0) {
        b1 = b1_req;
        if (b1 > 8) b1 = 8;
        if (b1 > bits - 1) b1 = bits - 1;
        if (b1 < bits - 8) b1 = bits - 8;
        if (b1 < 1) b1 = 1;
    }
    g->b1 = P == 2 ? b1 : bits;
    g->b2 = bits - g->b1;
    if (g->b1 > 8 || g->b2 > 8) return HJ_E_INVAL;
    g->F1 = 1 << g->b1;
    g->F2 = 1 << g->b2;
    return HJ_OK;
}

// The lowest bits that bring build partitions to kSingleTarget tuples on average, at least
// kSingleMinBits (items for every SM), at most what the caller asked for. Above 2^kSingleMaxBits
// partitions of kSingleMaxAvg tuples the two-pass pipelines run, and with 2^11 partitions also from
// kSingleManyTuples tuples: the scatter visits every page of its output once per tile, and those visits
// grow with the output (2^24 x 2^24, 12 bits: 0.57 ms in one pass, 0.74 in two; 2^24 x 2^26: 1.34 and 1.32;
// 2^24 x 2^28: 4.50 and 3.38). First-match joins stay up to twice that size: two passes may have to run
// again in order where build keys repeat (2^24 x 2^26, four a key: 1.55 ms against 2 x 1.4 and more). So do
// materialising joins, which have words in one pass only (`lp` covers both).
constexpr uint64_t kSingleTarget = 6144, kSingleMaxAvg = 8192, kSingleManyTuples = 80000000;
constexpr int kSingleMinBits = 8;

bool radix_geom_single(int bits, bool lp, size_t nR, size_t nS, RadixGeom *g) {
    if ((nR >> kSingleMaxBits) > kSingleMaxAvg || nR >= (1ull << 32) || nS >= (1ull << 32)) return false;
    int b = kSingleMinBits;
    while (b < kSingleMaxBits && (nR >> b) > kSingleTarget) b++;
    if (b == kSingleMaxBits && (uint64_t)nR + nS > (lp ? 2 : 1) * kSingleManyTuples) return false;
    if (b > bits) b = bits;
    g->bits = b;
    g->req_bits = bits;
    g->passes = 1;
    g->b1 = b;
    g->b2 = 0;
    g->F1 = 1 << b;
    g->F2 = 1;
    g->single = true;
    return true;
}

static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Pass-1 work items: about kSubPerChunk sub-chunks per chunk (two per warp of the histogram kernel).
constexpr int kSubPerChunk = 32;

static ChunkGeom chunk_geom(size_t nR, size_t nS, int num_sms) {
    // About three chunks per SM (the scatter kernel's residency), each a whole number of tiles.
    const uint64_t tiles = (uint64_t)ceil_div_u64(nR, kTile) + ceil_div_u64(nS, kTile);
    const uint64_t target = (uint64_t)(num_sms > 0 ? num_sms : 148) * 3;
    uint64_t ct = (tiles + target - 1) / target;
    if (ct < 1) ct = 1;
    // Pass 1 takes sub-chunks as work items, so that CTAs that run ahead take more of them instead of
    // idling while the slowest chunk finishes.
    const uint64_t st = (ct + kSubPerChunk - 1) / kSubPerChunk;
    ChunkGeom cg;
    cg.chunk = ct * kTile;
    cg.cR = ceil_div_u64(nR, cg.chunk);
    cg.cS = ceil_div_u64(nS, cg.chunk);
    cg.sub = st * kTile;
    cg.spc = (uint32_t)((ct + st - 1) / st);
    cg.pad = 0;
    return cg;
}

struct PhjSizes {
    size_t chunk_hist, prefix, total, start, units_off, units_cnt, subhist, counters, items, large, large_table,
        tmp1, tmp2, seg_head, seg_next, ors;
    size_t max_items, max_large, large_table_words;
    uint32_t max_segs, seg_grid, it_tiles;
    ChunkGeom cg;
};

// With fewer bits than asked for, keys that share low bits would overfill the partitions they fall into (2^24 x 2^26
// multiples of 4: 1.5 ms with 14 bits, 5.8 with 12), so the partitions are then those of mix_key.
// The two-pass pipelines' geometry: the lowest bits that bring build partitions to kSingleTarget tuples, at
// most what the caller asked for. Fewer digits make longer runs and fewer, fuller units (2^24 x 2^26 in
// segment mode: 1.32 ms with 12 bits, 1.40 with 13, 2.00 with 14; 2^24 x 2^28 3.38 / 3.47 / 4.09). Pass 2
// takes eight of them (pass 1 at least kMinBits1), unless the caller split them: a unit of pass 2 is a (pass-1
// CTA, digit) chain, and fewer pass-1 digits leave less of its last tile empty (2^26 x 2^28, 14 bits: 4.15 ms
// with 6 + 8, 4.41 with 7 + 7; 2^25 x 2^26, 13 bits: 1.39 with 5 + 8, 1.51 with 6 + 7; 2^24 x 2^27, 12 bits:
// 1.77 with 5 + 7, 1.82 with 4 + 8; 16-byte tuples prefer one bit more in pass 1, by 4%). From
// kWideSplitTuples on pass 2 takes seven: what its CTAs write at a time spreads over more memory with the size
// (2^26 x 2^28: 4.04 ms with 6 + 8, 4.07 with 7 + 7; 2^27 x 2^28: 4.80 and 4.68; 2^27 x 2^29: 7.73 and 7.49).
constexpr int kMinBits1 = 5;
constexpr uint64_t kWideSplitTuples = 400000000;
void radix_geom_by_size(size_t nR, size_t nS, bool split_given, RadixGeom *g) {
    if (g->passes != 2) return;
    const int req = g->req_bits;
    int b = 2;
    while (b < g->bits && (nR >> b) > kSingleTarget) b++;
    if (b < g->bits || !split_given) {
        const int bits2 = (uint64_t)nR + nS >= kWideSplitTuples ? 7 : 8;
        radix_geom(b, 2, g, b - bits2 > kMinBits1 ? b - bits2 : kMinBits1);
    }
    g->mix = b < req;
    g->req_bits = req;
}

// Segment mode from 2^26 tuples. Its pass 2 has one unit per (pass-1 CTA, relation, digit) and a
// partial tile per unit whatever the size, its pass 1 runs at two CTAs per SM, and the partly filled
// segments reserve storage (2 * CTAs * F1 * kTile tuples); the histogram read it saves grows with the
// size. Fewest bits, unique keys: 2^24 x 2^24 0.86 ms against 0.74 in the exact-offset pipeline, 2^25 x
// 2^25 1.25 against 1.34 (63-bit keys 1.52 against 1.67), 2^26 x 2^28 4.61 against 5.01 (6.41 / 7.09).
constexpr uint64_t kSegMinTuples = 1ull << 26;

bool phj_seg_applies(const RadixGeom &g, bool, size_t nR, size_t nS) {
    return g.passes == 2 && g.bits <= kSegMaxBits && (uint64_t)nR + nS >= kSegMinTuples;
}

static PhjSizes phj_sizes(const RadixGeom &g, size_t nR, size_t nS, int num_sms, bool seg) {
    PhjSizes z;
    const size_t np = (size_t)g.nparts();
    const int sms = num_sms > 0 ? num_sms : 148;
    if (seg) {
        // "Chunks" are the pass-1 CTAs, one per relation each.
        z.seg_grid = (uint32_t)(sms * kSegCtasPerSm);
        z.cg.chunk = 0;
        z.cg.cR = z.cg.cS = z.seg_grid;
        z.cg.sub = 0;
        z.cg.spc = 0;
        z.cg.pad = 0;
        const uint64_t tiles = (uint64_t)ceil_div_u64(nR, kTile) + ceil_div_u64(nS, kTile);
        uint64_t it = tiles / ((uint64_t)z.seg_grid * 8);
        z.it_tiles = (uint32_t)(it < 1 ? 1 : it > 16 ? 16 : it);
        // Every segment but the current one of each (CTA, relation, digit) is full; each CTA leaves
        // fewer than kSegSlab ids of its last slab unused.
        const uint64_t segs = (uint64_t)(nR + nS) / kTile + 2ull * z.seg_grid * g.F1 + (uint64_t)z.seg_grid * kSegSlab;
        z.max_segs = (uint32_t)segs;
    } else if (g.single) {
        z.seg_grid = z.it_tiles = z.max_segs = 0;
        z.cg.chunk = z.cg.sub = 0;
        z.cg.cR = z.cg.cS = single_grid(nR, nS, sms);
        z.cg.spc = 0;
        z.cg.pad = 0;
    } else {
        z.cg = chunk_geom(nR, nS, num_sms);
        z.seg_grid = 0;
        z.it_tiles = 0;
        z.max_segs = 0;
    }
    const size_t nchunks = (size_t)z.cg.cR + z.cg.cS;
    z.chunk_hist = align_up(nchunks * np * 4, 256);
    z.prefix = g.single ? 0 : z.chunk_hist;  // the one-pass pipeline's prefixes replace its histogram rows
    z.ors = g.single ? align_up((size_t)z.cg.cR * 3 * 8, 256) : 0;
    z.total = align_up(2 * np * 4, 256);
    z.start = align_up(2 * (np + 1) * 8, 256);
    z.units_off = g.single ? 0 : align_up(nchunks * (size_t)g.F1 * 8, 256);
    z.units_cnt = g.single ? 0 : align_up(nchunks * (size_t)g.F1 * 4, 256);
    z.subhist = align_up(nchunks * (size_t)z.cg.spc * g.F1 * 4, 256);
    z.counters = 256;
    z.max_items = np + nS / kProbeChunk + 2;
    z.items = align_up(z.max_items * sizeof(JoinItem), 256);
    const size_t min_large = g.single ? kFirstCap : kSmemCap;
    z.max_large = np < nR / min_large + 1 ? np : nR / min_large + 1;
    z.large = align_up(z.max_large * sizeof(LargePart), 256);
    z.tmp1 = seg ? align_up((size_t)z.max_segs * kTile * 16, 256) : align_up((nR + nS) * 16, 256);
    z.tmp2 = g.passes == 2 ? align_up((nR + nS) * 16, 256) : 0;
    z.seg_head = seg ? align_up((size_t)2 * z.seg_grid * g.F1 * 4, 256) : 0;
    z.seg_next = seg ? align_up((size_t)z.max_segs * 4, 256) : 0;
    // Large-partition tables: chains take head <= 2*|R_p| words and next = |R_p| words; key-aggregated
    // tables another 4*|R_p| words plus one word of alignment each. With two passes they reuse the
    // pass-1 buffer, which is dead once pass 2 has run (tables that do not fit it fall back to chains).
    z.large_table_words = 7 * nR + 2 * z.max_large + 2;
    z.large_table = g.passes == 2 ? 0 : align_up(z.large_table_words * 4, 256);
    return z;
}

size_t phj_scratch_bytes(const RadixGeom &g, size_t nR, size_t nS, int num_sms, bool seg) {
    PhjSizes z = phj_sizes(g, nR, nS, num_sms, seg);
    return z.chunk_hist + z.prefix + z.total + z.start + z.units_off + z.units_cnt + z.subhist + z.counters + z.items +
           z.large + z.large_table + z.tmp1 + z.tmp2 + z.seg_head + z.seg_next + z.ors;
}

void phj_carve(const RadixGeom &g, size_t nR, size_t nS, int num_sms, char *base, PhjScratch *s, bool seg) {
    PhjSizes z = phj_sizes(g, nR, nS, num_sms, seg);
    char *p = base;
    s->seg = seg;
    s->seg_grid = z.seg_grid;
    s->max_segs = z.max_segs;
    s->it_tiles = z.it_tiles;
    s->chunk = z.cg.chunk;
    s->cR = z.cg.cR;
    s->cS = z.cg.cS;
    s->sub = z.cg.sub;
    s->spc = z.cg.spc;
    s->chunk_hist = reinterpret_cast<uint32_t *>(p); p += z.chunk_hist;
    s->prefix = reinterpret_cast<uint32_t *>(p); p += z.prefix;
    s->total = reinterpret_cast<uint32_t *>(p); p += z.total;
    s->start = reinterpret_cast<uint64_t *>(p); p += z.start;
    s->unit_off = reinterpret_cast<uint64_t *>(p); p += z.units_off;
    s->unit_cnt = reinterpret_cast<uint32_t *>(p); p += z.units_cnt;
    s->subhist = reinterpret_cast<uint32_t *>(p); p += z.subhist;
    s->seg_head = reinterpret_cast<uint32_t *>(p); p += z.seg_head;
    s->seg_next = reinterpret_cast<uint32_t *>(p); p += z.seg_next;
    s->ors = reinterpret_cast<unsigned long long *>(p); p += z.ors;
    s->counters = reinterpret_cast<uint32_t *>(p); p += z.counters;
    s->items = p; p += z.items;
    s->max_items = z.max_items;
    s->large = p; p += z.large;
    s->max_large = z.max_large;
    s->tmp1 = reinterpret_cast<ulonglong2 *>(p); p += z.tmp1;
    if (g.passes == 2) {
        s->tmp2 = reinterpret_cast<ulonglong2 *>(p); p += z.tmp2;
        s->large_table = reinterpret_cast<uint32_t *>(s->tmp1);
        s->large_table_words = z.tmp1 / 4;
    } else {
        s->tmp2 = s->tmp1;
        s->large_table = reinterpret_cast<uint32_t *>(p); p += z.large_table;
        s->large_table_words = z.large_table_words;
    }
}

#define HJ_CU(call)                                                                   \
    do {                                                                              \
        cudaError_t e_ = (call);                                                      \
        if (e_ != cudaSuccess) {                                                      \
            fprintf(stderr, "hjscm: %s failed: %s\n", #call, cudaGetErrorString(e_)); \
            return HJ_E_DEVICE;                                                       \
        }                                                                             \
    } while (0)

// Dynamic shared memory of scatter_kernel: tile buffers (word tiles: 16 spare bytes each), gbase, running,
// tdstart, and the digit counts (per warp for the stable rank).
static constexpr size_t scatter_smem_bytes(bool stable) {
    return (size_t)kScatterBufs * (kTile * 16 + 16) + 256 * 8 * 2 + 256 * 4 +
           (stable ? (size_t)(kScatterThreads / 32) * 256 * 2 : (size_t)256 * 4);
}

// The exact-offset pipeline's kernels that partition by mix_key.
static int prepare_mixed() {
    HJ_CU(cudaFuncSetAttribute(hist_chunk_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 136 * 1024));
    HJ_CU(cudaFuncSetAttribute(
        scatter_kernel<kScatterThreads, kScatterItems, true, kScatterBufs, kScatterCtasPerSm, false, true>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_smem_bytes(true)));
    HJ_CU(cudaFuncSetAttribute(
        scatter_kernel<kScatterThreads, kScatterItems, false, kScatterBufs, kScatterCtasPerSm, false, true>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_smem_bytes(false)));
    return HJ_OK;
}

static int prepare_all() {
    HJ_CU(cudaFuncSetAttribute(hist_chunk_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 136 * 1024));
    HJ_CU(cudaFuncSetAttribute(plan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)((size_t)2 * (1u << kPlanStageBits) * 4)));
    HJ_CU(cudaFuncSetAttribute(scatter_kernel<kScatterThreads, kScatterItems, true, kScatterBufs, kScatterCtasPerSm>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_smem_bytes(true)));
    HJ_CU(cudaFuncSetAttribute(scatter_kernel<kScatterThreads, kScatterItems, false, kScatterBufs, kScatterCtasPerSm>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_smem_bytes(false)));
    HJ_CU(cudaFuncSetAttribute(
        scatter_kernel<kScatterThreads, 2 * kScatterItems, false, kScatterBufs, scatter_word_ctas(false), true>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_smem_bytes(false)));
    HJ_CU(cudaFuncSetAttribute(
        scatter_kernel<kScatterThreads, 2 * kScatterItems, true, kScatterBufs, scatter_word_ctas(true), true>,
        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scatter_smem_bytes(true)));
    HJ_CU(cudaFuncSetAttribute(join_small_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kJoinSmem));
    HJ_CU(cudaFuncSetAttribute(join_small_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kJoinSmem));
    HJ_CU(cudaFuncSetAttribute(join_compact_kernel<false, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kCompactSmem));
    HJ_CU(cudaFuncSetAttribute(join_compact_kernel<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kCompactSmem));
    HJ_CU(cudaFuncSetAttribute(join_compact_kernel<true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kCompactSmem));
    HJ_CU(cudaFuncSetAttribute(join_words_kernel<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kOaSmem));
    HJ_CU(cudaFuncSetAttribute(join_words_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOaSmem));
    HJ_CU(cudaFuncSetAttribute(join_first_words_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kFwSmem));
    HJ_CU(cudaFuncSetAttribute(join_words_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOaSmem));
    HJ_CU(cudaFuncSetAttribute(join_words_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOaSmem));
    HJ_CU(cudaFuncSetAttribute(join_first_words_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwSmem));
    HJ_CU(cudaFuncSetAttribute(join_first_words_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwSmem));
    HJ_CU(cudaFuncSetAttribute(join_first_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFirstSmem));
    HJ_CU(cudaFuncSetAttribute(join_small_kernel<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kJoinSmem));
    HJ_CU(cudaFuncSetAttribute(join_first_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFirstSmem));
    HJ_CU(cudaFuncSetAttribute(join_first_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFirstSmem));
    HJ_CU(cudaFuncSetAttribute(join_small_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kJoinSmem));
    HJ_CU(cudaFuncSetAttribute(join_compact_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kCompactSmem));
    HJ_CU(cudaFuncSetAttribute(join_compact_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kCompactSmem));
    {
        int rc = single_prepare_device();
        if (!rc) rc = small_prepare_device();
        if (rc) return rc;
    }
    return nphj_prepare_device();
}

// In parts, as setting an attribute loads the kernel (a process's first server took 24 ms to create with all of them,
// 16 without the pass-1 forms that it does not use).
int phj_prepare_device(bool seg, bool mix) {
    static std::atomic<unsigned> done[64];
    int cur_dev = 0;
    HJ_CU(cudaGetDevice(&cur_dev));
    if (cur_dev < 0 || cur_dev >= 64) return HJ_E_INVAL;
    const unsigned want = 1u | (!seg && mix ? 2u : 0u) | (seg ? (mix ? 8u : 4u) : 0u), have = done[cur_dev].load();
    int rc = HJ_OK;
    if (want & ~have & 1u) rc = prepare_all();
    if (!rc && (want & ~have & 2u)) rc = prepare_mixed();
    if (!rc && (want & ~have & 4u)) rc = seg_prepare_device(false);
    if (!rc && (want & ~have & 8u)) rc = seg_prepare_device(true);
    if (!rc) done[cur_dev].fetch_or(want);
    return rc;
}

JoinArgs join_args(const RadixGeom &g, bool lp, bool skip0, const ulonglong2 *R, size_t nR, const PhjScratch &s,
                          JoinAccum *acc, const MatOut *mat, int ci_ok, int w8_b1, JoinAccum *host_out) {
    JoinArgs ja = {};
    ja.items = reinterpret_cast<const JoinItem *>(s.items);
    ja.large = reinterpret_cast<const LargePart *>(s.large);
    ja.counters = s.counters;
    ja.finR = s.tmp2;
    ja.finS = s.tmp2 + nR;
    ja.large_table = s.large_table;
    ja.bits = g.bits;
    ja.lp = lp ? 1 : 0;
    ja.skip0 = skip0 ? 1 : 0;
    ja.acc = acc;
    ja.mat = mat ? *mat : MatOut{nullptr, 0};
    ja.ci = ci_ok;
    ja.finR8 = reinterpret_cast<const unsigned long long *>(s.tmp2);
    ja.finS8 = g.single ? single_probe_words(s, nR, lp) : ja.finR8 + nR;
    ja.lp_pos = g.single && lp ? 1 : 0;
    ja.relR = R;
    ja.nR = nR;
    ja.flag_bits = g.req_bits;
    ja.w8_b1 = w8_b1;
    ja.all_items = g.single ? 1 : 0;
    ja.host_out = host_out;
    return ja;
}

// Partitions beyond shared memory, then the error word of all kernels.
static int large_launch(const JoinArgs &ja, bool mat, const PhjScratch &s, JoinAccum *acc, cudaStream_t st, int num_sms) {
    join_large_clear<<<num_sms * 2, 256, 0, st>>>(ja);
    join_large_build<<<num_sms * 2, 256, 0, st>>>(ja);
    if (mat)
        join_large_probe<true><<<num_sms * 2, 256, 0, st>>>(ja);
    else
        join_large_probe<false><<<num_sms * 2, 256, 0, st>>>(ja);
    copy_error<<<1, 32, 0, st>>>(s.counters, acc);
    HJ_CU(cudaGetLastError());
    return HJ_OK;
}

int multi_join_launch(const MultiJob *jobs, const uint2 *every_map, unsigned every_blocks, const uint2 *first_map,
                      unsigned first_blocks, const uint2 *large_map, unsigned large_blocks, cudaStream_t st,
                      uint32_t *launches) {
    const JoinArgs none = {};
    const MultiRef every = {jobs, every_map}, first = {jobs, first_map}, large = {jobs, large_map};
    if (every_blocks) {
        join_words_kernel<true><<<every_blocks, kCompactThreads, kOaSmem, st>>>(none, every);
        join_small_kernel<false, false, true><<<every_blocks, kJoinThreads, kJoinSmem, st>>>(none, every);
        *launches += 2;
    }
    if (first_blocks) {
        join_first_words_kernel<true><<<first_blocks, kJoinThreads, kFwSmem, st>>>(none, first);
        join_first_kernel<false, true><<<first_blocks, kJoinThreads, kFirstSmem, st>>>(none, first);
        *launches += 2;
    }
    multi_large<<<large_blocks, kMultiLargeThreads, 0, st>>>(large);
    *launches += 1;
    HJ_CU(cudaGetLastError());
    return HJ_OK;
}

int phj_large_enqueue(const RadixGeom &g, bool lp, bool skip0, const ulonglong2 *R, size_t nR, size_t nS,
                      const PhjScratch &s, JoinAccum *acc, cudaStream_t st, int num_sms, uint32_t *launches) {
    (void)nS;
    *launches += 4;
    return large_launch(join_args(g, lp, skip0, R, nR, s, acc, nullptr, 1, -1, nullptr), false, s, acc, st, num_sms);
}

int phj_enqueue(const RadixGeom &g, bool lp, bool skip0, const ulonglong2 *R, size_t nR, const ulonglong2 *S,
                size_t nS, const PhjScratch &s, JoinAccum *acc, cudaStream_t st, cudaEvent_t ev_mid,
                int num_sms, cudaEvent_t *ph, uint32_t *launches, const MatOut *mat, int test_flags,
                bool ordered, JoinAccum *host_out) {
    uint32_t nlaunch = 0;
    // Stable ranks of the build relation: first-match joins that keep the input order.
    const bool stable = lp && ordered && !g.single;
#define HJ_PH(i) \
    if (ph) HJ_CU(record_event(ph[i], st))
    if (nR >= (1ull << 32) || nS >= (1ull << 32)) return HJ_E_INVAL;
    const int np = g.nparts();
    const int F1 = g.F1, F2 = g.F2;
    const size_t hist_smem = (size_t)np * 4 + (size_t)16 * F1 * 4;  // 16 warps
    ChunkGeom cg;
    cg.chunk = s.chunk;
    cg.cR = s.cR;
    cg.cS = s.cS;
    cg.sub = s.sub;
    cg.spc = s.spc;
    cg.pad = 0;
    const uint32_t nchunks = cg.cR + cg.cS;
    // A segment-mode scratch holds the segment storage, not the exact-offset pipeline's buffers.
    const bool segm = s.seg;
    // 8-byte words in the partitions (compact final partitions, and in segment mode an 8-byte pass 1):
    // joins without per-match output (all but the materialising ones), unless the caller asked for
    // tuples (test_flags bit 2), when the widths allow them (decided on the device).
    const int ci_ok = ((!mat || g.single) && !(test_flags & 2)) ? 1 : 0;
    const bool seg_words = segm && ci_ok;
    // The exact-offset pipeline with two passes stores pass 1 as words too (when w8_fits holds, which
    // the histogram pass's ORs decide before pass 1) when its pass-2 units (chunk, pass-1 digit) average
    // a full 4096-word tile, or when asked (test_flags bit 4). Pass 2 over 4096-word tiles is slower than
    // over 2048-tuple tiles when most tiles are partial (2^24 x 2^26: 1.91 against 1.82 ms; 2^27 x 2^29:
    // 9.01 against 10.68 ms).
    const bool exact_words =
        !segm && ci_ok && g.passes == 2 && ((test_flags & 4) || cg.chunk / (uint64_t)F1 >= 2ull * kTile);
    if (segm && (g.passes != 2 || g.bits > kSegMaxBits || (g.mix && F1 > 128))) return HJ_E_INVAL;
    {
        const int rc = phj_prepare_device(segm, g.mix);
        if (rc) return rc;
    }
    if (!g.single) HJ_CU(cudaMemsetAsync(s.counters, 0, kNumCounters * 4, st));  // the one-pass count clears them

    HJ_PH(0);
    if (g.single) {
        const int rc = single_partition_enqueue(g, lp, skip0, ci_ok != 0, R, nR, S, nS, s, acc, host_out && !mat, st, !mat,
                                                ph, &nlaunch);
        if (rc) return rc;
    } else if (segm) {
        // 1'. pass 1 into segment chains, with the per-CTA histograms
        const int rc = seg_pass1_enqueue(g, R, nR, S, nS, s, seg_words, stable, (test_flags & 1) != 0, st, &nlaunch);
        if (rc) return rc;
    } else {
        // 1. per-chunk histograms
        if (g.mix)
            hist_chunk_kernel<true><<<nchunks, 512, hist_smem, st>>>(R, nR, S, nS, g.bits, F1, cg, s.chunk_hist, s.subhist,
                                                                     s.counters + kCtrMaxKey);
        else
            hist_chunk_kernel<false><<<nchunks, 512, hist_smem, st>>>(R, nR, S, nS, g.bits, F1, cg, s.chunk_hist, s.subhist,
                                                                      s.counters + kCtrMaxKey);
        HJ_CU(cudaGetLastError());
    }
    if (!g.single) {
    HJ_PH(1);
    // 2. prefix over chunks, 3. plan, 4. units
    colscan_kernel<<<(8 * np + 255) / 256, 256, 0, st>>>(s.chunk_hist, s.prefix, s.total, np, cg);
    PlanArgs pa;
    pa.bits = g.bits;
    pa.passes = g.passes;
    pa.b1 = g.b1;
    pa.F1 = F1;
    pa.F2 = F2;
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
    pa.agg_ok = mat ? 0 : 1;
    pa.small_cap = kSmemCap;
    plan_kernel<<<1, 1024, g.bits <= kPlanStageBits ? (size_t)2 * np * 4 : 0, st>>>(pa);
    {
        const int ut = F1 < 32 ? 32 : F1;
        units_kernel<<<nchunks, ut, 0, st>>>(s.chunk_hist, s.prefix, s.start, g.bits, g.b1, F1, g.passes == 2 ? F2 : 1,
                                             cg, s.unit_off, s.unit_cnt, s.subhist, s.counters + kCtrErr);
    }
    HJ_CU(cudaGetLastError());
    nlaunch += segm ? 3 : 4;
    HJ_PH(2);
    }

    // 5. scatter passes (segment mode: pass 2 only, its units are the pass-1 chains)
    const int scatter_grid = num_sms * kScatterCtasPerSm;
    for (int pass = segm ? 1 : 0; pass < g.passes && !g.single; pass++) {
        ScatterArgs sa;
        sa.pass = pass;
        sa.F = pass == 0 ? F1 : F2;
        sa.logF = pass == 0 ? g.b1 : g.b2;
        sa.shift = pass == 0 ? 0 : g.b1;
        sa.bits = g.bits;
        sa.b1 = g.b1;
        sa.F1 = F1;
        sa.F2 = g.passes == 2 ? F2 : 1;
        sa.cg = cg;
        sa.inR = pass == 0 ? R : s.tmp1;
        sa.inS = pass == 0 ? S : s.tmp1 + nR;
        tuple_v *out = pass == 0 ? s.tmp1 : s.tmp2;
        sa.outR = out;
        sa.outS = out + nR;
        sa.nR = nR;
        sa.nS = nS;
        sa.prefix = s.prefix;
        sa.start = s.start;
        sa.unit_off = s.unit_off;
        sa.unit_cnt = s.unit_cnt;
        sa.subpre = s.subhist;
        sa.seg_head = segm ? s.seg_head : nullptr;
        sa.seg_next = segm ? s.seg_next : nullptr;
        sa.max_segs = segm ? s.max_segs : 0;
        sa.test_stall = (pass == 0 && (test_flags & 1)) ? 1 : 0;
        sa.counters = s.counters;
        sa.ctr_item = pass == 0 ? kCtrItem1 : kCtrItem2;
        sa.item_base = sa.item_end = 0;
        sa.ci_out = (pass == g.passes - 1) ? ci_ok : 0;
        sa.ci_z0 = skip0 ? 1 : 0;
        sa.outR8 = reinterpret_cast<unsigned long long *>(out);
        sa.outS8 = sa.outR8 + nR;
        sa.w8 = 0;
        sa.w8_out = (exact_words && pass == 0) ? 1 : 0;
        sa.inR8 = reinterpret_cast<const unsigned long long *>(s.tmp1);
        sa.inS8 = sa.inR8 + nR;
        const bool words_in = (segm && seg_words) || (exact_words && pass == 1);
        // One pass over [item_base, item_end): after a pass 1 that may have stored words, the launch over
        // 4096-word tiles and the tuple launch after it (which runs only if pass 1 stored tuples).
        auto launch_scatter = [&](bool stable) {
#define HJ_SCATTER(ST)                                                                                         \
    if (words_in) {                                                                                            \
        sa.w8 = 1;                                                                                             \
        scatter_kernel<kScatterThreads, 2 * kScatterItems, ST, kScatterBufs, scatter_word_ctas(ST), true>       \
            <<<num_sms * scatter_word_ctas(ST), kScatterThreads, scatter_smem_bytes(ST), st>>>(sa);            \
        nlaunch++;                                                                                             \
        sa.w8 = 2;                                                                                             \
    }                                                                                                          \
    if (g.mix && pass == 0)                                                                                     \
        scatter_kernel<kScatterThreads, kScatterItems, ST, kScatterBufs, kScatterCtasPerSm, false, true>         \
            <<<scatter_grid, kScatterThreads, scatter_smem_bytes(ST), st>>>(sa);                               \
    else                                                                                                       \
        scatter_kernel<kScatterThreads, kScatterItems, ST, kScatterBufs, kScatterCtasPerSm>                      \
            <<<scatter_grid, kScatterThreads, scatter_smem_bytes(ST), st>>>(sa)
            if (stable) {
                HJ_SCATTER(true);
            } else {
                HJ_SCATTER(false);
            }
#undef HJ_SCATTER
        };
        if (stable) {
            // Ordered first-match joins need each final build partition in input order (the join keeps
            // the lowest position among equal keys), so the build relation's items take the stable rank.
            // The probe relation's order inside a partition changes nothing (each probe tuple finds its
            // first match on its own), so its items take the cheaper atomic rank, in a second launch.
            const uint32_t per_chunk = pass == 0 ? cg.spc : (uint32_t)F1;
            const uint32_t r_items = cg.cR * per_chunk, all_items = (cg.cR + cg.cS) * per_chunk;
            sa.item_end = r_items;
            if (r_items) {
                launch_scatter(true);
                nlaunch++;
            }
            sa.item_base = r_items;
            sa.item_end = all_items;
            sa.ctr_item = pass == 0 ? kCtrItem1S : kCtrItem2S;
            sa.test_stall = 0;
            sa.w8 = 0;
            if (all_items > r_items) launch_scatter(false);
        } else {
            launch_scatter(false);
        }
        HJ_CU(cudaGetLastError());
        nlaunch++;
        HJ_PH(segm ? 3 : 3 + pass);
    }
    if (ph && g.passes == 1 && !g.single) HJ_CU(record_event(ph[4], st));
    if (ev_mid) HJ_CU(record_event(ev_mid, st));

    // 6. joins
    const JoinArgs ja = join_args(g, lp, skip0, R, nR, s, acc, mat, ci_ok, (seg_words || exact_words) ? g.b1 : -1,
                                  g.single && !mat ? host_out : nullptr);
    const MultiRef none = {};
    if (ja.lp_pos) {
        if (mat) {
            join_first_words_kernel<false, true><<<num_sms, kJoinThreads, kFwSmem, st>>>(ja, none);
            join_first_kernel<true><<<num_sms, kJoinThreads, kFirstSmem, st>>>(ja, none);
            nlaunch++;
        } else {
            // One launch per element layout; the one that does not match the device's choice returns at once.
            join_first_words_kernel<false><<<num_sms, kJoinThreads, kFwSmem, st>>>(ja, none);
            join_first_kernel<false><<<num_sms, kJoinThreads, kFirstSmem, st>>>(ja, none);
            nlaunch++;
        }
        nlaunch++;
    } else if (mat && g.single) {
        join_words_kernel<false, true><<<num_sms * 2, kCompactThreads, kOaSmem, st>>>(ja, none);
        join_small_kernel<true><<<num_sms, kJoinThreads, kJoinSmem, st>>>(ja, none);
        nlaunch += 2;
    } else if (mat) {
        if (lp)
            join_compact_kernel<true, false, true><<<num_sms * 2, kCompactThreads, kCompactSmem, st>>>(ja);
        else
            join_compact_kernel<true><<<num_sms * 2, kCompactThreads, kCompactSmem, st>>>(ja);
        join_small_kernel<true><<<num_sms, kJoinThreads, kJoinSmem, st>>>(ja, none);
        nlaunch += 2;
    } else if (g.single) {
        // One launch per element layout; the one that does not match the device's choice returns at once.
        join_words_kernel<false><<<num_sms * 2, kCompactThreads, kOaSmem, st>>>(ja, none);
        join_small_kernel<false, false><<<num_sms, kJoinThreads, kJoinSmem, st>>>(ja, none);
        nlaunch += 2;
    } else {
        // One launch per partition layout (tuples, compact words); the one that does not match the
        // device's choice returns at once.
        if (lp)
            join_compact_kernel<false, false, true><<<num_sms * 2, kCompactThreads, kCompactSmem, st>>>(ja);
        else
            join_compact_kernel<false, false><<<num_sms * 2, kCompactThreads, kCompactSmem, st>>>(ja);
        join_small_kernel<false, false><<<num_sms, kJoinThreads, kJoinSmem, st>>>(ja, none);
        nlaunch += 2;
        if (ci_ok) {
            if (lp && !ordered) {
                join_words_kernel<false, false, true><<<num_sms * 2, kCompactThreads, kOaSmem, st>>>(ja, none);
            } else if (lp) {
                join_compact_kernel<false, true, true><<<num_sms * 2, kCompactThreads, kCompactSmem, st>>>(ja);
                join_small_kernel<false, true><<<num_sms, kJoinThreads, kJoinSmem, st>>>(ja, none);
                nlaunch++;
            } else {
                join_words_kernel<false><<<num_sms * 2, kCompactThreads, kOaSmem, st>>>(ja, none);  // items of every size
            }
            nlaunch++;
        }
    }
    HJ_CU(cudaGetLastError());
    HJ_PH(segm ? 4 : 5);
    if (!ja.host_out) {
        const int rc = large_launch(ja, mat != nullptr, s, acc, st, num_sms);
        if (rc) return rc;
        nlaunch += 4;
    }
    HJ_PH(segm ? 5 : 6);
    if (launches) *launches = nlaunch;
#undef HJ_PH
    return HJ_OK;
}

}  // namespace hj
