// hj_partition.cuh - plan structures, compact words and counters shared by the kernels of the radix
// joins: the two-pass pipelines (hj_partition.cu) and the one-pass pipeline (hj_single.cu).
#pragma once

#include "hj_common.cuh"
#include "hj_internal.h"

namespace hj {

// ------------------------------------------------------------------------------------------------
// Device-side plan structures
// ------------------------------------------------------------------------------------------------
struct JoinItem {
    uint64_t r_begin;  // index into the final R buffer
    uint64_t s_begin;  // index into the final S buffer
    uint32_t r_len;
    uint32_t s_len;
    uint32_t part0;    // 1: the partition of the keys whose radix bits are 0 (key 0's partition)
    uint32_t pad;
};

struct LargePart {
    uint64_t r_begin, s_begin;
    uint64_t r_len, s_len;
    uint64_t table_off;  // u32 words into the large table: head[nb] then next[r_len]
    uint64_t r_flat, s_flat;
    uint32_t nb_log;
    uint32_t part0;  // as JoinItem::part0
};

// counters[] slots
enum : int {
    kCtrItem1 = 0,       // scatter pass-1 work-item counter
    kCtrItem2 = 1,       // scatter pass-2 work-item counter
    kCtrNItemsA = 2,     // join items whose build side fits the compact shared-memory table (listed first)
    kCtrItemA = 3,       // compact join work-item counter
    kCtrSegAlloc = 4,    // segment mode: segment ids handed out
    kCtrLargeAgg = 5,    // 1: large partitions use key-aggregated tables (see join_large_build)
    kCtrNItems = 6,
    kCtrNLarge = 7,
    kCtrItem = 8,        // join work-item counter
    kCtrLargeR = 9,      // total R tuples in large partitions (u32 pairs: lo, hi)
    kCtrLargeS = 11,     // total S tuples in large partitions (lo, hi)
    kCtrLargeWords = 13, // table words used (lo, hi)
    kCtrErr = 15,
    kCtrMaxKey = 16,     // u64: OR of all R keys (words 16-17)
    kCtrMaxRid = 18,     // u64: OR of all R row ids (words 18-19)
    kCtrOrRidS = 20,     // u64: OR of all S row ids (words 20-21)
    kCtrItem1S = 22,     // first-match joins: pass-1 work-item counter of the probe relation's items
    kCtrItem2S = 23,     // first-match joins: pass-2 work-item counter of the probe relation's items
    kCtrTicket = 24,     // one-pass pipeline: CTAs of single_plan that have written their totals
    kCtrTicketJoin = 25, // one-pass pipeline: CTAs of the partition join that have finished
    kCtrSegWide = 26,    // segment mode: the word pass 1 met a value too wide for words and stopped
    kNumCounters = 28
};

// Compact final partitions. When every build key shifted right by the radix bits is below 2^31 and
// every row id (build and probe) below 2^32, the last partition pass stores each tuple as one 8-byte
// word, (key >> bits) << 32 | row id, and the joins read 8 bytes per tuple instead of 16. Inside a
// final partition the low `bits` key bits are equal, so comparing key >> bits compares keys. A probe
// key whose high part is 2^31 or more is stored as 0xffffffff: no build key has that high part. Joins
// where a build key 0 never matches (lp_join's empty-slot rule): a last pass that reads tuples stores
// that key's words with high part 0x80000000, which no build key and no probe word has (ci_word_z0);
// from segment-mode pass-1 words it keeps high part 0, and since key 0 lies in the partition of the
// keys whose radix bits are 0, where a high part of 0 means key 0, the joins skip such build words
// there (JoinItem::part0). The widths are ORed together by the pass that reads the relations first (hist_chunk_kernel or
// seg_pass1_kernel), so the choice is made on the device, before the last pass.
__device__ __forceinline__ bool ci_applies(const uint32_t *counters, int bits) {
    const unsigned long long *mx = reinterpret_cast<const unsigned long long *>(counters + kCtrMaxKey);
    return (mx[0] >> bits) < (1ull << 31) && mx[1] < (1ull << 32) && mx[2] < (1ull << 32);
}

// Segment mode can go further: pass 1 stores (key >> b1) << 32 | row id (w8_word) in segments of 4096
// words (the same 32 KB as 2048 tuples) when every build key >> b1 is below 2^31 and every row id below
// 2^32; pass 2 then reads 8-byte words in tiles of 4096 and writes compact final partitions. A probe
// key whose key >> b1 does not fit keeps its low 31 bits and gets bit 31 set: its pass-2 digit stays
// right, and after pass 2's shift its high part is still above every build key's.
__device__ __forceinline__ bool w8_fits(const uint32_t *counters, int b1) {
    const unsigned long long *mx = reinterpret_cast<const unsigned long long *>(counters + kCtrMaxKey);
    return (mx[0] >> b1) < (1ull << 31) && mx[1] < (1ull << 32) && mx[2] < (1ull << 32);
}

__device__ __forceinline__ unsigned long long w8_word(unsigned long long key, unsigned long long rid, int b1) {
    const unsigned long long hi = key >> b1;
    const unsigned long long h32 = hi < (1ull << 31) ? hi : (0x80000000ull | (hi & 0x7fffffffull));
    return (h32 << 32) | (rid & 0xffffffffull);
}

// Build relations whose key 0 never matches (z0), in the exact-offset pipeline's word pass 1: key 0's
// word takes the high part 0x80000000, which no other build word has; the last pass keeps it
// (store_elem) and stores every probe word whose high part has bit 31 set as 0xffffffff, so nothing
// matches it. (Segment mode's pass 1 stores key 0 as any key; the joins skip it in its partition.)
__device__ __forceinline__ unsigned long long w8_word_z0(unsigned long long key, unsigned long long rid, int b1,
                                                         bool z0) {
    return z0 && key == 0 ? (0x80000000ull << 32) | (rid & 0xffffffffull) : w8_word(key, rid, b1);
}

__device__ __forceinline__ unsigned long long ci_word(unsigned long long key, unsigned long long rid, int bits) {
    const unsigned long long hi = key >> bits;
    return ((hi < 0x80000000ull ? hi : 0xffffffffull) << 32) | (rid & 0xffffffffull);
}

__device__ __forceinline__ unsigned long long ci_word_z0(unsigned long long key, unsigned long long rid, int bits,
                                                         bool z0) {
    return z0 && key == 0 ? (0x80000000ull << 32) | (rid & 0xffffffffull) : ci_word(key, rid, bits);
}

// Build partitions up to this size whose keys (above the radix bits) and row ids fit 32 bits are
// joined with a 4-byte-per-field shared-memory table, two CTAs per SM.
constexpr int kCompactCap = 8192;
constexpr int kCompactThreads = 512;
// Largest build partition of the one-pass pipeline's first-match join.
constexpr int kFirstCap = 9216;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// Bounded wait for the completion of phase `parity` of an mbarrier.
__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for an mbarrier phase: gives up after kWaitNs of wall time (try_wait may suspend the
// thread for a hardware-defined time per call, so an iteration count alone is no time bound).
constexpr uint64_t kWaitNs = 2000000000ull;
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity) {
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t it = 0; it < (1u << 30); it++) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 63u) == 63u && globaltimer_ns() - t0 > kWaitNs) return false;
    }
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    return mbar_try(bar, parity) || mbar_wait_slow(bar, parity);
}

// TMA bulk copy global -> shared of `bytes` (a multiple of 16, <= 1 MiB per phase), completing on
// `bar`. Issued by one thread.
__device__ __forceinline__ void tma_load_1d(void *dst_smem, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    const char *s = reinterpret_cast<const char *>(src);
    const uint32_t d = smem_addr(dst_smem);
    for (uint32_t off = 0; off < bytes; off += 32768u) {
        const uint32_t sz = bytes - off < 32768u ? bytes - off : 32768u;
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(d + off),
            "l"(s + off), "r"(sz), "r"(bar)
            : "memory");
    }
}

// Segment mode (hj_segments.cu).
constexpr uint32_t kSegSlab = 32;          // segment ids a CTA takes from the global counter at once
constexpr int kSegCtasPerSm = 2;           // shared memory: two tile buffers + 32 KB of counters
constexpr int kSegMaxBits = 14;
int seg_prepare_device(bool mix);
// Pass 1 into segment chains, with the per-CTA histograms. words_too: in 8-byte words where the widths allow them;
// stable: every build partition keeps input order (ordered first-match joins); stall: the test hook.
int seg_pass1_enqueue(const RadixGeom &g, const ulonglong2 *R, size_t nR, const ulonglong2 *S, size_t nS,
                      const PhjScratch &s, bool words_too, bool stable, bool stall, cudaStream_t st, uint32_t *launches);

// Lanes of the warp whose digit equals this lane's: one ballot per digit bit (NB bits).
template <int NB>
__device__ __forceinline__ unsigned digit_peers(uint32_t d) {
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const unsigned bit = (d >> b) & 1u;
        const unsigned bal = __ballot_sync(0xffffffffu, bit);
        peers &= bal ^ (bit - 1u);  // bit ? bal : ~bal
    }
    return peers;
}

// Chunking of the two relations (identical for the histogram and both scatter passes).
struct ChunkGeom {
    uint64_t chunk;  // tuples per chunk (a multiple of the tile)
    uint32_t cR, cS; // chunks of R, chunks of S (R's come first)
    uint64_t sub;    // tuples per sub-chunk (a multiple of the tile): the pass-1 work item
    uint32_t spc;    // sub-chunks per chunk
    uint32_t pad;
};

// The key that a pass partitions by and stores where the geometry says so (RadixGeom::mix): the low `bits` bits
// changed by a hash of those above, which stay, so equal keys stay equal, distinct ones distinct, 0
// stays 0, and a run of 2^bits consecutive keys still takes every digit once. Keys with a stride, or with their
// ids in the high half, then spread over the partitions evenly (strides of 1..64 and of powers of 2 and 10 up to
// 2^43, 2^20 to 6e6 keys: the largest partition at most 1.11 times the average), where their own low bits put them
// into a few that no longer fit shared memory. Two 32-bit products (a 64-bit one costs the one-pass scatter 6%,
// these 4%), with odd multipliers taken for that evenness out of a dozen pairs, and because the runs that such keys
// make in the joins' tables, which hash the same bits, stay below 13 slots (others: up to 135).
constexpr uint32_t kMixLow = 0x7feb352du, kMixHigh = 0x846ca68bu;
__device__ __forceinline__ unsigned long long mix_key(unsigned long long key, int bits) {
    return key ^ ((((uint32_t)key >> bits) * kMixLow + (uint32_t)(key >> 32) * kMixHigh) >> (32 - bits));
}

__device__ __forceinline__ uint64_t ld_u64_pair(const uint32_t *p) {
    return (uint64_t)p[0] | ((uint64_t)p[1] << 32);
}
__device__ __forceinline__ void st_u64_pair(uint32_t *p, uint64_t v) {
    p[0] = (uint32_t)v;
    p[1] = (uint32_t)(v >> 32);
}

__host__ __device__ __forceinline__ uint32_t ceil_div_u64(uint64_t a, uint64_t b) {
    return (uint32_t)((a + b - 1) / b);
}

struct PlanArgs {
    int bits, passes, b1, F1, F2;
    uint64_t nR, nS;
    const uint32_t *total;  // [2][2^B]
    uint64_t *start;        // [2][2^B + 1]
    uint32_t *counters;
    JoinItem *items;
    uint64_t max_items;
    LargePart *large;
    uint64_t max_large;
    uint64_t large_table_words;
    uint64_t small_cap;  // build partitions above this many tuples are large
    int agg_ok;  // joins that need no per-match output may use key-aggregated large-partition tables
};

__device__ __forceinline__ uint32_t part_to_value(int f, int passes, int b1, int F2) {
    if (passes == 1) return (uint32_t)f;
    const uint32_t d1 = (uint32_t)f / (uint32_t)F2, d2 = (uint32_t)f % (uint32_t)F2;
    return d1 | (d2 << b1);
}

// u32 words of one large partition's table. Chains: head[nb] then next[r_len]. Key-aggregated:
// sum[r_len] (u64), head[nb], next[r_len], cnt[r_len], negpos[r_len], rounded to an even count so the
// next table's sums stay 8-byte aligned.
__device__ __forceinline__ uint64_t large_words_chain(const LargePart &L) { return (1ull << L.nb_log) + L.r_len; }
__device__ __forceinline__ uint64_t large_words_agg(const LargePart &L) {
    return ((1ull << L.nb_log) + 5 * L.r_len + 1) & ~1ull;
}

// Final partition starts, join work items and large partitions from the relation totals tot_all
// ([2][2^B], readable by the calling CTA of 1024 threads). tmp: 32 u32, s_run: 2 u64 of shared memory.
__device__ __forceinline__ void plan_body(const PlanArgs &a, const uint32_t *tot_all, uint32_t *tmp, uint64_t *s_run) {
    const int tid = threadIdx.x;
    const int nparts = 1 << a.bits;
    // Each thread owns a contiguous range of partitions.
    const int per = (nparts + 1023) / 1024;
    const int f0 = tid * per < nparts ? tid * per : nparts;
    const int f1 = f0 + per < nparts ? f0 + per : nparts;
    uint64_t base[2];  // start of this thread's first partition, per relation
    for (int rel = 0; rel < 2; rel++) {
        uint64_t *start = a.start + (size_t)rel * (nparts + 1);
        const uint32_t *tot = tot_all + (size_t)rel * nparts;
        uint32_t sum = 0;
        for (int f = f0; f < f1; f++) sum += tot[part_to_value(f, a.passes, a.b1, a.F2)];
        uint32_t all;
        uint64_t run = block_excl_scan_u32(sum, tmp, &all);
        base[rel] = run;
        for (int f = f0; f < f1; f++) {
            start[f] = run;
            run += tot[part_to_value(f, a.passes, a.b1, a.F2)];
        }
        if (tid == 0) start[nparts] = all;
    }

    // Join work items (partitions with both sides non-empty, src/algo/phj.c:459-491) and large
    // partitions. Partition sizes come from the totals, starts from the running sums above.
    const uint32_t *totR = tot_all, *totS = tot_all + nparts;
    const uint64_t small_cap = a.small_cap;
    uint32_t asum = 0, bsum = 0, lsum = 0;  // items with |R_p| <= compact cap, other small items, large
    for (int f = f0; f < f1; f++) {
        const uint32_t v = part_to_value(f, a.passes, a.b1, a.F2);
        const uint64_t nr = totR[v], ns = totS[v];
        if (nr > 0 && ns > 0) {
            if (nr <= (uint64_t)kCompactCap) asum += ceil_div_u64(ns, kProbeChunk);
            else if (nr <= small_cap) bsum += ceil_div_u64(ns, kProbeChunk);
            else lsum++;
        }
    }
    uint32_t atot, btot, ltot;
    uint64_t a_idx = block_excl_scan_u32(asum, tmp, &atot);
    uint64_t b_idx = block_excl_scan_u32(bsum, tmp, &btot) + atot;
    uint64_t large_idx = block_excl_scan_u32(lsum, tmp, &ltot);
    const uint32_t ktot = atot + btot;
    uint64_t rR = base[0], rS = base[1];
    for (int f = f0; f < f1; f++) {
        const uint32_t v = part_to_value(f, a.passes, a.b1, a.F2);
        const uint64_t nr = totR[v], ns = totS[v];
        const uint64_t sR = rR, sS = rS;
        rR += nr;
        rS += ns;
        if (!(nr > 0 && ns > 0)) continue;
        if (nr <= small_cap) {
            uint64_t &item_idx = nr <= (uint64_t)kCompactCap ? a_idx : b_idx;
            const uint32_t k = ceil_div_u64(ns, kProbeChunk);
            for (uint32_t q = 0; q < k; q++, item_idx++) {
                if (item_idx < a.max_items) {
                    JoinItem it;
                    it.r_begin = sR;
                    it.s_begin = sS + (uint64_t)q * kProbeChunk;
                    it.r_len = (uint32_t)nr;
                    const uint64_t rem = ns - (uint64_t)q * kProbeChunk;
                    it.s_len = (uint32_t)(rem < (uint64_t)kProbeChunk ? rem : (uint64_t)kProbeChunk);
                    it.part0 = v == 0 ? 1u : 0u;
                    it.pad = 0;
                    a.items[item_idx] = it;
                } else {
                    atomicOr(&a.counters[kCtrErr], kErrCapacity);
                }
            }
        } else {
            if (large_idx < a.max_large) {
                LargePart lp;
                lp.r_begin = sR;
                lp.s_begin = sS;
                lp.r_len = nr;
                lp.s_len = ns;
                uint32_t nb_log = 0;
                while ((1ull << nb_log) < nr) nb_log++;
                lp.nb_log = nb_log;
                lp.part0 = v == 0 ? 1u : 0u;
                lp.table_off = 0;
                lp.r_flat = lp.s_flat = 0;
                a.large[large_idx] = lp;
            } else {
                atomicOr(&a.counters[kCtrErr], kErrCapacity);
            }
            large_idx++;
        }
    }
    if (tid == 0) a.counters[kCtrNItemsA] = atot < a.max_items ? atot : (uint32_t)a.max_items;
    if (tid == 0) {
        s_run[0] = ktot;
        s_run[1] = ltot;
    }
    __syncthreads();
    const uint64_t item_run = s_run[0], large_run = s_run[1];
    __syncthreads();
    if (tid == 0) {
        const uint64_t nl = large_run < a.max_large ? large_run : a.max_large;
        // Key-aggregated tables (large_words_agg) when the join allows them and they fit the table
        // area, else plain chains (large_words_chain).
        uint64_t need_agg = 0;
        for (uint64_t l = 0; l < nl; l++) need_agg += large_words_agg(a.large[l]);
        const bool agg = a.agg_ok && need_agg <= a.large_table_words;
        a.counters[kCtrLargeAgg] = agg ? 1u : 0u;
        uint64_t off = 0, rf = 0, sf = 0;
        for (uint64_t l = 0; l < nl; l++) {
            LargePart &lp = a.large[l];
            lp.table_off = off;
            lp.r_flat = rf;
            lp.s_flat = sf;
            off += agg ? large_words_agg(lp) : large_words_chain(lp);
            rf += lp.r_len;
            sf += lp.s_len;
        }
        const bool fits = off <= a.large_table_words;
        if (!fits) atomicOr(&a.counters[kCtrErr], kErrCapacity);
        a.counters[kCtrNItems] = (uint32_t)(item_run < a.max_items ? item_run : a.max_items);
        a.counters[kCtrNLarge] = (uint32_t)nl;
        st_u64_pair(&a.counters[kCtrLargeR], fits ? rf : 0);
        st_u64_pair(&a.counters[kCtrLargeS], fits ? sf : 0);
        st_u64_pair(&a.counters[kCtrLargeWords], fits ? off : 0);
    }
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
    JoinAccum *acc;          // cleared by the count if clear_acc
    int clear_acc;
    int ci_ok;               // compact words allowed
    int lp;                  // first match: build elements carry their input position
    int z0;                  // build key 0 never matches
    tuple_v *outR, *outS;    // tuples
    unsigned long long *outR8, *outS8;  // compact words
};

struct JoinArgs {
    const JoinItem *items;
    const LargePart *large;
    uint32_t *counters;
    const tuple_v *finR, *finS;
    uint32_t *large_table;
    int bits;
    int lp;     // first match per probe tuple (lowest build position) instead of all matches
    int skip0;  // build tuples with key 0 never match (key 0 marks an empty slot in lp_join)
    JoinAccum *acc;
    MatOut mat; // materialising joins (MAT kernels): where the (r.row_id, s.row_id) pairs go
    int ci;     // the final partitions may be compact words (when ci_applies holds) at finR8 / finS8
    const unsigned long long *finR8, *finS8;
    // First-match joins of the one-pass pipeline: build elements are {ci_word or key, input position}, and
    // a wide match reads its row id from the build relation itself.
    int lp_pos;
    const tuple_v *relR;
    uint64_t nR;
    int flag_bits;  // HJ_RES_COMPACT_PARTITIONS tells whether words of this many radix bits fit
    // One-pass pipeline: one launch takes the items of every size; host_out: see join_finish.
    int all_items;
    JoinAccum *host_out;
    int w8_b1;  // a pass 1 that may store words (either pipeline): its shift (reported when w8_fits held); -1 otherwise
};

// Kernels of the one-pass pipeline run on one join (its arguments are the launch's) or on many (MULTI: a
// block's job and its index among the job's blocks come from a map; the job's arguments are copied to shared
// memory). One launch per step then serves a whole wave of joins.
struct MultiJob {
    SingleArgs sa;
    PlanArgs pa;
    JoinArgs ja;
    uint32_t grid;         // blocks of the count and the scatter
    uint32_t plan_blocks;  // blocks of the plan
    uint32_t join_blocks;  // blocks of the partition joins
    uint32_t large_blocks; // blocks of the large-partition probe
};
constexpr int kMultiLargeThreads = 256;
static_assert(sizeof(MultiJob) % 8 == 0 && sizeof(SingleArgs) % 8 == 0 && sizeof(PlanArgs) % 8 == 0 &&
              sizeof(JoinArgs) % 8 == 0, "copied by 8-byte words");

struct MultiRef {
    const MultiJob *jobs;
    const uint2 *map;  // [gridDim.x] {job, block of the job}
};

template <class T>
__device__ __forceinline__ void multi_copy(T *dst, const T *src) {
    static_assert(sizeof(T) % 8 == 0, "8-byte words");
    for (uint32_t i = threadIdx.x; i < sizeof(T) / 8; i += blockDim.x)
        reinterpret_cast<unsigned long long *>(dst)[i] = reinterpret_cast<const unsigned long long *>(src)[i];
}

// Compact words of the probe relation in the one-pass pipeline: behind the build relation's words, or
// behind its 16-byte elements for first-match joins.
inline unsigned long long *single_probe_words(const PhjScratch &s, size_t nR, bool lp) {
    return lp ? reinterpret_cast<unsigned long long *>(s.tmp1 + nR) : reinterpret_cast<unsigned long long *>(s.tmp1) + nR;
}

// Arguments of a radix join's partition joins (hj_partition.cu).
JoinArgs join_args(const RadixGeom &g, bool lp, bool skip0, const ulonglong2 *R, size_t nR, const PhjScratch &s,
                   JoinAccum *acc, const MatOut *mat, int ci_ok, int w8_b1, JoinAccum *host_out);
// Arguments of a one-pass join's partition phase (hj_single.cu).
void single_args(const RadixGeom &g, bool lp, bool skip0, bool ci_ok, const ulonglong2 *R, size_t nR,
                 const ulonglong2 *S, size_t nS, const PhjScratch &s, JoinAccum *acc, bool clear_acc, bool agg_ok,
                 SingleArgs *a, PlanArgs *pa);
// The steps of a wave of one-pass joins (hj_wave.cu): partition phase, partition joins (maps of the joins
// that count every match and of the first-match ones), large partitions and error words (a map of all).
int multi_partition_launch(const MultiJob *jobs, const uint2 *part_map, unsigned part_blocks, const uint2 *plan_map,
                           unsigned plan_blocks, int max_bits, cudaStream_t st, uint32_t *launches);
int multi_join_launch(const MultiJob *jobs, const uint2 *every_map, unsigned every_blocks, const uint2 *first_map,
                      unsigned first_blocks, const uint2 *large_map, unsigned large_blocks, cudaStream_t st,
                      uint32_t *launches);

}  // namespace hj
