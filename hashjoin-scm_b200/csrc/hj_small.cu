// hj_small.cu - joins whose build relation fits one CTA's shared memory, as one kernel.
//
// A build relation of at most kSmallMaxBuild tuples needs neither partitions nor a global table: every
// CTA builds the whole table in its own shared memory (from L2 after the first) and probes its share of
// the probe relation, which is read once. The pipelines' dozen launches, memsets and copies cost such a
// join 90-160 us, of which its data took a few. The CTA that finishes last adds up the CTAs' partial
// results and writes them to the caller's pinned host record, so there is nothing to clear before and
// nothing to copy after the kernel (whole calls: phj_radix_bc 1000 x 4000 158 -> 29 us).
//
// The table, where every match counts: tuples, 32-bit bucket heads and 16-bit chain links by build position (at
// most 176 KB, one CTA of 1024 threads per SM). Keys may share low bits, so buckets are taken from the top of a
// multiplicative hash. First-match joins need one place per key, not a walk over its duplicates (8192 build
// tuples on eight keys, 2^22 probes: 3050 us with chains, 42 with one place): an open-addressing table of
// build positions, at most half full, in which equal keys lower the position they share, and a bit per slot that
// tells which two tuples share (at most 194 KB). Bound by the read of the probe relation (four 16-byte
// loads per thread in flight) when that is large, else by the latency of its four dependent steps.
#include <cstdio>

#include "hj_common.cuh"
#include "hj_internal.h"
#include "hj_partition.cuh"
#include "hj_wave.cuh"

namespace hj {

constexpr int kSmallThreads = 1024;

struct SmallArgs {
    const tuple_v *R, *S;
    uint32_t nR;
    uint64_t nS;
    int nb_log;       // buckets
    int lp, skip0;
    int flag_bits;    // radix bits of the HJ_RES_COMPACT_PARTITIONS test; -1: not a radix join
    SmallPart *part;  // [gridDim.x]
    uint32_t *ticket; // 0 before and after every join
    JoinAccum *out;   // pinned host memory
};

// In dynamic shared memory: 2^nb_log heads with chains, or (lp) twice as many slots and their duplicate bits.
struct SmallTable {
    tuple_v *rt;        // [nR]
    uint32_t *head;     // [2^nb_log], or slots [2^(nb_log + 1)]
    uint16_t *nxt;      // [nR]
    uint32_t *dup;      // [slots / 32]
    uint32_t entries;   // heads or slots
    int shift;
    __device__ __forceinline__ SmallTable(unsigned char *smem, uint32_t nR, int nb_log, bool lp)
        : rt(reinterpret_cast<tuple_v *>(smem)), head(reinterpret_cast<uint32_t *>(rt + nR)),
          entries(1u << (nb_log + (lp ? 1 : 0))), shift(64 - nb_log - (lp ? 1 : 0)) {
        nxt = reinterpret_cast<uint16_t *>(head + entries);
        dup = head + entries;
    }
    __device__ __forceinline__ uint32_t bucket(unsigned long long key) const {
        return (uint32_t)((key * 0x9e3779b97f4a7c15ull) >> shift);
    }
};

struct SmallSums {
    unsigned long long cnt = 0, sum = 0, kor = 0, ror = 0, sor = 0;
    bool multi = false, over = false;
};

// Build the whole table and probe it with S[j0], S[j0 + stride], ... below end. All threads of the block.
__device__ __forceinline__ void small_block(const SmallTable &tb, const tuple_v *R, uint32_t nR, bool lp, bool skip0,
                                            const tuple_v *S, uint64_t j0, uint64_t stride, uint64_t end,
                                            SmallSums &o) {
    const int tid = threadIdx.x;
    constexpr int UR = kSmallMaxBuild / kSmallThreads, U = 4;
    // The first probe tuples are requested before the build.
    tuple_v s[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint64_t j = j0 + u * stride;
        s[u] = j < end ? ld_stream(S + j) : make_ulonglong2(0, 0);
    }
    tuple_v t[UR];
#pragma unroll
    for (int u = 0; u < UR; u++) {
        const uint32_t i = tid + u * kSmallThreads;
        if (i < nR) t[u] = __ldg(R + i);
    }
    for (uint32_t q = tid; q < tb.entries; q += kSmallThreads) tb.head[q] = 0;
    if (lp)
        for (uint32_t q = tid; q < (tb.entries + 31) / 32; q += kSmallThreads) tb.dup[q] = 0;
#pragma unroll
    for (int u = 0; u < UR; u++) {
        const uint32_t i = tid + u * kSmallThreads;
        if (i >= nR) break;
        tb.rt[i] = t[u];
        o.kor |= t[u].x;
        o.ror |= t[u].y;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < UR; u++) {
        const uint32_t i = tid + u * kSmallThreads;
        if (i >= nR) break;
        const unsigned long long k = tb.rt[i].x;
        if (skip0 && k == 0) continue;
        uint32_t h = tb.bucket(k);
        if (!lp) {
            tb.nxt[i] = (uint16_t)atomicExch(&tb.head[h], i + 1);
            continue;
        }
        for (uint32_t steps = 0;; h = (h + 1) & (tb.entries - 1)) {
            const uint32_t cur = atomicCAS(&tb.head[h], 0u, i + 1);
            if (!cur) break;
            if (tb.rt[cur - 1].x == k) {
                atomicMin(&tb.head[h], i + 1);
                atomicOr(&tb.dup[h >> 5], 1u << (h & 31));
                break;
            }
            if (++steps >= tb.entries) {
                o.over = true;
                break;
            }
        }
    }
    __syncthreads();
    for (; j0 < end; j0 += U * stride) {
        tuple_v nx[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint64_t j = j0 + (U + u) * stride;
            nx[u] = j < end ? ld_stream(S + j) : make_ulonglong2(0, 0);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (j0 + u * stride >= end) continue;
            o.sor |= s[u].y;
            uint32_t h = tb.bucket(s[u].x), steps = 0;
            uint32_t e = tb.head[h];
            while (e) {
                const tuple_v r = tb.rt[e - 1];
                if (r.x == s[u].x) {
                    o.cnt++;
                    o.sum += r.y + s[u].y;
                    if (lp) {
                        o.multi |= (tb.dup[h >> 5] >> (h & 31)) & 1u;
                        break;
                    }
                }
                h = (h + 1) & (tb.entries - 1);
                e = lp ? tb.head[h] : tb.nxt[e - 1];
                if (++steps > tb.entries) {
                    o.over = true;
                    break;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) s[u] = nx[u];
    }
}

// Many small joins: block b takes the probe range chunks[b] of its job.
__global__ void __launch_bounds__(kSmallThreads, 1) small_multi(const SmallJob *__restrict__ jobs,
                                                               const MChunk *__restrict__ chunks) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned long long red[64];
    const MChunk ch = chunks[blockIdx.x];
    const SmallJob J = jobs[ch.job];
    const SmallTable tb(smem, J.nR, J.nb_log, J.lp != 0);
    SmallSums o;
    small_block(tb, J.R, J.nR, J.lp != 0, J.skip0 != 0, J.S, ch.begin + threadIdx.x, kSmallThreads,
                ch.begin + ch.len, o);
    block_sum2_to(o.cnt, o.sum, red, &J.acc->matched, &J.acc->checksum);
    if (__syncthreads_or(o.over) && threadIdx.x == 0) set_error(&J.acc->error, kErrProbeLimit);
}

__global__ void __launch_bounds__(kSmallThreads, 1) small_join(SmallArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned long long s_red[5][kSmallThreads / 32];
    __shared__ bool s_last;
    const int tid = threadIdx.x;
    const SmallTable tb(smem, a.nR, a.nb_log, a.lp != 0);
    SmallSums o;
    small_block(tb, a.R, a.nR, a.lp != 0, a.skip0 != 0, a.S, (uint64_t)blockIdx.x * kSmallThreads + tid,
                (uint64_t)gridDim.x * kSmallThreads, a.nS, o);
    unsigned long long cnt = o.cnt, sum = o.sum, kor = o.kor, ror = o.ror, sor = o.sor;
    const bool multi = o.multi, over = o.over;
    // This CTA's partial result: sums, ORs and flags.
    const unsigned lane = lane_id(), w = tid >> 5;
    cnt = warp_sum_u64(cnt);
    sum = warp_sum_u64(sum);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        kor |= __shfl_xor_sync(0xffffffffu, kor, o);
        ror |= __shfl_xor_sync(0xffffffffu, ror, o);
        sor |= __shfl_xor_sync(0xffffffffu, sor, o);
    }
    if (lane == 0) {
        s_red[0][w] = cnt;
        s_red[1][w] = sum;
        s_red[2][w] = kor;
        s_red[3][w] = ror;
        s_red[4][w] = sor;
    }
    const bool any_multi = __syncthreads_or(multi), any_over = __syncthreads_or(over);
    if (w == 0) {
        cnt = warp_sum_u64(s_red[0][lane]);
        sum = warp_sum_u64(s_red[1][lane]);
        kor = s_red[2][lane];
        ror = s_red[3][lane];
        sor = s_red[4][lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            kor |= __shfl_xor_sync(0xffffffffu, kor, o);
            ror |= __shfl_xor_sync(0xffffffffu, ror, o);
            sor |= __shfl_xor_sync(0xffffffffu, sor, o);
        }
        if (lane == 0) {
            SmallPart p;
            p.cnt = cnt;
            p.sum = sum;
            p.sor = sor;
            p.multi = any_multi;
            p.over = any_over;
            a.part[blockIdx.x] = p;
            __threadfence();
            s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!s_last || w != 0) return;
    __threadfence();
    unsigned long long tc = 0, ts = 0, to = 0;
    bool tm = false, tv = false;
    for (uint32_t q = lane; q < gridDim.x; q += 32) {
        const volatile SmallPart *p = a.part + q;
        tc += p->cnt;
        ts += p->sum;
        to |= p->sor;
        tm |= p->multi != 0;
        tv |= p->over != 0;
    }
    tc = warp_sum_u64(tc);
    ts = warp_sum_u64(ts);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) to |= __shfl_xor_sync(0xffffffffu, to, o);
    tm = __any_sync(0xffffffffu, tm);
    tv = __any_sync(0xffffffffu, tv);
    if (lane == 0) {
        JoinAccum r = {};
        r.matched = tc;
        r.checksum = ts;
        r.error = tv ? kErrProbeLimit : 0u;
        r.dup_flag = tm ? 1u : 0u;
        // Every CTA has seen the whole build relation, so kor and ror are its ORs.
        if (a.flag_bits >= 0 && (kor >> a.flag_bits) < (1ull << 31) && ror < (1ull << 32) && to < (1ull << 32))
            r.flags = HJ_RES_COMPACT_PARTITIONS;
        *a.out = r;
        *a.ticket = 0;
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

static int small_buckets_log(size_t nR) {
    int b = 1;
    while ((1u << b) < nR) b++;
    return b;
}

// Shared memory of a join: tuples, then heads and links, or (lp) slots and their duplicate bits. A wave takes the
// larger form for its largest build side.
static size_t small_smem(size_t nR, bool lp) {
    const size_t heads = (size_t)1 << small_buckets_log(nR);
    return nR * 16 + (lp ? 2 * heads * 4 + (2 * heads + 31) / 32 * 4 : heads * 4 + nR * 2);
}

int small_prepare_device() {
    const int most = (int)small_smem(kSmallMaxBuild, true);
    HJ_CU(cudaFuncSetAttribute(small_multi, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    HJ_CU(cudaFuncSetAttribute(small_join, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    return HJ_OK;
}

void small_job(bool lp, bool skip0, const ulonglong2 *R, size_t nR, const ulonglong2 *S, JoinAccum *acc, SmallJob *j) {
    j->R = R;
    j->S = S;
    j->acc = acc;
    j->nR = (uint32_t)nR;
    j->nb_log = small_buckets_log(nR);
    j->lp = lp ? 1u : 0u;
    j->skip0 = skip0 ? 1u : 0u;
}

int small_multi_launch(const SmallJob *jobs, const MChunk *chunks, unsigned nchunks, size_t max_build, cudaStream_t st) {
    small_multi<<<nchunks, kSmallThreads, small_smem(max_build, true), st>>>(jobs, chunks);
    HJ_CU(cudaGetLastError());
    return HJ_OK;
}

int small_enqueue(bool lp, bool skip0, int flag_bits, const ulonglong2 *R, size_t nR, const ulonglong2 *S, size_t nS,
                  SmallPart *part, uint32_t *ticket, JoinAccum *out_host, cudaStream_t st, int num_sms) {
    if (nR > kSmallMaxBuild) return HJ_E_INVAL;
    SmallArgs a;
    a.R = R;
    a.S = S;
    a.nR = (uint32_t)nR;
    a.nS = nS;
    a.nb_log = small_buckets_log(nR);
    a.lp = lp ? 1 : 0;
    a.skip0 = skip0 ? 1 : 0;
    a.flag_bits = flag_bits;
    a.part = part;
    a.ticket = ticket;
    a.out = out_host;
    const uint64_t want = ((uint64_t)nS + kSmallThreads - 1) / kSmallThreads;
    const uint64_t sms = (uint64_t)(num_sms < kSmallMaxGrid ? num_sms : kSmallMaxGrid);
    const unsigned grid = (unsigned)(want < 1 ? 1 : want < sms ? want : sms);
    small_join<<<grid, kSmallThreads, small_smem(nR, lp), st>>>(a);
    HJ_CU(cudaGetLastError());
    return HJ_OK;
}

}  // namespace hj
