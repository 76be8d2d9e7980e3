// hj_shard.cu - routing of tuples to the ranks of a sharded join.
//
// A join sharded over G GPUs sends every tuple to the rank that owns its key, joins locally and adds up
// the G results. Co-partitions of a radix join are independent (src/algo/phj.c:1257-1311), and so are
// the key ranges of any key -> rank function, so one exchange step suffices. The owner of a key is
// mulhi(mix(key ^ 0x5ca1ab1e5eed0001), G): a multiply-xorshift mix (the same family as the tables'
// hash, on a different input) reduced to [0, G) by a multiply-high, so neither the radix digits (the
// low key bits) nor the table hash of a rank's keys is skewed by the routing.
//
// hj_shard_route groups the tuples of one relation by owner, stably: within an owner's range the
// tuples keep their input order, so after an all-to-all that concatenates the ranks' pieces in rank
// order, each rank's build relation is in global input order (first-match joins stay exact).
//
// Kernels (all block ranges are contiguous slices of the input, in block order, four blocks per SM):
//   route_count    per block and owner: tuples. Every lane counts in a shared-memory column of its own, so
//                  that 32 lanes on a few owners do not serialise; four loads per thread in flight
//   route_offsets  one CTA: each block's start per owner (exclusive scan down the columns, then owner
//                  bases), and the owner totals
//   route_scatter  per block, tiles of 8 rows of 32 tuples per warp: a tuple's stable rank is the number of
//                  lanes before it with its owner (one ballot per bit of the owner) plus what its warp has
//                  seen; a prefix over the warps and the owners gives its place in the tile, which is
//                  staged by owner and written out coalesced
// Bound by the two reads and the write (48 bytes a tuple): 2^24 tuples to 8 owners 174 us, where one block scan
// per owner and tile, strided loads and a single load in flight took 462 us.
#include <cstdio>

#include "../host/hj_feistel.h"
#include "hj_common.cuh"
#include "hj_internal.h"

namespace hj {

constexpr int kRouteThreads = 256;
constexpr int kRouteItems = 8;
constexpr int kRouteMaxShards = 32;
constexpr int kRouteCtas = 4;  // blocks per SM

// The count's loads: the scatter reads the tuples again, so their lines keep the normal L2 priority.
__device__ __forceinline__ tuple_v ld_once_more(const tuple_v *p) {
    tuple_v v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ unsigned shard_of(unsigned long long key, unsigned nshards) {
    return (unsigned)__umul64hi(hj_mix64(key ^ 0x5ca1ab1e5eed0001ull), (unsigned long long)nshards);
}

__device__ __forceinline__ void route_block_range(unsigned long long n, unsigned long long *lo,
                                                  unsigned long long *hi) {
    // Whole tiles per block, so that a tile never straddles two blocks.
    constexpr unsigned long long T = (unsigned long long)kRouteThreads * kRouteItems;
    const unsigned long long tiles = (n + T - 1) / T;
    const unsigned long long per = (tiles + gridDim.x - 1) / gridDim.x * T;
    *lo = blockIdx.x * per < n ? blockIdx.x * per : n;
    *hi = *lo + per < n ? *lo + per : n;
}

__global__ void __launch_bounds__(kRouteThreads, kRouteCtas) route_count(const tuple_v *__restrict__ in,
                                                                         unsigned long long n, unsigned nshards,
                                                                         uint32_t *__restrict__ blk_cnt) {
    __shared__ uint32_t cnt[kRouteThreads / 32][kRouteMaxShards][32];  // [warp][owner][lane]
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (unsigned s = 0; s < nshards; s++) cnt[w][s][lane] = 0;
    unsigned long long lo, hi;
    route_block_range(n, &lo, &hi);
    constexpr int U = 4;
    for (unsigned long long i0 = lo + threadIdx.x; i0 < hi; i0 += U * kRouteThreads) {
        tuple_v v[U];
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = i0 + u * kRouteThreads < hi ? ld_once_more(in + i0 + u * kRouteThreads) : make_ulonglong2(0, 0);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * kRouteThreads < hi) cnt[w][shard_of(v[u].x, nshards)][lane]++;
    }
    __syncthreads();
    for (unsigned s = w; s < nshards; s += kRouteThreads / 32) {
        uint32_t c = 0;
#pragma unroll
        for (int q = 0; q < kRouteThreads / 32; q++) c += cnt[q][s][lane];
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) blk_cnt[(size_t)blockIdx.x * nshards + s] = c;
    }
}

// One CTA of 1024 threads; lane = owner, warp w sums a contiguous run of block rows.
__global__ void __launch_bounds__(1024) route_offsets(const uint32_t *__restrict__ blk_cnt, unsigned nblocks,
                                                      unsigned nshards, unsigned long long *__restrict__ blk_off,
                                                      unsigned long long *__restrict__ totals) {
    __shared__ unsigned long long part[32][33];
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool valid = lane < nshards;
    const unsigned rpw = (nblocks + 31) / 32;
    const unsigned r0 = w * rpw, r1 = min(nblocks, r0 + rpw);
    unsigned long long sum = 0;
    for (unsigned r = r0; r < r1 && valid; r++) sum += blk_cnt[(size_t)r * nshards + lane];
    part[w][lane] = sum;
    __syncthreads();
    if (w == 0) {
        unsigned long long run = 0;
        for (int q = 0; q < 32; q++) {
            const unsigned long long v = part[q][lane];
            part[q][lane] = run;
            run += v;
        }
        // Owner bases: exclusive scan of the owner totals across the lanes.
        unsigned long long incl = valid ? run : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (unsigned)o) incl += v;
        }
        const unsigned long long base = incl - (valid ? run : 0);
        if (valid) totals[lane] = run;
        for (int q = 0; q < 32; q++) part[q][lane] += base;
    }
    __syncthreads();
    unsigned long long run = part[w][lane];
    for (unsigned r = r0; r < r1 && valid; r++) {
        const size_t q = (size_t)r * nshards + lane;
        blk_off[q] = run;
        run += blk_cnt[q];
    }
}

__global__ void __launch_bounds__(kRouteThreads, kRouteCtas) route_scatter(const tuple_v *__restrict__ in,
                                                                           unsigned long long n, unsigned nshards,
                                                                           int owner_bits,
                                                                           const unsigned long long *__restrict__ blk_off,
                                                                           tuple_v *__restrict__ out, unsigned int *err) {
    constexpr int NW = kRouteThreads / 32;
    constexpr unsigned T = kRouteThreads * kRouteItems;
    __shared__ __align__(16) tuple_v stage[T];
    __shared__ uint8_t own_of[T];                         // owner of each staged tuple
    __shared__ uint32_t wcnt[NW][kRouteMaxShards];        // a warp's tuples per owner, then its start in the tile
    __shared__ unsigned long long gofs[kRouteMaxShards];  // output index of a staged tuple - its staged index
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned ltmask = lanemask_lt();
    // Warp 0, lane = owner: the block's next output index.
    unsigned long long base = 0;
    if (w == 0 && lane < nshards) base = blk_off[(size_t)blockIdx.x * nshards + lane];
    unsigned long long lo, hi;
    route_block_range(n, &lo, &hi);
    for (unsigned long long t0 = lo; t0 < hi; t0 += T) {
        const unsigned m = hi - t0 < T ? (unsigned)(hi - t0) : T;
        tuple_v v[kRouteItems];
        unsigned pr[kRouteItems];  // owner << 16 | rank within the warp; owner kRouteMaxShards: no tuple
#pragma unroll
        for (int u = 0; u < kRouteItems; u++) {
            const unsigned j = (w * kRouteItems + u) * 32 + lane;
            v[u] = j < m ? ld_stream(in + t0 + j) : make_ulonglong2(0, 0);
        }
        wcnt[w][lane] = 0;
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kRouteItems; u++) {
            const bool live = (w * kRouteItems + u) * 32 + lane < m;
            const unsigned d = live ? shard_of(v[u].x, nshards) : 0u;
            unsigned peers = __ballot_sync(0xffffffffu, live);
            for (int b = 0; b < owner_bits; b++) {
                const unsigned bit = (d >> b) & 1u;
                peers &= __ballot_sync(0xffffffffu, bit) ^ (bit - 1u);  // bit ? ballot : ~ballot
            }
            const unsigned before = wcnt[w][d];
            __syncwarp();
            if (live && (peers & ltmask) == 0) wcnt[w][d] = before + __popc(peers);
            __syncwarp();
            pr[u] = ((live ? d : (unsigned)kRouteMaxShards) << 16) | (before + __popc(peers & ltmask));
        }
        __syncthreads();
        if (w == 0) {
            // Lane = owner: each warp's start within the owner's run, then the runs' starts in the tile.
            uint32_t run = 0;
#pragma unroll
            for (int q = 0; q < NW; q++) {
                const uint32_t c = wcnt[q][lane];
                wcnt[q][lane] = run;
                run += c;
            }
            uint32_t incl = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (unsigned)o) incl += y;
            }
            const uint32_t start = incl - run;
#pragma unroll
            for (int q = 0; q < NW; q++) wcnt[q][lane] += start;
            gofs[lane] = base - start;
            base += run;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kRouteItems; u++) {
            const unsigned d = pr[u] >> 16;
            if (d == (unsigned)kRouteMaxShards) continue;
            const unsigned p = wcnt[w][d] + (pr[u] & 0xffffu);
            stage[p] = v[u];
            own_of[p] = (uint8_t)d;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kRouteItems; u++) {
            const unsigned j = u * kRouteThreads + threadIdx.x;
            if (j >= m) continue;
            const unsigned long long dst = gofs[own_of[j]] + j;
            if (dst < n)
                out[dst] = stage[j];
            else
                set_error(err, kErrBounds);
        }
        __syncthreads();
    }
}

}  // namespace hj

namespace {
size_t route_blocks(size_t n, int num_sms) {
    const size_t T = (size_t)hj::kRouteThreads * hj::kRouteItems;
    const size_t tiles = (n + T - 1) / T;
    size_t b = (size_t)num_sms * hj::kRouteCtas;
    if (tiles < b) b = tiles ? tiles : 1;
    return b;
}
size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }
}  // namespace

extern "C" {

size_t hj_shard_route_scratch_bytes(size_t n, int nshards) {
    if (nshards < 1) nshards = 1;
    // Enough for any device's SM count (up to 512 SMs at kRouteCtas blocks each).
    const size_t blocks = route_blocks(n, 512);
    return a256(blocks * nshards * 4) + a256(blocks * nshards * 8) + 256;
}

int hj_shard_route(const hj_tuple_t *in_dev, size_t n, int nshards, hj_tuple_t *out_dev, uint64_t *counts_dev,
                   void *scratch_dev, size_t scratch_bytes, void *stream) {
    if (nshards < 1 || nshards > hj::kRouteMaxShards || !counts_dev || (n && (!in_dev || !out_dev))) return HJ_E_INVAL;
    if (scratch_bytes < hj_shard_route_scratch_bytes(n, nshards) || !scratch_dev) return HJ_E_INVAL;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return HJ_E_DEVICE;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned blocks = (unsigned)route_blocks(n, sms);
    char *p = reinterpret_cast<char *>(scratch_dev);
    uint32_t *blk_cnt = reinterpret_cast<uint32_t *>(p);
    unsigned long long *blk_off = reinterpret_cast<unsigned long long *>(p + a256((size_t)blocks * nshards * 4));
    unsigned int *err = reinterpret_cast<unsigned int *>(p + a256((size_t)blocks * nshards * 4) +
                                                         a256((size_t)blocks * nshards * 8));
    if (cudaMemsetAsync(err, 0, 4, st) != cudaSuccess) return HJ_E_DEVICE;
    if (n == 0) return cudaMemsetAsync(counts_dev, 0, sizeof(uint64_t) * nshards, st) == cudaSuccess ? HJ_OK : HJ_E_DEVICE;
    const hj::tuple_v *in = reinterpret_cast<const hj::tuple_v *>(in_dev);
    hj::route_count<<<blocks, hj::kRouteThreads, 0, st>>>(in, n, (unsigned)nshards, blk_cnt);
    hj::route_offsets<<<1, 1024, 0, st>>>(blk_cnt, blocks, (unsigned)nshards, blk_off,
                                          reinterpret_cast<unsigned long long *>(counts_dev));
    int owner_bits = 0;
    while ((1 << owner_bits) < nshards) owner_bits++;
    hj::route_scatter<<<blocks, hj::kRouteThreads, 0, st>>>(in, n, (unsigned)nshards, owner_bits, blk_off,
                                                            reinterpret_cast<hj::tuple_v *>(out_dev), err);
    return cudaGetLastError() == cudaSuccess ? HJ_OK : HJ_E_DEVICE;
}

}  // extern "C"
