// hj_wave.cu - waves of joins without global tables: sizes, descriptors and launches (see hj_wave.cuh).
#include <algorithm>
#include <cstring>

#include "hj_partition.cuh"
#include "hj_wave.cuh"

namespace hj {

namespace {

// Tuples per block of the partition steps and of the joins, and of a small join's probe range: enough to
// amortise the block's digit arrays and tables in a wave that fills the SMs, fewer in a small wave, whose
// time is that of its longest block.
constexpr uint64_t kWavePartTuples = 65536, kWaveJoinTuples = 32768, kWaveSmallTuples = 16384;
constexpr uint64_t kWavePartMin = 8192, kWaveJoinMin = 4096, kWaveSmallMin = 2048;
// Fewest radix bits: fewer digits make the lanes of a warp wait for each other's counters.
constexpr int kWaveMinBits = 4;
constexpr size_t kWaveTarget = 6144;

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

uint32_t blocks(uint64_t n, uint64_t per, uint32_t cap) {
    const uint64_t b = (n + per - 1) / per;
    return b < 1 ? 1u : b < cap ? (uint32_t)b : cap;
}

RadixGeom geom_of(const WaveJoin &j) {
    RadixGeom g = {};
    int b = kWaveMinBits;
    while (b < kSingleMaxBits && (j.nR >> b) > kWaveTarget) b++;
    g.bits = g.req_bits = g.b1 = b;
    g.passes = 1;
    g.F1 = 1 << b;
    g.F2 = 1;
    g.single = true;
    g.mix = true;
    return g;
}

bool is_small(const WaveJoin &j) { return j.nR <= kSmallMaxBuild; }

struct Pieces {
    uint64_t part, join, small;
};

Pieces pieces_of(const WaveJoin *joins, size_t n, int num_sms) {
    uint64_t total = 0;
    for (size_t q = 0; q < n; q++) total += (uint64_t)joins[q].nR + joins[q].nS;
    auto clamp = [](uint64_t v, uint64_t lo, uint64_t hi) { return v < lo ? lo : v > hi ? hi : v; };
    Pieces p;
    p.part = clamp(total / (2 * (uint64_t)num_sms), kWavePartMin, kWavePartTuples);
    p.join = clamp(total / (4 * (uint64_t)num_sms), kWaveJoinMin, kWaveJoinTuples);
    p.small = clamp(total / (4 * (uint64_t)num_sms), kWaveSmallMin, kWaveSmallTuples);
    return p;
}

// Blocks of a join's partition steps (the grid that its scratch is carved for).
uint32_t part_grid(const WaveJoin &j, const Pieces &pc, int num_sms) {
    return single_grid(j.nR, j.nS, (int)blocks((uint64_t)j.nR + j.nS, pc.part, (uint32_t)num_sms));
}

uint32_t join_blocks(const WaveJoin &j, const Pieces &pc, int num_sms) {
    return blocks((uint64_t)j.nR + j.nS, pc.join, 2 * (uint32_t)num_sms);
}

// Blocks of a join's large-partition probe, which return at once for most joins: few, up to what fills the GPU.
uint32_t large_blocks(const WaveJoin &j, int num_sms) {
    return blocks((uint64_t)j.nR + j.nS, kWavePartTuples, 4 * (uint32_t)num_sms);
}

// Probe tuples per block of a small join: no fewer than twice its build side, which every block reads.
uint64_t small_range(const WaveJoin &j, const Pieces &pc) { return std::max<uint64_t>(pc.small, 2 * j.nR); }

}  // namespace

bool wave_takes(size_t nR, size_t nS) {
    return nR <= ((size_t)kWaveTarget << kSingleMaxBits) && nS < (1ull << 32);
}

void wave_plan(const WaveJoin *joins, size_t n, int num_sms, WavePlan *wp) {
    *wp = WavePlan();
    const Pieces pc = pieces_of(joins, n, num_sms);
    for (size_t q = 0; q < n; q++) {
        const WaveJoin &j = joins[q];
        if (!j.nR || !j.nS) continue;
        if (is_small(j)) {
            wp->n_small++;
            wp->n_chunks += blocks(j.nS, small_range(j, pc), ~0u);
            wp->max_build = std::max(wp->max_build, j.nR);
            continue;
        }
        const RadixGeom g = geom_of(j);
        wp->n_jobs++;
        wp->n_part += part_grid(j, pc, num_sms);
        wp->n_plan += (2u * (unsigned)g.F1 + 31) / 32;
        (j.lp ? wp->n_first : wp->n_every) += join_blocks(j, pc, num_sms);
        wp->n_large += large_blocks(j, num_sms);
        wp->max_bits = std::max(wp->max_bits, g.bits);
        wp->scratch_bytes += a256(phj_scratch_bytes(g, j.nR, j.nS, (int)part_grid(j, pc, num_sms)));
    }
    size_t o = 0;
    auto put = [&](size_t bytes) {
        const size_t at = o;
        o += a256(bytes);
        return at;
    };
    wp->jobs_off = put(sizeof(MultiJob) * wp->n_jobs);
    wp->small_off = put(sizeof(SmallJob) * wp->n_small);
    wp->chunk_off = put(sizeof(MChunk) * wp->n_chunks);
    wp->part_off = put(8 * (size_t)wp->n_part);
    wp->plan_off = put(8 * (size_t)wp->n_plan);
    wp->every_off = put(8 * (size_t)wp->n_every);
    wp->first_off = put(8 * (size_t)wp->n_first);
    wp->large_off = put(8 * (size_t)wp->n_large);
    wp->image_bytes = o;
}

int wave_image(const WaveJoin *joins, size_t n, int num_sms, const WavePlan &wp, char *scratch, char *image) {
    MultiJob *mj = reinterpret_cast<MultiJob *>(image + wp.jobs_off);
    SmallJob *sj = reinterpret_cast<SmallJob *>(image + wp.small_off);
    MChunk *ch = reinterpret_cast<MChunk *>(image + wp.chunk_off);
    uint2 *part = reinterpret_cast<uint2 *>(image + wp.part_off), *plan = reinterpret_cast<uint2 *>(image + wp.plan_off);
    uint2 *every = reinterpret_cast<uint2 *>(image + wp.every_off);
    uint2 *first = reinterpret_cast<uint2 *>(image + wp.first_off), *large = reinterpret_cast<uint2 *>(image + wp.large_off);
    const Pieces pc = pieces_of(joins, n, num_sms);
    unsigned nj = 0, ns = 0, nc = 0, npt = 0, npl = 0, ne = 0, nf = 0, nl = 0;
    for (size_t q = 0; q < n; q++) {
        const WaveJoin &j = joins[q];
        if (!j.nR || !j.nS) continue;
        if (is_small(j)) {
            const uint64_t per = small_range(j, pc);
            for (uint64_t b = 0; b < j.nS; b += per) {
                MChunk c;
                c.job = ns;
                c.begin = b;
                c.len = (unsigned)std::min<uint64_t>(per, j.nS - b);
                ch[nc++] = c;
            }
            small_job(j.lp, j.skip0, j.R, j.nR, j.S, j.acc, &sj[ns++]);
            continue;
        }
        const RadixGeom g = geom_of(j);
        const uint32_t G = part_grid(j, pc, num_sms);
        PhjScratch s;
        phj_carve(g, j.nR, j.nS, (int)G, scratch, &s);
        scratch += a256(phj_scratch_bytes(g, j.nR, j.nS, (int)G));
        if (s.cR != G) return HJ_E_INVAL;
        MultiJob m;
        memset(&m, 0, sizeof(m));
        single_args(g, j.lp, j.skip0, true, j.R, j.nR, j.S, j.nS, s, j.acc, false, true, &m.sa, &m.pa);
        m.ja = join_args(g, j.lp, j.skip0, j.R, j.nR, s, j.acc, nullptr, 1, -1, nullptr);
        m.grid = G;
        m.plan_blocks = (2u * (unsigned)g.F1 + 31) / 32;
        for (uint32_t b = 0; b < G; b++) part[npt++] = make_uint2(nj, b);
        for (uint32_t b = 0; b < m.plan_blocks; b++) plan[npl++] = make_uint2(nj, b);
        m.join_blocks = join_blocks(j, pc, num_sms);
        m.large_blocks = large_blocks(j, num_sms);
        for (uint32_t b = 0; b < m.large_blocks; b++) large[nl++] = make_uint2(nj, b);
        const uint32_t jb = m.join_blocks;
        for (uint32_t b = 0; b < jb; b++) {
            if (j.lp)
                first[nf++] = make_uint2(nj, b);
            else
                every[ne++] = make_uint2(nj, b);
        }
        mj[nj++] = m;
    }
    const bool same = nj == wp.n_jobs && ns == wp.n_small && nc == wp.n_chunks && npt == wp.n_part && npl == wp.n_plan &&
                      ne == wp.n_every && nf == wp.n_first && nl == wp.n_large;
    return same ? HJ_OK : HJ_E_INVAL;
}

int wave_enqueue(const WavePlan &wp, const char *image_dev, cudaStream_t st, uint32_t *launches) {
    uint32_t l = 0;
    int rc = HJ_OK;
    if (wp.n_chunks) {
        rc = small_multi_launch(reinterpret_cast<const SmallJob *>(image_dev + wp.small_off),
                                reinterpret_cast<const MChunk *>(image_dev + wp.chunk_off), wp.n_chunks, wp.max_build, st);
        l++;
    }
    if (!rc && wp.n_jobs) {
        const MultiJob *jobs = reinterpret_cast<const MultiJob *>(image_dev + wp.jobs_off);
        auto map = [&](size_t off) { return reinterpret_cast<const uint2 *>(image_dev + off); };
        rc = multi_partition_launch(jobs, map(wp.part_off), wp.n_part, map(wp.plan_off), wp.n_plan, wp.max_bits, st, &l);
        if (!rc)
            rc = multi_join_launch(jobs, map(wp.every_off), wp.n_every, map(wp.first_off), wp.n_first, map(wp.large_off),
                                   wp.n_large, st, &l);
    }
    if (launches) *launches += l;
    return rc;
}

}  // namespace hj
