// hj_wave.cuh - waves: many independent joins with one launch per step over flat lists of (join, range) items, so
// that the launch count does not grow with the number of joins.
//
// Two forms. In the first (MJob, WaveDev) each join has its own global hash table: one multi-join build kernel
// and one multi-join probe kernel. In the second (WaveJoin, WavePlan, below) joins have no global table: shared-memory
// tables for small build sides, the one-pass radix pipeline for the others. Batches (hj_batch.cu) pack their joins
// into waves at plan time, of the first form only when the second's scratch cannot be had; the join server
// (hj_server.cu) forms a wave from the requests queued at each dispatch (continuous batching).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "hj_common.cuh"
#include "hj_internal.h"

namespace hj {

struct MSide {
    unsigned long long cnt, sum;  // build tuples whose key is the empty pattern: count, row-id sum
    unsigned long long notpos;    // max of ~position over them (0 = none), i.e. ~(smallest position)
    unsigned int dup;             // an equal key was inserted twice
    unsigned int pad;
};

struct MJob {
    const tuple_v *R, *S;
    unsigned long long nR, nS;
    tuple_v *table;
    unsigned long long cap;
    MSide *side;
    JoinAccum *acc;
    unsigned int lp, skip0;
};

// A piece of one job's build or probe side: the multi-join kernels take these as work items, so a
// block always works on a single job.
struct MChunk {
    unsigned int job;
    unsigned int len;
    unsigned long long begin;
};

constexpr unsigned kBuildChunk = 8192, kProbeChunkMJ = 16384;

// Chunk length for `total` tuples of a wave: the fixed piece, or a smaller one (a multiple of 256, at
// least 256) when the wave is too small to give every SM four chunks; a lone small request would
// otherwise run on a handful of CTAs, each working through thousands of dependent table accesses.
inline unsigned mj_piece(unsigned long long total, unsigned max_piece, int num_sms) {
    const unsigned long long want = (unsigned long long)(num_sms > 0 ? num_sms : 148) * 4;
    unsigned long long p = (total + want - 1) / want;
    p = (p + 255) / 256 * 256;
    return p < 256 ? 256u : p > max_piece ? max_piece : (unsigned)p;
}

// Table slots of one job (load factor 0.5, two spare slots).
inline unsigned long long mj_slots(size_t nR) { return (unsigned long long)((double)nR / 0.5) + 2; }

// Device view of one wave: descriptors, prefix sums of build / probe / table sizes over the jobs (count
// + 1 entries each), and the tables and side records the wave clears before building.
struct WaveDev {
    const MJob *jobs;
    int count;
    const MChunk *r_chunks, *s_chunks;
    int n_r_chunks, n_s_chunks;
    const unsigned long long *r_flat, *t_flat;
    unsigned long long total_r, total_t;
    bool any_lp;
    void *tables;
    MSide *sides;
};

// Enqueue a wave on `st`: clear its tables and side records, build, resolve first-match joins with
// duplicate build keys, probe. Results accumulate into each job's JoinAccum (which the caller zeroes).
int mj_launch_wave(const WaveDev &w, int num_sms, cudaStream_t st, uint32_t *launches);

// ------------------------------------------------------------------------------------------------
// Waves without global tables. Joins of at most kSmallMaxBuild build tuples take one shared-memory table
// per probe range (hj_small.cu); the others run the one-pass pipeline (hj_single.cu), each step as one
// launch over all joins of the wave. A wave needs 16 bytes of scratch per tuple (and 28 per build tuple),
// where table waves need 32 bytes per build tuple; the server falls back to those when its pool is short.
// ------------------------------------------------------------------------------------------------
struct SmallJob {
    const tuple_v *R, *S;
    JoinAccum *acc;
    uint32_t nR;
    int nb_log;
    unsigned int lp, skip0;
};
void small_job(bool lp, bool skip0, const ulonglong2 *R, size_t nR, const ulonglong2 *S, JoinAccum *acc, SmallJob *j);
int small_multi_launch(const SmallJob *jobs, const MChunk *chunks, unsigned nchunks, size_t max_build, cudaStream_t st);

struct WaveJoin {
    bool lp, skip0;
    const ulonglong2 *R;
    size_t nR;
    const ulonglong2 *S;
    size_t nS;
    JoinAccum *acc;  // device, zeroed by the caller before the wave
};

// Whether a join may be part of such a wave.
bool wave_takes(size_t nR, size_t nS);

// Sizes and launches of one wave, from the joins' sizes alone; the descriptor image and the scratch are the
// caller's (image: host copy of what goes to the device).
struct WavePlan {
    size_t scratch_bytes = 0, image_bytes = 0;
    size_t jobs_off, small_off, chunk_off, part_off, plan_off, every_off, first_off, large_off;
    unsigned n_jobs = 0, n_small = 0, n_chunks = 0, n_part = 0, n_plan = 0, n_every = 0, n_first = 0, n_large = 0;
    int max_bits = 0;
    size_t max_build = 0;
};
void wave_plan(const WaveJoin *joins, size_t n, int num_sms, WavePlan *wp);
// Fill the image for scratch at `scratch` (device, 256-byte aligned).
int wave_image(const WaveJoin *joins, size_t n, int num_sms, const WavePlan &wp, char *scratch, char *image);
// Enqueue the wave; image_dev: the image on the device.
int wave_enqueue(const WavePlan &wp, const char *image_dev, cudaStream_t st, uint32_t *launches);

}  // namespace hj
