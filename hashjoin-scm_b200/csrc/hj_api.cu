// hj_api.cu - the C ABI: contexts, scratch arena, and the synchronous join entry points.
//
// The reference's join_init_run (src/algo/phj.c:1875-2512) and nphj_sc/nphj_lp
// (src/algo/nphj.c:677-1037, 1487-...) each allocate their buffers, spawn thread pools, join and free
// everything per call. Here a context keeps a stream, events and a grow-only device arena; a join
// carves its scratch out of the arena and enqueues the whole kernel pipeline on one stream, reading
// back only the 64-byte accumulator at the end.
#include <cstdio>
#include <chrono>
#include <cstring>
#include <thread>
#include <mutex>

#include "hj_common.cuh"
#include "hj_ctx.h"
#include "hj_internal.h"

using hj::JoinAccum;

#define CU_OR(call, code)                                                                   \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess) {                                                            \
            fprintf(stderr, "hjscm: %s failed: %s\n", #call, cudaGetErrorString(e_));       \
            return (code);                                                                  \
        }                                                                                   \
    } while (0)

namespace {

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

std::mutex g_default_mu;
hj_ctx *g_default[64] = {};

constexpr size_t kAccBytes = 256;
constexpr size_t kSmallBufBytes = 256 + hj::kSmallMaxGrid * sizeof(hj::SmallPart);

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

void resolve_params(const hj_params_t *p, hj_params_t *out) {
    hj_params_init(out);
    if (p) *out = *p;
    if (out->num_radix_bits == 0) out->num_radix_bits = 14;
    if (out->num_passes == 0) out->num_passes = 2;
    if (!(out->table_load > 0.0)) out->table_load = 0.0;  // the size-dependent default (nphj_default_load)
}

bool is_phj(hj_algo_t a) { return hj::algo_is_phj(a); }

// Segment mode for a radix join (see HJ_F_SEGMENTS): by size unless a flag decides.
bool want_seg(hj_algo_t algo, const hj_params_t &p, const hj::RadixGeom &g, size_t nR, size_t nS) {
    if ((p.flags & HJ_F_EXACT) || g.single) return false;
    if (p.flags & HJ_F_SEGMENTS) return hj::phj_seg_applies(g, hj::algo_lp(algo), 1ull << 40, 0);
    return hj::phj_seg_applies(g, hj::algo_lp(algo), nR, nS);
}

// Flags that name a pipeline or its element layout: the two-pass pipelines run as asked.
constexpr uint32_t kPipelineFlags = HJ_F_SEGMENTS | HJ_F_EXACT | HJ_F_WIDE | HJ_F_WORDS | HJ_F_TEST_STALL;

// One-pass radix joins of at most kRawDigitsMaxBuild build tuples partition by the key's own low bits, as asked, larger
// ones by mix_key (which a materialising join, whose large partitions walk every duplicate, always does). Keys
// that share low bits overfill a few of the raw partitions; a join that finds most of its build tuples in partitions
// beyond shared memory is run again by mix_key (2^21 x 2^23 multiples of 4: 809 us with the global tables of such
// partitions, 332 run again, 480 in two passes of 14 bits; dense keys 155). At kRerunMinBuild build tuples and
// below the tables are as fast (multiples of 2^14, 2^16 x 2^18: 103 us and 106 run again, 2^18 x 2^20: 161 and 127).
// Mixing costs dense keys 1% in one pass, 2.5% in two.
constexpr size_t kRawDigitsMaxBuild = 1u << 21, kRerunMinBuild = 1u << 16;

// The geometry of a radix join: the one-pass pipeline where the build relation needs few partitions,
// unless the flags name another, else as asked.
int join_geom(hj_algo_t algo, const hj_params_t &p, size_t nR, size_t nS, bool mat, hj::RadixGeom *g) {
    const int rc = hj::radix_geom(p.num_radix_bits, p.num_passes, g, p.radix_bits_pass1);
    if (rc) return rc;
    if (p.flags & kPipelineFlags) return HJ_OK;
    if (hj::radix_geom_single(p.num_radix_bits, hj::algo_lp(algo) || mat, nR, nS, g))
        g->mix = mat || nR > kRawDigitsMaxBuild;
    else
        hj::radix_geom_by_size(nR, nS, p.radix_bits_pass1 > 0, g);
    return HJ_OK;
}

// Non-partitioned joins of these sizes run a radix pipeline (14 bits, or the one-pass geometry; partitions of
// mix_key, so that the keys' low bits matter as little as to the table's hash): what a join reports does not
// depend on how it was computed, and beyond L2 partitioning both sides beats one random table access per tuple
// (wall clock, radix then table; nphj_sc 2^22 x 2^23 dense 193 / 247 us, multiples of 4 209 / 247, 63-bit keys 290 /
// 460; nphj_lp 2^24 x 2^26 with four tuples a key 1.45 / 1.82 ms). The line lies where every measured form of the
// keys gains, which a skewed probe side decides: it finds the table's hot lines in L2. With at most two
// probe tuples a build tuple, Zipf 1.5, dense / 63-bit: nphj_sc 2^21 x 2^22 144 176 / 139 212, 2^23 x 2^24
// 396 539 / 427 804, nphj_lp 463 767 / 557 821. With up to four, nphj_sc takes the table below 2^25 build
// tuples (12e6 x 48e6 787 / 737, 2^24 x 2^26 1527 / 1279), nphj_lp below 12e6 (2^23 x 2^25 with 63-bit keys
// 1004 / 927; 12e6 x 48e6 Zipf 1.0 1657 / 1690, dense 868 / 920). With
// more, both take it (2^24 x 2^28: 3086 3864 / 2755 3383, nphj_lp 5309 / 3005). Below 2^21 the table sits in
// L2 (300000 x 300000 Zipf 1.5 96 / 73). First matches take the table beyond one pass (plan_join). A load factor asks
// for the table itself; build partitions above 6144 tuples on average, and scratch that cannot be had, take it too.
constexpr size_t kNphjRadixMinBuild = 1u << 21, kNphjScWide = 1u << 25, kNphjLpWide = 12000000;
constexpr size_t kNphjRadixMaxBuild = (size_t)6144 << 14;
bool nphj_by_radix(const hj_params_t &p, bool lp, size_t nR, size_t nS) {
    if (p.table_load > 0.0 || nR < kNphjRadixMinBuild || nR > kNphjRadixMaxBuild || nS >= (1ull << 32)) return false;
    return nS <= 2 * nR || (nS <= 4 * nR && nR >= (lp ? kNphjLpWide : kNphjScWide));
}

// How a join runs: by a radix pipeline (radix, geom, seg) or on the non-partitioned table.
struct JoinPlan {
    bool radix = false, seg = false;
    hj::RadixGeom geom = {};
};

int plan_join(hj_algo_t algo, hj_params_t *p, size_t nR, size_t nS, JoinPlan *jp, bool mat = false) {
    *jp = JoinPlan();
    if (is_phj(algo)) {
        const int rc = join_geom(algo, *p, nR, nS, mat, &jp->geom);
        if (rc) return rc;
    } else if (nphj_by_radix(*p, hj::algo_lp(algo), nR, nS)) {
        hj::radix_geom(14, 2, &jp->geom);
        if (!hj::radix_geom_single(14, hj::algo_lp(algo) || mat, nR, nS, &jp->geom)) {
            // Two passes join first matches in partition order, where a probe walks all duplicates of its key.
            if (hj::algo_lp(algo)) return HJ_OK;
            hj::radix_geom_by_size(nR, nS, false, &jp->geom);
        }
        p->flags &= ~(kPipelineFlags | HJ_F_ORDERED);  // radix joins' flags
        jp->geom.mix = true;  // as the table's hash, whatever bits the keys share
    } else {
        return HJ_OK;
    }
    jp->radix = true;
    jp->seg = want_seg(algo, *p, jp->geom, nR, nS);
    return HJ_OK;
}

size_t scratch_need(const JoinPlan &jp, const hj_params_t &p, size_t nR, size_t nS, bool host_inputs, int num_sms) {
    size_t need = kAccBytes;
    if (host_inputs) need += align256(nR * 16) + align256(nS * 16);
    if (jp.radix)
        need += hj::phj_scratch_bytes(jp.geom, nR, nS, num_sms, jp.seg);
    else
        need += align256(hj::nphj_scratch_bytes(nR, p.table_load));
    return need;
}

// Drop the context's join graphs (they address the arena).
void drop_graphs(hj_ctx *c) {
    for (hj_graph_entry &e : c->graphs)
        if (e.exec) cudaGraphExecDestroy(e.exec);
    c->graphs.clear();
    c->last_key = hj_graph_key();
}

constexpr size_t kMaxJoinGraphs = 4;

hj_graph_entry *find_graph(hj_ctx *c, const hj_graph_key &k) {
    for (hj_graph_entry &e : c->graphs)
        if (e.key == k) {
            e.used = ++c->graph_tick;
            return &e;
        }
    return nullptr;
}

void refuse_arena(hj_ctx *c, size_t bytes) {
    c->refused_bytes = bytes;
    c->refused_at = std::chrono::steady_clock::now();
}

int ensure_arena(hj_ctx *c, size_t bytes) {
    if (c->arena_bytes >= bytes) return HJ_OK;
    CU_OR(cudaStreamSynchronize(c->stream), HJ_E_DEVICE);
    drop_graphs(c);
    if (c->arena) cudaFree(c->arena);
    c->arena = nullptr;
    c->arena_bytes = 0;
    if (cudaMalloc(&c->arena, bytes) != cudaSuccess) {
        cudaGetLastError();
        c->arena = nullptr;
        refuse_arena(c, bytes);
        return HJ_E_OOM;
    }
    c->arena_bytes = bytes;
    return HJ_OK;
}

// Whether the arena can be as large as this: it is, or the device has the memory for it. A plan that has a smaller one
// to fall back to asks first, so that an arena which serves that one is not given up for an allocation that
// fails, with the join graphs, at every call. Asking the driver takes 0.07 to 1 ms, so a refusal stands for a second.
bool arena_may_grow(hj_ctx *c, size_t bytes) {
    if (c->arena_bytes >= bytes) return true;
    if (c->refused_bytes && bytes >= c->refused_bytes &&
        std::chrono::steady_clock::now() - c->refused_at < std::chrono::seconds(1))
        return false;
    c->refused_bytes = 0;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    if (bytes <= free_b + c->arena_bytes) return true;
    refuse_arena(c, bytes);
    return false;
}

// Scratch for the plan (need: its bytes); one that cannot be had falls back to a plan that needs less (segment mode to
// the exact-offset pipeline, a non-partitioned join's radix pipeline to the table).
template <class Need>
int ensure_plan(hj_ctx *c, hj_algo_t algo, JoinPlan *jp, const Need &need) {
    const bool table = jp->radix && !is_phj(algo);  // a plan to fall back to
    auto attempt = [&](bool last) { return last || arena_may_grow(c, need()) ? ensure_arena(c, need()) : (int)HJ_E_OOM; };
    int rc = attempt(!jp->seg && !table);
    if (rc == HJ_E_OOM && jp->seg) {
        jp->seg = false;
        rc = attempt(!table);
    }
    if (rc == HJ_E_OOM && table) {
        *jp = JoinPlan();
        rc = ensure_arena(c, need());
    }
    return rc;
}

int map_error_bits(unsigned bits) {
    if (!bits) return HJ_OK;
    if (bits & hj::kErrSpinLimit) return HJ_E_TIMEOUT;
    if (bits & hj::kErrProbeLimit) return HJ_E_PROBE_LIMIT;
    if (bits & hj::kErrOutput) return HJ_E_CAPACITY;
    if (bits & hj::kErrRowId) return HJ_E_ROWID;
    return HJ_E_OVERFLOW;
}

}  // namespace

extern "C" {

void hj_params_init(hj_params_t *p) {
    if (!p) return;
    memset(p, 0, sizeof(*p));
    p->num_radix_bits = 14;
    p->num_passes = 2;
    p->table_load = 0.0;
}

const char *hj_status_str(int s) {
    switch (s) {
        case HJ_OK: return "ok";
        case HJ_E_INVAL: return "invalid argument";
        case HJ_E_OOM: return "out of memory";
        case HJ_E_DEVICE: return "CUDA error";
        case HJ_E_PROBE_LIMIT: return "table walk exceeded capacity";
        case HJ_E_TIMEOUT: return "bounded wait gave up";
        case HJ_E_NOT_FOUND: return "unknown algorithm";
        case HJ_E_IO: return "i/o error";
        case HJ_E_OVERFLOW: return "device bound check fired";
        case HJ_E_BUDGET: return "over the HBM budget";
        case HJ_E_CAPACITY: return "the pair buffer is too small (matched_cnt = pairs needed)";
        case HJ_E_ROWID: return "a matched row id is not a 1-based position of its relation";
        default: return "unknown status";
    }
}

static const char *const k_algo_names[HJ_ALGO_COUNT] = {"nphj_sc",      "nphj_lp",      "phj_radix_bc", "phj_radix_lp",
                                                        "phj_radix_sc", "phj_radix_hr", "phj_radix_hro"};

const char *hj_algo_name(hj_algo_t a) {
    return ((int)a >= 0 && a < HJ_ALGO_COUNT) ? k_algo_names[a] : "?";
}

int hj_algo_from_name(const char *name, hj_algo_t *algo) {
    if (!name || !algo) return HJ_E_INVAL;
    for (int i = 0; i < HJ_ALGO_COUNT; i++)
        if (strcmp(name, k_algo_names[i]) == 0) {
            *algo = (hj_algo_t)i;
            return HJ_OK;
        }
    // Bandwidth-regulated variants compute identical results (src/algo/phj_bw_reg.c:2874-2893); the
    // asymmetric-radix variants too (the bit split is hj_params_t.radix_bits_pass1).
    static const char *const prefixes[] = {"phj_radix_bw_reg_", "phj_asymm_radix_bw_reg_", "phj_asymm_radix_"};
    for (const char *pre : prefixes) {
        const size_t n = strlen(pre);
        if (strncmp(name, pre, n) != 0) continue;
        const char *suf = name + n;
        static const char *const sufs[] = {"bc", "lp", "sc", "hr", "hro"};
        static const hj_algo_t algs[] = {HJ_ALGO_PHJ_RADIX_BC, HJ_ALGO_PHJ_RADIX_LP, HJ_ALGO_PHJ_RADIX_SC,
                                         HJ_ALGO_PHJ_RADIX_HR, HJ_ALGO_PHJ_RADIX_HRO};
        for (int i = 0; i < 5; i++)
            if (strcmp(suf, sufs[i]) == 0) {
                // The reference has no phj_asymm_radix_lp (src/main.c:80-82, 114-116, 128, 138).
                if (i == 1 && pre[4] == 'a') return HJ_E_NOT_FOUND;
                *algo = algs[i];
                return HJ_OK;
            }
    }
    return HJ_E_NOT_FOUND;
}

int hj_ctx_create(int device, hj_ctx_t **out) {
    if (!out) return HJ_E_INVAL;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return HJ_E_DEVICE;
    }
    DeviceGuard g(device);
    hj_ctx *c = new hj_ctx();
    c->device = device;
    CU_OR(cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device), HJ_E_DEVICE);
    CU_OR(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking), HJ_E_DEVICE);
    CU_OR(cudaEventCreate(&c->ev_h2d), HJ_E_DEVICE);
    CU_OR(cudaEventCreate(&c->ev_start), HJ_E_DEVICE);
    CU_OR(cudaEventCreate(&c->ev_mid), HJ_E_DEVICE);
    CU_OR(cudaEventCreate(&c->ev_end), HJ_E_DEVICE);
    CU_OR(cudaEventCreate(&c->ev_ret), HJ_E_DEVICE);
    CU_OR(cudaEventCreateWithFlags(&c->ev_done, cudaEventDisableTiming), HJ_E_DEVICE);
    for (int i = 0; i <= HJ_PH_COUNT; i++) CU_OR(cudaEventCreate(&c->ev_ph[i]), HJ_E_DEVICE);
    CU_OR(cudaMallocHost(&c->acc_host, sizeof(JoinAccum)), HJ_E_OOM);
    CU_OR(cudaMalloc(&c->small_buf, kSmallBufBytes), HJ_E_OOM);
    CU_OR(cudaMemset(c->small_buf, 0, kSmallBufBytes), HJ_E_DEVICE);
    c->tuner.nphj_max_table_bytes = 64e6;
    c->tuner.wave_table_bytes = 64e6;
    c->tuner.partition_target = 6144;
    c->tuner.calibrated = 0;
    *out = c;
    return HJ_OK;
}

int hj_ctx_destroy(hj_ctx_t *c) {
    if (!c) return HJ_E_INVAL;
    {
        DeviceGuard g(c->device);
        std::lock_guard<std::mutex> lk(c->mu);
        if (c->stream) cudaStreamSynchronize(c->stream);
        drop_graphs(c);
        if (c->arena) cudaFree(c->arena);
        if (c->acc_host) cudaFreeHost(c->acc_host);
        if (c->small_buf) cudaFree(c->small_buf);
        hj::free_copy_buffers(c);
        cudaEventDestroy(c->ev_h2d);
        cudaEventDestroy(c->ev_start);
        cudaEventDestroy(c->ev_mid);
        if (c->ev_ret) cudaEventDestroy(c->ev_ret);
        if (c->ev_done) cudaEventDestroy(c->ev_done);
        cudaEventDestroy(c->ev_end);
        for (int i = 0; i <= HJ_PH_COUNT; i++) cudaEventDestroy(c->ev_ph[i]);
        if (c->stream) cudaStreamDestroy(c->stream);
    }
    delete c;
    return HJ_OK;
}

size_t hj_ctx_scratch_bytes(const hj_ctx_t *c) { return c ? c->arena_bytes : 0; }

int hj_ctx_reserve(hj_ctx_t *c, hj_algo_t algo, const hj_params_t *pin, size_t nR, size_t nS) {
    if (!c || (int)algo < 0 || algo >= HJ_ALGO_COUNT) return HJ_E_INVAL;
    hj_params_t p;
    resolve_params(pin, &p);
    JoinPlan jp;
    const int rc = plan_join(algo, &p, nR, nS, &jp);
    if (rc) return rc;
    DeviceGuard g(c->device);
    std::lock_guard<std::mutex> lk(c->mu);
    return ensure_plan(c, algo, &jp, [&] { return scratch_need(jp, p, nR, nS, !p.inputs_on_device, c->num_sms); });
}

int hj_join_ctx(hj_ctx_t *c, hj_algo_t algo, const hj_params_t *pin, const hj_tuple_t *R, size_t nR,
                const hj_tuple_t *S, size_t nS, hj_result_t *out) {
    if (!c || !out || (int)algo < 0 || algo >= HJ_ALGO_COUNT) return HJ_E_INVAL;
    memset(out, 0, sizeof(*out));
    if ((nR && !R) || (nS && !S)) return out->status = HJ_E_INVAL;
    hj_params_t p;
    resolve_params(pin, &p);
    if (p.device != c->device) return out->status = HJ_E_INVAL;
    JoinPlan jp;
    int rc = plan_join(algo, &p, nR, nS, &jp);
    if (rc) return out->status = rc;
    if (is_phj(algo)) out->physical_passes = jp.geom.passes;
    if (nR == 0 || nS == 0) return out->status = HJ_OK;  // no join task (src/algo/phj.c:1290)

    DeviceGuard g(c->device);
    std::lock_guard<std::mutex> lk(c->mu);
    const bool host_in = !p.inputs_on_device;
    // Few build tuples: one kernel, without scratch.
    const bool small = nR <= hj::kSmallMaxBuild && !(p.flags & kPipelineFlags);
    if (small) {
        out->physical_passes = 0;
        if (host_in) rc = ensure_arena(c, kAccBytes + align256(nR * 16) + align256(nS * 16));
    } else {
        rc = ensure_plan(c, algo, &jp, [&] { return scratch_need(jp, p, nR, nS, host_in, c->num_sms); });
    }
    if (rc) return out->status = rc;
    const bool radix = jp.radix, seg = jp.seg && !small;
    const hj::RadixGeom &geom = jp.geom;
    cudaStream_t st = p.stream ? (cudaStream_t)p.stream : c->stream;
    // A join that a watchdog gave up on may still run; its arena use must end before this one starts.
    if (c->gave_up) {
        CU_OR(cudaStreamWaitEvent(st, c->ev_done, 0), out->status = HJ_E_DEVICE);
        c->gave_up = false;
    }
    const bool timing = !(p.flags & HJ_F_NO_TIMING);
    const bool phases = (p.flags & HJ_F_PHASE_TIMES) != 0;
    cudaEvent_t *ph = phases ? c->ev_ph : nullptr;
    uint32_t launches = 0;

    char *cur = c->arena;
    JoinAccum *acc = reinterpret_cast<JoinAccum *>(cur);
    cur += kAccBytes;
    const ulonglong2 *dR = reinterpret_cast<const ulonglong2 *>(R);
    const ulonglong2 *dS = reinterpret_cast<const ulonglong2 *>(S);
    if (host_in) {
        ulonglong2 *r = reinterpret_cast<ulonglong2 *>(cur);
        cur += align256(nR * 16);
        ulonglong2 *s = reinterpret_cast<ulonglong2 *>(cur);
        cur += align256(nS * 16);
        if (timing) CU_OR(cudaEventRecord(c->ev_h2d, st), out->status = HJ_E_DEVICE);
        const hj::HostCopy copies[2] = {{r, R, nR * 16}, {s, S, nS * 16}};
        rc = hj::copy_in(c, copies, 2, (p.flags & HJ_F_PINNED_HOST) != 0, st);
        if (rc) {
            cudaStreamSynchronize(st);
            return out->status = rc;
        }
        dR = r;
        dS = s;
    }
    // phj_radix_lp: first with unordered partition passes (phj_radix_bc's ranks), then, only if a probe
    // tuple matched two build tuples (the first match then depends on the order inside a partition),
    // again with ordered ones. The second run needs the first one's flag on the host, so these joins
    // are not captured into a graph; a build relation that needed it runs ordered at once next time.
    // The one-pass pipeline needs neither: its build elements carry their input position. It reports
    // HJ_RES_ORDERED_PASSES for the joins that the two-pass pipelines would have run ordered.
    const bool lp_first = radix && hj::algo_lp(algo) && !(p.flags & (HJ_F_ORDERED | HJ_F_TEST_STALL)) &&
                          p.watchdog_ms <= 0 && !(c->lp_ordered_R == (const void *)R && c->lp_ordered_nR == nR);
    const bool lp_try = lp_first && !geom.single && !small;
    const bool lp_ordered = radix && hj::algo_lp(algo) && !lp_first;
    bool lp_rerun = false;
    // The one-pass pipeline writes its result to acc_host itself and leaves large partitions, if any, to a
    // second step below (a watchdog's deadline covers one step only, so such a join has none).
    const bool one_pass = radix && geom.single && !small && p.watchdog_ms <= 0;
    // Everything from the result reset to the result copy; a repeated device-resident join replays it
    // from a CUDA graph (the key holds every input of the enqueued work).
    auto enqueue = [&]() -> int {
        if (small) {
            // The build and the probe are one kernel, timed as the probe.
            if (timing && hj::record_event(c->ev_start, st) != cudaSuccess) return HJ_E_DEVICE;
            for (int i = 0; ph && i < HJ_PH_LARGE; i++)
                if (hj::record_event(ph[i], st) != cudaSuccess) return HJ_E_DEVICE;
            int erc = hj::phj_prepare_device(false, false);
            if (!erc)
                erc = hj::small_enqueue(hj::algo_lp(algo), hj::algo_skip0(algo), is_phj(algo) ? geom.req_bits : -1, dR,
                                        nR, dS, nS, reinterpret_cast<hj::SmallPart *>(c->small_buf + 256),
                                        reinterpret_cast<uint32_t *>(c->small_buf), c->acc_host, st, c->num_sms);
            if (erc) return erc;
            launches = 1;
            for (int i = HJ_PH_LARGE; ph && i <= HJ_PH_COUNT; i++)
                if (hj::record_event(ph[i], st) != cudaSuccess) return HJ_E_DEVICE;
            if (timing && hj::record_event(c->ev_end, st) != cudaSuccess) return HJ_E_DEVICE;
            return HJ_OK;
        }
        if (!one_pass && cudaMemsetAsync(acc, 0, sizeof(JoinAccum), st) != cudaSuccess) return HJ_E_DEVICE;
        if (timing && hj::record_event(c->ev_start, st) != cudaSuccess) return HJ_E_DEVICE;
        int erc;
        if (radix) {
            hj::PhjScratch s;
            hj::phj_carve(geom, nR, nS, c->num_sms, cur, &s, seg);
            const int tf = ((p.flags & HJ_F_TEST_STALL) ? 1 : 0) | ((p.flags & HJ_F_WIDE) ? 2 : 0) |
                           ((p.flags & HJ_F_WORDS) ? 4 : 0);
            uint32_t first = 0;
            if (lp_try) {
                erc = hj::phj_enqueue(geom, true, hj::algo_skip0(algo), dR, nR, dS, nS, s, acc, st,
                                      timing ? c->ev_mid : nullptr, c->num_sms, ph, &first, nullptr, tf, false);
                if (erc) return erc;
                if (cudaMemcpyAsync(c->acc_host, acc, sizeof(JoinAccum), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                    cudaStreamSynchronize(st) != cudaSuccess)
                    return HJ_E_DEVICE;
                lp_rerun = c->acc_host->dup_flag != 0;
                if (lp_rerun && cudaMemsetAsync(acc, 0, sizeof(JoinAccum), st) != cudaSuccess) return HJ_E_DEVICE;
            }
            if (!lp_try || lp_rerun)
                erc = hj::phj_enqueue(geom, hj::algo_lp(algo), hj::algo_skip0(algo), dR, nR, dS, nS, s, acc, st,
                                      timing ? c->ev_mid : nullptr, c->num_sms, ph, &launches, nullptr, tf, true,
                                      one_pass ? c->acc_host : nullptr);
            launches += first;
        } else {
            const size_t tb = c->arena_bytes - (size_t)(cur - c->arena);
            erc = hj::nphj_enqueue(hj::algo_lp(algo), false, dR, nR, dS, nS, cur, tb, p.table_load, acc, st,
                                   timing ? c->ev_mid : nullptr, c->num_sms, ph, &launches);
        }
        if (erc) return erc;
        if (timing && hj::record_event(c->ev_end, st) != cudaSuccess) return HJ_E_DEVICE;
        if (one_pass) return HJ_OK;  // its last kernel writes the result to acc_host
        if (cudaMemcpyAsync(c->acc_host, acc, sizeof(JoinAccum), cudaMemcpyDeviceToHost, st) != cudaSuccess)
            return HJ_E_DEVICE;
        return HJ_OK;
    };
    hj_graph_key key;
    const bool graphable = !host_in && st == c->stream && !(p.flags & HJ_F_TEST_STALL) && !lp_try && !small;
    if (graphable) {
        key.algo = (int)algo;
        key.R = R;
        key.S = S;
        key.nR = nR;
        key.nS = nS;
        key.flags = p.flags;
        key.bits = p.num_radix_bits;
        key.passes = p.num_passes;
        key.bits_pass1 = p.radix_bits_pass1;
        key.table_load = p.table_load;
        key.seg = seg;
        key.radix = radix;
        key.one_pass = one_pass;  // differs between calls with and without a watchdog
        key.arena = c->arena;
        key.arena_bytes = c->arena_bytes;
    }
    if (hj_graph_entry *ge = graphable ? find_graph(c, key) : nullptr) {
        CU_OR(cudaGraphLaunch(ge->exec, st), out->status = HJ_E_DEVICE);
        launches = ge->launches;
    } else if (graphable && key == c->last_key) {
        // Second identical call in a row: capture, instantiate, launch; keep the graph. If the capture
        // or the instantiation fails, the join runs its kernels directly instead.
        bool ran = false;
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            const int crc = enqueue();
            cudaGraph_t graph = nullptr;
            const cudaError_t ce = cudaStreamEndCapture(st, &graph);
            cudaGraphExec_t exec = nullptr;
            if (!crc && ce == cudaSuccess && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess &&
                cudaGraphLaunch(exec, st) == cudaSuccess) {
                if (c->graphs.size() >= kMaxJoinGraphs) {
                    size_t lru = 0;
                    for (size_t i = 1; i < c->graphs.size(); i++)
                        if (c->graphs[i].used < c->graphs[lru].used) lru = i;
                    cudaGraphExecDestroy(c->graphs[lru].exec);
                    c->graphs.erase(c->graphs.begin() + (long)lru);
                }
                hj_graph_entry e;
                e.key = key;
                e.exec = exec;
                e.launches = launches;
                e.used = ++c->graph_tick;
                c->graphs.push_back(e);
                ran = true;
            } else if (exec) {
                cudaGraphExecDestroy(exec);
            }
            if (graph) cudaGraphDestroy(graph);
            if (crc && crc != HJ_E_DEVICE) {  // an argument the enqueue rejects: the same without a graph
                cudaGetLastError();
                return out->status = crc;
            }
        }
        cudaGetLastError();
        if (!ran) {
            launches = 0;
            rc = enqueue();
            if (rc) {
                cudaStreamSynchronize(st);
                return out->status = rc;
            }
        }
    } else {
        rc = enqueue();
        if (rc) {
            cudaStreamSynchronize(st);
            return out->status = rc;
        }
    }
    if (graphable) c->last_key = key;
    if (p.watchdog_ms > 0) {
        // Host watchdog: poll the join's completion against a deadline instead of blocking.
        CU_OR(cudaEventRecord(c->ev_done, st), out->status = HJ_E_DEVICE);
        const auto deadline = std::chrono::steady_clock::now() + std::chrono::milliseconds(p.watchdog_ms);
        for (;;) {
            const cudaError_t q = cudaEventQuery(c->ev_done);
            if (q == cudaSuccess) break;
            if (q != cudaErrorNotReady) return out->status = HJ_E_DEVICE;
            if (std::chrono::steady_clock::now() > deadline) {
                c->gave_up = true;
                return out->status = HJ_E_TIMEOUT;
            }
            std::this_thread::sleep_for(std::chrono::microseconds(50));
        }
    } else {
        CU_OR(cudaStreamSynchronize(st), out->status = HJ_E_DEVICE);
    }
    JoinAccum res = *c->acc_host;
    unsigned long long raw_large = 0;  // large partitions of the digits asked for, when the join ran again by mix_key
    hj::RadixGeom run_geom = geom;
    if (one_pass && !geom.mix && nR > kRerunMinBuild && res.large_build > nR / 2) {
        raw_large = res.large_parts;
        run_geom.mix = true;
        hj::PhjScratch s;
        hj::phj_carve(run_geom, nR, nS, c->num_sms, cur, &s, false);
        uint32_t again = 0;
        rc = hj::phj_enqueue(run_geom, hj::algo_lp(algo), hj::algo_skip0(algo), dR, nR, dS, nS, s, acc, st,
                             timing ? c->ev_mid : nullptr, c->num_sms, ph, &again, nullptr, 0, true, c->acc_host);
        launches += again;
        if (rc) {
            cudaStreamSynchronize(st);
            return out->status = rc;
        }
        if (timing) CU_OR(cudaEventRecord(c->ev_end, st), out->status = HJ_E_DEVICE);
        CU_OR(cudaStreamSynchronize(st), out->status = HJ_E_DEVICE);
        res = *c->acc_host;
    }
    if (one_pass && res.large_parts) {
        // Partitions beyond shared memory (rare: a hot build key, or keys that share their low bits) are
        // joined by a second batch of kernels, launched only now that there are some.
        hj::PhjScratch s;
        hj::phj_carve(run_geom, nR, nS, c->num_sms, cur, &s, false);
        rc = hj::phj_large_enqueue(run_geom, hj::algo_lp(algo), hj::algo_skip0(algo), dR, nR, nS, s, acc, st, c->num_sms,
                                   &launches);
        if (rc) return out->status = rc;
        if (phases) CU_OR(cudaEventRecord(c->ev_ph[HJ_PH_COUNT], st), out->status = HJ_E_DEVICE);
        if (timing) CU_OR(cudaEventRecord(c->ev_end, st), out->status = HJ_E_DEVICE);
        CU_OR(cudaMemcpyAsync(c->acc_host, acc, sizeof(JoinAccum), cudaMemcpyDeviceToHost, st),
              out->status = HJ_E_DEVICE);
        CU_OR(cudaStreamSynchronize(st), out->status = HJ_E_DEVICE);
        res.matched += c->acc_host->matched;
        res.checksum += c->acc_host->checksum;
        res.error |= c->acc_host->error;
        res.dup_flag |= c->acc_host->dup_flag;
    }
    out->matched_cnt = res.matched;
    out->checksum = res.checksum;
    out->large_partitions = !is_phj(algo) ? 0 : raw_large ? raw_large : res.large_parts;
    out->flags = is_phj(algo) ? (uint32_t)res.flags : 0u;
    if (lp_first && !lp_try) lp_rerun = res.dup_flag != 0;
    if (is_phj(algo) && (lp_ordered || lp_rerun)) out->flags |= HJ_RES_ORDERED_PASSES;
    if (lp_rerun) {
        c->lp_ordered_R = R;
        c->lp_ordered_nR = nR;
    }
    if (timing) {
        float a = 0, b = 0, h = 0;
        if (!small) cudaEventElapsedTime(&a, c->ev_start, c->ev_mid);
        cudaEventElapsedTime(&b, small ? c->ev_start : c->ev_mid, c->ev_end);
        if (host_in) cudaEventElapsedTime(&h, c->ev_h2d, c->ev_start);
        out->buildpart = a * 1e-3;
        out->probejoin = b * 1e-3;
        out->total = out->buildpart + out->probejoin;
        out->h2d = h * 1e-3;
    }
    if (phases) {
        for (int i = 0; i < HJ_PH_COUNT; i++) {
            float ms = 0;
            int from = 0, to = 0;
            if (!is_phj(algo) && radix) {
                // Non-partitioned joins report a build and a probe phase: partitioning and the joins.
                from = i == HJ_PH_JOIN ? (seg ? 3 : 4) : 0;
                to = i == HJ_PH_JOIN ? (seg ? 5 : 6) : (seg ? 3 : 4);
                if (i == HJ_PH_HIST || i == HJ_PH_JOIN) cudaEventElapsedTime(&ms, c->ev_ph[from], c->ev_ph[to]);
            } else if (hj::phj_phase_span(seg, i, &from, &to)) {
                cudaEventElapsedTime(&ms, c->ev_ph[from], c->ev_ph[to]);
            }
            out->phase[i] = ms * 1e-3;
        }
    }
    out->kernel_launches = launches;
    out->status = map_error_bits(res.error);
    return out->status;
}

// Materialising joins (the reference's ptr_* joins, src/algo/ptr_phj.c, ptr_nphj.c): the join writes
// one (r.row_id, s.row_id) pair per match, and a retrieve phase recomputes the checksum by gathering
// R[r_row_id - 1].row_id + S[s_row_id - 1].row_id (src/inc/utils.c:712-724).
static int join_mat(hj_ctx *c, hj_algo_t algo, hj_params_t p, const hj_tuple_t *R, size_t nR,
                    const hj_tuple_t *S, size_t nS, hj_pair_t *user_pairs, size_t user_cap,
                    unsigned long long cap_guess, hj_result_t *out) {
    JoinPlan jp;
    int rc = plan_join(algo, &p, nR, nS, &jp, true);
    if (rc) return out->status = rc;
    if (is_phj(algo)) out->physical_passes = jp.geom.passes;
    if (nR == 0 || nS == 0) return out->status = HJ_OK;
    const bool host_in = !p.inputs_on_device;
    // Pairs land in the caller's device buffer, or in the arena (library-owned, or staged for a host
    // buffer).
    const bool pairs_in_arena = !user_pairs || host_in;
    const unsigned long long cap = user_pairs ? (unsigned long long)user_cap : cap_guess;
    auto need_of = [&]() {
        size_t need = kAccBytes;
        if (host_in) need += align256(nR * 16) + align256(nS * 16);
        if (jp.radix)
            need += hj::phj_scratch_bytes(jp.geom, nR, nS, c->num_sms, jp.seg);
        else
            need += align256(hj::nphj_scratch_bytes(nR, p.table_load, true));
        if (pairs_in_arena) need += align256(cap * 16);
        return need;
    };
    rc = ensure_plan(c, algo, &jp, need_of);
    if (rc) return out->status = rc;
    const bool seg = jp.seg;
    const hj::RadixGeom &geom = jp.geom;
    cudaStream_t st = p.stream ? (cudaStream_t)p.stream : c->stream;
    CU_OR(cudaStreamWaitEvent(st, c->ev_done, 0), out->status = HJ_E_DEVICE);
    const bool timing = !(p.flags & HJ_F_NO_TIMING);
    uint32_t launches = 0;

    char *cur = c->arena;
    JoinAccum *acc = reinterpret_cast<JoinAccum *>(cur);
    cur += kAccBytes;
    const ulonglong2 *dR = reinterpret_cast<const ulonglong2 *>(R);
    const ulonglong2 *dS = reinterpret_cast<const ulonglong2 *>(S);
    if (host_in) {
        ulonglong2 *r = reinterpret_cast<ulonglong2 *>(cur);
        cur += align256(nR * 16);
        ulonglong2 *s = reinterpret_cast<ulonglong2 *>(cur);
        cur += align256(nS * 16);
        if (timing) CU_OR(cudaEventRecord(c->ev_h2d, st), out->status = HJ_E_DEVICE);
        const hj::HostCopy copies[2] = {{r, R, nR * 16}, {s, S, nS * 16}};
        rc = hj::copy_in(c, copies, 2, (p.flags & HJ_F_PINNED_HOST) != 0, st);
        if (rc) {
            cudaStreamSynchronize(st);
            return out->status = rc;
        }
        dR = r;
        dS = s;
    }
    hj::MatOut mat;
    mat.cap = cap;
    if (pairs_in_arena) {
        mat.pairs = reinterpret_cast<ulonglong2 *>(cur);
        cur += align256(cap * 16);
    } else {
        mat.pairs = reinterpret_cast<ulonglong2 *>(user_pairs);
    }
    CU_OR(cudaMemsetAsync(acc, 0, sizeof(JoinAccum), st), out->status = HJ_E_DEVICE);
    if (timing) CU_OR(cudaEventRecord(c->ev_start, st), out->status = HJ_E_DEVICE);
    void *dead = cur;  // scratch that the retrieve phase may use: the join's partitions, or its table
    size_t dead_bytes = c->arena_bytes - (size_t)(cur - c->arena);
    if (jp.radix) {
        hj::PhjScratch s;
        hj::phj_carve(geom, nR, nS, c->num_sms, cur, &s, seg);
        dead = s.tmp1;
        dead_bytes = (nR + nS) * 16;
        rc = hj::phj_enqueue(geom, hj::algo_lp(algo), hj::algo_skip0(algo), dR, nR, dS, nS, s, acc, st,
                             timing ? c->ev_mid : nullptr, c->num_sms, nullptr, &launches, &mat);
    } else {
        const size_t tb = c->arena_bytes - (size_t)(cur - c->arena);
        rc = hj::nphj_enqueue(hj::algo_lp(algo), false, dR, nR, dS, nS, cur, tb, p.table_load, acc, st,
                              timing ? c->ev_mid : nullptr, c->num_sms, nullptr, &launches, &mat);
    }
    if (!rc) {
        if (timing) CU_OR(cudaEventRecord(c->ev_end, st), out->status = HJ_E_DEVICE);
        rc = hj::mat_retrieve_enqueue(mat.pairs, &acc->pairs, cap, dR, nR, dS, nS, dead, dead_bytes, acc, st,
                                      c->num_sms, &launches);
    }
    if (rc) {
        cudaStreamSynchronize(st);
        return out->status = rc;
    }
    if (timing) CU_OR(cudaEventRecord(c->ev_ret, st), out->status = HJ_E_DEVICE);
    CU_OR(cudaMemcpyAsync(c->acc_host, acc, sizeof(JoinAccum), cudaMemcpyDeviceToHost, st),
          out->status = HJ_E_DEVICE);
    CU_OR(cudaStreamSynchronize(st), out->status = HJ_E_DEVICE);
    const unsigned long long n = c->acc_host->pairs;
    if (user_pairs && host_in && n)
        CU_OR(cudaMemcpy(user_pairs, mat.pairs, (size_t)(n < cap ? n : cap) * 16, cudaMemcpyDeviceToHost),
              out->status = HJ_E_DEVICE);
    out->matched_cnt = n;
    out->checksum = c->acc_host->checksum;
    if (is_phj(algo)) {
        out->large_partitions = c->acc_host->large_parts;
        out->flags = (uint32_t)c->acc_host->flags;
    }
    if (timing) {
        float a = 0, b = 0, r = 0, h = 0;
        cudaEventElapsedTime(&a, c->ev_start, c->ev_mid);
        cudaEventElapsedTime(&b, c->ev_mid, c->ev_end);
        cudaEventElapsedTime(&r, c->ev_end, c->ev_ret);
        if (host_in) cudaEventElapsedTime(&h, c->ev_h2d, c->ev_start);
        out->buildpart = a * 1e-3;
        out->probejoin = b * 1e-3;
        out->retrieve = r * 1e-3;
        // The reference's ptr joins time partition/build + join/probe + retrieve (ptr_phj.c:3094-3096).
        out->total = out->buildpart + out->probejoin + out->retrieve;
        out->h2d = h * 1e-3;
    }
    out->kernel_launches = launches;
    out->status = map_error_bits(c->acc_host->error);
    return out->status;
}

int hj_join_mat_ctx(hj_ctx_t *c, hj_algo_t algo, const hj_params_t *pin, const hj_tuple_t *R, size_t nR,
                    const hj_tuple_t *S, size_t nS, hj_pair_t *pairs, size_t pair_cap, hj_result_t *out) {
    if (!c || !out || (int)algo < 0 || algo >= HJ_ALGO_COUNT) return HJ_E_INVAL;
    memset(out, 0, sizeof(*out));
    if ((nR && !R) || (nS && !S) || (pair_cap && !pairs)) return out->status = HJ_E_INVAL;
    hj_params_t p;
    resolve_params(pin, &p);
    if (p.device != c->device) return out->status = HJ_E_INVAL;
    DeviceGuard g(c->device);
    std::lock_guard<std::mutex> lk(c->mu);
    if (pairs) return join_mat(c, algo, p, R, nR, S, nS, pairs, pair_cap, 0, out);
    // Library-owned pairs: first-match joins write at most |S| pairs; for the others |S| is the
    // guess (exact for PK-FK joins), and one rerun with the exact count follows when it was short.
    int rc = join_mat(c, algo, p, R, nR, S, nS, nullptr, 0, nS ? nS : 1, out);
    if (rc == HJ_E_CAPACITY) {
        const unsigned long long need = out->matched_cnt;
        memset(out, 0, sizeof(*out));
        rc = join_mat(c, algo, p, R, nR, S, nS, nullptr, 0, need, out);
    }
    return rc;
}

int hj_join_mat(hj_algo_t algo, const hj_params_t *pin, const hj_tuple_t *R, size_t nR, const hj_tuple_t *S,
                size_t nS, hj_pair_t *pairs, size_t pair_cap, hj_result_t *out) {
    hj_params_t p;
    resolve_params(pin, &p);
    if (p.device < 0 || p.device >= 64) return HJ_E_INVAL;
    hj_ctx *c;
    {
        std::lock_guard<std::mutex> lk(g_default_mu);
        if (!g_default[p.device]) {
            int rc = hj_ctx_create(p.device, &g_default[p.device]);
            if (rc) return rc;
        }
        c = g_default[p.device];
    }
    return hj_join_mat_ctx(c, algo, &p, R, nR, S, nS, pairs, pair_cap, out);
}

int hj_join(hj_algo_t algo, const hj_params_t *pin, const hj_tuple_t *R, size_t nR, const hj_tuple_t *S,
            size_t nS, hj_result_t *out) {
    hj_params_t p;
    resolve_params(pin, &p);
    if (p.device < 0 || p.device >= 64) return HJ_E_INVAL;
    hj_ctx *c;
    {
        std::lock_guard<std::mutex> lk(g_default_mu);
        if (!g_default[p.device]) {
            int rc = hj_ctx_create(p.device, &g_default[p.device]);
            if (rc) return rc;
        }
        c = g_default[p.device];
    }
    return hj_join_ctx(c, algo, &p, R, nR, S, nS, out);
}

}  // extern "C"
