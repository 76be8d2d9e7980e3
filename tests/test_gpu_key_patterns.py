"""Build keys with structure (strides, ids in the high half, packed fields) through every route that partitions by
key bits, against the oracle. The tables of partitions beyond shared memory, the chains in shared memory and the
partitions themselves must not degenerate on them: a join here takes well under a millisecond, and one that
walks a chain of all its build tuples per tuple takes seconds, so the time is bounded far from both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ALGOS = ["phj_radix_bc", "phj_radix_lp", "nphj_sc", "nphj_lp"]
PATTERNS = {
    "x4": lambda k: k * np.uint64(4),
    "x2^11": lambda k: k << np.uint64(11),
    "x2^14": lambda k: k << np.uint64(14),
    "x2^32": lambda k: k << np.uint64(32),
    "packed": lambda k: ((k >> np.uint64(8)) << np.uint64(40)) | ((k & np.uint64(255)) << np.uint64(20)),
}


def relations(rng, nR, nS, pattern, dup=1, rid_bits=32):
    """Every build key `dup` times; a quarter of the probe tuples without a match."""
    f = PATTERNS[pattern]
    n = max(1, nR // dup)
    R, S = np.empty((nR, 2), dtype=np.uint64), np.empty((nS, 2), dtype=np.uint64)
    R[:, 0] = f(rng.permutation(nR).astype(np.uint64) % np.uint64(n))  # key 0 included
    S[:, 0] = f(rng.integers(0, n + n // 3 + 1, nS, dtype=np.uint64))
    R[:, 1] = rng.integers(0, 1 << rid_bits, nR, dtype=np.uint64)
    S[:, 1] = rng.integers(0, 1 << rid_bits, nS, dtype=np.uint64)
    return R, S


def dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("pattern", list(PATTERNS))
@pytest.mark.parametrize("nR", [9_000, 20_000, 300_000])
def test_single_joins(hj, oracle, cuda, nR, pattern, algo):
    """Partitions beyond shared memory whose keys share bits above the radix bits too."""
    rng = np.random.default_rng(nR)
    for dup in (1, 3):
        R, S = relations(rng, nR, 2 * nR + 7, pattern, dup)
        want = oracle.join(algo, R, S)
        for flags in (0, hj.HJ_F_EXACT) if algo.startswith("phj") else (0,):
            r = hj.join(algo, dev(cuda, R), dev(cuda, S), on_device=True, flags=flags)
            assert (r.matched_cnt, r.checksum) == want, (dup, flags)
            assert r.total < 0.1, (dup, flags)


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp"])
@pytest.mark.parametrize("pattern", ["x2^14", "x2^32"])
def test_materialised_large_partitions(hj, oracle, cuda, pattern, algo):
    rng = np.random.default_rng(5)
    R, S = relations(rng, 60_000, 90_000, pattern)
    R[:, 1] = np.arange(1, R.shape[0] + 1, dtype=np.uint64)
    S[:, 1] = np.arange(1, S.shape[0] + 1, dtype=np.uint64)
    want = oracle.join_pairs(algo, R, S)
    out = cuda.zeros((want.shape[0], 2), dtype=cuda.int64, device="cuda")
    r = hj.join_mat(algo, dev(cuda, R), dev(cuda, S), pairs=out, on_device=True)
    got = out.cpu().numpy().view(np.uint64)
    assert r.matched_cnt == want.shape[0]
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want)


@pytest.mark.parametrize("algo", ALGOS)
def test_partitions_of_keys_that_share_low_bits(hj, cuda, algo):
    """Partitions that fit shared memory, whose keys are equal in 24 bits above the radix bits: no slower than five
    times the same join of mixed keys (one chain per partition: over twenty times)."""
    nR, nS = 1 << 20, 1 << 21
    g = cuda.Generator(device="cuda")
    g.manual_seed(1)
    R = cuda.empty((nR, 2), dtype=cuda.int64, device="cuda")
    S = cuda.empty((nS, 2), dtype=cuda.int64, device="cuda")
    r, s = cuda.randperm(nR, generator=g, device="cuda"), cuda.randint(0, nR, (nS,), generator=g, device="cuda")
    R[:, 1], S[:, 1] = cuda.arange(nR, device="cuda") << 20, cuda.arange(nS, device="cuda")
    rid = cuda.empty(nR, dtype=cuda.int64, device="cuda")
    rid[r] = R[:, 1]
    want = (nS, int((rid[s] + S[:, 1]).sum()))
    times = []
    for f in (lambda k: k * 0x1E3779B97F4A7C15 & 0x7FFFFFFFFFFFFFFF, lambda k: (k << 32) | (k & 255)):
        R[:, 0], S[:, 0] = f(r + 1), f(s + 1)  # key 0 never matches in phj_radix_lp
        with hj.Context(0) as ctx:
            res = [hj.join(algo, R, S, on_device=True, ctx=ctx) for _ in range(5)]
        assert all((q.matched_cnt, q.checksum) == want for q in res)
        times.append(min(q.total for q in res))
    assert times[1] < 5 * times[0], times


@pytest.mark.parametrize("kind", ["x16", "hot"])
def test_batch_jobs_with_large_partitions(hj, cuda, kind):
    """Batch jobs of millions of tuples whose partitions exceed shared memory, or whose hot build key's does: the
    answer, and a time of the order of a single join's (one block per job for these partitions: 20 times it)."""
    nR, nS = 1 << 21, 1 << 23
    g = cuda.Generator(device="cuda")
    g.manual_seed(2)
    jobs, want, alone = [], [], []
    for i, algo in enumerate(("nphj_sc", "phj_radix_lp", "nphj_lp", "phj_radix_bc")):
        k = cuda.randperm(nR, generator=g, device="cuda") + 1
        s = cuda.randint(1, nR + nR // 4, (nS,), generator=g, device="cuda")
        if kind == "hot":
            k[nR // 4: 3 * nR // 4] = k[0]
            s[: nS // 2] = k[0]
        R, S = (cuda.empty((n, 2), dtype=cuda.int64, device="cuda") for n in (nR, nS))
        R[:, 1], S[:, 1] = cuda.randperm(nR, generator=g, device="cuda"), cuda.arange(nS, device="cuda")
        cnt = cuda.bincount(k, minlength=2 * nR)
        if algo.endswith("lp"):
            first = cuda.full((2 * nR,), nR, device="cuda").scatter_reduce_(0, k, cuda.arange(nR, device="cuda"), "amin")
            m = (cnt[s] > 0).to(cuda.int64)
            total = ((R[:, 1][first[s].clamp(max=nR - 1)] + S[:, 1]) * m).sum()
        else:
            m = cnt[s]
            total = (cuda.zeros(2 * nR, dtype=cuda.int64, device="cuda").index_add_(0, k, R[:, 1])[s] + m * S[:, 1]).sum()
        want.append((int(m.sum()), int(total) % 2**64))
        R[:, 0], S[:, 0] = (k, s) if kind == "hot" else (k * 16, s * 16)
        jobs.append((algo, R, S))
        with hj.Context(0) as ctx:
            alone.append(min(hj.join("phj_radix_" + ("lp" if algo.endswith("lp") else "bc"), R, S, on_device=True,
                                     ctx=ctx).total for _ in range(3)))
    with hj.Context(0) as ctx, hj.Batch(ctx, jobs) as b:
        stats = []
        for _ in range(3):
            res, st = b.run()
            assert [(r.status, r.matched_cnt, r.checksum) for r in res] == [(0, *w) for w in want]
            stats.append(st.seconds)
    assert min(stats) < 3 * sum(alone), (stats, alone)


@pytest.mark.parametrize("algo,nR", [("phj_radix_lp", 1 << 20), ("nphj_lp", (1 << 21) + 5)])
@pytest.mark.parametrize("copies", [2, 1000])
def test_first_match_of_repeated_wide_keys(hj, oracle, cuda, algo, nR, copies):
    """First matches over 16-byte tuples: one node per key, so that repeated keys cost a probe no walk; the joins'
    sums, the pairs' retrieved row ids, and a time of the order of distinct keys' (a walk over 1000: ten times)."""
    rng = np.random.default_rng(copies)
    nS, times = 1 << 21, []
    for c in (1, copies):
        n = nR // c
        R, S = np.empty((nR, 2), dtype=np.uint64), np.empty((nS, 2), dtype=np.uint64)
        R[:, 0] = (rng.permutation(nR).astype(np.uint64) % np.uint64(n) + np.uint64(1)) * np.uint64(0x1E3779B97F4A7C15)
        S[:, 0] = rng.integers(1, n + n // 4 + 2, nS, dtype=np.uint64) * np.uint64(0x1E3779B97F4A7C15)
        R[:, 1], S[:, 1] = np.arange(1, nR + 1, dtype=np.uint64), np.arange(1, nS + 1, dtype=np.uint64)
        want, dR, dS = oracle.join(algo, R, S), dev(cuda, R), dev(cuda, S)
        with hj.Context(0) as ctx:
            got = [hj.join(algo, dR, dS, on_device=True, ctx=ctx) for _ in range(4)]
            assert all((r.matched_cnt, r.checksum) == want for r in got)
            times.append(min(r.total for r in got))
            r = hj.join_mat(algo, dR, dS, on_device=True, ctx=ctx)
            assert (r.matched_cnt, r.checksum) == want
            if algo.startswith("phj"):
                assert bool(got[0].flags & hj.HJ_RES_ORDERED_PASSES) == (c > 1)
    assert times[1] < 3 * times[0], times


STRIDES = {"x1": lambda k: k, "x4": lambda k: k * 4, "x2^14": lambda k: k << 14, "x2^32": lambda k: k << 32}


@pytest.mark.parametrize("algo,nR,nS", [
    ("phj_radix_bc", 1 << 17, 1 << 18), ("phj_radix_lp", 1 << 21, 1 << 21),   # raw digits, run again by mix_key
    ("phj_radix_bc", (1 << 21) + 1, 1 << 22), ("phj_radix_lp", (1 << 21) + 1, 1 << 22),  # one pass by mix_key
    ("nphj_sc", 1 << 21, 1 << 22), ("nphj_lp", (1 << 21) + 7, 1 << 22),
    ("phj_radix_bc", (1 << 24) + 1, 1 << 24), ("phj_radix_lp", (1 << 24) + 1, 1 << 24),  # two passes, exact offsets
    ("phj_radix_bc", (1 << 24) + 1, 3 << 24), ("phj_radix_lp", (1 << 24) + 1, 3 << 24),  # two passes, segments
    ("nphj_sc", (1 << 24) + 1, 1 << 25), ("nphj_lp", (1 << 24) + 1, 1 << 25)])            # segments; the table
def test_strided_keys(hj, cuda, algo, nR, nS):
    """Distinct keys with a stride: the answer, no partition beyond shared memory where mix_key picks them, and no
    more than four times a dense join's time (raw digits of such keys: six to ten times)."""
    g = cuda.Generator(device="cuda")
    g.manual_seed(nR)
    R, S = (cuda.empty((n, 2), dtype=cuda.int64, device="cuda") for n in (nR, nS))
    r = cuda.randperm(nR, generator=g, device="cuda")
    s = cuda.randint(0, nR + nR // 4, (nS,), generator=g, device="cuda")
    R[:, 1], S[:, 1] = cuda.randperm(nR, generator=g, device="cuda"), cuda.arange(nS, device="cuda")
    rid = cuda.empty(nR, dtype=cuda.int64, device="cuda")
    rid[r] = R[:, 1]
    hit = s < nR
    want = (int(hit.sum()), int((rid[s[hit]] + S[:, 1][hit]).sum()))
    times = {}
    for name, f in STRIDES.items():
        R[:, 0], S[:, 0] = f(r + 1), f(s + 1)
        with hj.Context(0) as ctx:
            res = [hj.join(algo, R, S, on_device=True, ctx=ctx) for _ in range(4)]
        assert all((q.matched_cnt, q.checksum) == want for q in res), name
        raw = algo.startswith("phj") and nR <= 1 << 21
        assert raw or all(q.large_partitions == 0 for q in res), name
        times[name] = min(q.total for q in res)
    assert max(times.values()) < 4 * times["x1"], times


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp"])
@pytest.mark.parametrize("kind", ["strided", "hot"])
def test_run_again_by_mixed_keys(hj, oracle, cuda, algo, kind):
    """A join whose raw digits overfill most of the build side's partitions runs again: duplicates, key 0, wide row
    ids, the same partitions reported, with phase times, from a graph and from host memory; and a hot key, whose
    partition is too large by either digits."""
    rng = np.random.default_rng(77)
    nR, nS = 100_000, 230_000
    if kind == "strided":
        R, S = relations(rng, nR, nS, "x2^14", dup=3, rid_bits=40)
    else:
        R, S = relations(rng, nR, nS, "x4", rid_bits=32)
        R[20_000:90_000, 0] = R[1, 0]
        S[:3000, 0] = R[1, 0]
    want = oracle.join(algo, R, S)
    dR, dS = dev(cuda, R), dev(cuda, S)
    with hj.Context(0) as ctx:
        got = [hj.join(algo, dR, dS, on_device=True, ctx=ctx, flags=hj.HJ_F_PHASE_TIMES) for _ in range(4)]
        got += [hj.join(algo, R, S, ctx=ctx), hj.join(algo, dR, dS, on_device=True, ctx=ctx, watchdog_ms=60_000)]
    for r in got:
        assert (r.matched_cnt, r.checksum) == want
        assert r.large_partitions == got[0].large_partitions >= 1
        assert r.total > 0
