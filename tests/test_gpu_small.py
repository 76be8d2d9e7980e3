"""Joins of at most 8192 build tuples (one kernel) against the oracle and, for the radix joins, the two-pass
pipeline: every algorithm, sizes around the warp, block and build limits, duplicates, keys 0 and 2^64-1,
keys that share their low bits, wide row ids, repeated calls (the ticket is zero again), host inputs,
another stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ALGOS = ["phj_radix_bc", "phj_radix_lp", "nphj_sc", "nphj_lp", "phj_radix_hr"]


def dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


def relations(rng, nR, nS, kind):
    R = np.empty((nR, 2), dtype=np.uint64)
    S = np.empty((nS, 2), dtype=np.uint64)
    keys = max(2, nR // 4 if kind == "dup" else nR)
    R[:, 0] = rng.permutation(nR).astype(np.uint64) % np.uint64(keys)
    S[:, 0] = rng.integers(0, keys + keys // 3 + 1, nS, dtype=np.uint64)
    if kind == "shared_low_bits":
        R[:, 0] <<= np.uint64(40)
        S[:, 0] <<= np.uint64(40)
    if kind == "dup":
        R[::7, 0] = np.uint64(2**64 - 1)
        S[::5, 0] = np.uint64(2**64 - 1)
    rid = 64 if kind == "dup" else 32
    R[:, 1] = rng.integers(0, 2**rid - 1, nR, dtype=np.uint64)
    S[:, 1] = rng.integers(0, 2**rid - 1, nS, dtype=np.uint64)
    return R, S


@pytest.mark.parametrize("kind", ["plain", "dup", "shared_low_bits"])
@pytest.mark.parametrize("nR,nS", [(1, 1), (2, 4097), (31, 1024), (1023, 1025), (1024, 700_001), (8192, 33), (8191, 5000),
                                   (8193, 5000)])
def test_small_builds(hj, oracle, cuda, nR, nS, kind):
    rng = np.random.default_rng(nR * 7 + nS)
    R, S = relations(rng, nR, nS, kind)
    dR, dS = dev(cuda, R), dev(cuda, S)
    side = cuda.cuda.Stream()
    with hj.Context(0) as ctx:
        for algo in ALGOS:
            want = oracle.join(algo, R, S)
            got = [hj.join(algo, dR, dS, on_device=True, ctx=ctx) for _ in range(2)]
            got.append(hj.join(algo, R, S, ctx=ctx))
            got.append(hj.join(algo, dR, dS, on_device=True, ctx=ctx, stream=side.cuda_stream, flags=hj.HJ_F_PHASE_TIMES))
            for r in got:
                assert (r.matched_cnt, r.checksum) == want, algo
                assert r.large_partitions == 0
            if algo.startswith("phj"):
                two = hj.join(algo, dR, dS, on_device=True, ctx=ctx, flags=hj.HJ_F_EXACT)
                assert (two.matched_cnt, two.checksum) == want, algo
                assert two.flags == got[0].flags, algo


@pytest.mark.parametrize("nR", [2, 33, 1024, 8192])
@pytest.mark.parametrize("keys", [1, 8])
def test_first_match_of_few_keys(hj, oracle, cuda, nR, keys):
    """First-match joins with one place per key: a build relation on one or eight keys, in a join and in a batch,
    takes no longer for many probes than one of distinct keys (a walk over the duplicates: a hundred times)."""
    rng = np.random.default_rng(nR)
    nS = 1 << 19
    R, S = relations(rng, nR, nS, "plain")
    few = R.copy()
    few[:, 0] = rng.integers(1, keys + 1, nR, dtype=np.uint64) * np.uint64(1 << 33)
    fewS = S.copy()
    fewS[:, 0] = rng.integers(0, keys + 2, nS, dtype=np.uint64) * np.uint64(1 << 33)
    for algo in ("nphj_lp", "phj_radix_lp"):
        times = []
        for r, s in ((R, S), (few, fewS)):
            dr, ds, want = dev(cuda, r), dev(cuda, s), oracle.join(algo, r, s)
            with hj.Context(0) as ctx:
                got = [hj.join(algo, dr, ds, on_device=True, ctx=ctx) for _ in range(4)]
                assert all((g.matched_cnt, g.checksum) == want for g in got), algo
                ordered = [g.flags & hj.HJ_RES_ORDERED_PASSES != 0 for g in got]
                assert not any(ordered) if r is R or algo == "nphj_lp" else ordered[-1] == (keys < nR), algo
                times.append(min(g.total for g in got))
                with hj.Batch(ctx, [(algo, dr, ds)] * 2) as b:
                    assert [(g.matched_cnt, g.checksum) for g in b.run()[0]] == [want] * 2
        assert times[1] < 5 * times[0] + 20e-6, times
