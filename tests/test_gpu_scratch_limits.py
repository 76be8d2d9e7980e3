"""Little device memory left: plans whose scratch does not fit run the form that needs less, with the same result, and
keep what they have for the next call. The memory is taken by one allocation of the test's own."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Leave:
    """Leaves about `free` bytes of device memory."""

    def __init__(self, cuda, free):
        self.cuda = cuda
        cuda.cuda.synchronize()
        cuda.cuda.empty_cache()
        self.block = cuda.empty(max(0, cuda.cuda.mem_get_info()[0] - free), dtype=cuda.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        del self.block
        self.cuda.cuda.empty_cache()


def pkfk(hj, cuda, nR, nS, seed):
    R, S = (cuda.empty((n, 2), dtype=cuda.int64, device="cuda") for n in (nR, nS))
    hj.gen_fast_device(nR, nS, R.data_ptr(), S.data_ptr(), seed=seed)
    cuda.cuda.synchronize()
    return R, S


@pytest.mark.parametrize("mat", [False, True])
def test_non_partitioned_join_falls_back_to_the_table_once(hj, cuda, mat):
    """2^23 x 2^24 nphj_sc: 0.6 GB of radix scratch (one pass), 0.3 of table; with 0.45 free (0.75 with pairs) the table
    runs, and the next calls find its memory (and graph) where it was instead of freeing and asking again."""
    nR, nS = 1 << 23, 1 << 24
    R, S = pkfk(hj, cuda, nR, nS, 5)
    if mat:
        R[:, 1], S[:, 1] = cuda.arange(1, nR + 1, device="cuda"), cuda.arange(1, nS + 1, device="cuda")
    run = hj.join_mat if mat else hj.join
    with hj.Context(0) as roomy:
        want = run("nphj_sc", R, S, on_device=True, ctx=roomy)
        radix = roomy.scratch_bytes()
    with hj.Context(0) as table:
        run("nphj_sc", R, S, on_device=True, ctx=table, load=0.5)
        need = table.scratch_bytes()
    assert need < radix
    with hj.Context(0) as ctx, Leave(cuda, (need + radix) // 2):
        walls = []
        for _ in range(6):
            t0 = time.perf_counter()
            r = run("nphj_sc", R, S, on_device=True, ctx=ctx)
            walls.append(time.perf_counter() - t0 - r.total)
            assert (r.matched_cnt, r.checksum) == (want.matched_cnt, want.checksum)
            assert ctx.scratch_bytes() < radix
        assert min(walls[2:]) < 200e-6, walls


def dup_relations(cuda, nR, nS, dup, seed, stride=1):
    """dup build tuples a key; want(first) = (matches, checksum) where every match, or the first, counts."""
    g = cuda.Generator(device="cuda")
    g.manual_seed(seed)
    n = nR // dup
    R, S = (cuda.empty((m, 2), dtype=cuda.int64, device="cuda") for m in (nR, nS))
    k = cuda.randperm(nR, generator=g, device="cuda") % n
    s = cuda.randint(0, n + n // 4, (nS,), generator=g, device="cuda")
    R[:, 0], S[:, 0] = (k + 1) * stride, (s + 1) * stride
    R[:, 1], S[:, 1] = cuda.randperm(nR, generator=g, device="cuda"), cuda.arange(nS, device="cuda")

    def want(first):
        if first:
            at = cuda.full((2 * n,), nR, device="cuda").scatter_reduce_(0, k, cuda.arange(nR, device="cuda"), "amin")[s]
            hit = at < nR
            return int(hit.sum()), int((R[:, 1][at[hit]] + S[:, 1][hit]).sum())
        cnt = cuda.bincount(k, minlength=2 * n)[s]
        sums = cuda.zeros(2 * n, dtype=cuda.int64, device="cuda").index_add_(0, k, R[:, 1])[s]
        return int(cnt.sum()), int((sums + cnt * S[:, 1]).sum()) % 2**64

    return R, S, want


ALGOS = ("nphj_sc", "nphj_lp", "phj_radix_bc", "phj_radix_lp")


@pytest.mark.parametrize("tune", [False, True])
@pytest.mark.parametrize("budget", [1e12, 0.0])
def test_batch_table_waves(hj, cuda, tune, budget):
    """A batch whose one-pass scratch (1.1 GB here) cannot be had runs waves of global tables, and lanes for joins that
    the tuner sends there."""
    R, S, want = dup_relations(cuda, 20_000, 1 << 26, 2, 8)
    small = [dup_relations(cuda, n, 3 * n, d, n) for n, d in ((500, 1), (9_000, 3), (70_000, 1))]
    jobs = [(a, R, S) for a in ALGOS[:2]] + [(a, r, s) for a in ALGOS for r, s, _ in small]
    expect = [want(a.endswith("lp")) for a in ALGOS[:2]] + [w(a.endswith("lp")) for a in ALGOS for _, _, w in small]
    with hj.Context(0) as ctx:
        if budget:  # with no budget for tables every join is a lane's, and needs its scratch
            hj.tuner_set(ctx, nphj_max_table_bytes=budget)
        with Leave(cuda, 700 << 20):
            free = cuda.cuda.mem_get_info()[0]
            with hj.Batch(ctx, jobs, tune=tune) as b:
                assert free - cuda.cuda.mem_get_info()[0] < 500 << 20
                for _ in range(2):
                    assert [(r.status, r.matched_cnt, r.checksum) for r in b.run()[0]] == [(0, *w) for w in expect]


@pytest.mark.parametrize("budget", [1e12, 64e6])
@pytest.mark.parametrize("stride", [1, 4])
def test_batch_lanes(hj, cuda, budget, stride):
    """Joins beyond a wave's 12.58 M build tuples run pipelines of their own beside the waves, whatever the tuner says of
    them; with keys that share low bits too."""
    nR, nS = 12_600_000, 13_000_001
    big = [dup_relations(cuda, nR, nS, d, d, stride) for d in (1, 2)]
    few = dup_relations(cuda, 30_000, 90_000, 2, 3, stride)
    jobs = [(a, big[i % 2][0], big[i % 2][1]) for i, a in enumerate(ALGOS + ALGOS)][1:6] + [(a, *few[:2]) for a in ALGOS]
    expect = [big[i % 2][2](a.endswith("lp")) for i, a in enumerate(ALGOS + ALGOS)][1:6] + [few[2](a.endswith("lp")) for a in ALGOS]
    with hj.Context(0) as ctx:
        hj.tuner_set(ctx, nphj_max_table_bytes=budget)
        with hj.Batch(ctx, jobs) as b:
            stats = [b.run() for _ in range(3)]
    for res, _ in stats:
        assert [(r.status, r.matched_cnt, r.checksum) for r in res] == [(0, *w) for w in expect]
    assert min(st.seconds for _, st in stats) < 0.05
