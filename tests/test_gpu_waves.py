"""Waves without global tables (batches and bursts at the server): joins around the limit of the one-kernel
joins (8192 build tuples), of both semantics and layouts, hot build keys whose partitions do not fit shared
memory, joins with an empty side; against the oracle. A pool too small for a wave's scratch is served by
table waves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ALGOS = ["phj_radix_bc", "phj_radix_lp", "nphj_sc", "nphj_lp"]


def joins(rng):
    out = []
    for i, (nR, nS) in enumerate([(1, 5), (8192, 20_000), (8193, 20_000), (8200, 1), (30_000, 60_001), (100_003, 250_000),
                                  (70_000, 3_000), (0, 10), (10, 0), (8191, 40_000), (25_000, 50_000), (12_288, 12_289)]):
        for algo in ALGOS:
            R = np.empty((nR, 2), dtype=np.uint64)
            S = np.empty((nS, 2), dtype=np.uint64)
            keys = max(2, nR // (4 if i % 2 else 1))
            R[:, 0] = rng.permutation(nR).astype(np.uint64) % np.uint64(keys)
            S[:, 0] = rng.integers(0, keys + keys // 3 + 1, nS, dtype=np.uint64)
            if i in (5, 10) and nS:
                R[: nR // 2, 0] = R[0, 0]  # half of the build tuples on one key
                S[:40, 0] = R[0, 0]
            if i % 3 == 0 and nR:
                R[:, 0] |= np.uint64(1 << 50)
                S[:, 0] |= np.uint64(1 << 50)
                R[::97, 0] = np.uint64(2**64 - 1)
                S[::89, 0] = np.uint64(2**64 - 1)
            R[:, 1] = rng.integers(0, 1 << (40 if i % 4 == 1 else 32), nR, dtype=np.uint64)
            S[:, 1] = rng.integers(0, 1 << 32, nS, dtype=np.uint64)
            out.append((algo, R, S))
    return out


@pytest.mark.parametrize("graph", [True, False])
def test_batch_waves(hj, oracle, cuda, graph):
    host = joins(np.random.default_rng(61))
    dev = [(a, cuda.from_numpy(R.view(np.int64)).cuda(), cuda.from_numpy(S.view(np.int64)).cuda()) for a, R, S in host]
    want = [oracle.join(*j) for j in host]
    with hj.Context(0) as ctx:
        for budget in (64e6, 3e5):  # one wave, many waves on all branches
            hj.tuner_set(ctx, wave_table_bytes=budget)
            with hj.Batch(ctx, dev, graph=graph) as b:
                for _ in range(2):
                    res, _ = b.run()
                    for j, r, w in zip(host, res, want):
                        assert (r.status, r.matched_cnt, r.checksum) == (0, *w), (j[0], j[1].shape, j[2].shape)


@pytest.mark.parametrize("budget", [1e9, 20e6])
def test_server_bursts(hj, oracle, cuda, budget):
    host = joins(np.random.default_rng(62))
    dev = [(cuda.from_numpy(R.view(np.int64)).cuda(), cuda.from_numpy(S.view(np.int64)).cuda()) for _, R, S in host]
    with hj.Server(0, slots=4, hbm_budget_bytes=budget) as srv:
        for rep in range(2):
            ids = [srv.submit(a, *(d if (i + rep) % 3 else (R, S)), on_device=bool((i + rep) % 3))
                   for i, ((a, R, S), d) in enumerate(zip(host, dev))]
            got = srv.wait_all(ids)
            for i, (a, R, S) in enumerate(host):
                c = got[ids[i]]
                assert (c.status, c.matched_cnt, c.checksum) == (0, *oracle.join(a, R, S)), (a, R.shape, S.shape)
        assert srv.stats().in_use_bytes == 0


def test_server_full_bursts(hj, oracle, cuda):
    """Enough requests at once that waves hold more mid-size ones than the one-pass form asks for (32)."""
    host = [j for j in joins(np.random.default_rng(63)) if len(j[1]) > 8192]
    dev = [(cuda.from_numpy(R.view(np.int64)).cuda(), cuda.from_numpy(S.view(np.int64)).cuda()) for _, R, S in host]
    want = [oracle.join(*j) for j in host]
    with hj.Server(0, slots=4, hbm_budget_bytes=2e9) as srv:
        ids = [srv.submit(host[i][0], *dev[i], on_device=True) for _ in range(12) for i in range(len(host))]
        got = srv.wait_all(ids)
        for n, rid in enumerate(ids):
            c = got[rid]
            assert (c.status, c.matched_cnt, c.checksum) == (0, *want[n % len(host)]), host[n % len(host)][0]
