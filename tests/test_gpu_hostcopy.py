"""Joins of host relations in pageable memory (staged by the call's own threads from 4 MB), page-locked memory
and views that start off a page, at sizes around the staging threshold and its pieces: the result of the
device-resident join; a stream of the caller's; materialised pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nR,nS", [(1000, (1 << 18) - 1), (1 << 18, 1 << 18), ((1 << 18) + 1, (1 << 20) + 4097),
                                   (200_003, 3_000_001)])
def test_host_relations(hj, cuda, nR, nS):
    rng = np.random.default_rng(nR)
    base = np.empty((nR + nS + 3, 2), dtype=np.uint64)
    R, S = base[1: 1 + nR], base[2 + nR: 2 + nR + nS]
    R[:, 0] = rng.permutation(nR).astype(np.uint64) + np.uint64(1)
    S[:, 0] = rng.integers(1, nR + nR // 3 + 2, nS, dtype=np.uint64)
    R[:, 1] = np.arange(1, nR + 1, dtype=np.uint64)
    S[:, 1] = np.arange(1, nS + 1, dtype=np.uint64)
    dR, dS = (cuda.from_numpy(a.view(np.int64)).cuda() for a in (R, S))
    side = cuda.cuda.Stream()
    pR, pS = (cuda.from_numpy(a.view(np.int64)).pin_memory().numpy().view(np.uint64) for a in (R, S))
    with hj.Context(0) as ctx:
        for algo in ("phj_radix_bc", "nphj_lp"):
            want = hj.join(algo, dR, dS, on_device=True, ctx=ctx)
            for r in (hj.join(algo, R, S, ctx=ctx), hj.join(algo, R, S, ctx=ctx, stream=side.cuda_stream),
                      hj.join(algo, pR, pS, ctx=ctx), hj.join(algo, pR, pS, ctx=ctx, flags=hj.HJ_F_PINNED_HOST),
                      hj.join_mat(algo, R, S, ctx=ctx)):
                assert (r.matched_cnt, r.checksum) == (want.matched_cnt, want.checksum), algo
        # the buffers of one call are not overwritten by the next before they are read
        S2 = S.copy()
        S2[:, 1] += np.uint64(7)
        a, b = hj.join("phj_radix_bc", R, S, ctx=ctx), hj.join("phj_radix_bc", R, S2, ctx=ctx)
        assert (b.checksum - a.checksum) % 2**64 == 7 * a.matched_cnt % 2**64
