"""One-pass joins whose CTAs' ranges end on, before and after a tile of the scatter (10240 8-byte words or 5120 16-byte
tuples of a relation per CTA and tile, ranges rounded up to 8 tuples), on both sides of the join."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp"])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("per", [-8, 0, 1, 8])
@pytest.mark.parametrize("side", ["build", "probe"])
def test_ranges_around_a_tile(hj, oracle, cuda, algo, wide, per, side):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    tile = 5120 if wide or (algo.endswith("lp") and side == "build") else 10240  # first-match builds: 16 bytes
    n = sms * tile + per * sms
    nR, nS = (n, 700_003) if side == "build" else (100_003, n)
    rng = np.random.default_rng(n)
    R, S = np.empty((nR, 2), dtype=np.uint64), np.empty((nS, 2), dtype=np.uint64)
    R[:, 0] = rng.permutation(nR).astype(np.uint64) // np.uint64(2)
    S[:, 0] = rng.integers(0, nR // 2 + nR // 8, nS, dtype=np.uint64)
    if wide:
        R[:, 0] |= np.uint64(1 << 62)
        S[:, 0] |= np.uint64(1 << 62)
    R[:, 1], S[:, 1] = rng.integers(0, 1 << 32, nR, dtype=np.uint64), rng.integers(0, 1 << 32, nS, dtype=np.uint64)
    r = hj.join(algo, *(cuda.from_numpy(a.view(np.int64)).cuda() for a in (R, S)), on_device=True)
    assert (r.matched_cnt, r.checksum) == oracle.join(algo, R, S)
    assert r.physical_passes == 1
