"""hj_shard_route at the edges of its tiles (2048 tuples), blocks (four per SM) and owner counts, against the
oracle's routing: the same bytes, in the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shards", [1, 2, 3, 8, 17, 32])
@pytest.mark.parametrize("n", [1, 31, 2047, 2049, 70_001, 4 * 148 * 2048 + 5, 3_000_000])
def test_route_bytes(hj, oracle, cuda, n, shards):
    rng = np.random.default_rng(n + shards)
    T = rng.integers(0, 1 << 64, (n, 2), dtype=np.uint64)
    if n > 100:
        T[n // 3: n // 2, 0] = T[0, 0]  # one owner takes whole tiles
    routed, counts = hj.shard_route(cuda.from_numpy(T.view(np.int64)).cuda(), shards)
    want, want_counts = oracle.shard_route(T, shards)
    assert np.array_equal(counts.cpu().numpy(), np.asarray(want_counts, dtype=np.int64))
    assert np.array_equal(routed.cpu().numpy().view(np.uint64), want)
