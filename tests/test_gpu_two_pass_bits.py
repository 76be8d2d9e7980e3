"""Two-pass radix joins whose radix bits are lowered to what the build relation needs (build relations above
2^24 tuples, fewer than 14 bits), against the closed form and the pipelines with the bits asked for; and
the word pass 1 of segment mode that stops at the first value too wide for words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp"])
@pytest.mark.parametrize("nR,nS", [((1 << 24) + 1, 1 << 24), (1 << 25, (1 << 25) - 1), ((1 << 25) + 5, 1 << 25)])
def test_fewer_bits(hj, cuda, algo, nR, nS):
    R = cuda.empty((nR, 2), dtype=cuda.int64, device="cuda")
    S = cuda.empty((nS, 2), dtype=cuda.int64, device="cuda")
    hj.gen_fast_device(nR, nS, R.data_ptr(), S.data_ptr(), seed=nR)
    cuda.cuda.synchronize()
    want = hj.join(algo, R, S, on_device=True, flags=hj.HJ_F_EXACT)
    assert want.matched_cnt == nS
    got = hj.join(algo, R, S, on_device=True)
    seg = hj.join(algo, R, S, on_device=True, flags=hj.HJ_F_SEGMENTS)
    for r in (got, seg):
        assert (r.matched_cnt, r.checksum, r.large_partitions) == (want.matched_cnt, want.checksum, 0)
        assert r.flags & hj.HJ_RES_COMPACT_PARTITIONS


@pytest.mark.parametrize("where", ["first_tile", "last_build_tuple", "last_probe_row_id"])
@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp"])
def test_word_pass_that_stops(hj, oracle, cuda, algo, where):
    """One wide value among narrow ones, seen by one pass-1 CTA early or late: the others stop at their next
    claim and the tuple pass runs over everything."""
    rng = np.random.default_rng(17)
    nR, nS = 700_001, 1_900_003
    R = np.empty((nR, 2), dtype=np.uint64)
    S = np.empty((nS, 2), dtype=np.uint64)
    R[:, 0] = rng.permutation(nR).astype(np.uint64) + np.uint64(1)
    R[300_000:300_500, 0] = R[:500, 0]
    S[:, 0] = R[rng.integers(0, nR, nS), 0]
    R[:, 1] = rng.integers(0, 1 << 32, nR, dtype=np.uint64)
    S[:, 1] = rng.integers(0, 1 << 32, nS, dtype=np.uint64)
    if where == "first_tile":
        R[3, 0] = np.uint64(1 << 60)
    elif where == "last_build_tuple":
        R[-1, 0] = np.uint64((1 << 38) + 5)
    else:
        S[-1, 1] = np.uint64(1 << 32)
    S[::1000, 0] = np.uint64(1 << 60)
    to = lambda a: cuda.from_numpy(a.view(np.int64)).cuda()  # noqa: E731
    want = oracle.join(algo, R, S)
    for flags in (hj.HJ_F_SEGMENTS, hj.HJ_F_SEGMENTS | hj.HJ_F_ORDERED):
        r = hj.join(algo, to(R), to(S), on_device=True, flags=flags)
        assert (r.matched_cnt, r.checksum) == want, flags
        assert not r.flags & hj.HJ_RES_WORD_PASS1
