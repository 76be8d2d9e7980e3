"""Non-partitioned joins that run a radix pipeline (build relations of 2^21 tuples and more, on both sides of
each limit of the rule) against the oracle and against the table (an explicit load factor): both
semantics, duplicates, keys 0 and 2^64-1 (which first-match non-partitioned joins do match), wide keys;
the result carries no radix-join fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("nR,nS", [((1 << 21) - 1, 300_000), (1 << 21, 300_000), ((1 << 21) + 3, 10 * (1 << 21)),
                                   (5_000_001, 1_000_003), (1 << 21, (1 << 22) + 1), (12_000_001, 25_000_000)])
def test_radix_equals_table_and_oracle(hj, oracle, cuda, nR, nS, wide):
    rng = np.random.default_rng(nR)
    R = np.empty((nR, 2), dtype=np.uint64)
    R[:, 0] = rng.permutation(nR).astype(np.uint64)
    R[nR // 2: nR // 2 + 1000, 0] = R[:1000, 0]          # duplicates far apart
    R[5::100_003, 0] = 0
    R[7::200_003, 0] = np.uint64(2**64 - 1) if wide else np.uint64(1 << 33)
    S = np.empty((nS, 2), dtype=np.uint64)
    S[:, 0] = R[rng.integers(0, nR, nS), 0]
    S[::9, 0] += np.uint64(nR)
    S[::10_007, 0] = 0
    S[1::20_011, 0] = np.uint64(2**64 - 1)
    R[:, 1] = rng.integers(0, 1 << 32, nR, dtype=np.uint64)
    S[:, 1] = rng.integers(0, 1 << 32, nS, dtype=np.uint64)
    dR, dS = dev(cuda, R), dev(cuda, S)
    for algo in ("nphj_sc", "nphj_lp"):
        want = oracle.join(algo, R, S)
        for load in (0.0, 0.5):
            r = hj.join(algo, dR, dS, on_device=True, load=load, flags=hj.HJ_F_PHASE_TIMES)
            assert (r.matched_cnt, r.checksum) == want, (algo, load)
            assert (r.flags, r.physical_passes, r.large_partitions) == (0, 0, 0)
            assert r.phase[0] > 0 and r.phase[4] > 0


def test_two_pass_size(hj, cuda):
    """Beyond the one-pass pipeline (2^25 build tuples): closed form, both semantics."""
    nR, nS = 1 << 25, 1 << 26
    R = cuda.empty((nR, 2), dtype=cuda.int64, device="cuda")
    S = cuda.empty((nS, 2), dtype=cuda.int64, device="cuda")
    hj.gen_fast_device(nR, nS, R.data_ptr(), S.data_ptr(), seed=4)
    cuda.cuda.synchronize()
    for algo in ("nphj_sc", "nphj_lp"):
        r = hj.join(algo, R, S, on_device=True)
        assert (r.matched_cnt, r.checksum) == hj.pkfk_closed_form(nR, nS), algo
        assert (r.flags, r.physical_passes, r.large_partitions) == (0, 0, 0)
