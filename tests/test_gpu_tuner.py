"""The tuner measures and changes only what its decisions still decide."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tuning_a_batch_of_one_pass_waves_leaves_the_tuner(hj, oracle, cuda):
    """The table budget changes nothing about joins that one-pass waves take, so timing noise must not move it."""
    rng = np.random.default_rng(1)
    jobs, want = [], []
    for i, nR in enumerate((500, 9_000, 40_000, 150_000, 30_000, 70_001)):
        R, S = (np.empty((n, 2), dtype=np.uint64) for n in (nR, 3 * nR))
        R[:, 0], S[:, 0] = rng.permutation(nR) + 1, rng.integers(1, nR + 50, 3 * nR)
        R[:, 1], S[:, 1] = np.arange(nR), np.arange(3 * nR)
        algo = ("phj_radix_bc", "nphj_lp")[i % 2]
        want.append(oracle.join(algo, R, S))
        jobs.append((algo, *(cuda.from_numpy(a.view(np.int64)).cuda() for a in (R, S))))
    with hj.Context(0) as ctx:
        hj.tuner_set(ctx, nphj_max_table_bytes=1.5e6)
        before = bytes(hj.tuner_get(ctx))
        for _ in range(4):
            with hj.Batch(ctx, jobs, tune=True) as b:
                assert [(r.matched_cnt, r.checksum) for r in b.run()[0]] == want
            assert bytes(hj.tuner_get(ctx)) == before


def test_calibration_times_the_decided_pipeline(hj, cuda):
    """The partitioned side of the cost model is the pipeline that a decision for it runs (the exact-offset one with the
    decision's bits), not the one-pass pipeline that a join alone would take."""
    with hj.Context(0) as ctx:
        report = {n: t for n, _, t in hj.tuner_calibrate(ctx)}
    L = hj._bind_batch()
    with hj.Context(0) as ctx:
        hj.tuner_set(ctx, nphj_max_table_bytes=0.0)
        for nR in (1 << 16, 1 << 20, 1 << 22):
            impl, bits, passes = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
            L.hj_tuner_decide(ctx.handle, nR, 8 * nR, ctypes.byref(impl), ctypes.byref(bits), ctypes.byref(passes))
            R, S = (cuda.empty((n, 2), dtype=cuda.int64, device="cuda") for n in (nR, 8 * nR))
            hj.gen_fast_device(nR, 8 * nR, R.data_ptr(), S.data_ptr(), seed=4)
            cuda.cuda.synchronize()
            t = min(hj.join("phj_radix_bc", R, S, on_device=True, ctx=ctx, bits=bits.value, passes=passes.value,
                            flags=hj.HJ_F_EXACT).total for _ in range(4))
            assert 0.67 * t < report[nR] < 1.5 * t, (nR, t, report[nR])
