"""The non-partitioned joins' own tables at sizes where the default runs a radix pipeline: an explicit load factor asks for
the table, so its compact slots, sliced build and fallbacks run on the inputs that were made for them."""
import pytest
import test_gpu_nphj_compact as compact

pytestmark = pytest.mark.gpu


@pytest.fixture
def by_table(monkeypatch):
    def check(hj, oracle, cuda, R, S, algo="nphj_sc"):
        want = oracle.join(algo, R, S)
        with hj.Context(0) as ctx:
            r = hj.join(algo, compact.dev(cuda, R), compact.dev(cuda, S), on_device=True, load=0.4, ctx=ctx)
            assert (r.matched_cnt, r.checksum) == want, (algo, len(R), len(S))
            # no radix scratch of 16 bytes per tuple: the arena holds the table
            assert ctx.scratch_bytes() < 64 * len(R) + (1 << 22)
        h = hj.join(algo, R, S, load=0.4)
        assert (h.matched_cnt, h.checksum) == want

    monkeypatch.setattr(compact, "check", check)


def test_limits(by_table, hj, oracle, cuda):
    compact.test_compact_slots_limits(hj, oracle, cuda)


def test_duplicates(by_table, hj, oracle, cuda):
    compact.test_compact_slots_duplicates(hj, oracle, cuda)


def test_sliced_build_and_its_fallback(by_table, hj, oracle, cuda):
    compact.test_sliced_build_and_its_fallback(hj, oracle, cuda)


@pytest.mark.parametrize("algo", ["nphj_sc", "nphj_lp"])
def test_pkfk_sizes(hj, cuda, algo):
    for nR, nS in ((1 << 22, 1 << 23), ((1 << 21) + 5, 3 * ((1 << 21) + 5)), ((1 << 21) - 5, (1 << 21) - 5)):
        R, S = (cuda.empty((n, 2), dtype=cuda.int64, device="cuda") for n in (nR, nS))
        hj.gen_fast_device(nR, nS, R.data_ptr(), S.data_ptr(), seed=31)
        cuda.cuda.synchronize()
        r = hj.join(algo, R, S, on_device=True, load=0.4)
        assert (r.matched_cnt, r.checksum) == hj.pkfk_closed_form(nR, nS)
