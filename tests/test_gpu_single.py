"""One-pass radix pipeline (the default for build relations of up to 2^24 tuples) against the oracle and
against the two-pass exact-offset pipeline: sizes around the CTA, tile and chunk limits, both element
layouts, both match semantics, duplicates and key 0, few and many radix bits, skewed probes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


def relations(rng, nR, nS, layout, dup):
    """layout: word = keys and row ids that fit compact words, key / rid = one of them does not."""
    kmax = max(2, nR // dup)
    R = np.empty((nR, 2), dtype=np.uint64)
    S = np.empty((nS, 2), dtype=np.uint64)
    R[:, 0] = rng.permutation(nR).astype(np.uint64) % np.uint64(kmax)  # key 0 included
    S[:, 0] = rng.integers(0, kmax + kmax // 4, nS, dtype=np.uint64)
    S[: nS // 8, 0] = R[0, 0]  # a hot probe key
    if layout == "key":
        R[:, 0] |= (R[:, 0] & np.uint64(7)) << np.uint64(58)
        S[:, 0] |= (S[:, 0] & np.uint64(7)) << np.uint64(58)
    rid = 40 if layout == "rid" else 32
    R[:, 1] = rng.integers(0, 1 << rid, nR, dtype=np.uint64)
    S[:, 1] = rng.integers(0, 1 << rid, nS, dtype=np.uint64)
    return R, S


# nR x nS: one tuple; around the 8-tuple range rounding; one CTA; a chunk of the input ring more or less; more
# than one tile of words per CTA (148 x 12288 in all); build partitions above 6144 x 2^8 tuples
SIZES = [(1, 1), (7, 9), (1023, 3072), (9000, 1025), (30_001, 120_007), (1_600_003, 2_500_001)]


@pytest.mark.parametrize("layout", ["word", "key", "rid"])
@pytest.mark.parametrize("nR,nS", SIZES)
def test_one_pass_equals_oracle_and_two_pass(hj, oracle, cuda, nR, nS, layout):
    rng = np.random.default_rng(nR + nS)
    for dup in (1, 4):
        R, S = relations(rng, nR, nS, layout, dup)
        dR, dS = dev(cuda, R), dev(cuda, S)
        for algo in ("phj_radix_bc", "phj_radix_lp"):
            want = oracle.join(algo, R, S)
            for bits in (14, 3) if nR < 100_000 else (14,):
                with hj.Context(0) as ctx:
                    one = hj.join(algo, dR, dS, on_device=True, bits=bits, ctx=ctx)
                    two = hj.join(algo, dR, dS, on_device=True, bits=bits, ctx=ctx, flags=hj.HJ_F_EXACT)
                assert (one.matched_cnt, one.checksum) == want, (algo, dup, bits)
                assert (two.matched_cnt, two.checksum) == want, (algo, dup, bits)
                assert one.flags & hj.HJ_RES_COMPACT_PARTITIONS == two.flags & hj.HJ_RES_COMPACT_PARTITIONS
                assert one.flags & hj.HJ_RES_ORDERED_PASSES == two.flags & hj.HJ_RES_ORDERED_PASSES


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp"])
@pytest.mark.parametrize("n0", [8192, 8193, 9216, 9217, 10240, 10241])
def test_partitions_at_the_shared_memory_limits(hj, oracle, cuda, algo, n0):
    """One build partition of n0 tuples (duplicates among them) next to small ones: the limits of the
    shared-memory joins."""
    rng = np.random.default_rng(n0)
    R, S = relations(rng, 20_000, 50_000, "word", 1)
    p = np.empty((n0, 2), dtype=np.uint64)
    p[:, 0] = (rng.integers(0, 6000, n0, dtype=np.uint64) << np.uint64(14)) | np.uint64(5)
    p[:, 1] = rng.integers(0, 1 << 32, n0, dtype=np.uint64)
    R = R[(R[:, 0] & np.uint64(0xFF)) != np.uint64(5)]
    R = np.concatenate([R[:9000], p, R[9000:]])
    S = np.concatenate([S, p[:3000], p[:3000]])
    r = hj.join(algo, dev(cuda, R), dev(cuda, S), on_device=True)
    assert (r.matched_cnt, r.checksum) == oracle.join(algo, R, S)
    want_large = n0 > (10240 if algo == "phj_radix_bc" else 9216)
    assert (r.large_partitions > 0) == want_large


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp"])
def test_materialised_pairs(hj, oracle, cuda, algo):
    rng = np.random.default_rng(3)
    R, S = relations(rng, 30_000, 70_000, "word", 4)
    S[: S.shape[0] // 8, 0] = np.arange(S.shape[0] // 8, dtype=np.uint64)
    R[:, 1] = np.arange(1, R.shape[0] + 1, dtype=np.uint64)
    S[:, 1] = np.arange(1, S.shape[0] + 1, dtype=np.uint64)
    want = oracle.join_pairs(algo, R, S)
    out = cuda.zeros((want.shape[0], 2), dtype=cuda.int64, device="cuda")
    r = hj.join_mat(algo, dev(cuda, R), dev(cuda, S), pairs=out, on_device=True)
    got = out.cpu().numpy().view(np.uint64)
    assert r.matched_cnt == want.shape[0]
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want)


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp", "nphj_sc", "nphj_lp"])
@pytest.mark.parametrize("kind", ["unique", "dups", "hot", "wide_key", "wide_rid"])
def test_materialised_words(hj, oracle, cuda, algo, kind):
    """Pairs written from compact words and from tuples, with at most one match per probe and with many, a hot
    build key in a large partition, and a row id that is not a position (refused with HJ_E_ROWID)."""
    rng = np.random.default_rng(8)
    nR, nS = 50_001, 120_007
    R, S = relations(rng, nR, nS, "key" if kind == "wide_key" else "word", 3 if kind == "dups" else 1)
    S[: nS // 8, 0] = R[rng.integers(0, nR, nS // 8), 0]
    if kind == "hot":
        R[: 12_000, 0] = R[0, 0]
        S[(S[:, 0] == R[0, 0]), 0] += np.uint64(1)
        S[:3, 0] = R[0, 0]
    R[:, 1] = np.arange(1, nR + 1, dtype=np.uint64)
    S[:, 1] = np.arange(1, nS + 1, dtype=np.uint64)
    if kind == "wide_rid":
        R[0, 1] = np.uint64(1 << 40)
        S[0, 0] = R[0, 0]
        r = hj.join_mat(algo, dev(cuda, R), dev(cuda, S), on_device=True, check=False)
        assert r.status == hj.HJ_E_ROWID or (r.status == 0 and (R[0, 0] == 0 or R[0, 0] == 2**64 - 1))
        return
    want = oracle.join_pairs(algo, R, S)
    out = cuda.zeros((want.shape[0], 2), dtype=cuda.int64, device="cuda")
    r = hj.join_mat(algo, dev(cuda, R), dev(cuda, S), pairs=out, on_device=True)
    got = out.cpu().numpy().view(np.uint64)
    assert r.matched_cnt == want.shape[0]
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want)
    assert (r.matched_cnt, r.checksum) == oracle.join(algo, R, S)


@pytest.mark.parametrize("algo", ["phj_radix_bc", "phj_radix_lp", "nphj_sc", "nphj_lp"])
def test_retrieve_columns(hj, cuda, algo):
    """Relations beyond 64 MB gather from row-id columns: permuted row ids (in range, so retrieved), and one
    out of range."""
    nR, nS = (1 << 21) + 5, (1 << 22) + 3
    g = cuda.Generator(device="cuda")
    g.manual_seed(2)
    R = cuda.empty((nR, 2), dtype=cuda.int64, device="cuda")
    S = cuda.empty((nS, 2), dtype=cuda.int64, device="cuda")
    R[:, 0] = cuda.randperm(nR, generator=g, device="cuda") + 1
    S[:, 0] = cuda.randint(1, nR + nR // 4, (nS,), generator=g, device="cuda")
    R[:, 1] = cuda.randperm(nR, generator=g, device="cuda") + 1
    S[:, 1] = cuda.randperm(nS, generator=g, device="cuda") + 1
    rid = cuda.zeros(nR + nR // 4 + 1, dtype=cuda.int64, device="cuda")
    rid[R[:, 0]] = R[:, 1]
    hit = rid[S[:, 0]] > 0
    r_id, s_id = rid[S[:, 0]][hit], S[:, 1][hit]
    want = (int(hit.sum()), int((R[:, 1][r_id - 1] + S[:, 1][s_id - 1]).sum()))
    r = hj.join_mat(algo, R, S, on_device=True)
    assert (r.matched_cnt, r.checksum) == want
    S[5, 0], S[5, 1] = R[0, 0], 1 << 33
    r = hj.join_mat(algo, R, S, on_device=True, check=False)
    assert r.status == hj.HJ_E_ROWID
