"""The work that users of the join library have it do, as cases for a benchmark harness.

A case is a dict of plain values. `listed()` names the fixed ones, `draw(rng)` makes more of the same
ranges, `prepare(case, seed)` builds what a program has in hand before the call (relations, and a plan or
a server where such a program keeps one), `run(state)` is one pass through the public entry points,
`work(case)` the bytes that a pass cannot do without, and `exact(case, seed)` the answer computed with
plain torch from the definition of a join.

Kinds of work ("kind"):
  join   hj.join on device-resident relations, as bench.py's headline, C1 and skew workloads
  host   hj.join on numpy relations in host memory (the call's default)
  mat    hj.join_mat, the ptr_* joins: pairs, then the retrieve phase (bench.py --mode mat)
  batch  hj.Batch: independent joins of uneven sizes, planned once (bench.py --mode batch)
  serve  hj.Server: a burst of small requests (bench.py --mode serve)
  route  hj.shard_route: tuples grouped by owner rank before a sharded join's exchange
"""
from __future__ import annotations

import importlib.util
import pathlib
import random
import sys

import numpy as np
import torch


def _load():
    if "hashjoin_scm_b200" not in sys.modules:
        path = pathlib.Path("hashjoin-scm_b200").resolve() / "__init__.py"
        spec = importlib.util.spec_from_file_location("hashjoin_scm_b200", path)
        mod = importlib.util.module_from_spec(spec)
        sys.modules["hashjoin_scm_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["hashjoin_scm_b200"]


hj = _load()

ALGOS = ("phj_radix_bc", "phj_radix_lp", "nphj_sc", "nphj_lp", "phj_radix_hr", "phj_radix_sc", "phj_radix_hro")


def _join(kind, algo, nR, nS, keys="dense", dup=1, theta=0.0, hit=1.0):
    """keys: dense = 1..nR in random order (the reference's generator), sparse = 63-bit values; dup:
    build tuples per key; theta: Zipf exponent of the probe keys (0 = uniform); hit: share of probe
    tuples whose key is a build key."""
    return {"kind": kind, "algo": algo, "nR": nR, "nS": nS, "keys": keys, "dup": dup, "theta": theta, "hit": hit}


def _many(kind, jobs, min_log, max_log, sizes):
    """`jobs` joins, |R| log-uniform in [2^min_log, 2^max_log], |S| = 1..16 times that; sizes: seed of
    the sizes and algorithms."""
    return {"kind": kind, "jobs": jobs, "min_log": min_log, "max_log": max_log, "sizes": sizes}


def listed():
    return [
        # The smallest calls (a dimension table of a thousand rows): launches and latency.
        dict(_join("join", "phj_radix_bc", 1000, 4000), name="bc_1e3x4e3"),
        # Ordinary joins of millions of tuples with the default parameters (14 bits, two passes).
        dict(_join("join", "phj_radix_bc", 1 << 20, 1 << 22), name="bc_2e20x2e22"),
        # The first benchmark configuration: non-partitioned join, table about the size of L2.
        dict(_join("join", "nphj_sc", 1 << 22, 1 << 23), name="sc_2e22x2e23"),
        # Keys that are 63-bit ids, odd sizes, half of the probe tuples without a match.
        dict(_join("join", "phj_radix_hr", 3000017, 12000041, keys="sparse", hit=0.5), name="hr_sparse_3e6x12e6"),
        # First match among four duplicates of every build key, table beyond L2.
        dict(_join("join", "nphj_lp", 1 << 24, 1 << 26, dup=4), name="nlp_dup4_2e24x2e26"),
        # Skewed foreign keys, first match, radix-partitioned.
        dict(_join("join", "phj_radix_lp", 1 << 26, 1 << 28, theta=1.0), name="lp_zipf_2e26x2e28"),
        # The headline configuration and largest call.
        dict(_join("join", "phj_radix_bc", 1 << 27, 1 << 29), name="bc_2e27x2e29"),
        # Relations in pageable host memory: the copy is part of the call.
        dict(_join("host", "phj_radix_bc", 1 << 20, 1 << 22), name="host_bc_2e20x2e22"),
        # Materialising join: row-id pairs and the retrieve phase.
        dict(_join("mat", "phj_radix_bc", 1 << 24, 1 << 26), name="ptr_bc_2e24x2e26"),
        # A planned batch of uneven joins, the sizes of the batch configuration.
        dict(_many("batch", 96, 10, 22, 7), name="batch_96"),
        # A burst of small requests at the join server.
        dict(_many("serve", 64, 10, 18, 11), name="serve_64"),
        # Routing before the exchange of a join sharded over 8 ranks.
        {"kind": "route", "n": 1 << 24, "shards": 8, "name": "route8_2e24"},
    ]


def _log(rng, lo, hi):
    return int(round(2.0 ** rng.uniform(lo, hi)))


def draw(rng: random.Random):
    kind = rng.choice(("join", "join", "join", "join", "join", "join", "mat", "host", "batch", "serve", "route"))
    if kind == "route":
        return {"kind": "route", "n": _log(rng, 12, 26), "shards": rng.randint(2, 32)}
    if kind == "batch":
        return _many("batch", rng.randint(8, 128), 10, rng.choice((16, 18, 20, 22)), rng.randint(1, 1 << 20))
    if kind == "serve":
        return _many("serve", rng.randint(8, 128), 10, rng.choice((14, 16, 18)), rng.randint(1, 1 << 20))
    if kind == "join":
        nR = _log(rng, 8, 26)
        nS = min(1 << 28, int(nR * 2.0 ** rng.uniform(0, 4)) + rng.randint(0, 99))
    else:  # the retrieve phase and the host copy set the cost of these
        nR = _log(rng, 10, 24 if kind == "mat" else 22)
        nS = int(nR * 2.0 ** rng.uniform(0, 2)) + rng.randint(0, 99)
    return _join(kind, rng.choice(ALGOS), nR, nS, keys=rng.choice(("dense", "dense", "sparse")),
                 dup=rng.choice((1, 1, 1, 4)), theta=rng.choice((0.0, 0.0, 0.5, 1.0, 1.5)),
                 hit=rng.choice((1.0, 1.0, 0.5)))


# ------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------
_CHUNK = 1 << 26


def _spread(v):
    """A bijection of the 63-bit integers: distinct dense keys become distinct sparse ones."""
    v = (v * 0x1E3779B97F4A7C15) & 0x7FFFFFFFFFFFFFFF
    v = v ^ (v >> 29)
    return (v * 0x3F58476D1CE4E5B9) & 0x7FFFFFFFFFFFFFFF


def _relations(nR, nS, keys, dup, theta, hit, gen):
    """R and S as (n, 2) int64 CUDA tensors {key, row id}; row ids are 1-based positions."""
    dev = "cuda"
    nkeys = max(1, nR // dup)
    R = torch.empty((nR, 2), dtype=torch.int64, device=dev)
    S = torch.empty((nS, 2), dtype=torch.int64, device=dev)
    torch.remainder(torch.randperm(nR, generator=gen, device=dev), nkeys, out=R[:, 0])
    R[:, 0] += 1
    R[:, 1] = torch.arange(1, nR + 1, device=dev)
    cdf = None
    if theta > 0:
        # In whole numbers: a sum of floats on the GPU may differ from one call to the next.
        w = torch.arange(1, nkeys + 1, dtype=torch.float64, device=dev).pow_(-theta).mul_(2.0 ** 30)
        cdf = torch.cumsum(w.to(torch.int64).clamp_(min=1), 0)
        total = int(cdf[-1])
        alphabet = torch.randperm(nkeys, generator=gen, device=dev)
    for lo in range(0, nS, _CHUNK):
        n = min(_CHUNK, nS - lo)
        if cdf is None:
            k = torch.randint(0, nkeys, (n,), generator=gen, device=dev)
        else:
            u = torch.randint(0, total, (n,), generator=gen, device=dev)
            k = alphabet[torch.searchsorted(cdf, u, right=True)]
        if hit < 1.0:  # the others are keys above every build key
            k += (torch.rand(n, generator=gen, device=dev) >= hit).to(torch.int64) * nkeys
        S[lo:lo + n, 0] = k + 1
        S[lo:lo + n, 1] = torch.arange(lo + 1, lo + n + 1, device=dev)
    if keys == "sparse":
        R[:, 0] = _spread(R[:, 0])
        for lo in range(0, nS, _CHUNK):
            S[lo:lo + _CHUNK, 0] = _spread(S[lo:lo + _CHUNK, 0])
    return R, S


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _inputs(case, seed):
    return _relations(case["nR"], case["nS"], case["keys"], case["dup"], case["theta"], case["hit"], _gen(seed))


def _sizes(case):
    """(algorithm, |R|, |S|) of every join of a batch or burst."""
    rng = random.Random(case["sizes"])
    out = []
    for _ in range(case["jobs"]):
        nR = _log(rng, case["min_log"], case["max_log"])
        out.append((rng.choice(ALGOS[:4]), nR, nR * rng.randint(1, 16)))
    return out


def _jobs(case, seed):
    g = _gen(seed)
    return [(algo, *_relations(nR, nS, "dense", 1, 0.0, 1.0, g)) for algo, nR, nS in _sizes(case)]


class _Held:
    """A plan or server with the context and relations it needs, closed with the state."""

    def __init__(self, what, jobs, ctx=None):
        self.what, self.jobs, self.ctx = what, jobs, ctx

    def __del__(self):
        self.what.close()
        if self.ctx is not None:
            self.ctx.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "route":
        g = _gen(seed)
        T = torch.empty((case["n"], 2), dtype=torch.int64, device="cuda")
        T[:, 0] = torch.randint(1, 1 << 40, (case["n"],), generator=g, device="cuda")
        T[:, 1] = torch.arange(1, case["n"] + 1, device="cuda")
        return {"case": case, "T": T}
    if kind == "batch":
        jobs = _jobs(case, seed)
        torch.cuda.synchronize()
        ctx = hj.Context()
        return {"case": case, "held": _Held(hj.Batch(ctx, jobs), jobs, ctx)}
    if kind == "serve":
        jobs = _jobs(case, seed)
        torch.cuda.synchronize()
        return {"case": case, "held": _Held(hj.Server(hbm_budget_bytes=8e9), jobs)}
    R, S = _inputs(case, seed)
    if kind == "host":
        R, S = R.cpu().numpy().view(np.uint64), S.cpu().numpy().view(np.uint64)
    return {"case": case, "R": R, "S": S}


# ------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------
def _signed(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "route":
        routed, counts = hj.shard_route(state["T"], case["shards"])
        return {"routed": routed, "counts": counts}
    if kind == "batch":
        results, _ = state["held"].what.run()
        return {"matched": np.array([r.matched_cnt for r in results], dtype=np.uint64).view(np.int64),
                "checksum": np.array([r.checksum for r in results], dtype=np.uint64).view(np.int64)}
    if kind == "serve":
        srv = state["held"].what
        ids = [srv.submit(algo, R, S, on_device=True) for algo, R, S in state["held"].jobs]
        done = srv.wait_all(ids)
        return {"matched": np.array([done[i].matched_cnt for i in ids], dtype=np.uint64).view(np.int64),
                "checksum": np.array([done[i].checksum for i in ids], dtype=np.uint64).view(np.int64)}
    if kind == "mat":
        r = hj.join_mat("ptr_" + case["algo"], state["R"], state["S"], on_device=True)
    else:
        r = hj.join(case["algo"], state["R"], state["S"], on_device=kind == "join")
    return {"matched": _signed(r.matched_cnt), "checksum": _signed(r.checksum)}


def work(case):
    if case["kind"] == "route":
        n = 32.0 * case["n"]
    elif case["kind"] in ("batch", "serve"):
        n = sum(16.0 * (nR + nS) + 16.0 for _, nR, nS in _sizes(case))
    else:
        n = 16.0 * (case["nR"] + case["nS"]) + 16.0
        if case["kind"] == "mat":  # the pairs: hits, times the matches of each where all are written
            first = case["algo"] in ("phj_radix_lp", "nphj_lp")
            n += 16.0 * case["nS"] * case["hit"] * (1 if first else case["dup"])
    return {"bytes": n, "flops": 0.0}


# ------------------------------------------------------------------------------------------------
# The answer from the definition
# ------------------------------------------------------------------------------------------------
def _exact_join(algo, R, S):
    keys, order = torch.sort(R[:, 0], stable=True)
    rids = R[:, 1][order]
    total = torch.zeros(len(rids) + 1, dtype=torch.int64, device=R.device)
    torch.cumsum(rids, 0, out=total[1:])
    matched = checksum = 0
    for lo in range(0, S.shape[0], _CHUNK):
        sk, sr = S[lo:lo + _CHUNK, 0].contiguous(), S[lo:lo + _CHUNK, 1]
        a, b = torch.searchsorted(keys, sk), torch.searchsorted(keys, sk, right=True)
        if algo in ("phj_radix_lp", "nphj_lp"):  # the first build tuple in input order
            found = b > a
            m = found.to(torch.int64)
            part = (rids[a.clamp(max=len(rids) - 1)] + sr) * m
        else:
            m = b - a
            part = total[b] - total[a] + m * sr
        matched += int(m.sum())
        checksum += int(part.sum())
    return matched, _signed(checksum & ((1 << 64) - 1))


def _owner(key, shards):
    """mulhi(mix64(key ^ 0x5ca1ab1e5eed0001), shards), mix64 the splitmix64 output mix."""
    z = key.astype(np.uint64) ^ np.uint64(0x5CA1AB1E5EED0001)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z = z ^ (z >> np.uint64(31))
    hi, lo = z >> np.uint64(32), z & np.uint64(0xFFFFFFFF)
    g = np.uint64(shards)
    return ((hi * g + ((lo * g) >> np.uint64(32))) >> np.uint64(32)).astype(np.int64)


def exact(case, seed):
    kind = case["kind"]
    if kind == "route":
        if case["n"] > 1 << 25:
            return None
        T = prepare(case, seed)["T"].cpu().numpy()
        own = _owner(T[:, 0], case["shards"])
        return {"routed": T[np.argsort(own, kind="stable")], "counts": np.bincount(own, minlength=case["shards"])}
    if kind in ("batch", "serve"):
        got = [_exact_join(*job) for job in _jobs(case, seed)]
        return {"matched": np.array([m for m, _ in got], dtype=np.int64),
                "checksum": np.array([c for _, c in got], dtype=np.int64)}
    R, S = _inputs(case, seed)
    m, c = _exact_join(case["algo"], R, S)
    return {"matched": m, "checksum": c}
