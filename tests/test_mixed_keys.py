"""mix_key, the key that joins partition by where its own low bits are not taken as they are: restated from the kernels'
header, with the multipliers read from it. Bijective for every number of radix bits, 0 stays 0, the high bits stay,
and keys with structure spread evenly over the partitions."""
import pathlib
import re

import numpy as np
import pytest

HEADER = pathlib.Path(__file__).resolve().parents[1] / "hashjoin-scm_b200" / "csrc" / "hj_partition.cuh"
LOW, HIGH = (np.uint64(int(x, 16)) for x in
             re.search(r"kMixLow = (0x[0-9a-f]+)u, kMixHigh = (0x[0-9a-f]+)u", HEADER.read_text()).groups())
U32 = np.uint64(0xFFFFFFFF)


def mix(key, bits):
    low, high = (key & U32) >> np.uint64(bits), key >> np.uint64(32)
    with np.errstate(over="ignore"):
        return key ^ (((low * LOW + high * HIGH) & U32) >> np.uint64(32 - bits))


@pytest.mark.parametrize("bits", range(1, 16))
def test_bijective(bits):
    rng = np.random.default_rng(bits)
    k = np.concatenate([rng.integers(0, 2**64, 50_000, dtype=np.uint64), np.arange(1 << 17, dtype=np.uint64),
                        np.uint64(2**64 - 1) - np.arange(1 << 16, dtype=np.uint64)])
    m = mix(k, bits)
    assert np.array_equal(mix(m, bits), k)  # its own inverse: the high bits that decide the change stay
    assert np.array_equal(m >> np.uint64(bits), k >> np.uint64(bits))
    assert mix(np.zeros(1, dtype=np.uint64), bits)[0] == 0
    run = mix(np.arange(5 << bits, 6 << bits, dtype=np.uint64), bits) & np.uint64((1 << bits) - 1)
    assert np.array_equal(np.sort(run), np.arange(1 << bits, dtype=np.uint64))  # a run takes every digit once


@pytest.mark.parametrize("bits,n", [(4, 90_000), (8, 1 << 20), (10, 1 << 22), (11, 6_000_000), (12, 1 << 24)])
@pytest.mark.parametrize("stride", [1, 2, 3, 4, 10, 16, 60, 100, 1000, 1 << 11, 1 << 14, 10**6, 10**7, 1 << 20, 1 << 32, 3 << 32, 1 << 40])
def test_even_partitions(bits, n, stride):
    """The largest partition stays within shared memory's 10240 tuples where the average is 6144 at most."""
    with np.errstate(over="ignore"):
        k = (np.arange(n, dtype=np.uint64) + np.uint64(1)) * np.uint64(stride)
    c = np.bincount((mix(k, bits) & np.uint64((1 << bits) - 1)).astype(np.int64), minlength=1 << bits)
    assert c.max() <= 10240 / 6144 * n / (1 << bits)
