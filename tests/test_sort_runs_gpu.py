"""Keys in runs of equal digits are ranked another way than scattered ones, which
a warp decides from the first 32 of its 512 keys: runs of several lengths,
around the ends of warps and tiles, and keys that are of the other kind after
the first 32, against numpy's stable sort."""
import numpy as np
import pytest

from test_sort_gpu import expect, sort_gpu

pytestmark = pytest.mark.gpu


def runs(rng, n, length, mask):
    k = rng.integers(0, 2**32, n // length + 1, dtype=np.uint64).astype(np.uint32) & mask
    return np.repeat(k, length)[:n].copy()


@pytest.mark.parametrize("n", [1, 31, 33, 511, 513, 4095, 4097, 100_003])
@pytest.mark.parametrize("length", [2, 3, 16, 31, 33, 600, 5000])
@pytest.mark.parametrize("bits", [4, 8, 29, 32])
def test_runs(sky, n, length, bits):
    mask = np.uint32(0xFFFFFFFF if bits == 32 else (1 << bits) - 1)
    rng = np.random.default_rng(n * 31 + length + bits)
    keys = runs(rng, n, length, mask)
    vals = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    ko, vo = sort_gpu(sky, keys, vals, bits)
    ke, ve = expect(keys, vals, bits)
    assert np.array_equal(ko, ke) and np.array_equal(vo, ve)


@pytest.mark.parametrize("runs_first", [True, False])
@pytest.mark.parametrize("n", [500, 4100, 70_001])
def test_other_kind_after_the_first_round(sky, runs_first, n):
    rng = np.random.default_rng(n)
    mask = np.uint32(0xFFFFFFFF)
    scattered, in_runs = runs(rng, n, 1, mask), runs(rng, n, 40, mask)
    keys = np.where((np.arange(n) % 512 < 32) == runs_first, in_runs, scattered)
    ko, vo = sort_gpu(sky, keys, None, 32)
    ke, ve = expect(keys, None, 32)
    assert np.array_equal(ko, ke) and np.array_equal(vo, ve)
