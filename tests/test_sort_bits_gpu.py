"""The digit passes' ranking by ballots over the bits that vary: segments whose
digits differ in no bit, in low, high or all bits, sizes around a warp's
rounds and a tile, and ragged tails.  Stable order: values break ties."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 511, 4095, 4096, 4097, 70001])
@pytest.mark.parametrize("mask,bits", [(0x00000000, 32), (0x0000000F, 16), (0x000000F0, 8), (0x00FF0003, 32),
                                       (0xFFFFFFFF, 32), (0x00001FFF, 13), (0x80000001, 32)])
def test_stable_sort_over_varying_bits(sky, n, mask, bits):
    rng = np.random.default_rng(n)
    keys = (rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32) & np.uint32(mask)) | np.uint32(0x00200000 & ~mask)
    if bits < 32:
        keys &= np.uint32((1 << bits) - 1)
    vals = rng.permutation(n).astype(np.uint32)
    d = [torch.from_numpy(a.view(np.int32)).cuda() for a in (keys, vals)]
    out = [torch.empty_like(t) for t in d]
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    sky._lib.check(sky.lib().sky_sort_pairs(ptr(d[0]), ptr(d[1]), ptr(out[0]), ptr(out[1]), n, bits, None))
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(out[0].cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(out[1].cpu().numpy().view(np.uint32), vals[order])
