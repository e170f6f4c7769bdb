"""The device-pointer sorts on arrays that start at any element of larger ones:
the element's own alignment is all that they may assume."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("fn", ["sky_sort_pairs", "sky_sort_pairs_noalloc"])
@pytest.mark.parametrize("n", [1, 4, 7, 129, 4099, 100_003])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_any_first_element(sky, fn, n, offset):
    rng = np.random.default_rng(7 * n + offset)
    keys = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    vals = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    order = np.argsort(keys, kind="stable")
    for with_vals in (True, False):
        # the four arrays at four different offsets, each 3 elements short of its buffer's end
        bufs = [torch.full((n + 6,), -1, dtype=torch.int32, device="cuda") for _ in range(4)]
        first = [(offset + k) % 4 for k in range(4)]
        kin, vin, kout, vout = (b[o:o + n] for b, o in zip(bufs, first))
        kin.copy_(torch.from_numpy(keys.view(np.int32)))
        vin.copy_(torch.from_numpy(vals.view(np.int32)))
        p = [C.c_void_p(t.data_ptr()) for t in (kin, vin, kout, vout)]
        assert p[0].value % 16 == 4 * first[0]
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        sky._lib.check(getattr(sky.lib(), fn)(p[0], p[1] if with_vals else None, p[2], p[3], n, 32, st))
        torch.cuda.synchronize()
        want = [keys, vals, keys[order], vals[order] if with_vals else order.astype(np.uint32)]
        for b, o, w in zip(bufs, first, want):
            got = b.cpu().numpy().view(np.uint32)
            assert np.array_equal(got[o:o + n], w)
            assert (got[:o] == 0xFFFFFFFF).all() and (got[o + n:] == 0xFFFFFFFF).all()
