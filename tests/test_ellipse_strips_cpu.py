"""The forward's block masks take E's y-extent per strip of pixel columns
(band_extent with x and y exchanged).  A dropped 8x4 block may hold no pixel
whose f32 s passes the pre-filter, at the block positions of a 16x16 tile,
exact and with every square root and quotient moved adversarially."""
import numpy as np
import pytest

from test_ellipse_cull_cpu import band_extent, f, kernel_s, random_splats


def strip_dropped(a, b, c, mx, my, smax, x0, y0, bw, bh, rel, vr_sign):
    cond = (a > 0) & (c > 0) & (b * b <= f(0.98) * (a * c)) & (smax > 0)
    with np.errstate(invalid="ignore", divide="ignore"):
        cx, cy = f(x0) + f(0.5), f(y0) + f(0.5)
        meets, ul, ur = band_extent(c, b, a, my, mx, smax, cx - mx, (cx + f(bw - 1)) - mx, rel, vr_sign)
        kept = meets & (my + ur >= cy) & (my + ul <= cy + f(bh - 1))
    return cond & ~kept


@pytest.mark.parametrize("rel,vr_sign", [(0.0, 1.0), (2e-6, 1.0), (2e-6, -1.0)])
def test_dropped_blocks_hold_no_pixel_within_smax(rel, vr_sign):
    rng = np.random.default_rng(51)
    for x0, y0 in ((0, 0), (8, 12), (1000, 504), (3832, 2156)):
        a, b, c, mx, my, smax = random_splats(rng, 40000, x0, y0)
        live = smax > 0
        drop = strip_dropped(a, b, c, mx, my, smax, x0, y0, 8, 4, rel, vr_sign) & live
        reach = np.zeros_like(drop)
        for yy in range(4):
            for xx in range(8):
                s = kernel_s(a, b, c, mx, my, f(x0 + xx) + f(0.5), f(y0 + yy) + f(0.5))
                reach |= (s >= 0) & (s <= smax)
        assert not (drop & reach).any()
        assert drop.sum() >= 0.95 * (live & ~reach).sum()
