"""The forward's walk over pairs of listed splats: odd and even list lengths,
lists past a chunk of 32 and a batch of 256, a pixel that ends at the first or
the second splat of a pair, every tile size and batch depth, and infinite
colours.  Images, alpha and last contributors are the oracle's bit for bit."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


def one_view(sky, orc, P, w, h, ts, fb):
    cam = scenes.camera_fov((0.0, 0.0, -3.0), w, h)
    with sky.GaussianRenderer(sh_degree=0, tile_size=ts, fwd_batch=fb) as r:
        r.load_points(P)
        r.setTrainingCameras([cam])
        rgba, alpha = r.render([0])
        last = r.read_buffer("last_ids")
    s = orc.settings(tile_size=ts)
    pr = orc.project(P, cam, s, 0)
    fw = orc.forward(pr, orc.tiles(pr, cam, s), cam, s)
    return rgba, alpha, last, fw


@pytest.mark.parametrize("ts,fb", [(8, 0), (16, 0), (16, 64), (16, 128), (32, 0), (32, 64)])
@pytest.mark.parametrize("n,opaque", [(1, False), (2, True), (33, False), (65, True), (700, False), (4001, True)])
def test_forward_matches_oracle(sky, orc, ts, fb, n, opaque):
    P = scenes.scene_uniform(n, seed=70 + n)
    P[0:2] *= 0.1                      # long lists in a few tiles
    P[3:6] = -2.0
    if opaque:
        P[10] = 4.0                    # pixels end after a few splats
        P[10, ::3] = 9.0               # alpha clamped
    rgba, alpha, last, fw = one_view(sky, orc, P, 70, 50, ts, fb)
    assert np.array_equal(rgba, fw["rgba"])
    assert np.array_equal(alpha, fw["alpha"])
    assert np.array_equal(last, fw["last"])


def test_infinite_colours_stay_with_the_pixels_they_cover(sky, orc):
    P = scenes.scene_uniform(300, seed=90)
    P[3:6] = -2.5
    P[11, 5] = 7.0e4                   # infinite once read through f16
    P[12, 250] = 7.0e4
    rgba, alpha, last, fw = one_view(sky, orc, P, 64, 48, 16, 0)
    assert np.isinf(rgba).any() and np.isfinite(rgba[:, :3]).all(axis=1).any()
    assert np.array_equal(rgba, fw["rgba"], equal_nan=True)
    assert np.array_equal(alpha, fw["alpha"])
