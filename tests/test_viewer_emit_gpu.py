"""Viewer key emission: a warp of 32 Gaussians (in depth order) stages at most 384
tile keys in shared memory; a warp with more writes them directly.  Frames
whose warps hold fewer, exactly as many, more, and both in turn, and partly
filled warps, equal the oracle's."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


# 64x48: 12 tiles; 32 quads over all of them are 384 keys, 12 x 33 is a warp and one
@pytest.mark.parametrize("w,h,n,big", [(64, 48, 1, 1), (64, 48, 32, 1), (64, 48, 33, 1), (64, 48, 70, 2),
                                       (80, 48, 64, 1), (200, 120, 500, 40), (200, 120, 500, 9)])
def test_frame_matches_oracle(sky, orc, w, h, n, big):
    P = scenes.scene_uniform(n, seed=130 + n)
    P[0:2] *= 0.3
    P[3:6] = -4.0
    P[3:6, ::big] = 1.0        # quads over every tile
    cam = scenes.camera_fov((0.0, 0.0, -3.0), w, h)
    with sky.GaussianRenderer(sh_degree=0) as r:
        r.load_points(P)
        img = r.frame(cam, sh_degree=0)
    ref = orc.view_render(P, cam, 1.0, 0, 1)
    assert np.array_equal(img, ref["rgba"].reshape(img.shape)) and img.any()
