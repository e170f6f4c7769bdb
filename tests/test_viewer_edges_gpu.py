"""Viewer coverage at the edges of its 8x4 pixel blocks and 16x16 tiles, and
lists longer than a staged batch: every (pixel, quad) pair and its order are
the oracle's, so images are identical."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n,scaling", [(1, 1, 64, 1.0), (8, 4, 300, 1.0), (17, 16, 257, 2.0),
                                           (33, 21, 3000, 1.0), (48, 48, 20000, 0.3)])
def test_frame_matches_oracle_at_block_edges(sky, orc, w, h, n, scaling):
    P = scenes.scene_uniform(n, seed=61)
    P[3, ::7] = 0.5      # thin splats: exponents below the exp range inside the quad
    P[4, ::7] = -6.0
    P[10, ::5] = 20.0    # opacity 1
    cam = scenes.camera_fov((0.1, -0.2, -2.0), w, h)
    with sky.GaussianRenderer(sh_degree=0) as r:
        r.load_points(P)
        img = r.frame(cam, gaussian_scaling=scaling, sh_degree=0)
    ref = orc.view_render(P, cam, scaling, 0, 1)
    assert np.array_equal(img, ref["rgba"].reshape(img.shape))


@pytest.mark.parametrize("w,h", [(1, 1), (17, 5), (97, 61)])
def test_bytes_are_the_rounded_image(sky, w, h):
    P = scenes.scene_uniform(3000, seed=62)
    P[11:14, ::2] *= 3.0       # colours past 1
    cam = scenes.camera_fov((0.1, -0.2, -2.0), w, h)
    with sky.GaussianRenderer(sh_degree=0) as r:
        r.load_points(P)
        img = r.frame(cam, sh_degree=0)
        u8 = r.frame(cam, sh_degree=0, as_u8=True)
        again = r.read_buffer("view_rgba").reshape(img.shape)
    scaled = np.clip(img, 0.0, 1.0) * np.float32(255.0)
    assert np.array_equal(u8, np.floor(scaled.astype(np.float64) + 0.5).astype(np.uint8))
    assert np.array_equal(again, img)
