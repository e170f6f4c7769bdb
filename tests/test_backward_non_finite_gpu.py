"""The 16x16-tile backward composites without a branch per pixel: what does not
contribute, and the clamp's zero slope, have alpha 0.  Where a product is not
finite, 0 times it is not 0, and the gradients have to be those of the
8x8-tile kernel, which branches."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


def gradients(sky, P, cam, tgt, **cfg):
    with sky.GaussianRenderer(sh_degree=0, w_ssim=0.0, **cfg) as r:
        r.load_points(P)
        r.setTrainingCameras([cam])
        r.setTrainingImages([tgt])
        r.forward([0])
        alpha = r.read_buffer("alpha").copy()
        return r.backward(), alpha


@pytest.mark.parametrize("res", [(65, 49), (1, 1), (1, 3), (17, 33)])  # (entries of many lanes, and of one)
@pytest.mark.parametrize("value", [np.inf, -np.inf, 1e30, np.nan])
def test_clamped_pair_with_a_residual_that_is_not_finite(sky, res, value):
    w, h = res
    P = scenes.scene_uniform(7, seed=120)
    P[0:3] = 0.0                       # the first on the middle pixel, its alpha clamped there
    P[0, 1:] = [2.0, -2.0, 2.0, -2.0, 1.6, -1.6]   # the others clear of it
    P[1, 1:] = [1.2, 1.2, -1.2, -1.2, 0.0, 0.0]
    P[3:6] = -1.5
    P[3:6, 1:] = -3.0
    P[10] = 12.0                       # opacity 1 - 6e-6
    if w == 1:                         # (every splat reaches so small an image: the first alone)
        P = P[:, :1].copy()
    cam, tgt = scenes.camera_fov((0.0, 0.0, -3.0), w, h), scenes.target_uniform(w, h, seed=121)
    tgt[h // 2, w // 2, 1] = value
    g16, alpha = gradients(sky, P, cam, tgt, w_l2=1.0, w_l1=0.2, tile_size=16)
    g8, _ = gradients(sky, P, cam, tgt, w_l2=1.0, w_l1=0.2, tile_size=8)
    assert alpha[(h // 2) * w + w // 2] == np.float32(0.999)
    # the clamp passes nothing on to the opacity, the mean and the covariance
    assert np.isfinite(g8[:11]).all()
    fin = np.isfinite(g8)
    assert np.array_equal(fin, np.isfinite(g16))
    scale = np.abs(g8[:11]).max()
    assert np.all(np.abs(g16[fin] - g8[fin]) <= 1e-3 * np.abs(g8[fin]) + 1e-6 * scale)
