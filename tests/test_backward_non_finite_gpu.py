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
        alpha, records = r.read_buffer("alpha").copy(), r.read_buffer("records").reshape(-1, 12).copy()
        return r.backward(), alpha, records


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
    g16, alpha, _ = gradients(sky, P, cam, tgt, w_l2=1.0, w_l1=0.2, tile_size=16)
    g8, _, _ = gradients(sky, P, cam, tgt, w_l2=1.0, w_l1=0.2, tile_size=8)
    assert alpha[(h // 2) * w + w // 2] == np.float32(0.999)
    # the clamp passes nothing on to the opacity, the mean and the covariance
    assert np.isfinite(g8[:11]).all()
    fin = np.isfinite(g8)
    assert np.array_equal(fin, np.isfinite(g16))
    scale = np.abs(g8[:11]).max()
    assert np.all(np.abs(g16[fin] - g8[fin]) <= 1e-3 * np.abs(g8[fin]) + 1e-6 * scale)


@pytest.mark.parametrize("bb", [0, 32, 64, 128])
def test_finite_batches_in_front_of_an_overflow(sky, bb):
    n, w, h = 400, 48, 48
    P = scenes.scene_uniform(n, seed=122)
    P[0:2] *= 0.25
    P[2] = np.minimum(P[2], 0.8)       # whole depths below 4
    P[3:6] = -4.5                      # a pixel or two
    P[10] = -4.0                       # thin: the lists are walked to their ends
    P[0:2, n // 2] = 0.0               # behind all of them, in the first batch walked, a splat whose
    P[2, n // 2] = 1.5                 # colours are finite and their product with the residual is not
    P[3:6, n // 2] = -3.0
    P[10, n // 2] = 2.0
    P[11:14, n // 2] = 3.0e38
    cam, tgt = scenes.camera_fov((0.0, 0.0, -3.0), w, h), scenes.target_uniform(w, h, seed=123)
    cfg = dict(w_l2=0.0, w_l1=20.0, round_params_f16=0)
    g16, _, rec = gradients(sky, P, cam, tgt, tile_size=16, bwd_batch=bb, **cfg)
    g8, _, _ = gradients(sky, P, cam, tgt, tile_size=8, **cfg)
    # the pixels a splat reaches, with some to spare
    dx = (np.arange(w) + 0.5)[None, None, :] - rec[:, 0, None, None]
    dy = (np.arange(h) + 0.5)[None, :, None] - rec[:, 1, None, None]
    s = 0.5 * (rec[:, 2, None, None] * dx * dx + rec[:, 4, None, None] * dy * dy) + rec[:, 3, None, None] * dx * dy
    reach = rec[:, 5, None, None] * np.exp(-s) > 0.99 / 255
    clear = ~(reach & reach[n // 2]).any(axis=(1, 2))
    beside = clear & (reach[:, 16:32, 16:32].any(axis=(1, 2)))  # in a tile with the splat behind
    assert beside.sum() > 30 and (~clear).sum() > 30
    assert not np.isfinite(g16[:11, n // 2]).all()
    assert np.isfinite(g8[:, clear]).all() and np.isfinite(g16[:, clear]).all()
    scale = np.abs(g8[:11, clear]).max()
    assert np.all(np.abs(g16[:, clear] - g8[:, clear]) <= 1e-3 * np.abs(g8[:, clear]) + 1e-6 * scale)
