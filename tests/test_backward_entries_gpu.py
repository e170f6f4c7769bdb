"""The 16x16-tile backward's entries: reduced four at a time in shared memory,
so list lengths around multiples of four, entries of one lane and of none,
batches of every depth, and non-finite or huge colours and residuals, which
take the variant that clears what does not contribute.  Partial sums against
the oracle's f64 sums (2e-5 of the summed magnitudes); depths against each
other bit for bit; non-finite cases against the 8x8-tile kernel."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


def renderer(sky, P, cam, tgt, **cfg):
    r = sky.GaussianRenderer(sh_degree=0, w_l2=1.0, w_l1=0.2, w_ssim=0.0, **cfg)
    r.load_points(P)
    r.setTrainingCameras([cam])
    r.setTrainingImages([tgt])
    r.forward([0])
    return r


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 63, 65, 130, 700])
@pytest.mark.parametrize("size", [-2.0, -5.5])
def test_partials_match_oracle(sky, orc, n, size):
    P = scenes.scene_uniform(n, seed=95 + n)
    P[0:2] *= 0.15
    P[3:6] = size              # splats over whole tiles, splats of a pixel or two
    P[10, ::3] = 9.0           # clamped alphas
    cam, tgt = scenes.camera_fov((0.0, 0.0, -3.0), 41, 35), scenes.target_uniform(41, 35, seed=96)
    got = []
    for bb in (0, 32, 128):
        with renderer(sky, P, cam, tgt, tile_size=16, bwd_batch=bb) as r:
            r.backward()
            part = r.read_buffer("partials").reshape(-1, 12)[:, :9].astype(np.float64)
            emitted = r.read_buffer("counts").astype(np.int64)[r.read_buffer("item_order")]
            sums = np.zeros((n, 9))
            np.add.at(sums, np.repeat(r.read_buffer("item_order"), emitted), part)
            got.append((part, sums))
    s = orc.settings(tile_size=16, w_l2=1.0, w_l1=0.2, w_ssim=0.0)
    ref = orc.view_pipeline(P, cam, tgt, s, 0, mode=0)["bw"]
    assert np.all(np.abs(got[0][1] - ref["gsum9"]) <= 2e-5 * ref["gabs9"] + 1e-9)
    for part, _ in got[1:]:
        assert np.array_equal(part, got[0][0])


@pytest.mark.parametrize("kind", ["infinite colour", "infinite target", "huge target", "nan target"])
def test_non_finite_values_stay_with_what_they_touch(sky, kind):
    P = scenes.scene_uniform(400, seed=97)
    cam, tgt = scenes.camera_fov((0.0, 0.0, -3.0), 64, 48), scenes.target_uniform(64, 48, seed=98)
    if kind == "infinite colour":
        P[11, 7] = 7.0e4       # infinite once read through f16
    else:
        tgt[10:14, 20:30, 1] = {"infinite target": np.inf, "huge target": 1e20, "nan target": np.nan}[kind]
    with renderer(sky, P, cam, tgt, tile_size=16) as r:
        g16 = r.backward()
    with renderer(sky, P, cam, tgt, tile_size=8) as r:
        g8 = r.backward()
    fin = np.isfinite(g8)
    assert np.array_equal(fin, np.isfinite(g16))
    if kind != "huge target":
        assert not fin.all() and fin.mean() > 0.5
    scale = np.abs(g8[:14][fin[:14]]).max()
    assert np.all(np.abs(g16[fin] - g8[fin]) <= 1e-3 * np.abs(g8[fin]) + 1e-6 * scale)
