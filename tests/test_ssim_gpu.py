"""The SSIM term at the edges of its 64x16 pixel tiles: views smaller than a
window, one pixel short of and past a tile, and views of different aspect in
one step.  Both sides add the window in row-major order in f32, so the
residuals are identical."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(1, 1)], [(5, 3)], [(63, 15)], [(64, 16)], [(65, 17)],
                                   [(130, 33), (20, 211), (257, 9)]])
def test_ssim_residual_matches_oracle(sky, orc, sizes):
    P = scenes.scene_uniform(4096, seed=41)
    cams = [scenes.camera_fov((0.3 * k, 0.1, -3.0), w, h) for k, (w, h) in enumerate(sizes)]
    tgt = [scenes.target_uniform(w, h, seed=42 + k) for k, (w, h) in enumerate(sizes)]
    with sky.GaussianRenderer(sh_degree=0, w_l2=0.5, w_l1=0.8, w_ssim=0.2) as r:
        r.load_points(P)
        r.setTrainingCameras(cams)
        r.setTrainingImages(tgt)
        r.forward(list(range(len(cams))))
        res = r.read_buffer("residual").reshape(-1, 4)
    s = orc.settings(w_l2=0.5, w_l1=0.8, w_ssim=0.2)
    want = [orc.view_pipeline(P, c, t, s, 0, mode=0)["ls"]["residual"] for c, t in zip(cams, tgt)]
    assert np.array_equal(res, np.concatenate(want))
