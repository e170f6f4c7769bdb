"""Multi-view scores: a warp counts its list 32 entries at a time, so lists around
multiples of 32 and of a staged batch of 256, every splat over every pixel.
Hits are integers and identical to the oracle's."""
import numpy as np
import pytest

from oracle import densify as D
from skyfall import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 65, 255, 257, 300])
def test_hits_match_oracle(sky, orc, n):
    w, h = 24, 20
    P = scenes.scene_uniform(n, seed=140 + n)
    P[0:2] *= 0.1
    P[3:6] = -1.0              # over the whole image
    P[10] = -4.0               # thin: no pixel ends early
    cam, tgt = scenes.camera_fov((0.0, 0.0, -3.0), w, h), scenes.target_uniform(w, h, seed=141)
    with sky.GaussianRenderer(sh_degree=0, tile_size=16) as r:
        r.load_points(P)
        r.setTrainingCameras([cam])
        r.setTrainingImages([tgt])
        hits, _ = r.scoreViews([0])
    ref = orc.view_pipeline(P, cam, None, orc.settings(tile_size=16), 0)
    want, _ = D.combine_scores([D.metric_view(ref["fw"]["rgba"], tgt, ref["fw"]["last"], ref["tl"]["offsets"],
                                              ref["tl"]["gidx_sorted"], ref["pr"]["rec"], w, h, 16, n)])
    assert want.min() > 0 and np.array_equal(hits, want)
