"""Multi-view scores tile by tile: every tile size, views of different and odd
sizes in one batch, lists past a staged batch, ill-conditioned conics, a
camera given twice.  Hits are integers and identical to the oracle's; the
pruning scores' mean is an f64 sum in another order (1e-6 relative)."""
import numpy as np
import pytest

from oracle import densify as D
from skyfall import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts", [8, 16, 32])
@pytest.mark.parametrize("n,sizes", [(40, [(9, 5)]), (3000, [(33, 17), (64, 32), (33, 17)]), (6000, [(50, 41)])])
def test_scores_match_oracle(sky, orc, ts, n, sizes):
    P = scenes.scene_uniform(n, seed=81)
    P[0:2] *= 0.5
    P[3, ::4] = -0.5       # long and thin
    P[4:6, ::4] = -6.5
    cams = [scenes.camera_fov((0.4 * k, 0.1, -3.0), w, h) for k, (w, h) in enumerate(sizes)]
    tgts = [scenes.target_uniform(w, h, seed=82 + k) for k, (w, h) in enumerate(sizes)]
    views = list(range(len(cams))) + [0]
    with sky.GaussianRenderer(sh_degree=0, tile_size=ts) as r:
        r.load_points(P)
        r.setTrainingCameras(cams)
        r.setTrainingImages(tgts)
        hits, score = r.scoreViews(views)
    s = orc.settings(tile_size=ts)
    out = []
    for v in views:
        ref = orc.view_pipeline(P, cams[v], None, s, 0)
        out.append(D.metric_view(ref["fw"]["rgba"], tgts[v], ref["fw"]["last"], ref["tl"]["offsets"],
                                 ref["tl"]["gidx_sorted"], ref["pr"]["rec"], *sizes[v], ts, n))
    want_hits, want_score = D.combine_scores(out)
    assert hits.sum() > 0
    assert np.array_equal(hits, want_hits)
    np.testing.assert_allclose(score, want_score, rtol=1e-6, atol=1e-12)
