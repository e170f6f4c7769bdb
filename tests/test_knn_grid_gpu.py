"""The k-NN grid search where its skipped rows and cells could matter: far from
the origin, outliers many cells away, points on a line or in a plane, dense
clumps in a wide grid.  Distances are those of the all-pairs scan, bit for
bit."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


def positions(kind, n):
    rng = np.random.default_rng(7)
    x = rng.normal(size=(3, n))
    if kind == "offset":
        x = x * 3.0 + np.array([[30000.0], [-500.0], [60000.0]])
    elif kind == "outliers":
        x *= 0.01
        x[:, ::97] = rng.uniform(-50, 50, size=x[:, ::97].shape)
    elif kind == "line":
        x[1:] = 0.25
    elif kind == "plane":
        x[2] = -1.5
    elif kind == "clumps":
        x = 0.002 * x + rng.uniform(-8, 8, size=(3, 5))[:, rng.integers(0, 5, n)]
    return x


@pytest.mark.parametrize("kind", ["offset", "outliers", "line", "plane", "clumps"])
def test_knn_matches_all_pairs_on_awkward_grids(sky, orc, kind):
    n = 4000
    P = scenes.scene_uniform(n, seed=1410)
    P[0:3] = positions(kind, n)
    with sky.GaussianRenderer() as r:
        r.load_points(P)
        dens = r.initializeKnnAndSync(scene_extent=3.0)
        ls = r.params()[3]
    want_d, want_ls = orc.knn_init(P, 3.0)
    assert np.array_equal(dens, want_d)
    assert np.array_equal(ls, want_ls)
