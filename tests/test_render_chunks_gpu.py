"""Renders large enough to leave chunk by chunk while later tiles are rendered:
the host images are those of the views rendered one at a time, and of the
buffers a forward pass leaves, for views of different sizes, with either
output alone, and for a first pass as for later ones."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts", [8, 16])
@pytest.mark.parametrize("sizes", [[(1290, 1001)], [(700, 513), (1280, 720), (33, 17), (900, 901)]])
def test_chunked_render_equals_the_passes_buffers(sky, ts, sizes):
    P = scenes.scene_uniform(20000, seed=65)
    cams = [scenes.camera_fov((0.2 * k, 0.1, -3.0), w, h) for k, (w, h) in enumerate(sizes)]
    with sky.GaussianRenderer(sh_degree=0, tile_size=ts) as r:
        r.load_points(P)
        r.setTrainingCameras(cams)
        views = list(range(len(cams)))
        first = r.render(views)
        again = r.render(views)
        assert np.array_equal(r.read_buffer("color").reshape(-1, 4), again[0])
        assert np.array_equal(r.read_buffer("alpha"), again[1])
        rgba_only, none = r.render(views, with_alpha=False)
        single = [r.render([v]) for v in views]
    assert none is None and np.array_equal(rgba_only, again[0])
    for a, b in zip(first, again):
        assert np.array_equal(a, b)
    assert np.array_equal(again[0], np.concatenate([s[0] for s in single]))
    assert np.array_equal(again[1], np.concatenate([s[1] for s in single]))
    assert (again[1] > 0).mean() > 0.05
