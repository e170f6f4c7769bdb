"""Renders large enough to leave chunk by chunk while later tiles are rendered:
the host images are those of the views rendered one at a time, and of the
buffers a forward pass leaves, for views of different sizes, with either
output alone, and for a first pass as for later ones.  Only page-locked images
leave so; pageable ones are copied whole, with the same result."""
import ctypes

import numpy as np
import pytest

from skyfall import _lib, scenes

pytestmark = pytest.mark.gpu


def render_into(r, views, rgba, alpha):
    v = np.ascontiguousarray(views, dtype=np.uint32)
    _lib.check(_lib.lib().sky_render(r._h, _lib.ptr(v), len(v), ctypes.c_void_p(rgba.data_ptr() if rgba is not None else None),
                                     ctypes.c_void_p(alpha.data_ptr() if alpha is not None else None)))


@pytest.mark.parametrize("ts", [8, 16])
@pytest.mark.parametrize("sizes", [[(1290, 1001)], [(700, 513), (1280, 720), (33, 17), (900, 901)]])
@pytest.mark.parametrize("locked", [(True, True), (True, False), (False, True), (True, None), (None, True)])
def test_page_locked_images(sky, ts, sizes, locked):
    torch = pytest.importorskip("torch")
    px = sum(w * h for w, h in sizes)
    P = scenes.scene_uniform(20000, seed=66)
    cams = [scenes.camera_fov((0.2 * k, 0.1, -3.0), w, h) for k, (w, h) in enumerate(sizes)]
    out = [None if lock is None else torch.zeros(shape, dtype=torch.float32, pin_memory=lock)
           for lock, shape in zip(locked, ((px, 4), (px,)))]
    with sky.GaussianRenderer(sh_degree=0, tile_size=ts) as r:
        r.load_points(P)
        r.setTrainingCameras(cams)
        views = list(range(len(cams)))
        want = r.render(views)
        for _ in range(2):
            render_into(r, views, *out)
            for o, w in zip(out, want):
                assert o is None or np.array_equal(o.numpy(), w)
                if o is not None:
                    o.zero_()
    with sky.GaussianRenderer(sh_degree=0, tile_size=ts) as r:  # a first pass
        r.load_points(P)
        r.setTrainingCameras(cams)
        render_into(r, views, *out)
    for o, w in zip(out, want):
        assert o is None or np.array_equal(o.numpy(), w)


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
