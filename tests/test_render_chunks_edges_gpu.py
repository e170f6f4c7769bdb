"""Renders that leave in chunks, where the chunks can go wrong: alpha alone (a
quarter of the bytes per pixel, so larger views), 32x32 tiles, and a first
large view whose lists outgrow what a small one sized: its pass is discarded
before anything is copied and run again."""
import ctypes

import numpy as np
import pytest

from skyfall import _lib, scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MB = 1 << 20


def render_into(r, views, rgba, alpha):
    v = np.ascontiguousarray(views, dtype=np.uint32)
    p = [ctypes.c_void_p(t.data_ptr() if t is not None else None) for t in (rgba, alpha)]
    _lib.check(_lib.lib().sky_render(r._h, _lib.ptr(v), len(v), *p))


def chunks(sizes, ts, bytes_per_px):  # at least two: the views are large enough
    tiles = sum(-(-w // ts) * -(-h // ts) for w, h in sizes)
    return min(16, sum(w * h for w, h in sizes) * bytes_per_px // (4 * MB), tiles // 2048)


def pinned(px, rgba, alpha):
    return (torch.full((px, 4), -1.0, pin_memory=True) if rgba else None,
            torch.full((px,), -1.0, pin_memory=True) if alpha else None)


def renderer(sky, sizes, ts, P):
    r = sky.GaussianRenderer(sh_degree=0, tile_size=ts)
    r.load_points(P)
    r.setTrainingCameras([scenes.camera_fov((0.2 * k, 0.1, -3.0), w, h) for k, (w, h) in enumerate(sizes)])
    return r


@pytest.mark.parametrize("ts,sizes", [(8, [(1290, 1001), (1277, 903)]), (16, [(1290, 1001), (1277, 903)]),
                                      (16, [(700, 513), (1921, 1080), (33, 17), (900, 901)]),
                                      (32, [(2111, 1093), (2111, 1125)])])
@pytest.mark.parametrize("rgba,alpha", [(False, True), (True, False), (True, True)])
def test_each_output(sky, ts, sizes, rgba, alpha):
    assert chunks(sizes, ts, 16 * rgba + 4 * alpha) >= 2
    out = pinned(sum(w * h for w, h in sizes), rgba, alpha)
    views = list(range(len(sizes)))
    with renderer(sky, sizes, ts, scenes.scene_uniform(20000, seed=131)) as r:
        for k in range(2):  # a first pass, which sizes the lists, and a later one
            for o in out:
                if o is not None:
                    o.fill_(-1.0)
            render_into(r, views, *out)
            if k == 0:
                single = [r.render([v]) for v in views]  # pageable: one copy each
            for o, which in zip(out, (0, 1)):
                assert o is None or np.array_equal(o.numpy(), np.concatenate([s[which] for s in single]))


@pytest.mark.parametrize("ts", [8, 16, 32])
def test_lists_that_outgrow_the_sized_ones(sky, ts):
    sizes = [(64, 48), (2111, 1093), (2111, 1125)]
    P = scenes.scene_uniform(20000, seed=132)
    P[3:6] = -2.8  # (over 160 pixels wide in the large views)
    out = pinned(2111 * (1093 + 1125), True, True)
    assert chunks(sizes[1:], ts, 20) >= 2
    with renderer(sky, sizes, ts, P) as r:
        r.render([0])
        small = int(r.read_buffer("counts").astype(np.int64).sum())
        render_into(r, [1, 2], *out)
        large = int(r.read_buffer("counts").astype(np.int64).sum())
        assert large > 1.5 * max(small, 65536) + 4096  # beyond the capacity after the first
        again = pinned(2111 * (1093 + 1125), True, True)
        render_into(r, [1, 2], *again)
    with renderer(sky, sizes, ts, P) as r:
        want = r.render([1, 2])
    for o, a, w in zip(out, again, want):
        assert np.array_equal(o.numpy(), w) and np.array_equal(a.numpy(), w)
