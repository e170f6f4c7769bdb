"""Key emission: a warp of 32 items stages at most 384 keys in shared memory and
writes them side by side; a warp with more writes item by item.  The same
Gaussians in orders that put their warps on either side of the limit, at it, and
in partly filled warps must be listed in the same tiles, each of them once, and
in the order of their depths and indices."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


def lists(sky, P, cam, tgt, cull):
    with sky.GaussianRenderer(sh_degree=0, tile_size=16, w_l2=1.0, w_l1=0.0, w_ssim=0.0) as r:
        r.load_points(P)
        r.setTrainingCameras([cam])
        r.setTrainingImages([tgt])
        r.setTileCull(cull)
        r.forward([0])
        if cull:
            r.backward()
        return (r.read_buffer("tile_offsets").astype(np.int64), r.read_buffer("flatten").astype(np.int64),
                r.read_buffer("counts").astype(np.int64))


@pytest.mark.parametrize("cull", [False, True])
@pytest.mark.parametrize("n,big,res", [(96, 6, (320, 240)), (71, 40, (64, 48)), (64, 64, (64, 48)),
                                       (32, 32, (64, 48)), (33, 1, (400, 300)), (300, 3, (640, 480))])
def test_order_of_items_does_not_change_lists(sky, cull, n, big, res):
    P = scenes.scene_uniform(n, seed=120 + n)
    P[0:2] *= 0.5
    P[3:6] = -4.5
    # over every tile: a radius of about 400 pixels, below the 512 that are culled
    P[3:6, :big] = np.log(400.0 / 3.0 * (3.0 + P[2, :big]) / (0.866 * res[1]))
    P[10] = 0.0
    cam, tgt = scenes.camera_fov((0.0, 0.0, -3.0), *res), scenes.target_uniform(*res, seed=121)
    rng = np.random.default_rng(122)
    spread = np.argsort(np.concatenate([np.linspace(0, 1, big), np.linspace(0, 1, max(n - big, 1))[:n - big]]),
                        kind="stable")
    ref, totals = None, []
    for order in (np.arange(n), np.arange(n)[::-1], spread, rng.permutation(n)):
        off, flat, counts = lists(sky, np.ascontiguousarray(P[:, order]), cam, tgt, cull)
        assert off[-1] == counts.sum() and off[-1] > 0
        totals += [counts[k:k + 32].sum() for k in range(0, n, 32)]
        flat = flat[:off[-1]]
        tile = np.repeat(np.arange(off.size - 1), np.diff(off))
        depth = np.trunc(3.0 + P[2, order[flat]])
        assert np.array_equal(np.lexsort((flat, depth, tile)), np.arange(flat.size))
        got = (off, np.sort(tile * n + order[flat]))
        if ref is None:
            ref = got
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
        assert np.unique(got[1]).size == got[1].size
    if big in (6, 3):
        assert min(totals) <= 384 < max(totals)
    if n == 32:
        assert totals[0] == 32 * 12  # exactly the limit
