"""The 16x16-tile backward of steps with few tiles stages 128 splats per batch
and loads the next batch ahead; larger steps stage 64.  Lists around multiples
of its batch, a step of one tile, and steps at both sides of the tile count
that separates the two: partial sums equal to those of the 64-deep batches,
bit for bit (a sum's order does not depend on the batches)."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,res", [(1, (16, 16)), (127, (16, 16)), (128, (16, 16)), (129, (16, 16)), (255, (33, 17)),
                                   (257, (16, 31)), (385, (48, 16)), (1500, (320, 608)), (1500, (321, 608)),
                                   (1500, (336, 608))])
def test_few_tiles_equal_many(sky, n, res):
    P = scenes.scene_uniform(n, seed=110 + n)
    P[0:2] *= 0.15
    P[3:6] = -2.5              # every splat over much of the image
    P[10] = np.minimum(P[10], -3.0)  # thin: the lists are walked to their ends
    cam, tgt = scenes.camera_fov((0.0, 0.0, -3.0), *res), scenes.target_uniform(*res, seed=111)
    got = []
    for bb in (0, 64, 128):
        with sky.GaussianRenderer(sh_degree=0, w_l2=1.0, w_l1=0.2, w_ssim=0.0, tile_size=16, bwd_batch=bb) as r:
            r.load_points(P)
            r.setTrainingCameras([cam])
            r.setTrainingImages([tgt])
            r.forward([0])
            r.backward()
            got.append(r.read_buffer("partials"))
    assert got[0].any()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[2], got[1])
