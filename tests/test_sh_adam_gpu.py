"""Adam of a training step against the gradients of the op pair on the same
state: the SH planes go through a kernel of their own for at most 16 views (in
groups of four Gaussians), through the geometry kernel beyond.  Counts that
are not multiples of four or of the plane padding, every SH degree, steps with
and without an SH update, and a second step on the first one's moments.  Both
sides apply the same f32 operations to the same gradients: identical bits."""
import numpy as np
import pytest

from skyfall import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,views,deg,every", [(1, 1, 3, 1), (255, 1, 0, 1), (513, 2, 1, 1), (1030, 1, 2, 2),
                                               (2049, 5, 3, 1), (700, 16, 3, 1), (700, 17, 3, 1)])
def test_train_step_applies_adam_to_the_op_pairs_gradients(sky, orc, n, views, deg, every):
    P = scenes.scene_clusters(n, seed=91, clusters=4, center_range=0.5, logscale_mean=-3.0, sh_degree=deg)
    cams = scenes.cameras_orbit(views, 3.5, 70, 50)
    tgt = [scenes.target_uniform(70, 50, seed=92 + k) for k in range(views)]
    groups = [(0, 3, 0), (3, 6, 1), (6, 10, 2), (10, 11, 3), (11, 59, 4)]
    with sky.GaussianRenderer(sh_degree=deg, sh_degree_interval=0, sh_update_interval=every, w_l2=1.0, w_l1=0.2,
                              w_ssim=0.0, max_views_per_step=64) as r:
        r.load_points(P)
        r.setTrainingCameras(cams)
        r.setTrainingImages(tgt)
        for step in (1, 2):
            p0, (m1, m2) = r.params(), r.moments()
            r.forward(list(range(views)))
            g = r.backward()
            st = r.trainStep(list(range(views)))
            assert st.sh_updated == (step % every == 0)
            sc = r.read_buffer("step_scalars")
            for lo, hi, k in groups:
                if k == 4 and not st.sh_updated:
                    continue
                p, a, b = (np.ascontiguousarray(x[lo:hi]) for x in (p0, m1, m2))
                orc.adam(p, a, b, np.ascontiguousarray(g[lo:hi]), sc[k], *sc[5:10])
                p0[lo:hi], m1[lo:hi], m2[lo:hi] = p, a, b
            got1, got2 = r.moments()
            assert np.array_equal(m1, got1) and np.array_equal(m2, got2)
            assert np.array_equal(p0, r.params())
            assert np.abs(g).max() > 0
