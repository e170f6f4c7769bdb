"""A render that leaves in chunks and fails on the way has no copy in flight when
it returns: the caller's memory is the caller's again.  (SKY_FAULT=copy:N, in a
process of its own: the N-th copy fails on the host before it is issued.)"""
import pytest

from test_faults_gpu import run_child

pytestmark = pytest.mark.gpu


# 8 views of 1280x720 leave in 14 chunks, the last of them within the last view
@pytest.mark.parametrize("at,with_alpha", [(1, True), (14, False), (27, True)])
def test_nothing_is_written_after_the_call(sky, at, with_alpha):
    out = run_child(f"copy:{at}", f"""
        import torch
        W, H, V = 1280, 720, 8
        P = scenes.scene_uniform(20000, seed=130)
        r = sky.GaussianRenderer(sh_degree=0)
        r.load_points(P)
        r.setTrainingCameras([scenes.camera_fov((0.2 * k, 0.1, -3.0), W, H) for k in range(V)])
        views = np.arange(V, dtype=np.uint32)
        want = r.render(list(range(V)))            # pageable memory: one copy, not counted
        rgba = torch.full((V * H * W, 4), -1.0, pin_memory=True)
        alpha = torch.full((V * H * W,), -1.0, pin_memory=True) if {with_alpha} else None
        p = lambda t: C.c_void_p(t.data_ptr() if t is not None else None)
        mine = rgba[7 * H * W - W:7 * H * W].numpy()   # a row of a chunk before the last
        args = (r._h, E.ptr(views), V, p(rgba), p(alpha))
        render = lambda: L.sky_render(*args)
        rc1 = render()
        mine[:] = -5.0
        msg = L.sky_last_error().decode()
        torch.cuda.synchronize()
        kept = bool((mine == -5.0).all())
        first = rgba[0].tolist()
        rc2 = render()
        same = bool(np.array_equal(rgba.numpy(), want[0]) and
                    (alpha is None or np.array_equal(alpha.numpy(), want[1])))
        print(json.dumps(dict(rc1=rc1, msg=msg, kept=kept, begun=first != [-1.0] * 4, rc2=rc2, same=same)))
    """)
    assert out["rc1"] == sky._lib.SKY_ERR_INJECTED and "copy" in out["msg"]
    assert out["begun"] == (at > 1)
    assert out["kept"]
    assert out["rc2"] == 0 and out["same"]
