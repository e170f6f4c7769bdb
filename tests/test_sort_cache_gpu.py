"""sky_sort_pairs keeps its scratch for the next call.  A call that needs more
and cannot get it leaves nothing of the old one behind: smaller sorts after it
allocate anew and are right.  (SKY_FAULT=alloc:2, in a process of its own: the
second device allocation fails on the host.)"""
import pytest

from test_faults_gpu import run_child

pytestmark = pytest.mark.gpu


def test_smaller_sorts_after_a_growth_that_failed(sky):
    out = run_child("alloc:2", """
        import torch
        def sort(n, seed):
            keys = np.random.default_rng(seed).integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
            kin = torch.from_numpy(keys.view(np.int32)).cuda()
            kout = torch.full_like(kin, -1); vout = torch.full_like(kin, -1)
            p = lambda t: C.c_void_p(t.data_ptr())
            rc = L.sky_sort_pairs(p(kin), None, p(kout), p(vout), n, 32, C.c_void_p(torch.cuda.current_stream().cuda_stream))
            torch.cuda.synchronize()
            order = np.argsort(keys, kind="stable")
            ok = bool(np.array_equal(kout.cpu().numpy().view(np.uint32), keys[order]) and
                      np.array_equal(vout.cpu().numpy().view(np.uint32), order.astype(np.uint32)))
            return rc, ok
        torch.zeros(1, device="cuda")
        first = sort(50_000, 1)            # allocation 1
        failed = sort(3_000_000, 2)        # allocation 2
        again = [sort(n, 3 + n) for n in (50_000, 1_000, 50_000, 3_000_000, 4_097)]
        print(json.dumps(dict(first=first, failed=failed, again=again)))
    """)
    assert out["first"] == [0, True]
    assert out["failed"] == [sky._lib.SKY_ERR_INJECTED, False]
    assert out["again"] == [[0, True]] * 5
