"""GPU: the all-ones word in lists that only the kernels check (the pipelined
end-to-end call, lists read in place, the no-allocation entry) is reported
like any other bad entry, in every list kind and at either end of a list."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("in_host", [False, True], ids=["copied", "in_place"])
@pytest.mark.parametrize("kind", [0, 1, 2, 3], ids=["points", "quadrupole", "order4", "correction"])
def test_all_ones_word_is_reported(kind, in_host):
    from pgrav import gravcuda as gc, host, ics
    pos, m = ics.grf_box(16, seed=3, rms_disp=0.3)
    t = host.Tree(pos, m, box=1.0, leaf_max=16, group_max=32, p2cut=7, p4cut=8, tol=1e-4)
    eps2 = (1.0 / 16 / 50) ** 2
    n = len((t.plist, t.qlist, t.hlist, t.clist)[kind])
    assert n > 2
    for at in (0, n // 2, n - 1):
        pp = gc.pinned_problem(t, lists_in_host=in_host)
        p = pp.problem
        addr = (p.plist, p.qlist, p.hlist, p.clist)[kind]
        (ctypes.c_uint32 * n).from_address(addr)[at] = 0xffffffff
        with pytest.raises(gc.GravError, match="device error word 0x2"):
            gc.groups_eval_problem(pp, eps2, 1.0, ewald=True)
        gc.lib().gravcuda_clear_status()
    gc.groups_eval_problem(gc.pinned_problem(t, lists_in_host=in_host), eps2, 1.0, ewald=True)
    gc.lib().grav_groups_release_CUDA()


def test_all_ones_word_is_reported_without_allocations():
    import torch
    from pgrav import gravcuda as gc, host, ics
    pos, m = ics.plummer(2000, seed=3)
    t = host.Tree(pos, m, leaf_max=16, group_max=32, p2cut=7, p4cut=0, tol=1e-4)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()

    plist = t.plist.copy()
    plist[len(plist) // 3] = 0xffffffff
    out = torch.empty((t.n, 4), dtype=torch.float32, device="cuda")
    keep = [dev(t.points), dev(t.groups), dev(t.ptr[0]), dev(plist)]
    p = gc.Problem()
    p.nbodies, p.ncells, p.ngroups, p.eps2, p.quad_phi_sign = t.n, t.ncells, t.ngroups, 1e-4, 1.0
    p.points, p.groups, p.pptr, p.plist = (k.data_ptr() for k in keep)
    torch.cuda.synchronize()
    with pytest.raises(gc.GravError, match="device error word 0x2"):
        gc.check(gc.lib().grav_groups_eval_dev_CUDA(ctypes.byref(p), out.data_ptr(), None))
