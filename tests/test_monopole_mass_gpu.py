"""GPU: a cell monopole's mass is the point table's, also where the cell tables
carry another one, in every entry that takes a problem, and after a refit, which
makes the two the same again."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p2cut,p4cut", [(7, 0), (7, 20), (0, 8)], ids=["quadrupole", "both", "order4"])
def test_point_table_masses_count(p2cut, p4cut):
    import torch
    from pgrav import gravcuda as gc, host, ics
    pos, m = ics.plummer(4000, seed=8)
    t = host.Tree(pos, m, leaf_max=16, group_max=32, p2cut=p2cut, p4cut=p4cut, tol=1e-3)
    plain = gc.Plan(t, 1e-4)
    plain.eval()
    same = plain.download()
    plain.free()
    assert (t.plist & 0x7ffffff >= t.n).any()
    t.points[t.n:, 3] *= np.float32(1.5)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()

    # the no-allocation entry reads nothing but the point table for its monopoles
    keep = [dev(a) for a in (t.points, t.qcells, t.hcells, t.groups, *t.ptr[:3], t.plist,
                             t.qlist if len(t.qlist) else np.zeros(1, np.uint32),
                             t.hlist if len(t.hlist) else np.zeros(1, np.uint32))]
    p = gc.Problem()
    p.nbodies, p.ncells, p.ngroups, p.eps2, p.quad_phi_sign = t.n, t.ncells, t.ngroups, 1e-4, 1.0
    (p.points, p.qcells, p.hcells, p.groups, p.pptr, p.qptr, p.hptr, p.plist, p.qlist,
     p.hlist) = (k.data_ptr() for k in keep)
    out = torch.empty((t.n, 4), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    gc.check(gc.lib().grav_groups_eval_dev_CUDA(ctypes.byref(p), out.data_ptr(), None))
    want = out.cpu().numpy()
    assert np.abs(want - same).max() > 1e-2 * np.abs(same).max()
    # its monopole centres are FP32: 1e-6 of a unit sphere's forces
    bound = 2e-6 * np.abs(want).max()
    plan = gc.Plan(t, 1e-4)
    plan.eval()
    assert np.abs(plan.download() - want).max() < bound
    got = gc.groups_eval_problem(gc.pinned_problem(t), 1e-4, 0.0)
    assert np.abs(got - want).max() < bound
    plan.set_tree(t)
    plan.refit()
    plan.eval()
    # a refit's moments are the bodies' (sums of children: another rounding)
    assert np.abs(plan.download() - same).max() < 1e-5 * np.abs(same).max()
    plan.free()
