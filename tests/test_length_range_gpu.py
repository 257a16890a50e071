"""GPU: the unit of length does not matter.  A system whose lengths are scaled
by a power of two gives the same forces, scaled, bit for bit, over eleven
decades, through every entry; the order-4 terms, whose largest intermediates go
as the eighth power of a length, among them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def evaluate(j):
    """acc and phi of the sphere scaled by 2^j, brought back to the unscaled one's units."""
    import torch
    from pgrav import gravcuda as gc, host, ics
    s = 2.0 ** j
    pos, m = ics.plummer(2000, seed=4)
    pos = (pos * np.float32(s)).astype(np.float32)
    m = (m * np.float32(2000)).astype(np.float32)  # unit masses
    kw = dict(leaf_max=8, group_max=32, p2cut=0, p4cut=8, tol=1.0 / s / s)
    eps2 = (0.01 * s) ** 2
    t = host.Tree(pos, m, **kw)
    assert len(t.hlist) > 1000
    out = []
    plan = gc.Plan(t, eps2)
    plan.eval()
    out.append(plan.download())
    plan.free()
    out.append(gc.groups_eval_problem(gc.pinned_problem(t), eps2, 0.0).copy())
    built = gc.Plan.build(pos, m, eps2, **kw)
    built.eval()
    out.append(built.download())
    built.free()
    keep = [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
            for a in (t.points, t.hcells, t.groups, t.ptr[0], t.ptr[2], t.plist, t.hlist)]
    p = gc.Problem()
    p.nbodies, p.ncells, p.ngroups, p.eps2, p.quad_phi_sign = t.n, t.ncells, t.ngroups, eps2, 1.0
    p.points, p.hcells, p.groups, p.pptr, p.hptr, p.plist, p.hlist = (k.data_ptr() for k in keep)
    dev = torch.empty((t.n, 4), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    gc.check(gc.lib().grav_groups_eval_dev_CUDA(ctypes.byref(p), dev.data_ptr(), None))
    out.append(dev.cpu().numpy())
    return [np.concatenate([f[:, :3].astype(np.float64) * s * s, f[:, 3:].astype(np.float64) * s], 1)
            for f in out]


@pytest.mark.parametrize("j", [-20, -10, 10, 17])
def test_forces_do_not_depend_on_the_unit_of_length(j):
    for a, b in zip(evaluate(j), evaluate(0)):
        assert np.isfinite(a).all()
        assert np.array_equal(a, b)
