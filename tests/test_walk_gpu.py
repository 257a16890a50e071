"""GPU: the warp-per-group walk at the sizes where its stack and its ordered
emission can go wrong, against the host walk (nln_walk_group), entry for
entry: single bodies, one round and one lane more, leaves longer than a warp,
one-body leaves (deep stacks), leaves whose bodies take their own images, and
correction lists with and without whole cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [
    (1, 0.0, dict(leaf_max=16, group_max=32)),
    (2, 0.0, dict(leaf_max=1, group_max=1)),
    (33, 0.0, dict(leaf_max=1, group_max=32)),
    (4097, 0.0, dict(leaf_max=1, group_max=7, tol=1e-7)),
    (3001, 0.0, dict(leaf_max=700, group_max=32)),
    (1, 2.5, dict(leaf_max=16, group_max=32)),
    (200, 2.5, dict(leaf_max=64, group_max=32)),          # leaves beyond the correction's domain
    (1777, 2.5, dict(leaf_max=1, group_max=32, tol=1e-6)),
    (3001, 2.5, dict(leaf_max=40, group_max=32, ewald_theta=0.0)),
    (3001, 2.5, dict(leaf_max=40, group_max=32, ewald_theta=0.6)),
]


@pytest.mark.parametrize("n,box,kw", EDGES, ids=[f"{n}-{b}-{i}" for i, (n, b, _) in enumerate(EDGES)])
def test_device_walk_equals_host_walk(n, box, kw):
    from pgrav import gravcuda as gc, host
    rng = np.random.default_rng(n)
    pos = rng.normal(0, 1, (n, 3)) ** 3 if box == 0 else rng.uniform(0, box, (n, 3)) * rng.uniform(0, 1, (n, 1))
    pos = pos.astype(np.float32)
    m = rng.uniform(0.5, 1.5, n).astype(np.float32)
    kw = dict(dict(p2cut=4, p4cut=12, tol=1e-3), **kw)
    t = host.Tree(pos, m, box=box, **kw)
    gp = gc.Plan.build(pos, m, 1e-4, box=box, ewald=box > 0, **kw)
    pr = gp.problem()
    gp.free()
    assert np.array_equal(pr["groups"].view(np.uint8), t.groups.view(np.uint8))
    for k, want in enumerate((t.plist, t.qlist, t.hlist, t.clist)):
        if k == 3 and box == 0:
            continue
        assert np.array_equal(pr["ptr"][k], t.ptr[k])
        assert np.array_equal(pr["lists"][k], want)
