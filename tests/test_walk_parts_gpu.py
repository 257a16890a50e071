"""GPU: wide groups walked in parts, one per child of the root, in a periodic
box, against the host walk entry for entry: groups that open a root spanning
the box, and groups that take the root itself into their correction list, so
that one part writes that entry and every part's first cell is covered."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = 2.5
CASES = [("spread", 2000, dict()), ("spread", 6000, dict(leaf_max=1)),
         ("spread", 6000, dict(ewald_theta=0.6)),
         ("compact", 20000, dict(ewald_theta=0.6)), ("compact", 20000, dict(ewald_theta=0.6, leaf_max=1))]


def bodies(kind, n):
    """A clump, and one body in fifty about it: over the whole box, or near enough for the
    root to count whole in the correction."""
    rng, k = np.random.default_rng(n), n // 50
    lo, hi, s = (0.0, 1.0, 0.004) if kind == "spread" else (0.42, 0.58, 0.003)
    x = np.concatenate([rng.normal(0.5, s, (n - k, 3)), rng.uniform(lo, hi, (k, 3))])
    return (np.clip(x, 0, 0.999) * BOX).astype(np.float32), rng.uniform(0.5, 1.5, n).astype(np.float32)


@pytest.mark.parametrize("kind,n,kw", CASES, ids=[f"{k}-{n}-{i}" for i, (k, n, _) in enumerate(CASES)])
def test_parts_of_a_periodic_walk_equal_the_host_walk(kind, n, kw):
    from pgrav import gravcuda as gc, host
    pos, m = bodies(kind, n)
    kw = dict(dict(p2cut=4, p4cut=12, tol=1e-3), **kw)
    t = host.Tree(pos, m, box=BOX, **kw)
    # the parts are used (the builder's rule), and on the case that they are tested for
    wide = np.flatnonzero(t.groups["radius"] >= BOX / 16)
    assert 0 < 4 * len(wide) <= len(t.groups)
    root = [int((t.clist[t.ptr[3][g]:t.ptr[3][g + 1]] & 0x7ffffff == t.n).sum()) for g in wide]
    assert root == [int(kind == "compact")] * len(wide)
    gp = gc.Plan.build(pos, m, 1e-4, box=BOX, ewald=True, **kw)
    pr = gp.problem()
    gp.free()
    assert np.array_equal(pr["groups"].view(np.uint8), t.groups.view(np.uint8))
    for k, want in enumerate((t.plist, t.qlist, t.hlist, t.clist)):
        assert np.array_equal(pr["ptr"][k], t.ptr[k])
        assert np.array_equal(pr["lists"][k], want)
