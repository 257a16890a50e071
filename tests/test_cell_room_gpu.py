"""GPU: trees on either side of the room that the builder first makes for
cells, 1024 + 7 n / leaf_max (2 n at most), against the host builder."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tight_pairs(n, seed):
    """n / 2 pairs closer than the keys' last levels resolve on the way down: long chains."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0, 1, (n // 2, 3))
    return np.concatenate([a, a + rng.uniform(-1, 1, a.shape) * 1e-5]).astype(np.float32)


@pytest.mark.parametrize("n,leaf_max,over", [(600, 1, 1), (3000, 1, 1), (200, 1, 1), (150, 1, 0), (8000, 16, 0)])
def test_trees_that_need_more_room(n, leaf_max, over):
    from pgrav import gravcuda as gc, host
    pos = tight_pairs(n, n)
    m = np.random.default_rng(n + 1).uniform(0.5, 1.5, n).astype(np.float32)
    kw = dict(leaf_max=leaf_max, group_max=32, p2cut=4, p4cut=12, tol=1e-3)
    t = host.Tree(pos, m, **kw)
    room, tries = 1024 + min(2 * n, 7 * n // leaf_max), 0
    while t.ncells > room:
        room, tries = 4 * room, tries + 1
    assert tries == over
    gp = gc.Plan.build(pos, m, 1e-4, **kw)
    pr = gp.problem()
    gp.free()
    assert np.array_equal(pr["groups"].view(np.uint8), t.groups.view(np.uint8))
    for k, want in enumerate((t.plist, t.qlist, t.hlist)):
        assert np.array_equal(pr["ptr"][k], t.ptr[k])
        assert np.array_equal(pr["lists"][k], want)
