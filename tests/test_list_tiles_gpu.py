"""GPU: the list kernels at the edges of their tiles (64, 128 and 256
records, two, four or eight per lane) and of their sink blocks (four sinks,
remainders of one to three), against the FP64 evaluation of the same lists.

Tolerance: an interaction is at most ~30 dependent FP32 roundings of 6e-8 on
moments stored in FP32, so a list of one entry is off by 2e-6 at worst and
longer ones by less."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 2e-6
LENGTHS = [0, 1, 2, 31, 63, 64, 65, 127, 128, 129, 192, 255, 256, 257, 511, 513]
COUNTS = [1, 2, 3, 4, 5, 6, 7, 8, 15, 16, 17, 29, 30, 31, 32]


def _tree(kind, box):
    """A walked tree with its groups and lists replaced: every list length of
    LENGTHS against every sink count of COUNTS, entries well away from their
    group (the list's own kind only)."""
    from pgrav import host, ics
    from pgrav.host import GROUP_DTYPE
    rng = np.random.default_rng(17 + kind)
    n = len(LENGTHS) * sum(COUNTS)
    pos = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    m = rng.uniform(0.5, 1.5, n).astype(np.float32) / n
    t = host.Tree(pos, m, box=box, leaf_max=16, group_max=32, p2cut=7, p4cut=20, tol=1e-4)
    x = t.sorted_pos.astype(np.float64)
    ng = len(LENGTHS) * len(COUNTS)
    groups = np.zeros(ng, GROUP_DTYPE)
    groups["count"] = np.tile(COUNTS, len(LENGTHS))
    groups["first"] = np.concatenate([[0], np.cumsum(groups["count"])[:-1]])
    cells = np.nonzero(t.hcells["R"] < 0.2)[0]
    lists, ptr = [], [0]
    for g in range(ng):
        f, c = groups["first"][g], groups["count"][g]
        groups["cen"][g] = x[f:f + c].mean(0)
        groups["radius"][g] = np.linalg.norm(x[f:f + c] - groups["cen"][g], axis=1).max() + 1e-6
        d = t.hcells["cen"][cells][:, None] - x[None, f:f + c]
        far = np.linalg.norm(d, axis=2).min(1) > 2.5 * t.hcells["R"][cells]
        pick = rng.choice(cells[far], LENGTHS[g // len(COUNTS)])
        if kind == 0:  # cell monopoles, and bodies for every other entry
            e = pick + t.n
            e[::2] = rng.integers(0, t.n, len(e[::2]))
        else:
            e = pick
        code = rng.integers(0, 27, len(e)) if box > 0 else np.full(len(e), 13)
        lists.append((e.astype(np.uint32) | (code.astype(np.uint32) << 27)))
        ptr.append(ptr[-1] + len(e))
    none = np.zeros(ng + 1, np.int64)
    t.groups, t.ngroups = groups, ng
    t.ptr = [np.array(ptr, np.int64) if k == kind else none for k in range(3)] + [none]
    full = np.concatenate(lists)
    t.plist, t.qlist, t.hlist = (full if k == kind else np.zeros(0, np.uint32) for k in range(3))
    t.clist = np.zeros(0, np.uint32)
    return t


def _eval(t, sign=1.0):
    from pgrav import gravcuda as gc
    plan = gc.Plan(t, 1e-4, quad_phi_sign=sign)
    plan.eval()
    out = plan.download()
    plan.free()
    return out


@pytest.mark.parametrize("box", [0.0, 1.0])
@pytest.mark.parametrize("kind", [0, 1, 2], ids=["points", "quadrupole", "order4"])
def test_tile_and_sink_edges(kind, box):
    t = _tree(kind, box)
    got = _eval(t)
    if kind == 0:  # a monopole entry carries its cell's mass at its centre
        b = t.points.astype(np.float64)
        b[t.n:, :3] = t.hcells["cen"]
        want = np.zeros((t.n, 4))
        for g in range(t.ngroups):
            e = t.plist[t.ptr[0][g]:t.ptr[0][g + 1]]
            s = b[e & (2 ** 27 - 1)]
            c = (e >> 27).astype(np.int64)
            s = s + np.stack([(c // 9 - 1) * box, (c // 3 % 3 - 1) * box, (c % 3 - 1) * box, 0 * c], 1)
            f, n = t.groups["first"][g], t.groups["count"][g]
            d = b[f:f + n, None, :3] - s[None, :, :3]
            r = 1 / np.sqrt((d * d).sum(-1) + 1e-4)
            want[f:f + n, :3] = -(s[None, :, 3:] * d * r[..., None] ** 3).sum(1)
            want[f:f + n, 3] = -(s[None, :, 3] * r).sum(1)
    else:
        want = O.ListsFP64(t, ewald=False).eval(t.sorted_pos, t.points[:t.n, 3], 1e-4)
    for k in range(len(LENGTHS)):  # every length by itself
        g = slice(k * len(COUNTS), (k + 1) * len(COUNTS))
        f = t.groups["first"][g]
        i = slice(f[0], f[-1] + t.groups["count"][g][-1])
        for cols in (slice(0, 3), slice(3, 4)):
            off = np.linalg.norm(got[i, cols] - want[i, cols])
            assert off <= TOL * np.linalg.norm(want[i, cols]), (LENGTHS[k], cols, off)


def test_order4_quadrupole_potential_sign():
    """quad_phi_sign = -1 turns the quadrupole potential around in the order-4
    kernel as in the quadrupole kernel, on the same cells, and nothing else."""
    h = _tree(2, 0.0)
    plus, minus = _eval(h), _eval(h, -1.0)
    h.qlist, h.hlist, h.ptr = h.hlist, h.qlist, [h.ptr[0], h.ptr[2], h.ptr[1], h.ptr[3]]
    qplus, qminus = _eval(h), _eval(h, -1.0)
    assert np.array_equal(plus[:, :3], minus[:, :3])
    assert np.abs((minus - plus)[:, 3] - (qminus - qplus)[:, 3]).max() <= TOL * np.abs(plus[:, 3]).max()
