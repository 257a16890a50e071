"""GPU: a drop-in list read in place from page-locked memory and one copied
to the device give the oracle's sums on both sides of each limit of the rule
(128 KiB of list, 256 sinks), and back to back on one slot, whose staging
buffers the in-place kernels still read."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
RMS_TOL = 1e-5  # the drop-in parity bar


def _records(kind, n, rng):
    sz = O.KIND_SZ[kind]
    rec = np.zeros((n, sz), np.float32)
    rec[:, 0] = rng.uniform(0.5, 1.5, n)
    rec[:, 1:4] = rng.normal(0, 1, (n, 3)) + 4.0
    if sz > 4:
        rec[:, 4] = 0.5
        rec[:, 8:] = rng.normal(0, 0.1, (n, sz - 8))
    return rec


@pytest.mark.parametrize("nsink", [1, 256, 257])
@pytest.mark.parametrize("routine,kind,nsrc", [
    ("pMp", O.MONO_PLUMMER, 8), ("pMp", O.MONO_PLUMMER, 8192), ("pMp", O.MONO_PLUMMER, 8200),
    ("pQp", O.QUAD_PLUMMER, 2520), ("pQp", O.QUAD_PLUMMER, 2528), ("pHp", O.HEXA_PLUMMER, 1136)])
def test_in_place_and_copied_lists(routine, kind, nsrc, nsink):
    from pgrav import gravcuda as gc
    rng = np.random.default_rng(nsrc + nsink)
    sinks = rng.normal(0, 0.3, (nsink, 3)).astype(np.float32)
    d = gc.DropIn(gc.body_table(sinks, 1.0))
    want = np.zeros((nsink, 4))
    look = sorted({0, nsink // 2, nsink - 1})
    for _ in range(3):  # the slot's two staging buffers, and one of them again
        f, nblk = O.pack_aosoa(_records(kind, nsrc, rng))
        p = d.btab.ctypes.data
        gc.lib().grav_mn_CUDA(routine.encode(), p, None, nsink, gc.BODY_STRIDE, f.ctypes.data, nblk * 8,
                              O.KIND_SZ[kind], 1e-4, None, 5)
        gc.check()
        for i in look:
            want[i] += O.list_eval(kind, f, nblk, sinks[i], 1e-4)
        f[:] = np.nan  # the list is the caller's again
    got = d.terminate()
    for i in look:
        assert np.linalg.norm(got[i, :3] - want[i, :3]) <= RMS_TOL * np.linalg.norm(want[i, :3])
        assert abs(got[i, 3] - want[i, 3]) <= RMS_TOL * abs(want[i, 3])
