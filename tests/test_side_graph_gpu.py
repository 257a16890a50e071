"""GPU: the periodic correction on a side stream inside a captured step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_side_stream_moments_in_a_captured_step():
    """The fork and the join of the side stream are captured with the step:
    replayed steps give the eager steps' positions and velocities, and those
    of the moments on the evaluation's own stream, bit for bit."""
    from pgrav import gravcuda as gc, ics
    from pgrav.step import Stepper
    pos, m = ics.grf_box(16, seed=9, rms_disp=0.25)
    vel = np.random.default_rng(9).normal(0, 0.01, pos.shape)
    out = []
    for graph, side in ((False, -2), (False, 2), (True, 2), (True, -2)):
        st = Stepper(pos, vel, m, (1.0 / 16 / 50) ** 2, box=1.0, rebuild=100, graph=graph,
                     tree_kw=dict(tol=1e-4, p2cut=7, p4cut=20))
        st.plan.retune(gc.Tuning(8, 0, 0, 0, 0, 0, side))
        st.run(4, 1e-3)
        out.append(st.state())
        st.free()
    for x, v in out[1:]:
        assert np.array_equal(x, out[0][0]) and np.array_equal(v, out[0][1])
