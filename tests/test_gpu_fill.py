"""The steps' one-launch ghost fill (k_fill_ghosts) against the axis-by-axis
fill restated here, bit for bit, on the state and face B that four steps leave:
every axis extent the fill treats on its own (1, 2 open, 3 and more), periodic
and open.  A periodic axis of one cell keeps two ghost layers of earlier steps
(its fill reads ghosts); those are compared with a run whose fills all went axis
by axis, which setting a stage of the face field before each step asks for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fill(a, n, bc):
    """In place on (..., n0+6, n1+6, n2+6); collapsed periodic axes: layers 2, 4, 5, 6."""
    for ax in range(3):
        b = np.moveaxis(a, a.ndim - 3 + ax, 0)
        m = n[ax]
        if bc[ax] == "open":
            src = [3] * 3 + [m + 2] * 3
        elif m == 1:
            b[2], b[4], b[5], b[6] = b[3], b[3], b[3], b[3]
            continue
        else:
            src = [m, m + 1, m + 2, 3, 4, 5]
        for d, s in zip([0, 1, 2, m + 3, m + 4, m + 5], src):
            b[d] = b[s]
    return a


@pytest.mark.parametrize("n,bc", [((5, 4, 3), "ppp"), ((9, 7, 1), "ppp"), ((9, 7, 1), "opo"), ((12, 1, 1), "ppp"),
                                  ((12, 1, 1), "opp"), ((7, 1, 5), "ppo"), ((6, 2, 5), "pop"), ((33, 3, 4), "oop")],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_steps_fill_as_the_axis_passes(n, bc):
    import how_mhd as hm
    bcs = ["open" if c == "o" else "periodic" for c in bc]
    p = hm.make_parameters(nx=n[0], ny=n[1], nz=n[2], nt=1, tend=10.0, gam=5.0 / 3.0, cour=0.3,
                           problem="uniform", x1bc=bcs[0], x2bc=bcs[1], x3bc=bcs[2])
    # (a uniform field: a 2-D run of the method with a varying out-of-plane B blows up)
    q = hm.problem_state(p)
    rng = np.random.default_rng(sum(n))
    for v, amp in ((0, 0.05), (1, 0.02), (2, 0.02), (3, 0.02)):
        a = q[v, 3:n[0] + 3, 3:n[1] + 3, 3:n[2] + 3]
        a += amp * rng.standard_normal(a.shape)
    out = []
    for axis_passes in (False, True):
        with hm.Domain(p) as d:
            d.set_state(q)
            d.bound(0)
            d.initialize_bfield_from_q()
            t = 0.0
            for _ in range(6):
                if axis_passes:
                    d.set_face_b(*d.get_face_b(5), stage=5)
                t, _, _ = d.run(t, 1)
            out.append([d.get_state(0), *d.get_face_b(0)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(a, _fill(a.copy(), n, bcs))
