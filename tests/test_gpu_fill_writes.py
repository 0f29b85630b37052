"""The steps' one-launch ghost fill after every entry point that writes fields
between steps, on periodic axes of one and two cells (whose fills read ghosts):
the runs must leave, ghosts included, what runs leave whose fills all went axis
by axis, which setting a stage of the face field before each step asks for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WRITES = {
    "init_bfield": lambda d: d.initialize_bfield_from_q(),
    "bound": lambda d: (d.bound(0), d.bound_bfield(0)),
    "prot": lambda d: d.prot(0),
    "sweep_fluxct": lambda d: (d.sweep(0 if d.params.nx > 1 else 1, 1e-4), d.fluxct(1, 1.0, 0.0)),
    "state": lambda d: d.set_state(d.get_state(0) * 1.0),
    "stage": lambda d: d.set_state(d.get_state(2), stage=3),
}


@pytest.mark.parametrize("write", WRITES)
@pytest.mark.parametrize("n,bc", [((9, 7, 1), "ppp"), ((1, 9, 7), "ppp"), ((6, 2, 5), "pop"), ((1, 12, 1), "ppp"),
                                  ((12, 1, 1), "ppp")],
                         ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_writes_between_steps(n, bc, write):
    import how_mhd as hm
    bcs = ["open" if c == "o" else "periodic" for c in bc]
    p = hm.make_parameters(nx=n[0], ny=n[1], nz=n[2], nt=1, tend=10.0, gam=5.0 / 3.0, cour=0.3,
                           problem="uniform", x1bc=bcs[0], x2bc=bcs[1], x3bc=bcs[2])
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
            t, seen = 0.0, []
            for step in range(9):
                if axis_passes:
                    d.set_face_b(*d.get_face_b(5), stage=5)
                if step in (3, 4, 7):
                    WRITES[write](d)
                t, _, _ = d.run(t, 1)
                seen += [d.get_state(0), *d.get_face_b(0)]
            out.append(seen)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
