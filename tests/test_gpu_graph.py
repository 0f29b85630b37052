"""The step as a CUDA graph (from the ninth step with each buffer role on) must
leave what the same launches leave one by one: a run of 40 steps against the
same run with the graph kept from forming (a precision change and back before
every second step resets it), bit for bit, and across a change of precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,problem", [((48, 1, 1), "brio_wu"), ((24, 20, 1), "orszag_tang"), ((12, 10, 9), "blast3d_b")],
                         ids=["1d", "2d", "3d"])
def test_graph_steps_equal_launched_steps(n, problem):
    import how_mhd as hm
    bc = "open" if problem == "brio_wu" else "periodic"
    p = hm.make_parameters(nx=n[0], ny=n[1], nz=n[2], nt=1, tend=10.0, gam=5.0 / 3.0, cour=0.4, problem=problem,
                           rhomin=1e-6, pgmin=1e-6, x1bc=bc, x2bc=bc, x3bc=bc)
    out = []
    for launched in (False, True):
        with hm.Domain(p) as d:
            d.init_problem()
            t = 0.0
            for block in range(20):
                if launched:      # a mixed step with each buffer role forgets the graphs
                    q, b = d.get_state(0), d.get_face_b(0)
                    d.set_precision("mixed")
                    d.ssprk(1e-9)
                    d.ssprk(1e-9)
                    d.set_precision("fp64")
                    d.set_state(q)
                    d.set_face_b(*b)
                t, s, _ = d.run(t, 2)
            for prec in ("mixed", "fp64"):
                d.set_precision(prec)
                t, s, _ = d.run(t, 3)
            out.append([t, d.get_state(0)[:, 3:-3, 3:-3, 3:-3], *[x[3:-3, 3:-3, 3:-3] for x in d.get_face_b(0)]])
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(a, b)
