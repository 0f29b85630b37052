"""The sweep kernel at the edges of its work items: a warp marches NL = 4 lines
in chunks of 8 cells, a launch cuts the lines into segments of whole chunks.
Sizes around one and two chunks and one and two line groups, each axis swept
and open or periodic, against the CPU oracle under the parity suite's bar
(relative L1 <= 1e-12 per conserved variable), with some cells below the
density and pressure floors in every run (the floors' own branch)."""
import numpy as np
import pytest

from howtest import CPUOracle, active, rel_l1

pytestmark = pytest.mark.gpu

SIZES = [(4, 4, 2), (5, 9, 3), (6, 7, 8), (7, 6, 9), (8, 8, 8), (9, 5, 14), (13, 15, 16),
         (14, 17, 7), (15, 31, 4), (16, 33, 6), (31, 3, 17), (33, 13, 15), (7, 1, 1), (9, 1, 1), (30, 1, 1), (8, 7, 1),
         (17, 30, 1), (61, 4, 1), (12, 1, 9), (1, 10, 9)]


@pytest.mark.parametrize("n", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
@pytest.mark.parametrize("mode", ["fp64", "all_full"])
def test_step_vs_oracle(n, mode):
    import how_mhd as hm
    import router_ref as rr
    bc = ("periodic", "open", "periodic") if sum(n) % 2 else ("open", "periodic", "open")
    p = hm.make_parameters(nx=n[0], ny=n[1], nz=n[2], nt=1, tend=10.0, gam=5.0 / 3.0, cour=0.4, rhomin=0.9,
                           pgmin=0.9, problem="mpi_smooth3d", x1bc=bc[0], x2bc=bc[1], x3bc=bc[2])
    q = hm.problem_state(p)
    rng = np.random.default_rng(100 + sum(n))
    a = active(q, *n)
    a *= 1.0 + 0.03 * rng.standard_normal(a.shape)
    low = rng.random(a.shape[1:]) < 0.1
    a[0][low] *= 0.85                 # below rhomin
    a[7][rng.random(a.shape[1:]) < 0.1] *= 0.85   # pressure below pgmin
    o = CPUOracle(*n, bc=bc, gam=5.0 / 3.0, rhomin=0.9, pgmin=0.9)
    o.set_state(q)
    rc, t, dts = o.run(10.0, 1, 2)
    with hm.Domain(p) as d:
        if mode == "all_full":        # the routed kernel with every face sent to full WENO
            d.set_router(rr.init_weights(0), "learned", threshold=-1e30)
        d.set_state(q)
        d.bound(0)
        d.initialize_bfield_from_q()
        t2, s, dts2 = d.run(0.0, 2, dts_cap=2)
        got = active(d.get_state(0), *n)
    np.testing.assert_allclose(dts2, dts, rtol=1e-13)
    err = rel_l1(got, active(o.get_q(0), *n))
    assert np.all(err <= 1e-12), err
