"""The routing pass of x sweeps at every length of its runs: a warp takes
`run` segments of 32 faces in a row, as long as every warp of a full chip has a
run.  The y pass walks its lines by another kernel, so the same state with its
axes rotated (x -> y, y -> z, z -> x) has to get the same decisions: the same
number of full and cheap faces, and the same sweep result up to the rounding of
the update's two forms (FP64: some 1e-16 of the largest value, held to 1e-12; one
face decided otherwise moves its cells by the WENO weights' departure times
dt/dx, 1e-6 and more in the noisy half)."""
import numpy as np
import pytest

from howtest import active

pytestmark = pytest.mark.gpu

# (lines' segments and the run at 148 SMs: 2 of 1, 8 of 2, 5 of 3 + 2, 4 of 4, 8 of 4)
SIZES = [(33, 9, 8), (230, 48, 30), (150, 60, 60), (100, 72, 72), (255, 56, 44)]


def _params(hm, n, **kw):
    return hm.make_parameters(nx=n[0], ny=n[1], nz=n[2], nt=1, tend=10.0, gam=5.0 / 3.0, cour=0.4, rhomin=1e-6,
                              pgmin=1e-6, problem="mpi_smooth3d", x1bc="periodic", x2bc="periodic",
                              x3bc="periodic", **kw)


@pytest.mark.parametrize("n", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
def test_x_decisions_equal_rotated_y(n):
    import how_mhd as hm
    q = hm.problem_state(_params(hm, n))   # smooth, with rough cells in one half
    rough = active(q, *n)[:, n[0] // 2:]
    rough *= 1.0 + 0.01 * np.random.default_rng(sum(n)).standard_normal(rough.shape)
    qa = np.array(active(q, *n))
    nr = (n[2], n[0], n[1])
    comp = [0, 3, 1, 2, 6, 4, 5, 7]                      # rotated (x, y, z) = old (z, x, y)
    qr = np.zeros((8,) + tuple(m + 6 for m in nr))
    active(qr, *nr)[...] = qa[comp].transpose(0, 3, 1, 2)
    out = []
    for m, state, d_sweep in ((n, q, 0), (nr, qr, 1)):
        with hm.Domain(_params(hm, m, router="on")) as d:
            d.set_state(state)
            d.bound(0)
            d.initialize_bfield_from_q()
            d.router_stats(reset=True)
            d.sweep(d_sweep, 1e-3)
            out.append((d.router_stats(), np.array(active(d.get_state(1), *m))))
    (sx, x), (sy, y) = out
    assert sx == sy and sx[0] > 0, (sx, sy)
    if n[0] >= 100:   # (33 cells do not resolve the smooth half: every face is full there)
        assert sx[1] > 0, sx
    back = y.transpose(0, 2, 3, 1)[[0, 2, 3, 1, 5, 6, 4, 7]]
    assert np.abs(x - back).max() <= 1e-12 * np.abs(x).max()
