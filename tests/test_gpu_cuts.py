"""The sweeps however their lines are cut: segments of one and of many chunks, a
shorter last one, warps that take several items, one and four lines per warp, 8
and 12 warps per SM, all precisions and routing modes.  The arithmetic is the
same in every form, so the results are, bit for bit: an x sweep against the y
sweep of the rotated state, whole domains against z slabs (whose sweeps are cut
otherwise) and against ensemble members at each of its shapes; and two steps at
such sizes against the CPU oracle under the parity suite's bar (relative L1
<= 1e-12, dt within 1e-13)."""
import numpy as np
import pytest

from howtest import CPUOracle, active, rel_l1

pytestmark = pytest.mark.gpu

# (at 148 SMs; chunks per item and items per quarter of an SM of the FP64 x sweep)
SIZES = [(33, 1, 9),       # one line per warp: 1 and 1
         (5000, 1, 1),     # 1 and 1
         (300, 1, 140),    # 1 and 3
         (2500, 1, 40),    # 2 and 3 (routed: 3 and 2), a shorter last segment
         (90, 2, 1100),    # 3 and 4
         (130, 3, 500),    # 5 and 3
         (33, 4, 9),       # four lines per warp: 1 and 1
         (5, 5, 40),       # 1 and 1
         (40, 37, 35),     # 2 and 2
         (107, 75, 53)]    # 3 and 9 (routed: 14 and 2), a shorter last segment


def _params(hm, n, bc=("periodic",) * 3, **kw):
    return hm.make_parameters(nx=n[0], ny=n[1], nz=n[2], nt=1, tend=10.0, gam=5.0 / 3.0, cour=0.4, rhomin=0.9,
                              pgmin=0.9, problem="mpi_smooth3d", x1bc=bc[0], x2bc=bc[1], x3bc=bc[2], **kw)


def _state(hm, n):
    """Smooth, with noise in one half and some cells below the floors there."""
    q = hm.problem_state(_params(hm, n))
    rng = np.random.default_rng(sum(n))
    a = active(q, *n)[:, n[0] // 2:]
    a *= 1.0 + 0.03 * rng.standard_normal(a.shape)
    a[0][rng.random(a.shape[1:]) < 0.1] *= 0.85
    a[7][rng.random(a.shape[1:]) < 0.1] *= 0.85
    return q


@pytest.mark.parametrize("mode", ["fp64", "mixed", "fp64-guard", "mixed-guard", "label"])
@pytest.mark.parametrize("n", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
def test_x_sweep_equals_rotated_y_sweep(n, mode):
    import how_mhd as hm
    q = _state(hm, n)
    nr = (n[2], n[0], n[1])                              # rotated (x, y, z) = old (z, x, y)
    qr = np.zeros((8,) + tuple(m + 6 for m in nr))
    active(qr, *nr)[...] = active(q, *n)[[0, 3, 1, 2, 6, 4, 5, 7]].transpose(0, 3, 1, 2)
    out = []
    for m, state, direction, ct in ((n, q, 0, (0, 1)), (nr, qr, 1, (3, 2))):
        with hm.Domain(_params(hm, m, precision="mixed" if "mixed" in mode else "fp64")) as d:
            if "guard" in mode:
                d.set_router(None, "guard")
            d.set_state(state)
            d.bound(0)
            d.initialize_bfield_from_q()
            if mode == "label":
                d.collect_begin(1000, 100)
            d.sweep(direction, 1e-3)
            s = np.array(active(d.get_state(1), *m))
            c = [d.get_ct_array(k) for k in ct]
            if direction == 0:
                out.append([s, *(x[2:m[0] + 3, 3:m[1] + 3, 3:m[2] + 3] for x in c)])
            else:
                out.append([s.transpose(0, 2, 3, 1)[[0, 2, 3, 1, 5, 6, 4, 7]],
                            *(x[3:m[0] + 3, 2:m[1] + 3, 3:m[2] + 3].transpose(1, 2, 0) for x in c)])
    for x, y in zip(*out):
        assert np.isfinite(x).all()
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [(40, 37, 35), (107, 30, 53)], ids=["40x37x35", "107x30x53"])
def test_slabs_equal_the_whole(n, precision):
    import how_mhd as hm
    p = _params(hm, n, precision=precision)
    q = _state(hm, n)
    with hm.Domain(p) as d:
        d.set_state(q)
        d.bound(0)
        d.initialize_bfield_from_q()
        t, _, _ = d.run(0.0, 2)
        want = active(d.get_state(0), *n)
    for parts in (2, 5):
        with hm.Group(p, parts) as g:
            g.set_state(q)
            assert g.run(0.0, 2)[0] == t
            np.testing.assert_array_equal(active(g.get_state(), *n), want)


def test_ensemble_shapes_equal_the_whole():
    import how_mhd as hm
    sizes = [(5000, 1, 1), (107, 75, 1), (40, 37, 35)]
    params, want = [_params(hm, n) for n in sizes], []
    for p in params:
        with hm.Domain(p) as d:
            d.init_problem()
            d.run(0.0, 2)
            want.append(d.get_state(0))
    for shape in range(3):
        with hm.Ensemble(params) as e:
            e.init()
            e.set_shapes(shape, shape, shape)
            e.run(2)
            for m, w in enumerate(want):
                np.testing.assert_array_equal(e.members[m].get_state(0), w)


@pytest.mark.parametrize("mode", ["fp64", "all_full"])
@pytest.mark.parametrize("n", [(5000, 1, 1), (300, 1, 40), (40, 37, 35), (107, 75, 53)],
                         ids=lambda n: "x".join(map(str, n)))
def test_steps_vs_oracle(n, mode):
    import how_mhd as hm
    import router_ref as rr
    bc = ("periodic", "open", "periodic") if n[0] % 2 else ("open", "periodic", "open")
    p = _params(hm, n, bc)
    q = _state(hm, n)
    o = CPUOracle(*n, bc=bc, gam=5.0 / 3.0, rhomin=0.9, pgmin=0.9)
    o.set_state(q)
    rc, t, dts = o.run(10.0, 1, 2)
    with hm.Domain(p) as d:
        if mode == "all_full":        # the routed kernel with every face sent to full WENO
            d.set_router(rr.init_weights(0), "learned", threshold=-1e30)
        d.set_state(q)
        d.bound(0)
        d.initialize_bfield_from_q()
        _, _, dts2 = d.run(0.0, 2, dts_cap=2)
        got = active(d.get_state(0), *n)
    np.testing.assert_allclose(dts2, dts, rtol=1e-13)
    err = rel_l1(got, active(o.get_q(0), *n))
    assert np.all(err <= 1e-12), err
