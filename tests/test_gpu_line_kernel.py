"""Segmented line solves (k_line) against the CPU oracle.

Lengths on both sides of every boundary of the segmentation: tiles of 16, 24
and 32 points, remainders (segments of two lengths), the smallest line with two
segments, lines spread over two to eight blocks; few and many lines; both end
kinds; in place; and a filter whose interface system decays too slowly for the
window (the generic kernel serves it).  The right-hand side and steps on grids
whose last direction carries the RK update in its store (1-D, 2-D, 3-D, odd
sizes).

Tolerances: 1e-12 of the largest value in FP64 and 5e-6 in FP32, those of the
other operator kernels (test_gpu_operators.py): the same sums in another order.
"""
import numpy as np
import pytest

import compactles_b200 as cl
import parity
from compactles_b200 import scenarios

pytestmark = pytest.mark.gpu


def _scheme(mod, name):
    return {"c6": mod.lele_d1_6, "c10": mod.lele_d1_10, "filt": lambda: mod.compact_filter(0.45),
            "pade": mod.pade_d1_4, "slow": lambda: mod.compact_filter(0.4995)}[name]()


def _line_form(ng, name, dim, periodic, dtype, count=1):
    """(warp-per-line form, segments a line, points a segment, blocks a cluster)"""
    import ctypes as C
    per = tuple(1 if (k != dim - 1 or periodic) else 0 for k in range(3))
    info = (C.c_int * 4)()
    cl.api._check(cl.lib().cles_selftest_line_form(C.byref(cl.grid(ng, per)), C.byref(_scheme(cl, name)), dim,
                                                   cl.abi.CLES_F64 if dtype == "f64" else cl.abi.CLES_F32, count, info))
    return tuple(info)


def _check(orc, name, ng, dim, periodic, dtype, tol, form=True):
    per = tuple(1 if (k != dim - 1 or periodic) else 0 for k in range(3))
    assert (_line_form(ng, name, dim, periodic, dtype)[1] > 0) == form   # k_line can take it
    g = orc.grid(ng, per)
    rng = np.random.default_rng(ng[dim - 1] + 10 * dim)
    f = np.zeros(orc.padded_shape(g))
    inner = orc.interior(g, f)
    z, y, x = np.meshgrid(*[np.arange(s) for s in inner.shape], indexing="ij")
    inner[...] = np.sin(0.3 * x + 0.2 * y + 0.1 * z) + 0.1 * rng.standard_normal(inner.shape)
    orc.exchange_halos(g, f)
    h = 0.9 / ng[dim - 1]
    ref = orc.interior(g, orc.Plan(g, _scheme(orc, name), dim, h).apply(f))
    plan = cl.plan_direction(cl.grid(ng, per), _scheme(cl, name), dim, h, dtype=dtype)
    fin = f if dtype == "f64" else f.astype(np.float32)
    out = np.zeros_like(fin)
    cl.apply_along(out, plan, fin)
    err = np.abs(orc.interior(g, out).astype(np.float64) - ref).max() / np.abs(ref).max()
    assert err < tol, (name, ng, dim, periodic, dtype, err)
    import torch
    t = torch.tensor(fin, device="cuda")   # in place, on the device
    cl.apply_along(t, plan, t)
    torch.cuda.synchronize()
    assert np.array_equal(orc.interior(g, t.cpu().numpy()), orc.interior(g, out))


@pytest.mark.parametrize("scheme", ["c6", "c10", "filt", "pade"])
@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("periodic", [True, False])
def test_lengths(orc, scheme, dim, periodic):
    for n in (18, 20, 21, 31, 32, 33, 35, 47, 49, 63, 65, 97, 129, 161, 255, 257, 1031):
        ng = tuple(n if k == dim - 1 else (7, 5, 6)[k] + 4 for k in range(3))
        _check(orc, scheme, ng, dim, periodic, "f64", 1e-12)
        _check(orc, scheme, ng, dim, periodic, "f32", 5e-6)


@pytest.mark.parametrize("scheme", ["c6", "c10", "filt"])
@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("n", [33, 161, 200])
def test_many_lines(orc, scheme, dim, n):
    # enough points for the long tile (more than 2^18): 2^21 and more
    o = int(np.ceil(np.sqrt((1 << 21) / n))) + 1
    ng = tuple(n if k == dim - 1 else o for k in range(3))
    for periodic in (True, False):
        _check(orc, scheme, ng, dim, periodic, "f64", 1e-12)
    _check(orc, scheme, ng, dim, False, "f32", 5e-6)


@pytest.mark.parametrize("ng,dim", [((7937, 1, 1), 1), ((8192, 1, 1), 1), ((9001, 1, 1), 1), ((12800, 1, 1), 1),
                                    ((12000, 16, 1), 1), ((3, 8999, 1), 2), ((4099, 40, 1), 1), ((37, 4099, 1), 2), ((300, 2049, 1), 2)])
def test_lines_over_clusters(orc, ng, dim):
    for scheme in ("c6", "c10", "filt"):
        for periodic in (True, False):
            _check(orc, scheme, ng, dim, periodic, "f64", 1e-12)


def test_slow_filter(orc):
    # 300 points: the window holds the whole line; 1000: no window is wide enough
    for n, form in ((300, True), (1000, False)):
        for dim in (1, 2):
            ng = tuple(n if k == dim - 1 else 9 for k in range(3))
            _check(orc, "slow", ng, dim, False, "f64", 1e-11, form)   # condition number of the filter about 2000


@pytest.mark.parametrize("n", [(333, 1, 1), (150, 67, 1), (45, 39, 51), (129, 40, 33)])
@pytest.mark.parametrize("walls", [True, False])
def test_rhs_and_steps(orc, n, walls):
    def desc(m):
        wall = (cl.SlipWallBC(), cl.SlipWallBC())
        bcs = tuple(wall if walls and n[k] > 1 else cl.PER3[k] for k in range(3))
        eos = cl.IdealMixture([cl.IdealSpecies("a", 1.0, 1.4), cl.IdealSpecies("b", 0.4, 1.3)])
        return cl.solver_desc(n, tuple(1.0 if v > 1 else 0.01 for v in n), bcs, m.lele_d1_6(), m.compact_filter(0.45),
                              eos=eos, transport=cl.Transport(mu0=1e-4))
    dg, do = desc(cl), desc(orc)
    tp = 2 * np.pi

    def ic(x, y, z):
        s = 0.7 * np.sin(tp * x + 0.7) * np.cos(tp * y + 0.4) + 0.3 * np.sin(tp * z + 0.2)
        Y = 0.5 + 0.3 * s
        return cl.Prim(u=(0.3 * s, 0.2 * s if n[1] > 1 else 0 * s, 0.1 * s if n[2] > 1 else 0 * s), p=2 + 0.2 * s,
                       rho=1 + 0.1 * s, Y=(Y, 1 - Y))
    Q0 = cl.initialize(dg, ic, eos=dg._eos)
    sl = (slice(None),) + cl.interior_slices(dg)
    S, O = cl.Solver(dg), orc.Solver(do)
    S.set_state(Q0)
    O.set_state(Q0)
    a, b = S.compute_rhs(), O.compute_rhs()
    plain, term = parity.rhs_errors(a[sl], b[sl], O.rhs_scales(cl.grid_spacing(dg)))
    assert max(term) < 1e-12, (plain, term)
    S.set_state(Q0)
    O.set_state(Q0)
    S.run(1e9, 5)
    assert O.run(1e9, 5)[0] == 0
    qa, qb = S.get_state()[sl], O.get_state()[sl]
    assert np.linalg.norm(qa - qb) < 1e-11 * np.linalg.norm(qb)


@pytest.mark.parametrize("n", [(333, 1, 1), (150, 67, 1), (1, 61, 1), (45, 39, 51)])
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 1e-5)])
def test_rhs_after_a_step(n, graph, precision, tol):
    """The right-hand side read after a step is that of its last stage, also where
    the update rides in the last direction's store.  A step of dt moves the stages by
    dt d(dQ)/dt, here 1e-9 of dQ: frequencies of these grids are below 1e4, dt is
    about 1e-13.  Mixed: single-precision fields may round the other way (6e-8 each), and
    a derivative raises that by the points a wave, up to 333 / 2."""
    import ctypes as C
    d = cl.solver_desc(n, tuple(1.0 if v > 1 else 0.01 for v in n), cl.PER3, cl.lele_d1_6(), cl.compact_filter(0.45),
                       cfl=1e-10, precision=precision)
    tp = 2 * np.pi
    Q0 = cl.initialize(d, lambda x, y, z: cl.Prim(
        u=(0.3 * np.sin(tp * (x + y)) + 0 * z, 0.2 * np.cos(tp * x) + 0 * y + 0 * z, 0 * x + 0 * y + 0.1 * np.sin(tp * z)),
        p=2 + 0.2 * np.sin(tp * (x + z)) + 0 * y, rho=1 + 0.1 * np.cos(tp * (y + z)) + 0 * x))
    R, S = cl.Solver(d), cl.Solver(d)
    R.set_state(Q0)
    S.set_state(Q0)
    ref = R.compute_rhs()
    if graph:
        S.run_graph(1.0, 1)
    else:
        S.step(1e-13)
    got = np.full_like(ref, np.nan)
    cl.api._check(cl.lib().cles_get_rhs(S.ptr, got.ctypes.data_as(C.c_void_p), S._layout("padded")))
    sl = (slice(None),) + cl.interior_slices(d)
    assert np.abs(got[sl] - ref[sl]).max() <= tol * np.abs(ref[sl]).max()


@pytest.mark.parametrize("n", [(1, 61, 1), (41, 1, 38), (1, 44, 39)])
def test_other_collapsed_dimensions(orc, n):
    """Grids whose collapsed dimension is not the last: every direction's code path runs."""
    test_rhs_and_steps(orc, n, True)


def test_mixed_faces_share_edges(orc):
    """Enforced faces of different kinds in one launch: cells on edges and corners
    get every face's condition in apply_bcs! order; an extrapolation face in between
    keeps its place.  Bitwise against one condition at a time would need the oracle's
    own rounding, hence 1e-14 of the largest value."""
    n = (20, 18, 17)
    D = cl.DirichletBC(cl.Prim(u=(0.1, 0.2, -0.1), p=1.3, rho=0.9))
    for bcs in (((cl.SlipWallBC(), cl.NoSlipWallBC()), (D, cl.SlipWallBC()), (cl.NoSlipWallBC(Twall=1.1), D)),
                ((cl.NoSlipWallBC(), cl.SlipWallBC()), (cl.ExtrapolationBC(), D), (cl.SlipWallBC(), cl.NoSlipWallBC()))):
        mk = lambda m: cl.solver_desc(n, (1.0, 1.0, 1.0), bcs, m.lele_d1_6(), m.compact_filter(0.45))
        dg, do = mk(cl), mk(orc)
        rng = np.random.default_rng(3)
        Q0 = cl.initialize(dg, lambda x, y, z: cl.Prim(u=tuple(0.3 * rng.standard_normal(n[::-1]) for _ in range(3)),
                                                       p=2 + 0.1 * rng.random(n[::-1]), rho=1 + 0.1 * rng.random(n[::-1])))
        sl = (slice(None),) + cl.interior_slices(dg)
        S, O = cl.Solver(dg), orc.Solver(do)
        S.set_state(Q0)
        O.set_state(Q0)
        S.apply_bcs()
        O.apply_bcs()
        a, b = S.get_state()[sl], O.get_state()[sl]
        assert np.abs(a - b).max() <= 1e-14 * np.abs(b).max()


@pytest.mark.parametrize("ny", [161, 300, 1031])
def test_gradient_groups_share_launches_on_long_lines(ny):
    """Velocity and scalar gradients along y ride in one launch wherever k_line serves
    the lines, also from 160 points on, where no tile kernel takes these lengths: as many
    launches a right-hand side as with 150 points."""
    def launches(n):
        d = cl.solver_desc((40, n, 1), (1.0, 1.0, 0.01), cl.PER3, cl.lele_d1_6(), cl.compact_filter(0.45))
        S = cl.Solver(d)
        S.set_state(cl.initialize(d, lambda x, y, z: cl.Prim(u=(0.1 * np.sin(2 * np.pi * y) + 0 * x + 0 * z,
                                                                0 * x + 0 * y + 0 * z, 0 * x + 0 * y + 0 * z),
                                                             p=2 + 0 * x + 0 * y + 0 * z, rho=1 + 0 * x + 0 * y + 0 * z)))
        before = cl.kernel_launches()
        S.compute_rhs(layout="interior")
        return cl.kernel_launches() - before
    assert launches(ny) == launches(150)
