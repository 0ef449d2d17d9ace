"""The work a user has this framework do, as measured cases.

Two layers are called, each through its public entry points:

* the directional compact operators (`plan_direction` / `apply_along`, or its
  batched form over several fields): gradients and the smoothing filter of
  device fields, as a host program that owns its own solver loop calls them;
* whole time steps: `Solver.run` and `Solver.run_graph` on 3-D boxes, 2-D
  shock-interface grids, 1-D tubes and a stretched channel, and `Batch.run` on
  an ensemble of uneven 2-D grids.

A solver pass advances the resident state by a few steps, so each pass starts
from where the last one ended, as a run does; its result is the conserved state
on the device and the clock.

`exact` restates the same numerics in plain torch, in FP64: every compact
operator as the dense matrix A^-1 B of its scheme, everything else as written
in the method's papers (Lele's C6 and C10, the Gaitonde-Visbal filter, Cook's
artificial properties, the LSRK(5,4) scheme).
"""
import ctypes
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch


def _package():
    if "compactles_b200" in sys.modules:
        return sys.modules["compactles_b200"]
    pkg = pathlib.Path.cwd() / "compactles.jl_b200"
    spec = importlib.util.spec_from_file_location("compactles_b200", pkg / "__init__.py",
                                                  submodule_search_locations=[str(pkg)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["compactles_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


# ------------------------------------------------------------------ cases ----
def listed():
    return [
        # One scalar's gradient on a small box: the smallest calls a user makes,
        # three launches whose latency is all there is.
        dict(name="grad_c6_64", kind="operator", scheme="c6", nx=64, ny=64, nz=64, fields=1, periodic=True, f32=False),
        # The gradient of five conserved fields on the benchmark's 256^3 box.
        dict(name="grad_c6_256", kind="operator", scheme="c6", nx=256, ny=256, nz=256, fields=5, periodic=True,
             f32=False),
        # The velocity gradient tensor with the tenth-order scheme between walls,
        # with the odd point counts that wall-to-wall grids have.
        dict(name="grad_c10_walls", kind="operator", scheme="c10", nx=201, ny=161, nz=129, fields=3, periodic=False,
             f32=False),
        # Smoothing five single-precision fields between walls.
        dict(name="filter_f32_walls", kind="operator", scheme="filter", nx=256, ny=192, nz=160, fields=5,
             periodic=False, f32=True),
        # Taylor-Green at 64^3: the README's quick start and the serving mix's box.
        dict(name="box_64", kind="box", nx=64, ny=64, nz=64, mixed=False, steps=4),
        # Taylor-Green at 256^3 in FP64: the headline benchmark.
        dict(name="box_256", kind="box", nx=256, ny=256, nz=256, mixed=False, steps=1),
        # The mixed-precision form of it on an ordinary box.
        dict(name="box_192_mixed", kind="box", nx=192, ny=192, nz=192, mixed=True, steps=2),
        # A closed box, whose wall-to-wall lines have odd point counts.
        dict(name="wallbox_129", kind="wallbox", nx=129, ny=129, nz=129, mixed=False, steps=2),
        # A viscous channel clustered towards its walls: the general metric path.
        dict(name="channel_160", kind="channel", nx=160, ny=129, nz=96, mixed=False, steps=2),
        # A well resolved 2-D He/CO2 shock-interface run (two species).
        dict(name="interface_2048", kind="interface", nx=2048, ny=1024, mixed=False, steps=2),
        # A long two-species shock tube in graph mode: the serving mix's longest request.
        dict(name="tube_5712", kind="tube", nx=5712, mixed=False, steps=20),
        # An ensemble of uneven 2-D shock-interface grids advanced together.
        dict(name="ensemble_8", kind="ensemble", members=8, nx=320, ny=112, mixed=True, steps=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator", "operator", "operator", "box", "box", "wallbox", "channel", "interface", "interface",
                       "tube", "ensemble"])
    if kind == "operator":
        while True:
            n = [_log(rng, 48, 320) for _ in range(3)]
            fields = rng.randint(1, 5)
            if 64 ** 3 <= n[0] * n[1] * n[2] * fields <= 5 * 256 ** 3:
                break
        return dict(kind=kind, scheme=rng.choice(["c6", "c10", "filter"]), nx=n[0], ny=n[1], nz=n[2], fields=fields,
                    periodic=rng.random() < 0.5, f32=rng.random() < 0.35)
    mixed = rng.random() < 0.35
    if kind == "box":
        n = [_log(rng, 48, 256) for _ in range(3)]
        if rng.random() < 0.5:
            n = [16 * max(3, round(v / 16)) for v in n]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], mixed=mixed, steps=1)
    if kind in ("wallbox", "channel"):
        n = [_log(rng, 40, 200) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], mixed=mixed, steps=1)
    if kind == "interface":
        nx = _log(rng, 192, 2048)
        return dict(kind=kind, nx=nx, ny=max(48, _log(rng, nx / 8, nx / 2)), mixed=mixed, steps=rng.randint(1, 2))
    if kind == "tube":
        return dict(kind=kind, nx=_log(rng, 300, 8192), mixed=mixed, steps=rng.randint(5, 20))
    return dict(kind=kind, members=rng.randint(3, 8), nx=_log(rng, 160, 512), ny=_log(rng, 64, 160), mixed=mixed,
                steps=rng.randint(5, 20))


# ------------------------------------------------------------------ inputs ---
def _rng(seed):
    return np.random.default_rng(1000003 * (int(seed) + 1))


def _modes(rng, shape_xyz, kmax, nmodes=8):
    """A seeded sum of Fourier modes, a / |k|^2 cos(k.x + phi), on the unit-periodic box (z, y, x)."""
    xs = [2 * math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n for n in shape_xyz]
    f = torch.zeros(shape_xyz[::-1], device="cuda", dtype=torch.float64)
    for _ in range(nmodes):
        k = rng.integers(1, kmax + 1, size=3) * rng.choice([-1, 1], size=3)
        a, ph = rng.standard_normal(), rng.uniform(0, 2 * math.pi)
        f += (a / float(np.dot(k, k))) * torch.cos((k[0] * xs[0] + ph)[None, None, :] + (k[1] * xs[1])[None, :, None] +
                                                   (k[2] * xs[2])[:, None, None])
    return f


def _operator_fields(case, seed):
    rng = _rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    kmax = max(2, min(n) // 8)
    f = torch.stack([_modes(rng, n, kmax) for _ in range(case["fields"])])
    return f.float() if case["f32"] else f


def _conserved(eos, u, p, rho, Y):
    cv = sum(y * (R / (g - 1)) for y, (R, g) in zip(Y, eos))
    Rm = sum(y * R for y, (R, _) in zip(Y, eos))
    E = rho * (cv * (p / (rho * Rm)) + 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2))
    return torch.stack([rho * y for y in Y] + [rho * u[0], rho * u[1], rho * u[2], E])


def _grid_case(n, L, periodic, wall, eos, Q0, *, mu0=0.0, cfl=0.5, stretch=None):
    return dict(n=n, L=L, periodic=periodic, wall=wall, eos=eos, Q0=Q0.contiguous(), mu0=mu0, cfl=cfl, stretch=stretch)


def _vortex(case, seed, L, x, y, z):
    """A Taylor-Green vortex with seeded amplitude and weak seeded large-scale perturbations."""
    rng = _rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    amp = rng.uniform(0.9, 1.1)
    u = (amp * torch.sin(x) * torch.cos(y) + 0 * z, -amp * torch.cos(x) * torch.sin(y) + 0 * z, 0 * x + 0 * y + 0 * z)
    u = tuple(c + 0.05 * _modes(rng, n, 3) for c in u)
    p = 71.43 * (1 + 0.01 * _modes(rng, n, 3))
    rho = 1 + 0.05 * _modes(rng, n, 3)
    return u, p, rho


def _axes(n, L, periodic):
    return [torch.arange(m, device="cuda", dtype=torch.float64) * (l / m if per else l / (m - 1))
            for m, l, per in zip(n, L, periodic)]


def _shape(ax):
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _box(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    walls = case["kind"] == "wallbox"
    L = (math.pi if walls else 2 * math.pi,) * 3
    per = (not walls,) * 3
    x, y, z = _shape(_axes(n, L, per))
    u, p, rho = _vortex(case, seed, L, x, y, z)
    if walls:   # no flow through any face
        s = (torch.sin(x), torch.sin(y), torch.sin(z))
        u = tuple(c * w for c, w in zip(u, s))
    return _grid_case(n, L, per, ["slip" if walls else None] * 3, [(1.0, 1.4)], _conserved([(1.0, 1.4)], u, p, rho, (1.0,)))


def _channel(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    L, per = (2 * math.pi, 2.0, math.pi), (True, False, True)
    a = 0.6   # spacing ratio (1 + a) / (1 - a) between the middle and the walls
    xi = torch.arange(n[1], device="cuda", dtype=torch.float64) / (n[1] - 1)
    yy = -1 + 2 * (xi - (a / (2 * math.pi)) * torch.sin(2 * math.pi * xi))
    m = 2 * (1 - a * torch.cos(2 * math.pi * xi))
    ax = _axes(n, L, per)
    ax[1] = yy
    x, y, z = _shape(ax)
    rng = _rng(seed)
    prof = 1 - y ** 2
    u = (prof * (1 + 0.1 * _modes(rng, n, 4)), 0.1 * prof * _modes(rng, n, 4), 0.1 * prof * _modes(rng, n, 4))
    p = 17.86 * (1 + 0.005 * prof * _modes(rng, n, 4))
    rho = 1 + 0.01 * prof * _modes(rng, n, 4)
    return _grid_case(n, L, per, [None, "noslip", None], [(1.0, 1.4)], _conserved([(1.0, 1.4)], u, p, rho, (1.0,)),
                      mu0=1e-3, stretch=(None, (yy.cpu().numpy(), m.cpu().numpy(), a), None))


_R = 8.31446261815324
_HE_CO2 = [(_R / 4.0026e-3, 5.0 / 3.0), (_R / 44.01e-3, 1.289)]


def _interface(nx, ny, seed):
    """A planar shock in helium about to hit a perturbed He/CO2 interface."""
    rng = _rng(seed)
    (R_he, g_he), (R_co2, _) = _HE_CO2
    Ly = 1.0
    h = Ly / ny
    Lx = h * (nx - 1)
    p1, T1 = 101325.0, 300.0
    rho1 = p1 / (R_he * T1)
    mach = rng.uniform(1.3, 2.2)
    c1 = math.sqrt(g_he * p1 / rho1)
    p2 = p1 * (1 + 2 * g_he / (g_he + 1) * (mach * mach - 1))
    rho2 = rho1 * (g_he + 1) * mach * mach / ((g_he - 1) * mach * mach + 2)
    u2 = c1 * 2 / (g_he + 1) * (mach - 1 / mach)
    per = (False, True, True)
    x, y, z = _shape(_axes((nx, ny, 1), (Lx, Ly, h), per))
    w = rng.uniform(0.2, 1.0, size=8) / np.arange(1, 9) ** 2
    A = rng.uniform(0.05, 0.15) * Ly * w / w.sum() * rng.choice([-1, 1], size=8)
    ph = rng.uniform(0, 2 * math.pi, size=8)
    xi = 0.4 * Lx + sum(float(A[m]) * torch.cos(2 * math.pi * (m + 1) * y / Ly + float(ph[m])) for m in range(8))
    ths = 0.5 * (1 + torch.tanh((x - 0.2 * Lx) / (3 * h)))
    co2 = 0.5 * (1 + torch.tanh((x - xi) / (3 * h))) + 0 * z
    he = 1 - co2
    p = (1 - ths) * p2 + ths * p1 + 0 * co2
    rho = (1 - ths) * rho2 + ths / (he / rho1 + co2 / (p1 / (R_co2 * T1)))
    u = ((1 - ths) * u2 + 0 * co2, 0 * co2, 0 * co2)
    return _grid_case((nx, ny, 1), (Lx, Ly, h), per, ["slip", None, None], _HE_CO2,
                      _conserved(_HE_CO2, u, p, rho, (he, co2)))


def _tube(case, seed):
    rng = _rng(seed)
    n = case["nx"]
    h = 1.0 / (n - 1)
    at = rng.uniform(0.2, 0.7)
    eos = [(1.0, 1.4), ((1 - at) / (1 + at), 1.4)]
    x, y, z = _shape(_axes((n, 1, 1), (1.0, h, h), (False, True, True)))
    th = 0.5 * (1 + torch.tanh((x - 0.5) / (2 * h))) + 0 * y + 0 * z
    p = (1 - th) * rng.uniform(4.0, 12.0) + th
    Y = (1 - th, th)
    rho = p / sum(yk * R for yk, (R, _) in zip(Y, eos))   # T = 1
    return _grid_case((n, 1, 1), (1.0, h, h), (False, True, True), ["slip", None, None], eos,
                      _conserved(eos, (0 * th, 0 * th, 0 * th), p, rho, Y), cfl=0.4)


def _members(case, seed):
    rng = _rng(seed + 77)
    out = []
    for m in range(case["members"]):   # sizes spread a factor of two around the case's, the same for every seed
        f = 2.0 ** ((m % 4) / 1.5 - 1)
        out.append(_interface(max(64, 2 * round(case["nx"] * f / 2)), max(32, 2 * round(case["ny"] / f ** 0.5 / 2)),
                              int(rng.integers(1 << 30))))
    return out


def _problem(case, seed):
    kind = case["kind"]
    if kind in ("box", "wallbox"):
        return _box(case, seed)
    if kind == "channel":
        return _channel(case, seed)
    if kind == "interface":
        return _interface(case["nx"], case["ny"], seed)
    return _tube(case, seed)


# ------------------------------------------------------------ the framework ---
class _DeviceArray:
    """Device memory of `owner` as a tensor source; the tensor keeps the owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=2)


def _descriptor(cl, g, mixed):
    walls = {"slip": cl.SlipWallBC, "noslip": cl.NoSlipWallBC}
    bcs = tuple((cl.PeriodicBC(), cl.PeriodicBC()) if w is None else (walls[w](), walls[w]()) for w in g["wall"])
    eos = cl.IdealMixture([cl.IdealSpecies(f"s{k}", R, gam) for k, (R, gam) in enumerate(g["eos"])])
    stretch = [None] * 3
    if g["stretch"]:
        for k, s in enumerate(g["stretch"]):
            if s is not None:
                stretch[k] = cl.Stretch(lambda xi, s=s: s[0], lambda xi, s=s: s[1])
    return cl.solver_desc(g["n"], g["L"], bcs, cl.lele_d1_6(), cl.compact_filter(0.45), eos=eos,
                          transport=cl.Transport(mu0=g["mu0"]), cfl=g["cfl"],
                          precision="mixed" if mixed else "fp64", stretch=tuple(stretch))


def _spacing(case):
    return [2 * math.pi / (n if case["periodic"] else n - 1) for n in (case["nx"], case["ny"], case["nz"])]


def prepare(case, seed):
    cl = _package()
    if case["kind"] == "operator":
        n = (case["nx"], case["ny"], case["nz"])
        scheme = {"c6": cl.lele_d1_6, "c10": cl.lele_d1_10, "filter": lambda: cl.compact_filter(0.45)}[case["scheme"]]()
        g = cl.grid(n, (case["periodic"],) * 3)
        plans = [cl.plan_direction(g, scheme, d + 1, h, dtype="f32" if case["f32"] else "f64", layout="interior")
                 for d, h in enumerate(_spacing(case))]
        f = _operator_fields(case, seed)
        return dict(case=case, cl=cl, plans=plans, f=f,
                    out=[torch.empty_like(f) for _ in range(1 if case["scheme"] == "filter" else 3)])
    if case["kind"] == "ensemble":
        gs = _members(case, seed)
        descs = [_descriptor(cl, g, case["mixed"]) for g in gs]
        B = cl.Batch(descs[0])
        ids = [B.add(d, g["Q0"].cpu().numpy(), 1e30, layout="interior") for d, g in zip(descs, gs)]
        return dict(case=case, cl=cl, batch=B, ids=ids)
    g = _problem(case, seed)
    S = cl.Solver(_descriptor(cl, g, case["mixed"]))
    ptr = ctypes.POINTER(ctypes.c_double)()
    cl.api._check(cl.lib().cles_state_device(S.ptr, ctypes.byref(ptr)))
    Q = torch.as_tensor(_DeviceArray(S, ctypes.cast(ptr, ctypes.c_void_p).value, tuple(g["Q0"].shape)), device="cuda")
    Q.copy_(g["Q0"])
    return dict(case=case, cl=cl, solver=S, Q=Q, ns=len(g["eos"]), done=0)


def _apply(cl, plan, f, out):
    if f.shape[0] == 1:
        cl.apply_along(out[0], plan, f[0])
        return
    cl.api._check(cl.lib().cles_apply_along_batch(plan.ptr, ctypes.c_void_p(f.data_ptr()),
                                                  ctypes.c_void_p(out.data_ptr()), f.shape[0], f[0].numel()))


def _named(Q, ns):
    return {"rho": Q[:ns], "momentum": Q[ns:ns + 3], "energy": Q[ns + 3]}


def run(state):
    case, cl = state["case"], state["cl"]
    if case["kind"] == "operator":
        src = state["f"]
        if case["scheme"] == "filter":   # one pass per direction, the later ones in place, as a smoothing is done
            out = state["out"][0]
            for plan in state["plans"]:
                _apply(cl, plan, src, out)
                src = out
            return [out]
        for plan, out in zip(state["plans"], state["out"]):
            _apply(cl, plan, src, out)
        return state["out"]
    if case["kind"] == "ensemble":
        B = state["batch"]
        B.run(case["steps"])
        return [B.fetch(i) for i in state["ids"]]
    S = state["solver"]
    state["done"] += case["steps"]
    res = (S.run_graph if case["kind"] == "tube" else S.run)(1e30, state["done"])
    return dict(_named(state["Q"], state["ns"]), t=res.t)


# -------------------------------------------------------------------- work ---
def _cells(case):
    if case["kind"] == "ensemble":
        tot = 0
        for m in range(case["members"]):
            f = 2.0 ** ((m % 4) / 1.5 - 1)
            tot += max(64, 2 * round(case["nx"] * f / 2)) * max(32, 2 * round(case["ny"] / f ** 0.5 / 2))
        return tot
    return case["nx"] * case.get("ny", 1) * case.get("nz", 1)


_FLOPS = {"c6": 12, "c10": 22, "filter": 22}   # per point of one line solve: stencil, sweeps


def work(case):
    if case["kind"] == "operator":
        pts = _cells(case) * case["fields"]
        el = 4 if case["f32"] else 8
        # the field read once; a gradient writes three results, a smoothing one
        return {"bytes": pts * el * (2 if case["scheme"] == "filter" else 4), "flops": 3 * pts * _FLOPS[case["scheme"]]}
    dims = 3 if "nz" in case else 2 if "ny" in case else 1
    ns = 1 if dims == 3 else 2
    nc = ns + 4
    # per right-hand side: gradients of u, v, w, T (and Y), the smoothed sensors,
    # the flux divergence, and the pointwise work; the state filter once a step
    gty = 1 if ns == 1 else 1 + ns
    sens = 2 if ns == 1 else 2 + ns
    rhs = dims * (_FLOPS["c6"] * (3 + gty + nc) + _FLOPS["filter"] * sens + 10 * sens + 12 * nc) + 60
    step = 5 * rhs + dims * _FLOPS["filter"] * nc + 40
    # the state read and written once a step
    return {"bytes": case["steps"] * _cells(case) * nc * 8 * 2, "flops": case["steps"] * _cells(case) * step}


def tolerance(case):
    # about four times the largest distance of the path from `exact` over the ranges
    if case["kind"] == "operator":
        return {"rel": 2.4e-6 if case["f32"] else 8e-15}
    if case["mixed"]:   # the clock follows the single-precision rate of one cell
        return {"rel": 1e-6 if "nz" in case else 4e-6}
    long = case["kind"] in ("tube", "ensemble")   # up to 20 steps past a shock
    return {"rel": 1.5e-13 if long else 3e-14}


# ------------------------------------------------------- the plain 64 bits ---
# (q, LHS off-diagonals, a0, stencil, symmetric, closure LHS rows, closure RHS rows)
def _scheme(name):
    if name == "c6":
        return (1, [1 / 3], 0.0, [7 / 9, 1 / 36], False, [[0, 1, 2], [1 / 4, 1, 1 / 4]],
                [[-5 / 2, 2, 1 / 2], [-3 / 4, 0, 3 / 4]])
    if name == "c10":
        return (2, [1 / 2, 1 / 20], 0.0, [17 / 24, 101 / 600, 1 / 600], False,
                [[0, 0, 1, 2, 0], [0, 1 / 4, 1, 1 / 4, 0], [0, 1 / 3, 1, 1 / 3, 0]],
                [[-5 / 2, 2, 1 / 2], [-3 / 4, 0, 3 / 4], [-1 / 36, -7 / 9, 0, 7 / 9, 1 / 36]])
    a = 0.45
    f2 = [(1 + 2 * a) / 2, (1 + 2 * a) / 2]
    f4 = [(5 + 6 * a) / 8, (1 + 2 * a) / 2, (-1 + 2 * a) / 8]
    f6 = [(11 + 10 * a) / 16, (15 + 34 * a) / 32, (-3 + 6 * a) / 16, (1 - 2 * a) / 32]

    def centred(c):
        return [v / 2 for v in c[:0:-1]] + [c[0]] + [v / 2 for v in c[1:]]
    return (1, [a], (93 + 70 * a) / 128,
            [(7 + 18 * a) / 32, (-7 + 14 * a) / 64, (1 - 2 * a) / 32, (-1 + 2 * a) / 256], True,
            [[0, 1, 0], [a, 1, a], [a, 1, a], [a, 1, a]], [[1.0], centred(f2), centred(f4), centred(f6)])


_dense = {}


def _matrix(name, n, periodic, h):
    """A^-1 B of one line of n points, on the GPU."""
    key = (name, n, periodic, h)
    if key in _dense:
        return _dense[key]
    q, lhs, a0, st, sym, clhs, crhs = _scheme(name)
    A, B = np.eye(n), np.zeros((n, n))
    sc = 1.0 if sym else 1.0 / h
    i = np.arange(n)
    for k, v in enumerate(lhs, 1):
        for s in (-k, k):
            ok = slice(None) if periodic else (i + s >= 0) & (i + s < n)
            A[i[ok], (i[ok] + s) % n] += v
    B[i, i] += a0 * sc
    for k, v in enumerate(st, 1):
        for s, sg in ((k, 1.0), (-k, 1.0 if sym else -1.0)):
            ok = slice(None) if periodic else (i + s >= 0) & (i + s < n)
            B[i[ok], (i[ok] + s) % n] += sg * v * sc
    if not periodic:
        end = 1.0 if sym else -1.0
        for j, (lr, rr) in enumerate(zip(clhs, crhs)):
            for row, step, sg in ((j, 1, 1.0), (n - 1 - j, -1, end)):
                A[row] = 0.0
                B[row] = 0.0
                for t, v in enumerate(lr):
                    if v != 0.0:
                        A[row, row + step * (t - q)] = v
                edge = 0 if step == 1 else n - 1
                for t, v in enumerate(rr):
                    B[row, edge + step * t] = sg * v * sc
    D = torch.linalg.solve(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda())
    if len(_dense) > 12:
        _dense.clear()
    _dense[key] = D
    return D


def _along(D, f, dim):
    """The line operator D along dimension dim (0 = x) of fields (..., z, y, x)."""
    if dim == 0:
        return f @ D.T
    if dim == 1:
        return D @ f
    sh = f.shape
    return (D @ f.reshape(*sh[:-3], sh[-3], -1)).reshape(sh)


class _Plain:
    """The solver's time step on one grid in plain torch."""
    A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
         -1275806237668 / 842570457699)
    B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
         3134564353537 / 4481467310338, 2277821191437 / 14882151754819)
    C_mu, C_beta, C_kappa, C_D, Pr, Sc = 0.002, 1.0, 0.01, 0.01, 0.7, 0.7

    def __init__(self, g):
        self.g, self.ns = g, len(g["eos"])
        self.act = [d for d in range(3) if g["n"][d] > 1]
        self.h, self.ih = [1.0] * 3, [1.0] * 3
        for d in self.act:
            n, L = g["n"][d], g["L"][d]
            s = g["stretch"][d] if g["stretch"] else None
            self.h[d] = 1.0 / (n - 1) if s is not None else (L / n if g["periodic"][d] else L / (n - 1))
            if s is not None:
                self.ih[d] = (1.0 / torch.from_numpy(s[1]).cuda()).reshape([-1 if 2 - e == d else 1 for e in range(3)])
        self.D = {d: _matrix("c6", g["n"][d], g["periodic"][d], self.h[d]) for d in self.act}
        self.F = {d: _matrix("filter", g["n"][d], g["periodic"][d], self.h[d]) for d in self.act}
        self.Q = g["Q0"].clone()
        self.R = torch.tensor([R for R, _ in g["eos"]], device="cuda", dtype=torch.float64).reshape(-1, 1, 1, 1)
        self.cv = torch.tensor([R / (k - 1) for R, k in g["eos"]], device="cuda", dtype=torch.float64).reshape(-1, 1, 1, 1)
        z = torch.zeros_like(self.Q[0])
        self.mu, self.be, self.ka, self.Dk = z, z, z, torch.zeros_like(self.Q[:self.ns])
        self.t = 0.0

    def walls(self):
        Q, ns = self.Q, self.ns
        for d in self.act:
            kind = self.g["wall"][d]
            for i in ((0, -1) if kind else ()):
                q = Q.select(3 - d, i)   # a view of the face plane
                r = q[:ns].sum(0)
                m = range(ns, ns + 3) if kind == "noslip" else (ns + d,)
                q[ns + 3] -= 0.5 * sum(q[c] ** 2 for c in m) / r
                for c in m:
                    q[c] = 0.0

    def prims(self):
        Q, ns = self.Q, self.ns
        self.rho = Q[:ns].sum(0)
        self.Y = Q[:ns] / self.rho
        self.Rm, self.cvm = (self.Y * self.R).sum(0), (self.Y * self.cv).sum(0)
        self.u = Q[ns:ns + 3] / self.rho
        self.e = Q[ns + 3] / self.rho - 0.5 * (self.u ** 2).sum(0)
        self.T = self.e / self.cvm
        self.p = self.rho * self.Rm * self.T
        self.cp = self.cvm + self.Rm
        self.c = torch.sqrt((1 + self.Rm / self.cvm) * self.Rm * self.T)

    def grad(self, f, d):
        return _along(self.D[d], f, d) * self.ih[d]

    def delta4(self, f, p):
        out = 0.0
        for d in self.act:
            n, ax = self.g["n"][d], 2 - d
            i = torch.arange(n, device="cuda")
            acc = 0.0
            for s, w in zip(range(-2, 3), (1.0, -4.0, 6.0, -4.0, 1.0)):
                j = (i + s) % n if self.g["periodic"][d] else (i + s).clamp(0, n - 1)
                acc = acc + w * f.index_select(ax, j)
            out = out + self.h[d] ** p * acc.abs()
        for d in self.act:
            out = _along(self.F[d], out, d)
        return out.clamp(min=0.0)

    def rhs(self):
        ns, u = self.ns, self.u
        G = torch.zeros((3, 3) + tuple(self.T.shape), device="cuda", dtype=torch.float64)   # G[d][j] = du_j/dx_d
        for d in self.act:
            G[d] = self.grad(u, d)
        S = 0.5 * (G + G.transpose(0, 1))
        s = self.rho * self.delta4(torch.sqrt((S * S).sum((0, 1))), 2)
        self.mu, self.be = self.C_mu * s, self.C_beta * s
        self.ka = self.C_kappa * self.rho * self.c / self.T * self.delta4(self.e, 1)
        if ns > 1:
            self.Dk = torch.stack([self.C_D * self.c * self.delta4(self.Y[k], 1) for k in range(ns)])
        mu0 = self.g["mu0"]
        mu, D = mu0 + self.mu, mu0 / (self.Sc * self.rho) + self.Dk
        ka = mu0 * self.cp / self.Pr + self.ka
        div = G[0, 0] + G[1, 1] + G[2, 2]
        h = (self.R + self.cv) * self.T
        E = self.Q[ns + 3]
        dQ = torch.zeros_like(self.Q)
        for d in self.act:
            tau = [mu * (G[d, j] + G[j, d]) + ((self.be - 2 * mu / 3) * div if j == d else 0.0) for j in range(3)]
            J = torch.zeros_like(self.Y)
            if ns > 1:
                gY = self.grad(self.Y, d)
                J = self.rho * (-D * gY + self.Y * (D * gY).sum(0))
            F = torch.empty_like(self.Q)
            F[:ns] = self.rho * self.Y * u[d] + J
            for j in range(3):
                F[ns + j] = self.rho * u[d] * u[j] + (self.p if j == d else 0.0) - tau[j]
            F[ns + 3] = ((E + self.p) * u[d] - sum(u[j] * tau[j] for j in range(3)) - ka * self.grad(self.T, d) +
                         (h * J).sum(0))
            dQ -= self.grad(F, d)
        return dQ

    def rate(self):
        acc, dsum = 0.0, 0.0
        for d in self.act:
            idx = self.ih[d] / self.h[d]
            acc = acc + (self.u[d].abs() + self.c) * idx
            dsum = dsum + idx * idx
        mu0 = self.g["mu0"]
        Dm = (mu0 / (self.Sc * self.rho) + self.Dk).amax(0)
        nu = (mu0 + self.mu + self.be) / self.rho + (mu0 * self.cp / self.Pr + self.ka) / self.rho / self.cp + Dm
        return float((acc + 2 * nu * dsum).max())

    def step(self):
        self.walls()
        self.prims()
        dt = self.g["cfl"] / self.rate()
        du = torch.zeros_like(self.Q)
        for s in range(5):
            if s:
                self.walls()
                self.prims()
            du = self.A[s] * du + dt * self.rhs()
            self.Q += self.B[s] * du
        self.walls()
        for d in self.act:
            self.Q = _along(self.F[d], self.Q, d)
        self.t += dt


def exact(case, seed):
    if case["kind"] == "operator":
        f = _operator_fields(case, seed).double()
        Ds = [_matrix(case["scheme"], n, case["periodic"], h)
              for n, h in zip((case["nx"], case["ny"], case["nz"]), _spacing(case))]
        if case["scheme"] == "filter":
            for d, D in enumerate(Ds):
                f = _along(D, f, d)
            return [f]
        return [_along(D, f, d) for d, D in enumerate(Ds)]
    if case["kind"] == "ensemble":
        out = []
        for g in _members(case, seed):
            s = _Plain(g)
            for _ in range(case["steps"]):
                s.step()
            out.append(s.Q)
        return out
    s = _Plain(_problem(case, seed))
    for _ in range(case["steps"]):
        s.step()
    return dict(_named(s.Q, s.ns), t=s.t)
