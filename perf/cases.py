"""Measured workloads of the finite-volume framework, through its public entry points.

Every case is a plain dict whose ``kind`` says what a user runs:

session    one Cartesian ``Simulation`` stepped with ``run(step_limit=...)``: how a
           solver script drives the framework (2D / 3D explosions, 1D shock tubes);
batch      independent grids advanced together by ``Batch`` with captured graphs, as a
           parameter sweep or the request server does (2D quadrant problems, 1D tubes,
           3D spheres of uneven sizes);
ignition   reactive grids (Arrhenius or ZND) through ``Grid`` / ``Batch``;
metric     a curvilinear ``Simulation`` (spherical wedge, annulus) with face boundaries;
stepfn     one call of the stateless step function on host arrays.

``exact`` restates the schemes in double precision with plain torch and shares no code
with the framework.
"""

import math

import numpy as np
import torch

import torch_gb300
from torch_gb300 import stepfn
from torch_gb300.batch import Batch, Grid

LIMITERS = ("VanLeer", "Albada", "MINBEE", "Superbee", "Unos")
FOREVER = dict(t_end=1e9, max_steps=10 ** 9)  # passes never run into the end of the solve
NONDIM = dict(q_heat=20.0, activation_energy=25.0, pre_exponential=1e3)
SI = dict(q_heat=141584000.0, activation_energy=17.15 * 4184.0, pre_exponential=1.76e5)


def listed():
    return [
        # the headline run: 3D spherical explosion, single precision, reflective box
        dict(name="explosion_3d_256_fp32", kind="session", nx=256, ny=256, nz=256,
             precision="fp32", limiter="Superbee", boundary="Reflective", cfl=0.6, steps=10),
        # the server's 3D batch: a few explosions of uneven sizes, odd ones among them,
        # both of the limiters that requests choose from
        dict(name="served_3d_mixed_fp32", kind="batch", dim=3, grids=6, lo=64, hi=190,
             precision="fp32", limiter="VanLeer", second="Superbee", cfl=0.4, steps=8, graph=4,
             layout=5),
        # one-step Arrhenius ignition of a 3D box, single precision
        dict(name="ignition_3d_192_fp32", kind="ignition", nx=192, ny=192, nz=192,
             precision="fp32", limiter="Albada", boundary="Open", model="arrhenius",
             closure="nondimensional", cfl=0.4, steps=10),
        # a sweep of 2D quadrant Riemann problems, one launch per stage for all of them
        dict(name="quadrants_2d_fp32", kind="batch", dim=2, grids=32, lo=64, hi=1024,
             precision="fp32", limiter="MINBEE", second="MINBEE", cfl=0.4, steps=10, graph=10,
             layout=4),
        # the server's 1D batch: Sod-type tubes of 1e3 to 1e5 cells, bound by launches
        dict(name="tubes_1d_fp32", kind="batch", dim=1, grids=16, lo=1000, hi=100000,
             precision="fp32", limiter="VanLeer", second="Superbee", cfl=0.4, steps=64, graph=8,
             layout=2),
        # the plain double-precision path, bit-faithful to the NumPy solver: the 2D
        # explosion of its documentation, and the 3D one
        dict(name="explosion_2d_256_fp64", kind="session", nx=256, ny=256, nz=0,
             precision="fp64", limiter="VanLeer", boundary="Open", cfl=0.8, steps=16),
        dict(name="explosion_3d_96_fp64", kind="session", nx=96, ny=96, nz=96,
             precision="fp64", limiter="Superbee", boundary="Reflective", cfl=0.6, steps=4),
        # curvilinear grids: a large single-precision wedge with a pressure outlet, and a
        # double-precision annulus with a periodic azimuth
        dict(name="wedge_3d_256x192x192_fp32", kind="metric", geometry="spherical", nx=256,
             ny=192, nz=192, precision="fp32", limiter="Superbee", cfl=0.4, steps=2),
        dict(name="annulus_2d_256x192_fp64", kind="metric", geometry="annular", nx=256, ny=192,
             nz=0, precision="fp64", limiter="VanLeer", cfl=0.4, steps=4),
        # the smallest call: one step of one shock tube, waited for (interactive stepping)
        dict(name="shock_tube_1d_1000_fp64", kind="session", nx=1000, ny=0, nz=0,
             precision="fp64", limiter="VanLeer", boundary="Open", cfl=0.4, steps=1),
        # detailed chemistry as the reference runs it: SI constants, two-stage ZND kinetics,
        # gamma(lambda) per cell, double precision
        dict(name="ignition_2d_znd_fp64", kind="ignition", nx=160, ny=144, nz=0,
             precision="fp64", limiter="VanLeer", boundary="Reflective", model="znd",
             closure="si", cfl=0.4, steps=6),
        # the step function on NumPy arrays, with the interface fluxes returned
        dict(name="stepfn_2d_192_fp64", kind="stepfn", nx=192, ny=192, nz=0, precision="fp64",
             limiter="VanLeer", boundary="Reflective"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """A case of the listed ranges: every extent, odd or even, with the options in use."""
    pick = rng.choice(["s3f", "s3f", "s3d", "s2f", "s2d", "s1", "b3", "b2", "b1", "r3", "r2",
                       "m3", "m2", "fn"])
    lim = rng.choice(LIMITERS)
    bnd = rng.choice(["Open", "Reflective", "Periodic"])
    common = dict(limiter=lim, boundary=bnd, cfl=round(rng.uniform(0.3, 0.5), 3))
    if pick == "s3f":
        n = [_log(rng, 24, 256) for _ in range(3)]
        return dict(kind="session", nx=n[0], ny=n[1], nz=n[2], precision="fp32",
                    steps=rng.randint(1, 8), **common)
    if pick == "s3d":
        n = [_log(rng, 12, 96) for _ in range(3)]
        return dict(kind="session", nx=n[0], ny=n[1], nz=n[2], precision="fp64",
                    steps=rng.randint(1, 4), **common)
    if pick in ("s2f", "s2d"):
        hi = 2048 if pick == "s2f" else 384
        return dict(kind="session", nx=_log(rng, 48, hi), ny=_log(rng, 48, hi), nz=0,
                    precision="fp32" if pick == "s2f" else "fp64", steps=rng.randint(1, 12),
                    **common)
    if pick == "s1":
        return dict(kind="session", nx=_log(rng, 500, 100000), ny=0, nz=0,
                    precision=rng.choice(["fp32", "fp64"]), steps=rng.randint(1, 32), **common)
    if pick in ("b1", "b2", "b3"):
        dim = int(pick[1])
        lo, hi = {1: (1000, 100000), 2: (64, 1024), 3: (64, 190)}[dim]
        graph = rng.choice([2, 4, 8])
        second = rng.choice([lim, rng.choice(LIMITERS)])
        return dict(kind="batch", dim=dim, grids=rng.randint(2, {1: 16, 2: 24, 3: 5}[dim]), lo=lo,
                    hi=hi, precision="fp32", limiter=lim, second=second,
                    cfl=round(rng.uniform(0.3, 0.45), 3), steps=graph * rng.randint(1, 2),
                    graph=graph, layout=rng.randint(0, 10 ** 6))
    if pick == "r3":
        n = [_log(rng, 32, 176) for _ in range(3)]
        return dict(kind="ignition", nx=n[0], ny=n[1], nz=n[2], precision="fp32",
                    model="arrhenius", closure="nondimensional", steps=rng.randint(2, 10),
                    **dict(common, boundary="Open"))
    if pick == "r2":
        return dict(kind="ignition", nx=_log(rng, 32, 160), ny=_log(rng, 32, 160), nz=0,
                    precision="fp64", model=rng.choice(["znd", "arrhenius"]), closure="si",
                    steps=rng.randint(2, 6), **common)
    if pick == "m3":
        return dict(kind="metric", geometry="spherical", nx=_log(rng, 24, 256),
                    ny=_log(rng, 24, 192), nz=_log(rng, 24, 160), precision="fp32", limiter=lim,
                    cfl=0.4, steps=rng.randint(1, 2))
    if pick == "m2":
        return dict(kind="metric", geometry="annular", nx=_log(rng, 32, 256),
                    ny=_log(rng, 32, 256), nz=0, precision=rng.choice(["fp32", "fp64"]),
                    limiter=lim, cfl=0.4, steps=rng.randint(1, 4))
    return dict(kind="stepfn", nx=_log(rng, 32, 256), ny=_log(rng, 32, 256), nz=0,
                precision="fp64", limiter=lim, boundary=bnd)


# -- inputs ------------------------------------------------------------------------------
def _counts(case):
    return [n for n in (case["nx"], case["ny"], case["nz"]) if n]


def _mesh(counts):
    """Cell centres of the unit box, [..., y, x] layout, x first."""
    axes = [(np.arange(n) + 0.5) / n for n in counts]
    return np.meshgrid(*axes[::-1], indexing="ij")[::-1]


def _blast(counts, rng, inside, outside, radius):
    """Gas at rest with a disc / sphere of other density and pressure (1D: a split tube)."""
    mesh = _mesh(counts)
    p = np.zeros((len(counts) + 2,) + tuple(counts[::-1]))
    if len(counts) == 1:
        hot = mesh[0] < rng.uniform(0.4, 0.6)
    else:
        hot = sum((m - rng.uniform(0.47, 0.53)) ** 2 for m in mesh) <= radius ** 2
    p[0] = np.where(hot, inside[0], outside[0])
    p[-1] = np.where(hot, inside[1], outside[1])
    return p


def _explosion(case, rng):
    inside = rng.uniform(0.8, 1.2, 2)
    outside = (rng.uniform(0.1, 0.15), rng.uniform(0.08, 0.12))
    return _blast(_counts(case), rng, inside, outside, rng.uniform(0.18, 0.24))


def _batch_sizes(case):
    """The batch's grid sizes, fixed by the case: like a sweep's, they are not input data."""
    rng = np.random.default_rng(case["layout"])
    if case["dim"] == 2:
        return [int(v) for v in rng.choice([64, 128, 256, 512, 1024], case["grids"])]
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [int(round(math.exp(rng.uniform(lo, hi)))) for _ in range(case["grids"])]


def _batch_grids(case, rng):
    """(primitive, limiter) per grid."""
    out = []
    for k, n in enumerate(_batch_sizes(case)):
        counts = [n] * case["dim"]
        if case["dim"] == 2:  # quadrant Riemann problem
            X, Y = _mesh(counts)
            v = np.stack([rng.uniform(0.1, 2, 4), rng.uniform(-1, 1, 4), rng.uniform(-1, 1, 4),
                          rng.uniform(0.1, 2, 4)])
            p = v[:, (X >= 0.5).astype(int) + 2 * (Y >= 0.5).astype(int)]
        else:
            p = _blast(counts, rng, rng.uniform(0.1, 2, 2), rng.uniform(0.1, 2, 2), 0.2)
        out.append((p, case["limiter"] if k % 2 == 0 else case["second"]))
    return out


def _ignition(case, rng):
    counts = _counts(case)
    if case["closure"] == "nondimensional":  # hot spot of width about 0.05, peak T about 3
        r2 = sum((m - rng.uniform(0.48, 0.52)) ** 2 for m in _mesh(counts))
        p = np.zeros((len(counts) + 2,) + tuple(counts[::-1]))
        p[0] = 1.0
        p[-1] = 1.0 + rng.uniform(1.9, 2.1) * np.exp(-r2 / (2 * rng.uniform(0.045, 0.055) ** 2))
        return p, 1.2, NONDIM
    p = _blast(counts, rng, (1.0, rng.uniform(2.8e6, 3.2e6)), (1.0, 101325.0),
               rng.uniform(0.2, 0.25))
    return p, 1.4, SI


def _metric(case, rng):
    """(primitive, lengths, origins, face boundaries) of a curvilinear case."""
    counts = _counts(case)
    mesh = _mesh(counts)
    p = np.zeros((len(counts) + 2,) + tuple(counts[::-1]))
    if case["geometry"] == "spherical":  # r in [0.5, 1.5], theta in [0.5, pi - 0.5]
        theta = 0.5 + mesh[1] * (math.pi - 1.0)
        p[0] = 1.0 + rng.uniform(0.03, 0.07) * np.cos(4 * theta)
        p[-1] = np.where(mesh[0] < rng.uniform(0.25, 0.35), rng.uniform(3.5, 4.5), 1.0)
        # the ambient gas at rest is at a higher pressure than the outlet: it flows out
        outlet = dict(type="pressure_outlet", pressure=0.9, backflow=[1.0, -0.1, 0.0, 0.0, 0.9])
        faces = dict(x_min="wall", x_max=outlet, y_min="wall", y_max="wall", z_min="wall",
                     z_max="wall")
        return p, [1.0, math.pi - 1.0, 1.0], [0.5, 0.5, 0.0], faces
    angle = 2 * math.pi * mesh[1] + rng.uniform(0, 2 * math.pi)  # full annulus, swirling gas
    p[0] = 1.0 + rng.uniform(0.1, 0.3) * np.cos(angle)
    p[1] = 0.1 * np.sin(angle)
    p[2] = rng.uniform(0.2, 0.4)
    p[3] = 1.0 + 0.1 * mesh[0]
    faces = dict(x_min="wall", x_max="wall", y_min="periodic", y_max="periodic")
    return p, [1.0, 2 * math.pi], [0.5, 0.0], faces


def _smooth(case, rng):
    """A conservative state with waves and a shock front, and a CFL step for it."""
    counts = _counts(case)
    X, Y = _mesh(counts)
    p = np.stack([1.0 + 0.3 * np.sin(2 * math.pi * (X + rng.uniform(0, 1))),
                  0.3 * np.cos(2 * math.pi * (Y + rng.uniform(0, 1))),
                  0.2 * np.sin(2 * math.pi * (X - Y)),
                  np.where(X < rng.uniform(0.3, 0.7), 1.5, 0.5)])
    state = p.copy()
    state[1:3] *= p[0]
    state[3] = p[3] / 0.4 + 0.5 * p[0] * (p[1] ** 2 + p[2] ** 2)
    return state, 1.0 / counts[0], 1.0 / counts[1], 0.2 / max(counts)


# -- passes -------------------------------------------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "session":
        counts = _counts(case)
        sim = torch_gb300.Simulation(
            _explosion(case, rng), [1.0] * len(counts), cfl=case["cfl"], limiter=case["limiter"],
            boundaries=[case["boundary"]] * len(counts), precision=case["precision"],
            strict_cfl=False, **FOREVER)
        return dict(case=case, sim=sim)
    if kind == "metric":
        p, lengths, origins, faces = _metric(case, rng)
        sim = torch_gb300.Simulation(
            p, lengths, geometry=case["geometry"], origins=origins, face_boundaries=faces,
            cfl=case["cfl"], limiter=case["limiter"], precision=case["precision"], **FOREVER)
        return dict(case=case, sim=sim)
    if kind == "batch":
        grids = [Grid(p, [1.0] * case["dim"], precision=case["precision"], cfl=case["cfl"],
                      limiter=lim, boundaries=["Open"] * case["dim"], **FOREVER)
                 for p, lim in _batch_grids(case, rng)]
        return dict(case=case, grids=grids, batch=Batch(grids, graph_steps=case["graph"]))
    if kind == "ignition":
        p, gamma, chem = _ignition(case, rng)
        dim = p.ndim - 1
        grid = Grid(p, [1.0] * dim, precision=case["precision"], cfl=case["cfl"], gamma=gamma,
                    limiter=case["limiter"], boundaries=[case["boundary"]] * dim, reactive=True,
                    kinetic_model=case["model"], chemistry=dict(chem, closure=case["closure"]),
                    **FOREVER)
        return dict(case=case, grids=[grid], batch=Batch([grid]))
    return dict(case=case, args=_smooth(case, rng))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("session", "metric"):
        sim = state["sim"]
        sim.run(step_limit=case["steps"])
        return dict(state=sim.device_state, time=sim.time, steps=sim.steps)
    if kind == "batch":
        state["batch"].advance(case["steps"])
        state["batch"].refresh()
        return [g.current for g in state["grids"]]
    if kind == "ignition":
        state["batch"].advance(case["steps"])
        state["batch"].refresh()
        g = state["grids"][0]
        out = dict(state=g.current, lam=g.lam_ring[g.report.current], time=g.time, steps=g.steps)
        if g.beta_ring is not None:
            out["beta"] = g.beta_ring[g.report.current]
        return out
    u, dx, dy, dt = state["args"]
    return list(stepfn.muscl_hancock_step_2d(
        u, dx, dy, dt, 1.4, case["limiter"], case["boundary"], case["boundary"],
        return_fluxes=True, precision=case["precision"]))


def work(case):
    """Bytes: the state read and written once per pass however many steps it holds, since a
    pass's outputs are its last step's.  Flops: about what a cell-update of the scheme needs."""
    size = 8 if case["precision"] == "fp64" else 4
    kind = case["kind"]
    if kind == "batch":
        dim, cells = case["dim"], sum(n ** case["dim"] for n in _batch_sizes(case))
    else:
        dim, cells = len(_counts(case)), math.prod(_counts(case))
    rows = dim + 2
    if kind == "ignition":
        rows += 2 if case["model"] == "znd" else 1
    per = {1: 200, 2: 450, 3: 1000}[dim]
    if kind == "metric":
        per = {2: 700, 3: 1500}[dim]
    moved = 2 * rows * size * cells
    if kind == "stepfn":  # and the two face arrays out
        moved += size * 4 * sum(cells // n * (n + 1) for n in _counts(case))
    return dict(bytes=moved, flops=per * cells * case.get("steps", 1))


# -- the schemes in double precision --------------------------------------------------------
class _Unsuited(Exception):
    """The inputs leave the part of the scheme that is restated here."""


def _dev(a):
    t = torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64)
    return t.cuda() if torch.cuda.is_available() else t


def _conserved(p, gamma):
    u = p.clone()
    u[1:-1] *= p[0]
    u[-1] = p[-1] / (gamma - 1) + 0.5 * p[0] * (p[1:-1] ** 2).sum(0)
    return u


def _pressure(u, gamma):
    return (gamma - 1) * (u[-1] - 0.5 * (u[1:-1] ** 2).sum(0) / u[0])


def _require(*tensors):
    for t in tensors:
        if not bool((t > 1e-12).all()):
            raise _Unsuited


def _ghosts(q, bcs, width, vector):
    """Pad every axis of q by the boundary rules (vector: mirror the normal momentum)."""
    for k, bc in enumerate(bcs):
        axis = q.ndim - 1 - k
        n = q.shape[axis]
        i = torch.arange(-width, n + width, device=q.device)
        if bc == "Periodic":
            src = i % n
        elif bc == "Reflective":
            src = torch.where(i < 0, -1 - i, torch.where(i >= n, 2 * n - 1 - i, i))
        else:
            src = i.clamp(0, n - 1)
        q = q.index_select(axis, src)
        if vector and bc == "Reflective":
            q[k + 1].narrow(axis - 1, 0, width).neg_()
            q[k + 1].narrow(axis - 1, n + width, width).neg_()
    return q


def _phi(r, limiter, third_bound=True):
    pos = r.clamp(min=0)
    if limiter == "VanLeer":
        return 2 * pos / (1 + pos)
    if limiter == "Albada":
        return (pos * pos + pos) / (pos * pos + 1)
    if limiter == "MINBEE":
        return r.clamp(0, 1)
    if limiter == "Superbee":
        return torch.maximum((2 * r).clamp(max=1), r.clamp(max=2)).clamp(min=0)
    v = torch.minimum((2 * r).clamp(max=2), (2 + r) / 3)
    if third_bound:
        v = torch.minimum(v, (1 + 2 * r) / 3)
    return v.clamp(min=0)


def _slope(minus, plus, limiter, third_bound=True):
    return _phi(minus / torch.where(plus.abs() < 1e-14, 1e-14, plus), limiter, third_bound) * plus


def _flux(u, p, d):
    v = u[d + 1] / u[0]
    f = u * v
    f[d + 1] += p
    f[-1] += v * p
    return f


def _hllc(ul, ur, gl, gr, d):
    pl, pr = _pressure(ul, gl), _pressure(ur, gr)
    rl, rr = ul[0], ur[0]
    vl, vr = ul[1:-1] / rl, ur[1:-1] / rr
    unl, unr = vl[d], vr[d]
    al, ar = (gl * pl / rl).sqrt(), (gr * pr / rr).sqrt()
    sql, sqr = rl.sqrt(), rr.sqrt()
    roe = (sql * vl + sqr * vr) / (sql + sqr)
    h = (sql * (ul[-1] + pl) / rl + sqr * (ur[-1] + pr) / rr) / (sql + sqr)
    a = ((0.5 * (gl + gr) - 1) * (h - 0.5 * (roe ** 2).sum(0))).clamp(min=1e-12).sqrt()
    sl, sr = torch.minimum(unl - al, roe[d] - a), torch.maximum(unr + ar, roe[d] + a)
    den = rl * (sl - unl) - rr * (sr - unr)
    den = torch.where(den.abs() < 1e-14, 1e-14, den)
    ss = (pr - pl + rl * unl * (sl - unl) - rr * unr * (sr - unr)) / den
    out = torch.full_like(ul, math.nan)
    for u, un, v, p, r, s, outer, star in (
            (ul, unl, vl, pl, rl, sl, 0 <= sl, (sl <= 0) & (0 <= ss)),
            (ur, unr, vr, pr, rr, sr, 0 >= sr, (ss <= 0) & (0 <= sr))):
        f = _flux(u, p, d)
        k = r * (s - un) / torch.where((s - ss).abs() < 1e-14, 1e-14, s - ss)
        us = torch.cat([k[None], k * v, k[None]])
        us[d + 1] = k * ss
        du = torch.where((s - un).abs() < 1e-14, 1e-14, s - un)
        us[-1] = k * (u[-1] / r + (ss - un) * (ss + p / (r * du)))
        fs = torch.where((s - ss).abs() < 1e-12, f, f + s * (us - u))
        out = torch.where(outer, f, torch.where(star, fs, out))
    return out


def _hydro(u, gamma, h, dt, limiter, bcs):
    """One MUSCL-Hancock / HLLC step; also the face fluxes per direction."""
    dim = u.ndim - 1
    P = _ghosts(u, bcs, 2, True)
    G = gamma
    if torch.is_tensor(gamma):
        G = _ghosts(gamma, bcs, 1, False)

    def cut(d, off):  # the cells and one ring around them, shifted along d
        at = [slice(None)] + [slice(1, -1)] * dim
        n = P.shape[dim - d]
        at[dim - d] = slice(1 + off, n - 1 + off)
        return P[tuple(at)]

    U = cut(0, 0)
    slopes = [_slope(U - cut(d, -1), cut(d, 1) - U, limiter, dim == 3) for d in range(dim)]
    bar = U.clone()
    for d, s in enumerate(slopes):
        hi, lo = U + 0.5 * s, U - 0.5 * s
        bar -= 0.5 * dt / h[d] * (_flux(hi, _pressure(hi, G), d) - _flux(lo, _pressure(lo, G), d))
    out, fluxes = u, []
    for d, s in enumerate(slopes):
        axis = dim - d
        at = [slice(None)] + [slice(1, -1)] * dim
        at[axis] = slice(None)
        hi, lo = (bar + 0.5 * s)[tuple(at)], (bar - 0.5 * s)[tuple(at)]
        _require(hi[0], lo[0], _pressure(hi, 1.4), _pressure(lo, 1.4))
        n = hi.shape[axis]
        left, right = hi.narrow(axis, 0, n - 1), lo.narrow(axis, 1, n - 1)
        gl = gr = gamma
        if torch.is_tensor(gamma):
            g = G[tuple(at[1:])]
            gl, gr = g.narrow(axis - 1, 0, n - 1), g.narrow(axis - 1, 1, n - 1)
        f = _hllc(left, right, gl, gr, d)
        fluxes.append(f)
        out = out - dt / h[d] * f.diff(dim=axis)
    _require(out[0], _pressure(out, 1.4))
    return out, fluxes


def _cfl_dt(u, gamma, h, cfl):
    a = (gamma * _pressure(u, gamma) / u[0]).sqrt()
    return cfl / sum(float(((u[d + 1] / u[0]).abs() + a).max()) / h[d]
                     for d in range(u.ndim - 1))


def _solve(u, h, cfl, limiter, bcs, steps):
    t = 0.0
    for _ in range(steps):
        dt = _cfl_dt(u, 1.4, h, cfl)
        u = _hydro(u, 1.4, h, dt, limiter, bcs)[0]
        t += dt
    return u, t


def _ends(u, bc, vector=True):
    """One ghost cell on either side of a tube."""
    lo, hi = (u[..., -1:], u[..., :1]) if bc == "Periodic" else (u[..., :1], u[..., -1:])
    if vector and bc == "Reflective":
        flip = torch.tensor([[1.0], [-1.0], [1.0]], dtype=u.dtype, device=u.device)
        lo, hi = lo * flip, hi * flip
    return torch.cat([lo, u, hi], -1)


def _waves(u, g):
    """Interface wave speeds from a pressure estimate (PVRS), per interface of padded cells."""
    rho, v, p = u[0], u[1] / u[0], _pressure(u, g)
    a = (g * p / rho).sqrt()
    mean = lambda q: 0.5 * (q[:-1] + q[1:])  # noqa: E731
    ps = (mean(p) - 0.5 * v.diff() * mean(rho) * mean(a)).clamp(min=0)
    q = lambda pk: torch.where(  # noqa: E731
        ps > pk, (1 + (g + 1) / (2 * g) * (ps / pk - 1)).clamp(min=0).sqrt(), 1.0)
    return v[:-1] - a[:-1] * q(p[:-1]), v[1:] + a[1:] * q(p[1:])


def _tube(u, dx, cfl, limiter, bc, steps, g=1.4):
    """The 1D chain: Sweby-bounded slopes, half-step predictor, HLLC with the cell states'
    wave speeds."""
    t = 0.0
    for _ in range(steps):
        P = _ends(u, bc)
        sl, sr = _waves(P, g)
        speed = (P[1] / P[0]).abs() + (g * _pressure(P, g) / P[0]).sqrt()
        dt = cfl * dx / max(float(sl.abs().max()), float(sr.abs().max()), float(speed.max()))
        up, down = u - P[:, :-2], P[:, 2:] - u
        mach = (u[1] / u[0]).abs() / (g * _pressure(u, g) / u[0]).sqrt()
        w = ((1 - mach) / (1 + mach)).clamp(-1, 1)
        r = torch.nan_to_num(up / down, nan=0.0, posinf=0.0, neginf=0.0)
        den = 1 - w + (1 + w) * r
        cap = 2 / torch.where(den.abs() < 1e-12, 1e-12, den)
        eps = _phi(r, limiter, False)
        if limiter == "MINBEE":
            eps = torch.where(r >= 1, torch.minimum(eps, cap), eps)
        else:
            eps = torch.where(r > 0, torch.minimum(eps, cap), 0.0)
        size = torch.minimum((eps.clamp(min=0) * 0.5 * (P[:, 2:] - P[:, :-2])).abs(),
                             2 * torch.minimum(up.abs(), down.abs()))
        s = torch.where(up * down > 0, down.sign() * size, 0.0)
        lo, hi = u - 0.5 * s, u + 0.5 * s
        half = 0.5 * dt / dx * (_flux(hi, _pressure(hi, g), 0) - _flux(lo, _pressure(lo, g), 0))
        lo, hi = lo - half, hi - half
        _require(lo[0], hi[0], _pressure(lo, g), _pressure(hi, g))
        ends = torch.stack([lo, hi], -1).reshape(3, -1)
        ends = _ends(ends, bc)
        L, R = ends[:, 0::2], ends[:, 1::2]
        pl, pr = _pressure(L, g), _pressure(R, g)
        vl, vr = L[1] / L[0], R[1] / R[0]
        den = L[0] * (sl - vl) - R[0] * (sr - vr)
        ss = (pr - pl + L[0] * vl * (sl - vl) - R[0] * vr * (sr - vr)) / torch.where(
            den.abs() < 1e-14, 1e-14, den)
        ss = torch.minimum(torch.maximum(ss, sl), sr)
        f = []
        for V, v, p, S in ((L, vl, pl, sl), (R, vr, pr, sr)):
            F = _flux(V, p, 0)
            ok = (S - ss).abs() > 1e-12
            star = V[0] * (S - v) / torch.where(ok, S - ss, 1.0) * torch.stack(
                [torch.ones_like(ss), ss, V[2] / V[0] + (ss - v) * (ss + p / (V[0] * (S - v)))])
            f += [F, F + S * (torch.where(ok, star, V) - V)]
        F = torch.where(sl > 0, f[0], torch.where(ss > 0, f[1], torch.where(sr >= 0, f[3], f[2])))
        u = u - dt / dx * F.diff(dim=-1)
        _require(u[0], _pressure(u, g))
        t += dt
    return u, t


def _react(u, lam, beta, dt, case, chem):
    """Exponential-midpoint source on the cell's normal projection."""
    si = case["closure"] == "si"
    side = 0.5 * (u[2:-1] ** 2).sum(0) / u[0]
    e = u[-1] - side

    def rate(q, energy):
        g = (4.5 - q) / (3.5 - q) if si else 1.2
        p = (g - 1) * (energy - 0.5 * u[1] ** 2 / u[0])
        if si:
            molar = q * (2 / 3) * 2.016 + q * (1 / 3) * 32.0 + (1 - q) * 18.016
            return chem["pre_exponential"] * torch.exp(
                -chem["activation_energy"] / (8.314 * p * molar / (u[0] * 8314.46)))
        return chem["pre_exponential"] * torch.exp(-chem["activation_energy"] * u[0] / p)

    def advance(k, span):
        if case["model"] == "znd":
            active = (span - beta / k.clamp(min=1e-300)).clamp(min=0)
            return lam * torch.exp(-5.0 * k * active), (beta - k * span).clamp(0, 1)
        return lam * torch.exp(-k * span), beta

    mid, _ = advance(rate(lam, e), 0.5 * dt)
    k = rate(mid, e + chem["q_heat"] * u[0] * (lam - mid))
    new, left = advance(k, dt)
    out = u.clone()
    out[-1] += chem["q_heat"] * u[0] * (lam - new)
    return out, new, left


def _transport(q, old, new, fluxes, dt, h, bcs):
    dim = q.ndim
    padded = _ghosts(q, bcs, 1, False)
    rq = old * q
    for d, f in enumerate(fluxes):
        axis = dim - 1 - d
        at = [slice(1, -1)] * dim
        at[axis] = slice(None)
        line = padded[tuple(at)]
        n = line.shape[axis]
        m = f[0]
        up = torch.where(m >= 0, line.narrow(axis, 0, n - 1), line.narrow(axis, 1, n - 1))
        rq = rq - dt / h[d] * (m * up).diff(dim=axis)
    return (rq / new).clamp(0, 1)


def _burn(case, p, gamma0, chem):
    """Strang-split reactive steps; an attempt may only halve dt (each counts as one)."""
    si = case["closure"] == "si"
    counts = _counts(case)
    h = [1.0 / n for n in counts]
    bcs = [case["boundary"]] * len(counts)
    gam = (lambda q: (4.5 - q) / (3.5 - q)) if si else (lambda q: gamma0)
    lam, beta = torch.ones_like(p[0]), torch.ones_like(p[0])
    u = _conserved(p, gam(lam))
    t, done, dt = 0.0, 0, _cfl_dt(u, gam(lam), h, case["cfl"])
    for _ in range(case["steps"]):
        a, la, ba = _react(u, lam, beta, 0.5 * dt, case, chem)
        allowed = _cfl_dt(a, gam(la), h, case["cfl"])
        if dt > allowed * (1 + 1e-12):
            dt = dt / 2 if dt / 2 <= allowed else allowed
            continue
        b, fluxes = _hydro(a, gam(la), h, dt, case["limiter"], bcs)
        lb = _transport(la, a[0], b[0], fluxes, dt, h, bcs)
        bb = _transport(ba, a[0], b[0], fluxes, dt, h, bcs)
        u, lam, beta = _react(b, lb, bb, 0.5 * dt, case, chem)
        t, done = t + dt, done + 1
        dt = _cfl_dt(u, gam(lam), h, case["cfl"])
    out = dict(state=u, lam=lam, time=t, steps=None)
    if case["model"] == "znd":
        out["beta"] = beta
    return out


class _Curved:
    """MUSCL-Rusanov-SSPRK2 on the wedge and the annulus."""

    def __init__(self, case, lengths, origins, faces):
        counts = _counts(case)
        ax = [np.linspace(o, o + w, n + 1) for o, w, n in zip(origins, lengths, counts)]
        wid = [np.diff(a) for a in ax]
        shell2 = np.diff(ax[0] ** 2) / 2
        if case["geometry"] == "spherical":
            solid = -np.diff(np.cos(ax[1]))
            vol = [np.diff(ax[0] ** 3) / 3, solid, wid[2]]
            area = [[ax[0] ** 2, solid, wid[2]], [shell2, np.sin(ax[1]), wid[2]],
                    [shell2, wid[1], np.ones(counts[2] + 1)]]
        else:
            vol = [shell2, wid[1]]
            area = [[ax[0], wid[1]], [wid[0], np.ones(counts[1] + 1)]]
        outer = lambda fs: _dev(  # noqa: E731
            math.prod(np.reshape(f, [-1] + [1] * k) for k, f in enumerate(fs)))
        self.dim, self.case = len(counts), case
        self.vol, self.area = outer(vol), [outer(f) for f in area]
        kind = lambda k: faces["xyz"[k // 2] + ("_min", "_max")[k % 2]]  # noqa: E731
        self.face = [kind(k) if isinstance(kind(k), dict) else dict(type=kind(k))
                     for k in range(2 * self.dim)]
        div = [a.diff(dim=self.dim - 1 - d) / self.vol for d, a in enumerate(self.area)]
        self.radial = div[0]
        self.cot = div[1] if case["geometry"] == "spherical" else None

    def plane(self, p, d, side):
        """The state beyond a boundary face."""
        axis = p.ndim - 1 - d
        face = self.face[2 * d + (side > 0)]
        n = p.shape[axis]
        if face["type"] == "periodic":
            return p.narrow(axis, n - 1 if side < 0 else 0, 1)
        q = p.narrow(axis, 0 if side < 0 else n - 1, 1).clone()
        if face["type"] == "wall":
            q[d + 1] = -q[d + 1]
            return q
        g, pb = 1.4, face["pressure"]  # pressure outlet
        a, un = (g * q[-1] / q[0]).sqrt(), side * q[d + 1]
        rho = q[0] * (pb / q[-1]) ** (1 / g)
        vel = un + 2 * (a - (g * pb / rho).sqrt()) / (g - 1)
        sub = un < a
        back = sub & ((vel < 0) | (un < 0))
        q[0], q[-1] = torch.where(sub, rho, q[0]), torch.where(sub, pb, q[-1])
        q[d + 1] = torch.where(sub, side * vel, q[d + 1])
        flow = torch.tensor(face["backflow"], dtype=q.dtype, device=q.device)
        return torch.where(back, flow.reshape([-1] + [1] * self.dim), q)

    def prim(self, u):
        p = u / u[0]
        p[0], p[-1] = u[0], _pressure(u, 1.4)
        return p

    def rhs(self, u):
        p = self.prim(u)
        k = torch.zeros_like(u)
        k[1] = p[-1] * self.radial
        if self.cot is not None:
            r = self.radial / 2
            k[1] += p[0] * (p[2] ** 2 + p[3] ** 2) * r
            k[2] = p[-1] * self.cot - p[0] * p[1] * p[2] * r + p[0] * p[3] ** 2 * self.cot
            k[3] = -p[0] * p[3] * (p[1] * r + p[2] * self.cot)
        else:
            k[1] += p[0] * p[2] ** 2 * self.radial
            k[2] = -p[0] * p[1] * p[2] * self.radial
        for d in range(self.dim):
            axis = p.ndim - 1 - d
            n = p.shape[axis]
            P = torch.cat([self.plane(p, d, -1), p, self.plane(p, d, 1)], axis)
            mid = P.narrow(axis, 1, n)
            s = torch.zeros_like(P)
            inner = _slope(mid - P.narrow(axis, 0, n), P.narrow(axis, 2, n) - mid,
                           self.case["limiter"])
            _require(*(mid[c] - 0.5 * inner[c].abs() for c in (0, -1)))
            s.narrow(axis, 1, n).copy_(inner)
            if self.face[2 * d]["type"] == "periodic":
                s.narrow(axis, 0, 1).copy_(inner.narrow(axis, n - 1, 1))
                s.narrow(axis, n + 1, 1).copy_(inner.narrow(axis, 0, 1))
            L = (P + 0.5 * s).narrow(axis, 0, n + 1).clone()
            R = (P - 0.5 * s).narrow(axis, 1, n + 1).clone()
            for at, to, of, f in ((0, L, R, self.face[2 * d]), (n, R, L, self.face[2 * d + 1])):
                if f["type"] == "wall":
                    edge = of.narrow(axis, at, 1).clone()
                    edge[d + 1] = -edge[d + 1]
                    to.narrow(axis, at, 1).copy_(edge)
            ul, ur = _conserved(L, 1.4), _conserved(R, 1.4)
            speed = torch.maximum(*(q[d + 1].abs() + (1.4 * q[-1] / q[0]).sqrt() for q in (L, R)))
            f = 0.5 * (_flux(ul, L[-1], d) + _flux(ur, R[-1], d) - speed * (ur - ul))
            k = k - (f * self.area[d]).diff(dim=axis) / self.vol
        return k

    def dt(self, u):
        p = self.prim(u)
        rate = 0.0
        for d in range(self.dim):
            axis = p.ndim - 1 - d
            P = torch.cat([self.plane(p, d, -1), p, self.plane(p, d, 1)], axis)
            s = P[d + 1].abs() + (1.4 * P[-1] / P[0]).sqrt()
            m = s.shape[axis - 1] - 1
            f = self.area[d] * torch.maximum(s.narrow(axis - 1, 0, m), s.narrow(axis - 1, 1, m))
            rate = rate + torch.maximum(f.narrow(axis - 1, 0, m - 1),
                                        f.narrow(axis - 1, 1, m - 1)) / self.vol
        return self.case["cfl"] / float(rate.max())

    def solve(self, p):
        u, t = _conserved(p, 1.4), 0.0
        for _ in range(self.case["steps"]):
            dt = self.dt(u)
            mid = u + dt * self.rhs(u)
            _require(mid[0], _pressure(mid, 1.4))
            u = 0.5 * (u + mid + dt * self.rhs(mid))
            t += dt
        return u, t


def exact(case, seed):
    """What run() returns on these inputs, in double precision; None where the inputs take a
    branch that is not restated here."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    try:
        if kind == "session":
            counts = _counts(case)
            u = _conserved(_dev(_explosion(case, rng)), 1.4)
            if len(counts) == 1:
                u, t = _tube(u, 1.0 / counts[0], case["cfl"], case["limiter"], case["boundary"],
                             case["steps"])
            else:
                u, t = _solve(u, [1.0 / n for n in counts], case["cfl"], case["limiter"],
                              [case["boundary"]] * len(counts), case["steps"])
            return dict(state=u, time=t, steps=None)
        if kind == "metric":
            p, lengths, origins, faces = _metric(case, rng)
            u, t = _Curved(case, lengths, origins, faces).solve(_dev(p))
            return dict(state=u, time=t, steps=None)
        if kind == "batch":
            out = []
            for p, lim in _batch_grids(case, rng):
                u, n, dim = _conserved(_dev(p), 1.4), p.shape[-1], case["dim"]
                try:
                    if dim == 1:
                        u = _tube(u, 1.0 / n, case["cfl"], lim, "Open", case["steps"])[0]
                    else:
                        u = _solve(u, [1.0 / n] * dim, case["cfl"], lim, ["Open"] * dim,
                                   case["steps"])[0]
                except _Unsuited:
                    u = None
                out.append(u)
            return out
        if kind == "ignition":
            p, gamma, chem = _ignition(case, rng)
            return _burn(case, _dev(p), gamma, chem)
        u, dx, dy, dt = _smooth(case, rng)
        new, fluxes = _hydro(_dev(u), 1.4, [dx, dy], dt, case["limiter"], [case["boundary"]] * 2)
        return [new] + fluxes
    except _Unsuited:
        return None
