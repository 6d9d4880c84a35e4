"""Performance cases: the work that a magnetotelluric modelling program has
this framework do, each through a public entry point.

Kinds
  survey    Survey.solve + Receivers.fields: all systems (frequencies x
            polarisations) of a survey from zero initial guesses to E and H at
            the receivers; the survey object is kept, the right-hand sides are
            new.  The solutions are iterated to 1e-9, a digit below the
            default, so that E and H are determined to ~1e-10.
  forward   ImpedanceProblem.forward: one model of an inversion, from the
            logarithms of the cell conductivities to E and H (assembly,
            right-hand sides, solver set-up, solve, receivers).
  dropin    pcocr_2x2_folded: the reference program's call, host arrays in
            and out, in double-float arithmetic; E and H of its solution.
  fp64      CocrContext.solve: the reference's algorithm in plain FP64.
  operator  Survey.spmv: A_k x_k for every system of a survey.
  assemble  Assembly + block2x2: BuildMatrix's work, the SLAE in host arrays.
  response  Receivers.fields + mt_response with the smoothed output.
  gradient  mtgpu_adjoint_gradient: the backward direction's reduction over
            cells, from forward and adjoint solutions.

Meshes are nx x ny x nz cells: a core of size h, `pad` cells growing by `ratio`
on the sides and below, `air` cells above; layered earth with random blocks.
nf frequencies are spread over f_lo .. f_hi (log scale), each with both
polarisations.  verify: iterate until the true residual is below eps too, as
the survey driver does; otherwise stop by the reference's rule.
"""
import ctypes
import math

import numpy as np
import torch

from mtcalc_with_dfp_cocr_gb300 import _lib, normal1d, solver
from mtcalc_with_dfp_cocr_gb300.adjoint import ImpedanceProblem
from mtcalc_with_dfp_cocr_gb300.assembly import Assembly
from mtcalc_with_dfp_cocr_gb300.mesh import Layer, layered_model, padded_lines, z_lines
from mtcalc_with_dfp_cocr_gb300.receivers import Receivers
from mtcalc_with_dfp_cocr_gb300.slae_io import mesh_to_solve_mesh
from mtcalc_with_dfp_cocr_gb300.survey import Survey

MU0 = 1.25663706143591729e-6
EPS = 1e-9
MAXITER = 20000


def _case(name, kind, nx, ny, nz, nf=1, f_lo=1.0, f_hi=1.0, h=100.0, pad=6, air=6, ratio=1.4,
          verify=True):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, nf=nf, f_lo=f_lo, f_hi=f_hi, h=h, pad=pad, air=air,
             ratio=ratio, verify=verify)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the plain benchmark mesh, one frequency: the smallest solve, bound by launches
        _case("survey_24_1f", "survey", 24, 24, 24, ratio=1.5),
        # the headline: a 1.8M-edge mesh at one frequency, both polarisations
        _case("survey_96_1f", "survey", 96, 96, 64, f_lo=0.1, f_hi=0.1, h=50.0, pad=10, air=10),
        # the mixed-precision configuration's frequencies (6 systems, a padded batch)
        _case("survey_64_3f", "survey", 64, 64, 48, 3, 0.01, 100.0, pad=8, air=8),
        # the adjoint configuration's mesh and frequencies
        _case("survey_48_8f", "survey", 48, 48, 32, 8, 0.01, 100.0),
        # a full batch of 32 systems on an odd mesh, the reference's stop rule
        _case("survey_37x45x29_16f", "survey", 37, 45, 29, 16, 0.01, 1000.0, verify=False),
        # one step of an inversion: everything from the model to E and H
        _case("forward_40x36x28_4f", "forward", 40, 36, 28, 4, 0.1, 100.0),
        # the reference program's call on one system
        _case("dropin_31x27x22", "dropin", 31, 27, 22, f_lo=0.3, f_hi=0.3),
        # the plain FP64 solver on the plain benchmark mesh
        _case("fp64_24", "fp64", 24, 24, 24, ratio=1.5),
        # operator products of a whole survey (residual checks, forward operators)
        _case("operator_64_16f", "operator", 64, 64, 48, 16, 0.01, 1000.0, pad=8, air=8),
        # the SLAE of one system as the reference's BuildMatrix hands it on
        _case("assemble_40x36x28", "assemble", 40, 36, 28),
        # receiver output of a survey's solutions
        _case("response_48_8f", "response", 48, 48, 32, 8, 0.01, 100.0),
        # the gradient's cell reduction of a survey
        _case("gradient_48_8f", "gradient", 48, 48, 32, 8, 0.01, 100.0),
    ]


def draw(rng):
    kind = rng.choice(["survey"] * 5 + ["forward", "dropin", "fp64", "operator", "assemble",
                                        "response", "gradient"])
    cells = math.exp(rng.uniform(math.log(12e3), math.log(250e3)))   # 23^3 .. 63^3
    if kind in ("dropin", "fp64"):
        cells = min(cells, 40e3)
    if kind in ("forward", "assemble", "response"):
        cells = min(cells, 80e3)
    side = cells ** (1.0 / 3.0)
    nx = max(20, round(side * rng.uniform(0.85, 1.25)))
    ny = max(20, round(side * rng.uniform(0.85, 1.25)))
    nz = max(20, round(cells / (nx * ny)))
    nf = 1
    if kind not in ("dropin", "fp64", "assemble"):
        # systems x edges up to about the largest listed case's
        most = max(1, min(16, int(1.8e6 / (3.0 * nx * ny * nz))))
        nf = round(math.exp(rng.uniform(0.0, math.log(most)))) if most > 1 else 1
    f_lo = 10.0 ** rng.uniform(-1.5, 0.5)
    f_hi = f_lo if nf == 1 else f_lo * 10.0 ** rng.uniform(1.0, 2.5)
    return _case(None, kind, nx, ny, nz, nf, round(f_lo, 4), round(f_hi, 4),
                 ratio=rng.choice([1.4, 1.5]), verify=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _model(case, rng):
    """Layered earth with random blocks; layer and block faces on mesh lines."""
    h, pad, air, ratio = case["h"], case["pad"], case["air"], case["ratio"]
    x = padded_lines(h, case["nx"] - 2 * pad, pad, ratio)
    y = padded_lines(h, case["ny"] - 2 * pad, pad, ratio)
    z = z_lines(h, case["nz"] - pad - air, pad, ratio, air, ratio)
    top = int(np.argmin(np.abs(z)))
    layers = [Layer(float(z[top - 6]), 10.0 ** rng.uniform(-3, -2)),
              Layer(float(z[top - 3]), 10.0 ** rng.uniform(-1.5, -0.5)),
              Layer(0.0, 10.0 ** rng.uniform(-2.2, -1.8))]
    blocks = []
    for _ in range(8):
        sx, sy, sz = (int(v) for v in rng.integers(2, 6, 3))
        ix = int(rng.integers(pad, case["nx"] - pad - sx + 1))
        iy = int(rng.integers(pad, case["ny"] - pad - sy + 1))
        it = top - int(rng.integers(0, 3))
        blocks.append((x[ix], x[ix + sx], y[iy], y[iy + sy], z[max(1, it - sz)], z[it],
                       10.0 ** rng.uniform(-3, 0)))
    return layered_model(x, y, z, layers, blocks=blocks)


def _receivers(h, n=9):
    c = h * (np.arange(n) - (n - 1) / 2.0)
    X, Y = np.meshgrid(c, c, indexing="xy")
    return np.stack([X.ravel(), Y.ravel(), np.zeros(n * n)], axis=1)


def _freqs(case, rng):
    f = np.geomspace(case["f_lo"], case["f_hi"], case["nf"])
    return f * 10.0 ** rng.uniform(-0.02, 0.02, case["nf"])


def _systems(mesh, freqs):
    """nu, alfa and the 1-D tables of every system (X then Y per frequency)."""
    tabs = [normal1d.solve_1d(f, [l.top for l in mesh.layers], [l.sigma for l in mesh.layers])
            for f in freqs]
    return (np.repeat(freqs, 2), np.tile(np.array([1, 0], np.int32), len(freqs)), tabs[0][0],
            np.repeat(np.stack([t[1] for t in tabs]), 2, axis=0),
            np.repeat(np.stack([t[2] for t in tabs]), 2, axis=0))


def _smooth_solution(mesh, S, rng):
    """A smooth complex field per system as edge values: plane waves across
    the core, decaying with distance from the surface."""
    X, Y, Z = (np.asarray(v) for v in (mesh.x, mesh.y, mesh.z))
    out = np.empty((S, mesh.nb), np.complex128)
    ids = [i.reshape(mesh.nz, mesh.ny, mesh.nx) for i in mesh._edge_ids()]
    kx, ky = rng.uniform(-2e-3, 2e-3, (2, S))
    amp = rng.standard_normal((S, 3)) + 1j * rng.standard_normal((S, 3))
    depth = rng.uniform(500.0, 3000.0, S)
    for d in range(3):
        e = ids[d] >= 0
        length = np.append(np.diff((X, Y, Z)[d]), 0.0)
        shape = [1, 1, 1]
        shape[2 - d] = -1
        half = 0.5 * length.reshape(shape)
        for k in range(S):
            v = (amp[k, d] * np.exp(1j * kx[k] * X)[None, None, :] *
                 np.exp(1j * ky[k] * Y)[None, :, None] *
                 np.exp(-np.abs(Z) / depth[k])[:, None, None])
            out[k, ids[d][e]] = (v * half)[e]
    return torch.from_numpy(out.view(np.float64)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"], case["nf"]])
    mesh = _model(case, rng)
    freqs = _freqs(case, rng)
    st = dict(case=case, mesh=mesh, freqs=freqs, points=_receivers(case["h"]))
    if kind == "forward":
        st["log_sigma"] = np.log(mesh.cell_sigma) + np.where(
            mesh.cell_sigma > 1e-6, 0.2 * rng.standard_normal(mesh.kpar), 0.0)
        st["problem"] = ImpedanceProblem(mesh, freqs, st["points"], eps=EPS, maxiter=MAXITER)
        return st
    st["sys"] = nus, alfas, z1d, usin, ucos = _systems(mesh, freqs)
    if kind == "assemble":
        return st
    S = len(nus)
    A = st["assembly"] = Assembly(mesh)
    if kind == "gradient":
        st["u"], st["lam"] = (_smooth_solution(mesh, S, rng) for _ in range(2))
        return st
    if kind == "response":
        st["u"] = _smooth_solution(mesh, S, rng)
        st["receivers"] = Receivers(A, st["points"], output="smooth")
        return st
    if kind == "operator":
        st["survey"] = Survey(A, nus)
        st["x"] = torch.from_numpy(rng.standard_normal((S, 2 * mesh.nb))).cuda()
        return st
    st["receivers"] = Receivers(A, st["points"])
    if kind == "dropin":
        st["sys"] = nus, alfas, z1d, usin, ucos = nus[:1], alfas[:1], z1d, usin[:1], ucos[:1]
        st["slae"] = A.block2x2(nus[0], alfas[0], z1d, usin[0], ucos[0], eps=EPS)
        st["solve_mesh"] = mesh_to_solve_mesh(mesh)
        return st
    if kind == "fp64":
        st["sys"] = nus, alfas, z1d, usin, ucos = nus[:1], alfas[:1], z1d, usin[:1], ucos[:1]
        S = 1
        st["context"] = A.cocr(nus[0])
    else:
        st["survey"] = Survey(A, nus)
    st["b"] = torch.empty(S, 2 * mesh.nb, dtype=torch.float64, device="cuda")
    A.rhs(nus, alfas, z1d, usin, ucos, st["b"])
    return st


# -------------------------------------------------------------------- runs
def _fields(st, x):
    E, H, _ = st["receivers"].fields(x, *st["sys"])
    return {"E": E, "H": H}


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "survey":
        x = torch.zeros_like(st["b"])
        st["survey"].solve(st["b"], x, eps=EPS, maxiter=MAXITER, verify=case["verify"])
        return _fields(st, x)
    if kind == "forward":
        s = st["problem"].forward(st["log_sigma"])[1]
        return {"E": s.E, "H": s.H}
    if kind == "dropin":
        x = solver.pcocr_2x2_folded(st["slae"], st["solve_mesh"], eps=EPS, maxiter=MAXITER,
                                    stop_on_true_residual=case["verify"], double_float=True)[1]
        return _fields(st, torch.from_numpy(x).cuda())
    if kind == "fp64":
        x = torch.zeros_like(st["b"])
        st["context"].solve(st["b"], x, eps=EPS, maxiter=MAXITER,
                            stop_on_true_residual=case["verify"])
        return _fields(st, x)
    if kind == "operator":
        y = torch.empty_like(st["x"])
        st["survey"].spmv(st["x"], y)
        return y
    if kind == "assemble":
        nus, alfas, z1d, usin, ucos = st["sys"]
        s = Assembly(st["mesh"]).block2x2(nus[0], alfas[0], z1d, usin[0], ucos[0])
        return {"ig": s.ig, "jg": s.jg, "idi": s.idi, "ijg": s.ijg, "di": s.di, "gg": s.gg,
                "pr": s.pr}
    if kind == "response":
        out = _fields(st, st["u"])
        n = 2 * len(st["freqs"])
        out["mt"] = st["receivers"].mt_response(st["freqs"], np.arange(0, n, 2),
                                                np.arange(1, n, 2), out["E"], out["H"])
        return out
    nus, alfas, z1d, usin, ucos = st["sys"]
    grad = torch.empty(st["mesh"].kpar, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().mtgpu_adjoint_gradient(
        st["assembly"]._h, len(nus), nus, alfas, len(z1d), z1d, usin, ucos,
        ctypes.c_void_p(st["u"].data_ptr()), ctypes.c_void_p(st["lam"].data_ptr()),
        ctypes.c_void_p(grad.data_ptr())), "mtgpu_adjoint_gradient")
    return grad


# ------------------------------------------------------------ minimal work
def work(case):
    """Bytes and operations of one pass.  A solve: one iteration reads and
    writes the recurrences' vectors (x, p, a, r, s and the smoothed residual)
    once and reads the diagonal preconditioner once, 13 vectors; the number
    of iterations to 1e-9 is about 10 per cell along the longest axis + 150."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cells = nx * ny * nz
    nb = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    S = 1 if case["kind"] in ("dropin", "fp64", "assemble") else 2 * case["nf"]
    vec = 16.0 * nb * S
    product = 8.0 * 9 * nb * S + 4.0 * 24 * nb * S    # complex and real entries of a row
    if case["kind"] in ("survey", "forward", "dropin", "fp64"):
        its = 10 * max(nx, ny, nz) + 150
        return {"bytes": its * 13 * vec, "flops": its * (product + 90.0 * nb * S)}
    if case["kind"] == "operator":
        return {"bytes": 2 * vec + 8.0 * cells, "flops": product}
    if case["kind"] == "assemble":
        return {"bytes": 12.0 * cells + (16 * 12 + 40.0) * nb, "flops": 12 * 12 * 10.0 * cells}
    if case["kind"] == "response":
        # the edges within five cells of the receivers' cells
        near = 3.0 * min(nx, 20) * min(ny, 20) * min(nz, 11)
        return {"bytes": 16.0 * near * S + 81 * (96 + 17 * 16.0) * S, "flops": 500.0 * near * S}
    return {"bytes": 2 * vec + 16.0 * cells, "flops": 12 * 20.0 * cells * S}


# ----------------------------------------------------- values in 64 bits
def _grid(mesh, v, d):
    """The +d edges of an edge vector as an array [z, y, x] (0 where a node has none)."""
    ids = mesh._edge_ids()[d].reshape(mesh.nz, mesh.ny, mesh.nx)
    return np.where(ids >= 0, v[np.maximum(ids, 0)], 0.0), ids


def _inner(mesh, d):
    """Whether an edge [z, y, x] of direction d is off the outer surface."""
    n = (mesh.nz, mesh.ny, mesh.nx)
    ok = np.ones(n, bool)
    for a in range(3):
        if a == 2 - d:      # no +d edge at the last node
            ok[tuple(slice(-1, None) if b == a else slice(None) for b in range(3))] = False
        else:
            for s in (slice(0, 1), slice(-1, None)):
                ok[tuple(s if b == a else slice(None) for b in range(3))] = False
    return ok


def _cut(a, axis, lo, hi):
    """a without its first lo and last hi entries along axis."""
    return a[tuple(slice(lo, a.shape[b] - hi) if b == axis else slice(None) for b in range(3))]


def _put(out, axis, side, v):
    """out += v shifted to the low (0) or high (1) nodes of axis."""
    n = out.shape[axis]
    out[tuple((slice(0, n - 1) if side == 0 else slice(1, n)) if b == axis else slice(None)
              for b in range(3))] += v


def _sizes(mesh):
    return (np.diff(mesh.x)[None, None, :], np.diff(mesh.y)[None, :, None],
            np.diff(mesh.z)[:, None, None])


def _cell_mass(t, axes):
    """The mass matrix [[2, 1], [1, 2]] / 3 along both transverse axes of a
    cell's four parallel edges t[(a, b)]."""
    m = {}
    for a in (0, 1):
        for b in (0, 1):
            m[a, b] = (4 * t[a, b] + 2 * t[1 - a, b] + 2 * t[a, 1 - b] + t[1 - a, 1 - b]) / 9.0
    return m


def _cell_edges(g, d):
    """The four +d edges of every cell, by their sides along the transverse axes."""
    ax = 2 - d
    p, q = 2 - (d + 1) % 3, 2 - (d + 2) % 3
    e = _cut(g, ax, 0, 1)
    return {(a, b): _cut(_cut(e, p, a, 1 - a), q, b, 1 - b) for a in (0, 1) for b in (0, 1)}, ax, p, q


def _apply(mesh, omega, v):
    """(K + i omega M) v with the outer surface's edges mapped to themselves."""
    h = _sizes(mesh)
    sig = mesh.mat_sigma[mesh.nvkat].reshape(mesh.nz - 1, mesh.ny - 1, mesh.nx - 1)
    inner = [_inner(mesh, d) for d in range(3)]
    g = [np.where(inner[d], _grid(mesh, v, d)[0], 0.0) for d in range(3)]
    out = [np.zeros((mesh.nz, mesh.ny, mesh.nx), np.complex128) for _ in range(3)]
    for n in range(3):
        # circulations of the faces of normal n, mass matrix along n, and back
        a, b = (n + 1) % 3, (n + 2) % 3
        ea, eb, en = 2 - a, 2 - b, 2 - n
        ga, gb = _cut(g[a], ea, 0, 1), _cut(g[b], eb, 0, 1)
        f = (_cut(ga, eb, 0, 1) + _cut(gb, ea, 1, 0) - _cut(ga, eb, 1, 0) - _cut(gb, ea, 0, 1))
        w = np.broadcast_to(2.0 * h[n] / (h[a] * h[b]) / MU0 / 3.0, sig.shape)
        lo, hi = _cut(f, en, 0, 1), _cut(f, en, 1, 0)
        r = np.zeros_like(f)
        _put(r, en, 0, w * (2 * lo + hi))
        _put(r, en, 1, w * (lo + 2 * hi))
        ta, tb = _cut(out[a], ea, 0, 1), _cut(out[b], eb, 0, 1)      # views
        _put(ta, eb, 0, r)
        _put(ta, eb, 1, -r)
        _put(tb, ea, 1, r)
        _put(tb, ea, 0, -r)
    for d in range(3):
        t, ax, p, q = _cell_edges(g[d], d)
        a, b = (d + 1) % 3, (d + 2) % 3
        w = 1j * omega * sig * (h[a] * h[b] / h[d])
        view = _cut(out[d], ax, 0, 1)
        for (i, j), m in _cell_mass(t, (p, q)).items():
            n = view.shape
            s = [slice(None)] * 3
            s[p] = slice(i, n[p] - 1 + i)
            s[q] = slice(j, n[q] - 1 + j)
            view[tuple(s)] += w * m
    y = v.astype(np.complex128).copy()
    for d in range(3):
        ids = _grid(mesh, v, d)[1]
        y[ids[inner[d]]] = out[d][inner[d]]
    return y


def _gradient(mesh, sys, u, lam):
    h = _sizes(mesh)
    nus, alfas, z1d, usin, ucos = sys
    sig = mesh.mat_sigma[mesh.nvkat].reshape(mesh.nz - 1, mesh.ny - 1, mesh.nx - 1)
    grad = np.zeros(sig.shape)
    for k, nu in enumerate(nus):
        a0 = np.interp(mesh.z, z1d, usin[k]) + 1j * np.interp(mesh.z, z1d, ucos[k])
        for d in range(3):
            t = _grid(mesh, u[k], d)[0].astype(np.complex128)
            if d == (0 if alfas[k] else 1):
                half = 0.5 * np.append(np.diff((mesh.x, mesh.y)[d]), 0.0)
                t = t + a0[:, None, None] * half.reshape((1, 1, -1) if d == 0 else (1, -1, 1))
            l = np.where(_inner(mesh, d), _grid(mesh, lam[k], d)[0], 0.0)
            te, _, p, q = _cell_edges(t, d)
            le = _cell_edges(l, d)[0]
            s = sum(le[i] * m for i, m in _cell_mass(te, (p, q)).items())
            w = h[(d + 1) % 3] * h[(d + 2) % 3] / h[d]
            grad += -2.0 * sig * w * np.real(1j * 2.0 * math.pi * nu * s)
    return grad.ravel()


def exact(case, seed):
    """Products and gradients in numpy; a solve's exact answer would take a
    direct factorisation of its matrix, minutes at these sizes."""
    if case["kind"] not in ("operator", "gradient"):
        return None
    st = prepare(case, seed)
    mesh = st["mesh"]
    cplx = lambda t: t.cpu().numpy().view(np.complex128)
    if case["kind"] == "operator":
        x = cplx(st["x"])
        y = np.stack([_apply(mesh, 2.0 * math.pi * nu, x[k])
                      for k, nu in enumerate(st["sys"][0])])
        return y.view(np.float64)
    return _gradient(mesh, st["sys"], cplx(st["u"]), cplx(st["lam"]))
