"""What is measured: the work that users of this package have it do.

A case is one pass of an electrical-resistivity operator through the public
classes, on seeded synthetic ground (log-normal resistivity, sigma 1, with
conductive and resistive bodies).  Kinds:

``line``     one 2.5-D electrode line with the banded direct solve: response
             and FP64 Jacobian of a Gauss-Newton iteration.
``batch``    several independent 2.5-D lines in one batched response.
``grid``     a 3-D electrode grid: response and Jacobian; the solver forms of
             the operator (plain FP64, mixed precision with its three
             preconditioners).
``cem``      the same with complete-electrode-model patches (total potential).
``complex``  induced polarisation on a 3-D grid: complex response and Jacobian.
``update``   the regularised model update of a Gauss-Newton iteration.
"""
from __future__ import annotations

import functools
import math
import os

import numpy as np
import torch

import pygimli_gb300
from pygimli_gb300 import DataContainerERT, ERTModelling, createData, create_box_mesh_3d, create_para_mesh_2d
from pygimli_gb300.batch import BatchedERTModelling
from pygimli_gb300.cem import mark_cem_electrodes
from pygimli_gb300.data import geometricFactors, grid_line_scheme, grid_scheme_3d
from pygimli_gb300.inversion import TransLog, cgls, smoothness_constraints

#: spacing of the 3-D electrode grids (m); the mesh cell size divides it
SPACING = 4.0


def listed():
    return [
        # a short Wenner line on a coarse mesh: the smallest calls, latency and launches
        {"name": "line_small", "kind": "line", "ne": 16, "dx": 0.5, "scheme": "wa", "sep": 999},
        # the 41-electrode line of the repository's first configuration: the ordinary 2-D survey
        {"name": "line_2d", "kind": "line", "ne": 41, "dx": 0.25, "scheme": "dd", "sep": 16},
        # a long line on a fine mesh: the largest 2-D survey
        {"name": "line_fine", "kind": "line", "ne": 72, "dx": 1.0 / 14.0, "scheme": "dd+wa", "sep": 12},
        # independent lines of different sizes solved together (a survey of parallel profiles)
        {"name": "batch_lines", "kind": "batch", "problems": 8, "ne": 24, "ne_step": 5, "dx": 0.25, "scheme": "dd+wa",
         "sep": 12},
        # the operator as it is constructed by default, on a 3-D grid with a coarse mesh
        {"name": "grid_default", "kind": "grid", "nx": 12, "ny": 8, "h": 4.0, "scheme": "full", "precision": "fp64",
         "precond": "jacobi", "jacobian": "float64"},
        # the 3-D operator's fast form: a coarse mesh for first inversions
        {"name": "grid_coarse", "kind": "grid", "nx": 12, "ny": 8, "h": 4.0, "scheme": "full", "precision": "mixed",
         "precond": "fsai", "jacobian": "float32"},
        # the 96-electrode box of the repository's second configuration
        {"name": "grid_box", "kind": "grid", "nx": 12, "ny": 8, "h": 4.0 / 3.0, "scheme": "full", "precision": "mixed",
         "precond": "fsai", "jacobian": "float32"},
        # the 256-electrode benchmark: the largest survey, learned preconditioner
        {"name": "grid_large", "kind": "grid", "nx": 16, "ny": 16, "h": 4.0 / 3.0, "scheme": "lines",
         "precision": "mixed", "precond": "learned", "jacobian": "float32"},
        # a small grid with an odd electrode count, mixed precision without a preconditioner of its own
        {"name": "grid_odd", "kind": "grid", "nx": 7, "ny": 5, "h": 2.0, "scheme": "full", "precision": "mixed",
         "precond": "jacobi", "jacobian": "float32"},
        # electrodes with an area and a contact impedance
        {"name": "cem_grid", "kind": "cem", "nx": 12, "ny": 8, "h": 2.0, "scheme": "inline"},
        # induced polarisation
        {"name": "complex_grid", "kind": "complex", "nx": 8, "ny": 6, "h": 2.0, "scheme": "inline"},
        # the model update from a Jacobian in FP32
        {"name": "update", "kind": "update", "nx": 12, "ny": 8, "h": 4.0, "scheme": "full", "iterations": 30},
    ]


def draw(rng):
    kind = rng.choice(["line", "line", "line", "batch", "grid", "grid", "grid", "grid", "cem", "complex", "update"])
    if kind == "line":
        ne = int(round(math.exp(rng.uniform(math.log(8), math.log(80)))))
        return {"kind": kind, "ne": ne, "dx": 1.0 / rng.randint(2, 14 if ne > 20 else 8),
                "scheme": rng.choice(["dd", "wa", "pd", "dd+wa"]), "sep": rng.randint(4, 16)}
    if kind == "batch":
        return {"kind": kind, "problems": rng.randint(2, 12), "ne": rng.randint(12, 32), "ne_step": rng.randint(1, 5),
                "dx": 1.0 / rng.randint(2, 5), "scheme": rng.choice(["dd", "wa", "dd+wa"]), "sep": rng.randint(4, 14)}
    nx, ny = rng.randint(5, 13), rng.randint(4, 9)
    if kind == "grid":
        h = rng.choice([4.0, 2.0, 4.0 / 3.0])
        form = rng.choice([("fp64", "jacobi"), ("mixed", "jacobi"), ("mixed", "fsai"), ("mixed", "fsai"),
                           ("mixed", "learned"), ("mixed", "learned")])
        if form[0] == "fp64":
            h = max(h, 2.0)
        return {"kind": kind, "nx": nx, "ny": ny, "h": h, "scheme": rng.choice(["full", "lines", "inline"]),
                "precision": form[0], "precond": form[1], "jacobian": "float64" if form[0] == "fp64" else "float32"}
    if kind == "cem":
        return {"kind": kind, "nx": nx, "ny": ny, "h": 2.0, "scheme": rng.choice(["lines", "inline"])}
    if kind == "complex":
        return {"kind": kind, "nx": min(nx, 9), "ny": min(ny, 7), "h": rng.choice([4.0, 2.0]), "scheme": "inline"}
    return {"kind": kind, "nx": nx, "ny": ny, "h": 4.0, "scheme": rng.choice(["full", "lines"]),
            "iterations": rng.randint(10, 40)}


# ------------------------------------------------------------- the surveys
@functools.lru_cache(maxsize=64)
def _line(ne, dx, scheme, sep):
    xs = np.arange(float(ne))
    mesh = create_para_mesh_2d(xs, para_dx=dx, para_depth=max(2.0, ne / 4.0))
    parts = [createData(xs, s, maxSeparation=sep) for s in scheme.split("+")]
    data = DataContainerERT(parts[0].sensorPositions(), np.vstack([p.abmn() for p in parts]))
    data.set("k", geometricFactors(data, 2))
    return mesh, data


@functools.lru_cache(maxsize=16)
def _grid(nx, ny, h, scheme, patches):
    e = np.array([(x, y) for x in np.arange(nx) * SPACING for y in np.arange(ny) * SPACING])
    mesh = create_box_mesh_3d(e, h=h)
    if scheme == "full":
        ab = grid_scheme_3d(nx, ny)
    else:
        ab = np.vstack([grid_line_scheme((nx, ny), s) for s in (("dd",) if scheme == "inline" else ("dd", "pd", "wa"))])
    data = DataContainerERT(np.column_stack([e, np.zeros(len(e))]), ab)
    data.set("k", geometricFactors(data, 3))
    if patches:  # the surface triangles within one cell diagonal of each electrode
        mesh = mark_cem_electrodes(mesh, data.sensorPositions()[:, :2], h * math.sqrt(2.0) * (1.0 + 1e-6))
    return mesh, data


def _batch(case):
    return [_line(case["ne"] + i * case["ne_step"], case["dx"], case["scheme"], case["sep"])
            for i in range(case["problems"])]


def _survey(case):
    if case["kind"] == "line":
        return _line(case["ne"], case["dx"], case["scheme"], case["sep"])
    return _grid(case["nx"], case["ny"], case["h"], case["scheme"], case["kind"] == "cem")


def _ground(mesh, data, rng):
    """Resistivity per cell: log-normal (median 100 Ohm m, sigma 1) with a
    conductive and a resistive body below the electrodes."""
    c = mesh.cellCenters()
    rho = np.exp(rng.normal(np.log(100.0), 1.0, mesh.cellCount()))
    p = data.sensorPositions()
    lo, hi = p.min(axis=0), p.max(axis=0)
    depth = 0.25 * float(np.max(hi - lo))
    for val in (10.0, 1000.0):
        ctr = lo + rng.uniform(0.15, 0.85, 3) * (hi - lo)
        ctr[mesh.dim() - 1] = -rng.uniform(0.1, 0.6) * depth
        ax = rng.uniform(0.25, 0.5, 3) * depth
        d = mesh.dim()
        rho[np.sum(((c[:, :d] - ctr[:d]) / ax[:d]) ** 2, axis=1) <= 1.0] = val
    return rho


def _operator(mesh, data, **kw):
    fop = ERTModelling(maxIter=200000, **kw)
    if mesh.dim() == 2:  # the default number of wavenumbers, at the exact quadrature points
        k, w = _wavenumbers(data)
        fop.setkValues(k)
        fop.setWeights(w)
    fop.setData(data)
    fop.setMesh(mesh, ignoreRegionManager=True)
    return fop


def _weights():
    return os.path.join(os.path.dirname(pygimli_gb300.__file__), "weights", "box_3d.npz")


# ----------------------------------------------------------------- a pass
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        probs = _batch(case)
        fops = [_operator(m, d, precond="band") for m, d in probs]
        return {"kind": kind, "op": BatchedERTModelling(fops), "models": [_ground(m, d, rng) for m, d in probs]}
    mesh, data = _survey(case)
    model = _ground(mesh, data, rng)
    st = {"kind": kind, "model": model}
    if kind == "line":
        st["op"] = _operator(mesh, data, precond="band")
        st["dtype"] = "float64"
    elif kind == "grid":
        more = {"weights": _weights()} if case["precond"] == "learned" else {}
        st["op"] = _operator(mesh, data, precision=case["precision"], precond=case["precond"], **more)
        st["dtype"] = case["jacobian"]
    elif kind == "cem":
        st["op"] = _operator(mesh, data, sr=False, precision="mixed", precond="fsai")
        st["dtype"] = "float32"
    elif kind == "complex":
        fop = _operator(mesh, data, precision="mixed")
        fop.setComplex(True)
        phase = -rng.uniform(0.005, 0.03, len(model))
        st["op"], st["model"] = fop, np.concatenate([model * np.cos(phase), model * np.sin(phase)])
        st["dtype"] = None
    else:
        # the Jacobian at the start model, data of the true ground with 3 % noise
        fop = _operator(mesh, data, precision="mixed", precond="fsai")
        obs = fop.response(model) * (1.0 + 0.03 * rng.standard_normal(data.size()))
        start = np.full(mesh.cellCount(), float(np.median(obs)))
        resp = fop.response(start)
        C = smoothness_constraints(mesh, fop.parameterCount)
        st = {"kind": kind, "J": fop.createJacobian(start, dtype="float32"), "C": C,
              "dweight": 1.0 / TransLog.error(obs, np.full(data.size(), 0.03)),
              "b": TransLog.trans(obs) - TransLog.trans(resp), "x0": np.zeros(len(start)),
              "wc": np.ones(len(C[0]) - 1), "wm": np.ones(len(start)), "tm": TransLog.deriv(start),
              "td": TransLog.deriv(resp), "rough": np.zeros(len(C[0]) - 1), "iterations": case["iterations"]}
    return st


def run(st):
    kind = st["kind"]
    if kind == "batch":
        return st["op"].response(st["models"])
    if kind == "update":
        return cgls(st["J"], st["C"], st["dweight"], st["b"], st["x0"], st["wc"], st["wm"], st["tm"], st["td"], 20.0,
                    st["rough"], max_iter=st["iterations"])[0]
    rhoa = st["op"].response(st["model"])
    if kind == "complex":
        return {"rhoa": rhoa, "J": st["op"].createJacobian(st["model"])}
    return {"rhoa": rhoa, "J": st["op"].createJacobian(st["model"], dtype=st["dtype"])}


# ------------------------------------------------------------------- work
def _line_work(mesh, data, jacobian):
    """One 2.5-D line: the banded factor of every wavenumber (b the smaller
    side of the structured mesh), two substitutions per source and
    wavenumber, the Jacobian's products."""
    n, C, ne, D = mesh.nodeCount(), mesh.cellCount(), data.sensorCount(), data.size()
    nk = len(_wavenumbers(data)[0])
    b = len(np.unique(mesh.nodes[:, 1]))
    flops = nk * n * b * (b + 1.0) + 4.0 * nk * ne * n * b + (D * C * (nk * 6.0 + 2.0) if jacobian else 0.0)
    nbytes = C * 8.0 + D * 8.0 + n * nk * (b + 1.0) * 8.0 + n * nk * ne * 8.0 + (D * C * 8.0 if jacobian else 0.0)
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_line_work(m, d, False) for m, d in _batch(case)]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    mesh, data = _survey(case)
    if kind == "line":
        nbytes, flops = _line_work(mesh, data, True)
        return {"bytes": nbytes, "flops": flops}
    n, C, ne, D = mesh.nodeCount(), mesh.cellCount(), data.sensorCount(), data.size()
    if kind == "update":
        passes = 2.0 * case["iterations"] + 2.0
        return {"bytes": passes * D * C * 4.0, "flops": passes * D * C * 2.0}
    # model in, potentials of every source out, J out; the solve's iterations are not counted
    width = {"complex": 16.0, "cem": 4.0}.get(kind) or (8.0 if case["jacobian"] == "float64" else 4.0)
    z = 2.0 if kind == "complex" else 1.0
    return {"bytes": z * (C * 8.0 + n * ne * 8.0 + D * 8.0) + D * C * width, "flops": z * z * D * C * 8.0}


# ------------------------------------------------- the same in 64 bits
# Abramowitz & Stegun 9.8.1-9.8.8, the Bessel functions that the operator's
# primary potentials and mixed boundaries are defined with
def _horner(y, c):
    out = torch.full_like(y, c[-1])
    for v in reversed(c[:-1]):
        out = out * y + v
    return out


def _k01(x):
    s = x <= 2.0
    xs = torch.where(s, x, torch.ones_like(x))
    xl = torch.where(s, torch.full_like(x, 2.0), x)
    t = (xs / 3.75) ** 2
    i0 = _horner(t, [1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813])
    i1 = xs * _horner(t, [0.5, 0.87890594, 0.51498869, 0.15084934, 0.02658733, 0.00301532, 0.00032411])
    y = xs * xs / 4.0
    lg = torch.log(xs / 2.0)
    k0 = -lg * i0 + _horner(y, [-0.57721566, 0.42278420, 0.23069756, 0.03488590, 0.00262698, 0.00010750, 0.0000074])
    k1 = lg * i1 + _horner(y, [1.0, 0.15443144, -0.67278579, -0.18156897, -0.01919402, -0.00110404, -0.00004686]) / xs
    y = 2.0 / xl
    f = torch.exp(-xl) / torch.sqrt(xl)
    k0l = f * _horner(y, [1.25331414, -0.07832358, 0.02189568, -0.01062446, 0.00587872, -0.00251540, 0.00053208])
    k1l = f * _horner(y, [1.25331414, 0.23498619, -0.03655620, 0.01504268, -0.00780353, 0.00325614, -0.00068245])
    return torch.where(s, k0, k0l), torch.where(s, k1, k1l)


def _wavenumbers(data):
    """Wavenumbers and weights of a 2.5-D line: Gauss-Legendre points for the
    small wavenumbers, four Gauss-Laguerre points for the others."""
    p = data.sensorPositions()
    d = np.linalg.norm(p[:, None, :] - p[None, :, :], axis=2)
    r_min, r_max = d[d > 0].min() / 2.0, d.max() * 2.0
    k0 = 1.0 / (2.0 * r_min)
    x, w = np.polynomial.legendre.leggauss(max(int(math.floor(6.0 * math.log10(r_max / r_min))), 4))
    x, w = 0.5 * (x + 1.0), 0.5 * w
    y, v = np.polynomial.laguerre.laggauss(4)
    return (np.concatenate([k0 * x * x, k0 * (y + 1.0)]),
            np.concatenate([2.0 * k0 * x * w / math.pi, k0 * np.exp(y) * v / math.pi]))


def _forward64(mesh, data, rho, with_jacobian):
    """Response (and Jacobian) of the singularity-removal operator: linear
    finite elements, dense Cholesky factors, everything in FP64."""
    dev = "cuda"
    d = mesh.dim()
    X = torch.from_numpy(np.ascontiguousarray(mesh.nodes)).to(dev)
    cells = torch.from_numpy(np.ascontiguousarray(mesh.cells)).long().to(dev)
    r = torch.from_numpy(rho).to(dev)
    n, C, nv = len(X), len(cells), d + 1
    ab = torch.from_numpy(np.ascontiguousarray(data.abmn())).long().to(dev)
    kf = torch.from_numpy(np.asarray(data["k"], np.float64)).to(dev)
    if d == 2:
        ks, ws = _wavenumbers(data)
    else:
        ks, ws = np.zeros(1), np.ones(1)
    # element matrices
    P = X[cells][:, :, :d]
    E = P[:, 1:] - P[:, :1]
    g = torch.linalg.inv(E).transpose(1, 2)
    g = torch.cat([-g.sum(1, keepdim=True), g], 1)
    V = torch.linalg.det(E).abs() / math.factorial(d)
    K = V[:, None, None] * (g @ g.transpose(1, 2))
    M = V[:, None, None] / (nv * (nv + 1.0)) * (torch.eye(nv, dtype=X.dtype, device=dev) + 1.0)
    # mixed boundaries
    mixed = np.flatnonzero(np.asarray(mesh.boundary_markers) == -2)
    bn = torch.from_numpy(np.ascontiguousarray(mesh.boundaries[mixed])).long().to(dev)
    bcell = torch.from_numpy(np.ascontiguousarray(mesh.boundary_cells[mixed])).long().to(dev)
    Q = X[bn]
    ctr = Q.mean(1)
    if d == 2:
        t = Q[:, 1] - Q[:, 0]
        size = t.norm(dim=1)
        nrm = torch.stack([t[:, 1], -t[:, 0], torch.zeros_like(t[:, 0])], 1) / size[:, None]
    else:
        nrm = torch.linalg.cross(Q[:, 1] - Q[:, 0], Q[:, 2] - Q[:, 0])
        size = 0.5 * nrm.norm(dim=1)
        nrm = nrm / (2.0 * size[:, None])
    Mb = size[:, None, None] / (d * (d + 1.0)) * (torch.eye(d, dtype=X.dtype, device=dev) + 1.0)
    # electrodes: nodes at the sensors
    s = torch.from_numpy(np.ascontiguousarray(data.sensorPositions())).to(dev)
    enode = torch.cdist(s, X).argmin(1)
    ep = X[enode]
    ne = len(ep)
    rad, rs = [], []
    for e in range(ne):
        near = (cells == enode[e]).any(1).nonzero()[:, 0]
        o = cells[near].reshape(-1)
        rad.append((X[o[o != enode[e]]] - ep[e]).norm(dim=1).min())
        rs.append(torch.exp(torch.log(r[near]).mean()))
    rad, rs = torch.stack(rad), torch.stack(rs)
    src = ep.mean(0)
    ax = 1 if d == 2 else 2
    mir = src.clone()
    mir[ax] = -mir[ax]

    def matrix(inv, kk, alpha):
        A = torch.zeros(n * n, dtype=X.dtype, device=dev)
        el = (K + kk * kk * M) * inv[:, None, None]
        A.index_add_(0, (cells[:, :, None] * n + cells[:, None, :]).reshape(-1), el.reshape(-1))
        el = Mb * (alpha * inv[bcell])[:, None, None]
        A.index_add_(0, (bn[:, :, None] * n + bn[:, None, :]).reshape(-1), el.reshape(-1))
        return A.view(n, n)

    U, sol = [], torch.zeros(ne, ne, dtype=X.dtype, device=dev)
    for kk, w in zip(ks, ws):
        a, b = (src - ctr).norm(dim=1), (mir - ctr).norm(dim=1)
        an, bm = ((src - ctr) * nrm).sum(1).abs(), ((mir - ctr) * nrm).sum(1).abs()
        dist = torch.cdist(X, ep, compute_mode="donot_use_mm_for_euclid_dist")
        dist[enode, torch.arange(ne, device=dev)] = 1.0
        if kk == 0.0:
            alpha = (b * b * an / a + a * a * bm / b) / (a * b * (a + b))
            up = 1.0 / (2.0 * math.pi * dist)
            up[enode, torch.arange(ne, device=dev)] = 1.0 / (math.pi * rad)
        else:
            (a0, a1), (b0, b1) = _k01(a * kk), _k01(b * kk)
            alpha = kk * (an / a * a1 + bm / b * b1) / (a0 + b0)
            alpha = torch.where((a0 < 1e-12) | (b0 < 1e-12), torch.zeros_like(alpha), alpha)
            up = _k01(dist * kk)[0] / math.pi
            up[enode, torch.arange(ne, device=dev)] = _k01(rad / 6.0 * kk)[0] / math.pi
        prim = up * rs
        S = matrix(1.0 / r, float(kk), alpha)
        rhs = (matrix(torch.ones_like(r), float(kk), alpha) @ prim) / rs - S @ prim
        L = torch.linalg.cholesky(S)
        x = torch.cholesky_solve(rhs, L)
        x = x + torch.cholesky_solve(rhs - S @ x, L) + prim
        del S, L
        sol += float(w) * x[enode].T
        U.append(x)
    U0 = torch.cat([sol, torch.zeros(ne, 1, dtype=X.dtype, device=dev)], 1)
    U0 = torch.cat([U0, torch.zeros(1, ne + 1, dtype=X.dtype, device=dev)], 0)
    i = torch.where(ab < 0, torch.full_like(ab, ne), ab)

    def volt(a, b, m, o):
        u = (U0[a, m] - U0[a, o]) - (U0[b, m] - U0[b, o])
        return torch.round(u / 1e-10) * 1e-10 * kf

    rhoa = torch.sqrt(torch.abs(volt(i[:, 0], i[:, 1], i[:, 2], i[:, 3]) * volt(i[:, 2], i[:, 3], i[:, 0], i[:, 1])))
    if not with_jacobian:
        return rhoa, None
    J = torch.zeros(len(ab), C, dtype=X.dtype, device=dev)
    for kk, w, x in zip(ks, ws, U):
        u = torch.cat([x, torch.zeros(n, 1, dtype=X.dtype, device=dev)], 1)[cells]  # C x nv x (ne + 1)
        # shifted by the first node: a constant has no gradient (exact for K)
        v = (K @ (u - u[:, :1])) + float(kk * kk) * (M @ u)
        for d0 in range(0, len(ab), 64):
            q = i[d0:d0 + 64]
            va = v[:, :, q[:, 0]] - v[:, :, q[:, 1]]
            um = u[:, :, q[:, 2]] - u[:, :, q[:, 3]]
            if kk == 0.0:
                um = um - um[:, :1]
            J[d0:d0 + 64] += float(w) * (va * um).sum(1).T
        del u, v
    J *= kf[:, None]
    J /= (r * r)[None, :]
    return rhoa, J


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        return [_forward64(m, d, rho, False)[0] if m.nodeCount() <= 5000 else None
                for m, d, rho in [(m, d, _ground(m, d, rng)) for m, d in _batch(case)]]
    if kind not in ("line", "grid"):
        return None
    mesh, data = _survey(case)
    if mesh.nodeCount() > (5000 if kind == "line" else 25000):
        return None
    rhoa, J = _forward64(mesh, data, _ground(mesh, data, rng), True)
    return {"rhoa": rhoa, "J": J}
