"""Performance cases: what a program that uses this library calls it for, through its public entry
points. Each case is a dict of plain values; `kind` is the entry point and the rest are its sizes and
options.

  eval     VolumetricFemEnergy.eval_device on tets, Q1 hexes or tricubic Hermite hexes: energy,
           gradient and (Exact or Projected) Hessian, or energy and gradient alone. FP64 with the
           gradient, as the Newton residual is; mixed precision with the Hessian alone, as the
           solvers ask for it.
  newton   solver.newton_solve of a box under gravity (bottom face held, block-Jacobi PCG).
  batch    solver.batch_newton_solve of many such boxes, of different sizes, in one call.
  adjoint  lpg_adjoint_theta: the equilibrium sensitivity in per-element [lambda, mu].

Meshes come from `mesh.make_box`, `mesh.make_hex_box` and `mesh.delaunay_ball`; a case names its
connectivity, the seed gives the material and the state. `exact` restates each case in FP64 with torch
alone (dense linear algebra for the solves).
"""

import ctypes
import functools
import math

import numpy as np
import torch

from litepgo_b200 import _native as N
from litepgo_b200 import dof, energy, fem, mesh, solver, workloads

DEVICE = "cuda"
EXACT_DOFS = 15000  # largest dense system of exact()


def listed():
    return [
        # A coarse block in an interactive tool: latency and launches, not arithmetic.
        {"name": "tet_tiny", "kind": "eval", "cell": "tet", "nx": 3, "ny": 4, "nz": 3, "hessian": "exact",
         "precision": "f64", "layout": "bsr", "plastic": False},
        # The residual of a line search or of an explicit step: energy and gradient alone.
        {"name": "tet_gradient", "kind": "eval", "cell": "tet", "nx": 48, "ny": 45, "nz": 41, "hessian": "none",
         "precision": "f64", "layout": "bsr", "plastic": False},
        # The repository's benchmark step: 64^3 cubes of five tets, FP64, block-CSR.
        {"name": "tet_exact_64", "kind": "eval", "cell": "tet", "nx": 64, "ny": 64, "nz": 64, "hessian": "exact",
         "precision": "f64", "layout": "bsr", "plastic": False},
        # A mixed-precision Hessian of a plastic block in the reference's scalar CSC order.
        {"name": "tet_plastic_mixed", "kind": "eval", "cell": "tet", "nx": 45, "ny": 39, "nz": 31, "hessian": "exact",
         "precision": "mixed", "layout": "csc", "plastic": True},
        # An unstructured mesh, eigenvalue-clamped Hessian: the default of newton_solve.
        {"name": "ball_projected", "kind": "eval", "cell": "ball", "points": 9000, "hessian": "projected",
         "precision": "f64", "layout": "bsr", "plastic": False},
        # The Hessian of one mixed-precision Newton iteration.
        {"name": "tet_projected_mixed", "kind": "eval", "cell": "tet", "nx": 40, "ny": 33, "nz": 27,
         "hessian": "projected", "precision": "mixed", "layout": "bsr", "plastic": False},
        # A Q1 hex block with the default (Projected) Hessian.
        {"name": "hex_projected", "kind": "eval", "cell": "hex", "nx": 20, "ny": 17, "nz": 22, "points_per_axis": 2,
         "hessian": "projected", "precision": "f64", "layout": "bsr"},
        # Tricubic Hermite hexes with four points per axis, the order their stiffness needs.
        {"name": "hermite_projected", "kind": "eval", "cell": "hermite", "nx": 5, "ny": 4, "nz": 4,
         "points_per_axis": 4, "hessian": "projected", "precision": "f64", "layout": "bsr"},
        # A small equilibrium, FP64: the solver's launches and round trips.
        {"name": "newton_small", "kind": "newton", "nx": 8, "ny": 8, "nz": 7, "precision": "f64"},
        # A large equilibrium on the mixed-precision path.
        {"name": "newton_mixed", "kind": "newton", "nx": 40, "ny": 40, "nz": 36, "precision": "mixed"},
        # Many different small bodies in one call.
        {"name": "batch_mixed", "kind": "batch", "count": 48, "lo": 4, "hi": 16, "dims_seed": 3, "precision": "mixed"},
        # The backward pass of a material fit.
        {"name": "adjoint", "kind": "adjoint", "nx": 16, "ny": 17, "nz": 15, "precision": "f64"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, lo, hi):
    n = _log(rng, lo, hi)
    return tuple(max(lo, min(hi, round(n * rng.uniform(0.75, 1.3)))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["tet", "tet", "tet", "ball", "hex", "hermite", "newton", "newton", "batch", "adjoint"])
    if kind in ("tet", "ball"):
        c = {"kind": "eval", "cell": kind}
        if kind == "tet":
            c["nx"], c["ny"], c["nz"] = _dims(rng, 3, 64)
        else:
            c["points"] = round(_log(rng, 150, 12000))
        c["precision"] = rng.choice(["f64", "mixed"])
        c["hessian"] = rng.choice(["none", "exact", "projected"] if c["precision"] == "f64" else ["exact", "projected"])
        c["layout"] = rng.choice(["bsr", "csc"])
        c["plastic"] = rng.random() < 0.3
        return c
    if kind in ("hex", "hermite"):
        four = rng.random() < (0.25 if kind == "hex" else 0.7)
        c = {"kind": "eval", "cell": kind}
        c["nx"], c["ny"], c["nz"] = _dims(rng, 3, 11 if four else 22) if kind == "hex" else _dims(rng, 2, 6)
        c["points_per_axis"] = 4 if four else 2
        c["precision"] = rng.choice(["f64", "f64", "mixed"])
        c["hessian"] = rng.choice(["exact", "projected"])
        c["layout"] = rng.choice(["bsr", "csc"])
        return c
    if kind == "batch":
        lo = rng.randint(3, 5)
        return {"kind": "batch", "count": round(_log(rng, 6, 48)), "lo": lo, "hi": lo + rng.randint(2, 11),
                "dims_seed": rng.randrange(1000), "precision": rng.choice(["f64", "mixed"])}
    c = {"kind": kind}
    # No taller than wide: a free-standing column of this material buckles under its own weight.
    c["nz"], c["nx"], c["ny"] = sorted(_dims(rng, 4, 36 if kind == "newton" else 20))
    c["precision"] = rng.choice(["f64", "mixed"])
    return c


# ---------------------------------------------------------------------------
# Inputs: meshes (kept by shape), materials and states (from the seed).
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _mesh(cell, nx, ny, nz, points):
    """(X, cells, h): the longest side of a box is 1 and its cells are cubes of side h."""
    if cell == "ball":
        X, cells = mesh.delaunay_ball(points, seed=points)
        return X, cells, float((4.19 / points) ** (1 / 3))
    h = 1.0 / max(nx, ny, nz)
    make = mesh.make_box if cell == "tet" else mesh.make_hex_box
    X, cells = make(nx, ny, nz, size=(nx * h, ny * h, nz * h))
    return X, cells, h


def _mesh_of(case):
    return _mesh(case.get("cell", "tet"), case.get("nx", 0), case.get("ny", 0), case.get("nz", 0),
                 case.get("points", 0))


def _material(rng, T):
    """Per-element [lambda, mu]: mu log-uniform in [1e3, 1e5], Poisson ratio in [0.30, 0.45]."""
    mu = np.exp(rng.uniform(math.log(1e3), math.log(1e5), T))
    lam, mu = workloads.lame(mu, rng.uniform(0.30, 0.45, T))
    return np.ascontiguousarray(np.stack([lam, mu], axis=1))


def _affine(rng):
    """A displacement gradient of stretch and shear up to 13 % per entry (det of I plus it > 0)."""
    A = 0.06 * rng.standard_normal((3, 3))
    return np.clip(A, -0.13, 0.13)


def _eval_inputs(case, seed):
    X, cells, h = _mesh_of(case)
    rng = np.random.default_rng([seed, 17])
    theta = _material(rng, cells.shape[0])
    A = _affine(rng)
    Fp = None
    if case["cell"] == "hermite":
        # u, its gradient and its mixed derivatives at every vertex (24 per vertex).
        u = np.zeros((X.shape[0], 8, 3))
        u[:, 0] = X @ A.T
        u[:, 1:4] = A.T
        scale = np.array([0.02 * h, 0.04, 0.04, 0.04, 0.05 / h, 0.05 / h, 0.05 / h, 0.1 / h**2])
        u += scale[:, None] * np.clip(rng.standard_normal(u.shape), -2, 2)
    else:
        k = rng.uniform(2.0, 4.0, 3)
        # The ball's slivers turn over where the gradient varies across them: a gentler ripple there.
        ripple = 0.02 if case["cell"] != "ball" else 2e-4 / h
        u = X @ A.T + ripple * np.sin(X @ np.diag(k) + rng.uniform(0, 6.28, 3))
        if case["cell"] != "ball":
            u += 0.04 * h * np.clip(rng.standard_normal(X.shape), -2, 2)
        if case.get("plastic"):
            d = 0.02 * rng.standard_normal((cells.shape[0], 3, 3))
            Fp = np.ascontiguousarray(np.swapaxes(np.eye(3) + d, 1, 2).reshape(-1, 9))
    return X, cells, theta, Fp, np.ascontiguousarray(u.ravel())


def _bottom(X):
    v = np.flatnonzero(X[:, 2] == X[:, 2].min())
    return (3 * v[:, None] + np.arange(3)).ravel().astype(np.int32)


def _newton_inputs(case, seed):
    X, cells, _ = _mesh_of(case)
    theta = _material(np.random.default_rng([seed, 23]), cells.shape[0])
    return X, cells, theta, _bottom(X), workloads.gravity_load(X, cells)


def _batch_dims(case):
    """Cube counts per axis of every box, no taller than wide."""
    dims = np.random.default_rng(case["dims_seed"]).integers(case["lo"], case["hi"] + 1, (case["count"], 3))
    return [(d[1], d[2], d[0]) for d in np.sort(dims, axis=1).tolist()]


def _batch_inputs(case, seed):
    """The boxes of newton, of different cube counts, as one union."""
    rng = np.random.default_rng([seed, 29])
    parts, fixed, f, theta, base = [], [], [], [], 0
    for d in _batch_dims(case):
        X, cells, load = _loaded_box(*d)
        parts.append((X, cells))
        fixed.append(3 * base + _bottom(X))
        f.append(load)
        theta.append(_material(rng, cells.shape[0]))
        base += X.shape[0]
    X, cells, voff, eoff = mesh.concatenate(parts)
    return X, cells, voff, eoff, np.concatenate(theta), np.concatenate(fixed), np.concatenate(f)


@functools.lru_cache(maxsize=256)
def _loaded_box(nx, ny, nz):
    h = 1.0 / max(nx, ny, nz)
    X, cells = mesh.make_box(nx, ny, nz, size=(nx * h, ny * h, nz * h))
    return X, cells, workloads.gravity_load(X, cells)


def _adjoint_inputs(case, seed):
    """A block hanging from its held face: stretched along z, with a small ripple; a loss gradient."""
    X, cells, h = _mesh_of(case)
    rng = np.random.default_rng([seed, 31])
    theta = _material(rng, cells.shape[0])
    u = np.zeros_like(X)
    u[:, 2] = 0.12 * X[:, 2] * (1.0 - 0.4 * X[:, 2])
    u += 0.004 * X[:, 2:] * np.sin(X @ np.diag(rng.uniform(2.0, 5.0, 3)) + rng.uniform(0, 6.28, 3))
    return X, cells, theta, _bottom(X), u.ravel(), rng.standard_normal(X.size)


# ---------------------------------------------------------------------------
# The calls.
# ---------------------------------------------------------------------------
_KINDS = {"none": None, "exact": energy.HessianKind.Exact, "projected": energy.HessianKind.Projected}


def _basis(case):
    if case["cell"] in ("tet", "ball"):
        return fem.VolumetricFemEnergy[fem.NeoHookean, fem.TetP1Basis, fem.TetCentroidQuadrature]
    basis = fem.HexQ1Basis if case["cell"] == "hex" else fem.HexHermiteBasis
    return fem.VolumetricFemEnergy[fem.NeoHookean, basis, fem.GaussLegendre3D[case["points_per_axis"]]]


def _load(f):
    """-f . x as a QuadraticEnergy (the pulling energy of no DOFs gives the empty matrix)."""
    none = energy.VertexPullingEnergy(f.size, [], [], 1.0).quadratic_form()[0]
    return energy.QuadraticEnergy(none, -f)


def _newton_options(case):
    return solver.NewtonOptions(gradient_tolerance=1e-11, stop_rule="relative", accept_rule="armijo",
                                precision=case["precision"], max_iterations=100, cg_tolerance=1e-2,
                                cg_max_iterations=20000)


def _on_gpu(a):
    return torch.as_tensor(a, device=DEVICE)


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "eval":
        X, cells, theta, Fp, u = _eval_inputs(case, seed)
        cls = _basis(case)
        e = cls.from_arrays(X, cells, theta, Fp=Fp) if Fp is not None else cls.from_arrays(X, cells, theta)
        s.update(energy=e, u=_on_gpu(u), hessian=_KINDS[case["hessian"]], grad=None, hess=None)
        if case["precision"] == "f64":
            s["grad"] = torch.empty(e.num_dofs, dtype=torch.float64, device=DEVICE)
        if s["hessian"] is not None:
            dtype = torch.float64 if case["precision"] == "f64" else torch.float32
            s["hess"] = torch.empty(e.nnz, dtype=dtype, device=DEVICE)
    elif case["kind"] == "newton":
        X, cells, theta, fixed, f = _newton_inputs(case, seed)
        e = fem.VolumetricFemEnergyTetP1.from_arrays(X, cells, theta)
        s.update(energy=energy.WeightedSumEnergy([(e, 1.0), (_load(f), 1.0)]),
                 fixed=dof.DofReduction(X.size, fixed), options=_newton_options(case),
                 x0=torch.zeros(X.size, dtype=torch.float64, device=DEVICE))
    elif case["kind"] == "batch":
        X, cells, voff, eoff, theta, fixed, f = _batch_inputs(case, seed)
        e = fem.VolumetricFemEnergyTetP1.from_arrays(X, cells, theta)
        s.update(energy=energy.WeightedSumEnergy([(e, 1.0), (_load(f), 1.0)]), voff=voff, eoff=eoff,
                 fixed=dof.DofReduction(X.size, fixed), options=_newton_options(case),
                 x0=torch.zeros(X.size, dtype=torch.float64, device=DEVICE))
    else:
        X, cells, theta, fixed, u, w = _adjoint_inputs(case, seed)
        e = fem.VolumetricFemEnergyTetP1.from_arrays(X, cells, theta)
        s.update(energy=e, fixed=np.ascontiguousarray(fixed, dtype=np.int32), u=_on_gpu(u), w=_on_gpu(w),
                 dtheta=torch.empty(2 * cells.shape[0], dtype=torch.float64, device=DEVICE),
                 lam=torch.empty(X.size, dtype=torch.float64, device=DEVICE),
                 precision=N.PRECISION_F64 if case["precision"] == "f64" else N.PRECISION_MIXED)
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "eval":
        E, g, H = s["energy"].eval_device(s["u"], gradient=s["grad"] is not None, hessian=s["hessian"],
                                          precision=case["precision"], layout=case["layout"], grad_out=s["grad"],
                                          hess_out=s["hess"])
        out = {"energy": E}
        if g is not None:
            out["gradient"] = g
        if H is not None:
            out["hessian"] = H
        return out
    if case["kind"] == "newton":
        r = solver.newton_solve(s["energy"], s["fixed"], s["x0"], s["options"])
        return {"x": r.x, "energy": r.energy}
    if case["kind"] == "batch":
        x, meshes, _ = solver.batch_newton_solve(s["energy"], s["voff"], s["eoff"], s["fixed"], s["x0"], s["options"])
        return {"x": x, "energy": np.array([m.energy for m in meshes])}
    e = s["energy"]
    N.check(N.lib.lpg_fem_set_stream(e.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    N.check(N.lib.lpg_adjoint_theta(e.handle, N.vptr(s["u"]), N.vptr(s["w"]), N.iptr(s["fixed"]), int(s["fixed"].size),
                                    N.MEM_DEVICE, s["precision"], 1e-11, 1, N.vptr(s["dtheta"]), N.vptr(s["lam"])))
    return {"dtheta": s["dtheta"], "lambda": s["lam"]}


def work(case):
    """Bytes and operations of one pass: mesh data and inputs read once, outputs written once, one
    evaluation of every element. A solve counts one evaluation and one product with its matrix."""
    word = 8 if case["precision"] == "f64" else 4
    if case["kind"] == "batch":
        counts = np.array([mesh.box_counts(*d) for d in _batch_dims(case)]).sum(axis=0)
        V, T, nnzb = (int(c) for c in counts)
    elif case.get("cell", "tet") == "tet":
        V, T, nnzb = mesh.box_counts(case["nx"], case["ny"], case["nz"])
    elif case["cell"] == "ball":
        V, T, nnzb = case["points"], 5.9 * case["points"], 15.2 * case["points"]
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        V, T = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
        nnzb = (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
    if case.get("cell") in ("hex", "hermite"):
        points, per = case["points_per_axis"] ** 3, 1 if case["cell"] == "hex" else 8
        nodes = 8 * per
        flops = T * points * (30 * nodes * (nodes + 1) / 2 + 40 * nodes)
        return {"bytes": T * (32 + 16) + V * (24 + 48 * per) + 9 * word * nnzb * per**2, "flops": flops}
    rest = T * (16 + 12 * word + (9 * word if case.get("plastic") else 0)) + V * 24
    if case["kind"] == "eval":
        out = (V * 24 if word == 8 else 0) + (9 * word * nnzb if case["hessian"] != "none" else 0)
        return {"bytes": rest + out, "flops": T * (300 if case["hessian"] == "none" else 900)}
    extra = V * 24 * 2 if case["kind"] != "adjoint" else V * 24 * 2 + T * 16
    return {"bytes": rest + extra + 9 * word * nnzb, "flops": T * 900 + 18 * nnzb}


# ---------------------------------------------------------------------------
# The same in 64 bits, with torch alone.
# ---------------------------------------------------------------------------
def _corner_gradients(cell, xi):
    """dN/dxi of the 8 (Q1) or 64 (tricubic Hermite, function 8 corner + slot) functions at xi."""
    corners = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    if cell == "hex":
        f, d = [[1 - t, t] for t in xi], [-1.0, 1.0]
        return np.array([[d[c[0]] * f[1][c[1]] * f[2][c[2]], f[0][c[0]] * d[c[1]] * f[2][c[2]],
                          f[0][c[0]] * f[1][c[1]] * d[c[2]]] for c in corners])
    orders = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)]
    f = [[2 * t**3 - 3 * t**2 + 1, t**3 - 2 * t**2 + t, 3 * t**2 - 2 * t**3, t**3 - t**2] for t in xi]
    d = [[6 * t**2 - 6 * t, 3 * t**2 - 4 * t + 1, 6 * t - 6 * t**2, 3 * t**2 - 2 * t] for t in xi]
    rows = []
    for c in corners:
        for o in orders:
            i = [2 * c[k] + o[k] for k in range(3)]
            rows.append([d[0][i[0]] * f[1][i[1]] * f[2][i[2]], f[0][i[0]] * d[1][i[1]] * f[2][i[2]],
                         f[0][i[0]] * f[1][i[1]] * d[2][i[2]]])
    return np.array(rows)


def _point(G, w, Fe, lam, mu, hessian):
    """w psi, w P G^T and w B^T A B of one quadrature point of every element (G: T x K x 3)."""
    Fi = torch.linalg.inv(Fe).transpose(1, 2)
    J = torch.linalg.det(Fe)
    L = torch.log(J)
    p = lam * L - mu
    E = w * (0.5 * mu * ((Fe * Fe).sum((1, 2)) - 3) - mu * L + 0.5 * lam * L * L)
    P = mu[:, None, None] * Fe + p[:, None, None] * Fi
    g = w[:, None, None] * (G @ P.transpose(1, 2))
    H = None
    if hessian:
        h = G @ Fi.transpose(1, 2)
        H = torch.einsum("t,tai,tbk->taibk", w * lam, h, h) - torch.einsum("t,tbi,tak->taibk", w * p, h, h)
        dn = (w * mu)[:, None, None] * (G @ G.transpose(1, 2))
        for i in range(3):
            H[:, :, i, :, i] += dn
    return E, g, H


def _tet_gradients(X, cells, Fp):
    """G (T x 4 x 3, times Fp^-1), the weights and Fp^-1."""
    x = X[cells]
    Dm = (x[:, 1:] - x[:, :1]).transpose(1, 2)
    w = torch.linalg.det(Dm) / 6
    G = torch.linalg.inv(Dm)
    G = torch.cat([-G.sum(1, keepdim=True), G], 1)
    Fi = torch.eye(3, dtype=X.dtype, device=X.device).expand(G.shape[0], 3, 3)
    if Fp is not None:
        F = Fp.reshape(-1, 3, 3).transpose(1, 2)
        Fi = torch.linalg.inv(F)
        w = w * torch.linalg.det(F)
        G = G @ Fi
    return G, w, Fi


def _elements(case, X, cells, theta, Fp, u, hessian):
    """(E, g, H, nodes) of every element, nodes the 3-DOF rows it touches."""
    lam, mu = theta[:, 0], theta[:, 1]
    if case.get("cell", "tet") in ("tet", "ball"):
        G, w, Fi = _tet_gradients(X, cells, Fp)
        F = Fi + u.reshape(-1, 3)[cells].transpose(1, 2) @ G
        return (*_point(G, w, F, lam, mu, hessian), cells)
    t, wt = np.polynomial.legendre.leggauss(case["points_per_axis"])
    t, wt = 0.5 + 0.5 * t, 0.5 * wt
    nodes = cells
    if case["cell"] == "hermite":
        nodes = (8 * cells[:, :, None] + torch.arange(8, device=cells.device)).reshape(-1, 64)
        size = X[cells[:, 6]] - X[cells[:, 0]]
        one = torch.ones_like(size[:, 0])
        hx, hy, hz = size.unbind(1)
        slot = torch.stack([one, hx, hy, hz, hx * hy, hx * hz, hy * hz, hx * hy * hz], 1).repeat(1, 8)
    d = u.reshape(-1, 3)[nodes]
    total = None
    for i, a in enumerate(t):
        for j, b in enumerate(t):
            for k, c in enumerate(t):
                dN = torch.as_tensor(_corner_gradients(case["cell"], (a, b, c)), device=X.device)
                if case["cell"] == "hex":
                    Jm = X[cells].transpose(1, 2) @ dN
                    w = torch.linalg.det(Jm)
                    G = dN @ torch.linalg.inv(Jm)
                else:
                    w = size.prod(1)
                    G = slot[:, :, None] * dN / size[:, None, :]
                F = torch.eye(3, dtype=X.dtype, device=X.device) + d.transpose(1, 2) @ G
                part = _point(G, wt[i] * wt[j] * wt[k] * w, F, lam, mu, hessian)
                total = list(part) if total is None else [None if s is None else s + q for s, q in zip(total, part)]
    return (*total, nodes)


def _gathered(nodes, g, rows):
    out = torch.zeros(rows, 3, dtype=g.dtype, device=g.device)
    return out.index_add_(0, nodes.reshape(-1), g.reshape(-1, 3)).reshape(-1)


def _matrix(nodes, H, rows, layout):
    """The block-CSR (rows ascending, columns sorted) or scalar CSC values."""
    T, K = nodes.shape
    key = (nodes[:, :, None] * rows + nodes[:, None, :]).reshape(-1)
    key, at = torch.unique(key, return_inverse=True)
    vals = torch.zeros(key.numel(), 9, dtype=H.dtype, device=H.device)
    vals.index_add_(0, at, H.permute(0, 1, 3, 2, 4).reshape(T * K * K, 9))
    if layout == "bsr":
        return vals.reshape(-1)
    row = torch.div(key, rows, rounding_mode="floor")
    nb = torch.bincount(row, minlength=rows)
    first = torch.cumsum(nb, 0) - nb
    q = torch.arange(key.numel(), device=key.device) - first[row]
    i, c = torch.arange(3, device=key.device)[:, None], torch.arange(3, device=key.device)[None, :]
    pos = 9 * first[row][:, None, None] + 3 * i * nb[row][:, None, None] + 3 * q[:, None, None] + c
    out = torch.empty(vals.numel(), dtype=H.dtype, device=H.device)
    out[pos.reshape(-1)] = vals.reshape(-1)
    return out


def _clamped(H):
    """Each element's Hessian with its negative eigenvalues set to zero."""
    shape, n = H.shape, H.shape[1] * 3
    A = H.reshape(-1, n, n).cpu()
    L, Q = torch.linalg.eigh(0.5 * (A + A.transpose(1, 2)))
    return ((Q * L.clamp(min=0)[:, None, :]) @ Q.transpose(1, 2)).to(H.device).reshape(shape)


def _dense(case, X, cells, theta, u):
    E, g, H, nodes = _elements(case, X, cells, theta, None, u, True)
    n = u.numel()
    dofs = (3 * nodes[:, :, None] + torch.arange(3, device=nodes.device)).reshape(nodes.shape[0], 12)
    at = (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1)
    K = torch.zeros(n * n, dtype=u.dtype, device=u.device).index_add_(0, at, H.reshape(-1)).reshape(n, n)
    return E.sum(), _gathered(nodes, g, X.shape[0]), K


def _equilibrium(case, X, cells, theta, fixed, f, x):
    """Damped Newton with a Cholesky solve of the free block (shifted until it is positive definite)."""
    free = torch.ones_like(x, dtype=torch.bool)
    free[fixed] = False
    eye = torch.arange(int(free.sum()), device=x.device)
    total = lambda E, y: E - f @ y  # noqa: E731
    first, shift = None, 0.0
    for _ in range(60):
        E, g, K = _dense(case, X, cells, theta, x)
        r = (g - f)[free]
        first = r.norm() if first is None else first
        if r.norm() <= 1e-13 * first:
            break
        A = K[free][:, free]
        del K
        scale = A.diagonal().abs().max()
        while True:
            B = A.clone()
            B[eye, eye] += shift * scale
            C, bad = torch.linalg.cholesky_ex(B)
            if int(bad) == 0:
                break
            shift = max(4 * shift, 1e-4)
        d = torch.zeros_like(x)
        d[free] = -torch.cholesky_solve(r[:, None], C)[:, 0]
        del A, B, C
        shift = 0.0 if shift < 1e-3 else 0.25 * shift
        base, slope, a = total(E, x), d[free] @ r, 1.0
        while a > 1e-8:
            Et = _elements(case, X, cells, theta, None, x + a * d, False)[0].sum()
            if torch.isfinite(Et) and total(Et, x + a * d) <= base + 1e-4 * a * slope + 1e-14 * base.abs():
                break
            a *= 0.5
        if a <= 1e-8:
            break
        x = x + a * d
    return x, total(_elements(case, X, cells, theta, None, x, False)[0].sum(), x)


def exact(case, seed):
    gpu = lambda *arrays: [None if a is None else _on_gpu(np.asarray(a)) for a in arrays]  # noqa: E731
    if case["kind"] == "eval":
        X, cells, theta, Fp, u = _eval_inputs(case, seed)
        if case["hessian"] == "projected" and cells.shape[0] > 400000:
            return None
        X, cells, theta, Fp, u = gpu(X, cells.astype(np.int64), theta, Fp, u)
        E, g, H, nodes = _elements(case, X, cells, theta, Fp, u, case["hessian"] != "none")
        out = {"energy": float(E.sum())}
        rows = u.numel() // 3
        if case["precision"] == "f64":
            out["gradient"] = _gathered(nodes, g, rows)
        if H is not None:
            out["hessian"] = _matrix(nodes, _clamped(H) if case["hessian"] == "projected" else H, rows, case["layout"])
        return out
    if case["kind"] == "newton":
        X, cells, theta, fixed, f = _newton_inputs(case, seed)
        if X.size > EXACT_DOFS:
            return None
        X, cells, theta, fixed, f = gpu(X, cells.astype(np.int64), theta, fixed.astype(np.int64), f)
        x, E = _equilibrium(case, X, cells, theta, fixed, f, torch.zeros_like(f))
        return {"x": x, "energy": float(E)}
    if case["kind"] == "batch":
        X, cells, voff, eoff, theta, fixed, f = _batch_inputs(case, seed)
        if 3 * int(np.diff(voff).max()) > EXACT_DOFS:
            return None
        xs, Es = [], []
        for m in range(case["count"]):
            v, e = slice(voff[m], voff[m + 1]), slice(eoff[m], eoff[m + 1])
            d = slice(3 * voff[m], 3 * voff[m + 1])
            held = fixed[(fixed >= d.start) & (fixed < d.stop)] - d.start
            a = gpu(X[v], cells[e].astype(np.int64) - voff[m], theta[e], held.astype(np.int64), f[d])
            x, E = _equilibrium(case, *a, torch.zeros_like(a[4]))
            xs.append(x)
            Es.append(float(E))
        return {"x": torch.cat(xs), "energy": np.array(Es)}
    X, cells, theta, fixed, u, w = _adjoint_inputs(case, seed)
    if X.size > EXACT_DOFS:
        return None
    X, cells, theta, fixed, u, w = gpu(X, cells.astype(np.int64), theta, fixed.astype(np.int64), u, w)
    free = torch.ones_like(u, dtype=torch.bool)
    free[fixed] = False
    K = _dense(case, X, cells, theta, u)[2][free][:, free]
    lam = torch.zeros_like(u)
    lam[free] = torch.cholesky_solve(w[free][:, None], torch.linalg.cholesky(K))[:, 0]
    G, vol, _ = _tet_gradients(X, cells, None)
    F = torch.eye(3, dtype=X.dtype, device=X.device) + u.reshape(-1, 3)[cells].transpose(1, 2) @ G
    Fi = torch.linalg.inv(F).transpose(1, 2)
    Gl = lam.reshape(-1, 3)[cells].transpose(1, 2) @ G
    hf, ff = (Fi * Gl).sum((1, 2)), (F * Gl).sum((1, 2))
    dtheta = -torch.stack([vol * torch.log(torch.linalg.det(F)) * hf, vol * (ff - hf)], 1)
    return {"dtheta": dtheta.reshape(-1), "lambda": lam}
