"""The solvers' PCG in one launch: the residual of a whole adjoint solve against the assembled Exact
Hessian, over part of one chunk of rows, full and ragged chunks, one and several chunks per block, rows
that several warps share, the largest mesh of one launch and the first past it, irregular valence, and
fixed components scattered over the rows. And batches: several meshes in a chunk, one and several launches,
and more than the launches of one solve, against the meshes' own solves."""

import numpy as np
import pytest

from litepgo_b200 import _native as N
from litepgo_b200 import dof, energy, fem, mesh, solver, workloads

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MESHES = {
    "part of a chunk": lambda: mesh.make_box(1),
    "one chunk": lambda: mesh.make_box(3, 3, 1),
    "two chunks": lambda: mesh.make_box(3, 3, 2),
    "ball": lambda: mesh.delaunay_ball(700, seed=4),
    "a chunk per block": lambda: mesh.make_box(15, 15, 17),
    "two chunks per block": lambda: mesh.make_box(15, 15, 18),
    "largest": lambda: mesh.make_box(40, 41, 43),
    "past it": lambda: mesh.make_box(40, 41, 44),
}


# The solvers refine until the FP64 residual, which they form anew, is below the tolerance; forming it
# here again differs by roundings of K x, some 1e-13 of |w| for these meshes' conditioning (1e2 n^2).
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("name", MESHES)
def test_residual_of_a_solve(name, precision):
    X, tets = MESHES[name]()
    rng = np.random.default_rng(3)
    T, n, tol = len(tets), X.size, 1e-9
    theta = np.stack([rng.uniform(1e4, 1e5, T), rng.uniform(1e3, 1e5, T)], axis=1)
    low = np.flatnonzero(X[:, 2] <= X[:, 2].min() + 0.1 * np.ptp(X[:, 2]))
    fixed = np.union1d((3 * low[:, None] + np.arange(3)).ravel(), rng.choice(n, n // 20, replace=False)).astype(np.int32)
    e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, theta)
    u, w, lam = np.zeros(n), rng.standard_normal(n), np.empty(n)
    N.check(N.lib.lpg_fem_set_stream(e.handle, None))
    for _ in range(2):  # the second solve finds the words of the first
        N.check(N.lib.lpg_adjoint_solve_terms(
            e.handle, None, N.vptr(u), N.vptr(w), N.iptr(fixed), int(fixed.size), N.MEM_HOST,
            N.PRECISION_F64 if precision == "f64" else N.PRECISION_MIXED, tol, N.vptr(lam)))
        _, _, K = e.eval(u, hessian=energy.HessianKind.Exact)
        free = np.ones(n, bool)
        free[fixed] = False
        assert np.all(lam[fixed] == 0)
        res = (K @ lam - w)[free]
        assert np.linalg.norm(res) <= 1.01 * tol * np.linalg.norm(w[free])
        w = rng.standard_normal(n)


# Cube counts of the batch's boxes (drawn in turn) and their number. A gradient of 1e-11 of its start leaves
# the displacement within 1e-11 of the stiffness' condition, 1e3 at 5 cubes a side: 1e-8, and ten times that.
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("sides,count", [((1, 2, 3), 3), ((1, 5, 2, 4), 40), ((1, 2), 400), ((1,), 3000)])
def test_batch_matches_its_meshes(sides, count, precision):
    boxes = [mesh.make_box(k, k, k, size=(k / 8,) * 3) for k in sides]
    X, tets, voff, eoff = mesh.concatenate([boxes[i % len(sides)] for i in range(count)])
    f = np.concatenate([workloads.gravity_load(*boxes[i % len(sides)]) for i in range(count)])
    fixed = (3 * np.flatnonzero(X[:, 2] == 0)[:, None] + np.arange(3)).ravel().astype(np.int32)
    theta = np.array([1.4e5, 3.4e4])
    opts = solver.NewtonOptions(gradient_tolerance=1e-11, stop_rule="relative", accept_rule="armijo", precision=precision,
                                max_iterations=100, cg_tolerance=1e-3)

    def total(X, tets, f):
        import scipy.sparse as sp

        e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, theta)
        return energy.WeightedSumEnergy([(e, 1.0), (energy.QuadraticEnergy(sp.csc_matrix((X.size,) * 2), -f), 1.0)])

    x, per, _ = solver.batch_newton_solve(total(X, tets, f), voff, eoff, dof.DofReduction(X.size, fixed),
                                          np.zeros(X.size), opts)
    assert all(p.status == solver.NewtonStatus.Converged for p in per)
    alone = []
    for Xm, tm in boxes:
        low = (3 * np.flatnonzero(Xm[:, 2] == 0)[:, None] + np.arange(3)).ravel().astype(np.int32)
        alone.append(solver.newton_solve(total(Xm, tm, workloads.gravity_load(Xm, tm)), dof.DofReduction(Xm.size, low),
                                         np.zeros(Xm.size), opts))
        assert alone[-1].status == solver.NewtonStatus.Converged
    for m in range(count):
        r = alone[m % len(sides)].x
        assert np.max(np.abs(x[3 * voff[m]:3 * voff[m + 1]] - r)) <= 1e-7 * np.max(np.abs(r))
