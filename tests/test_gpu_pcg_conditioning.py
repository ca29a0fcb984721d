"""The one-launch PCG on ill-conditioned positive definite systems: nearly incompressible blocks and slender
columns, at rest, held at the bottom. In FP32 a p.Ap that is not formed from p itself loses its sign there and the
solve ends as if the matrix were indefinite."""

import numpy as np
import pytest
import scipy.sparse as sp

from litepgo_b200 import _native as N
from litepgo_b200 import dof, energy, fem, mesh, solver, workloads

pytestmark = pytest.mark.gpu

# Cube counts (sides of 1/8) and lambda / mu.
SYSTEMS = {
    "nu 0.4999": ((8, 8, 8), 5e3),
    "nu 0.499975": ((8, 8, 8), 2e4),
    "nu 0.499995": ((8, 8, 8), 1e5),
    "column 1x1x50": ((1, 1, 50), 1.5),
    "column 2x2x60": ((2, 2, 60), 1.5),
}


def _system(name):
    d, ratio = SYSTEMS[name]
    X, tets = mesh.make_box(*d, size=tuple(k / 8 for k in d))
    fixed = (3 * np.flatnonzero(X[:, 2] == 0)[:, None] + np.arange(3)).ravel().astype(np.int32)
    return X, tets, fixed, fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, np.array([1e4 * ratio, 1e4]))


# The solver ends at an FP64 residual of 1e-9 |w| that it forms itself; forming it here again, in another order,
# differs by the rounding of two sums of at most 45 products per row, 90 eps |K| |lambda|.
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("name", SYSTEMS)
def test_adjoint_solve(name, precision):
    X, _, fixed, e = _system(name)
    n = X.size
    free = np.ones(n, bool)
    free[fixed] = False
    K = e.eval(np.zeros(n), hessian=energy.HessianKind.Exact)[2].tocsr()
    for seed in range(3):
        u, w, lam = np.zeros(n), np.random.default_rng(seed).standard_normal(n), np.empty(n)
        N.check(N.lib.lpg_adjoint_solve_terms(
            e.handle, None, N.vptr(u), N.vptr(w), N.iptr(fixed), int(fixed.size), N.MEM_HOST,
            N.PRECISION_F64 if precision == "f64" else N.PRECISION_MIXED, 1e-9, N.vptr(lam)))
        rounding = 90 * np.finfo(float).eps * np.linalg.norm((abs(K) @ abs(lam))[free])
        assert np.linalg.norm((K @ lam - w)[free]) <= 1e-9 * np.linalg.norm(w[free]) + rounding


# A load small enough that the block stays in its linear range: a few Newton steps, whatever the conditioning.
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("name", ["nu 0.4999", "nu 0.499975", "column 2x2x60"])
def test_newton(name, precision):
    X, tets, fixed, e = _system(name)
    load = energy.QuadraticEnergy(sp.csc_matrix((X.size,) * 2), -1e-6 * workloads.gravity_load(X, tets))
    r = solver.newton_solve(energy.WeightedSumEnergy([(e, 1.0), (load, 1.0)]), dof.DofReduction(X.size, fixed), np.zeros(X.size),
                            solver.NewtonOptions(gradient_tolerance=1e-8, stop_rule="relative", accept_rule="armijo",
                                                 precision=precision, max_iterations=40, cg_tolerance=1e-6,
                                                 cg_max_iterations=200000))
    assert r.status == solver.NewtonStatus.Converged
