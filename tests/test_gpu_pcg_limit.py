"""A wait between the blocks of the one-launch PCG that runs out: with no polls allowed every block gives up in
its first exchange, the solve returns an error, and the next one finds a handle as good as new. A mesh of one
block waits for no one."""

import numpy as np
import pytest
import scipy.sparse as sp

from litepgo_b200 import _native as N
from litepgo_b200 import dof, energy, fem, mesh, solver, workloads

pytestmark = pytest.mark.gpu
LIMIT = 1 << 22


def _problem(boxes, precision):
    X, tets, voff, eoff = mesh.concatenate(boxes)
    e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, np.array([1.4e5, 3.4e4]))
    f = np.concatenate([workloads.gravity_load(*b) for b in boxes])
    total = energy.WeightedSumEnergy([(e, 1.0), (energy.QuadraticEnergy(sp.csc_matrix((X.size,) * 2), -f), 1.0)])
    fixed = (3 * np.flatnonzero(X[:, 2] == 0)[:, None] + np.arange(3)).ravel().astype(np.int32)
    opts = solver.NewtonOptions(gradient_tolerance=1e-8, stop_rule="relative", accept_rule="armijo", precision=precision,
                                max_iterations=50, cg_tolerance=1e-3)
    return e, total, voff, eoff, fixed, opts, X.size


def _solves(problem):
    e, total, voff, eoff, fixed, opts, n = problem

    def newton():
        return solver.newton_solve(total, dof.DofReduction(n, fixed), np.zeros(n), opts).x

    def batch():
        return solver.batch_newton_solve(total, voff, eoff, dof.DofReduction(n, fixed), np.zeros(n), opts)[0]

    def adjoint():
        w, lam = np.random.default_rng(1).standard_normal(n), np.empty(n)
        N.check(N.lib.lpg_adjoint_solve_terms(
            e.handle, None, N.vptr(np.zeros(n)), N.vptr(w), N.iptr(fixed), int(fixed.size), N.MEM_HOST,
            N.PRECISION_F64 if opts.precision == "f64" else N.PRECISION_MIXED, 1e-9, N.vptr(lam)))
        return lam

    return newton, batch, adjoint


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_a_wait_runs_out(precision):
    boxes = [mesh.make_box(9, 9, 7, size=(1, 1, 7 / 9)), mesh.make_box(11, 10, 8, size=(1, 10 / 11, 8 / 11))]
    problem = _problem(boxes, precision)
    for solve in _solves(problem):
        before = solve()
        N.check(N.lib.lpg_fem_set_poll_limit(problem[0].handle, 0))
        for _ in range(2):
            with pytest.raises(RuntimeError, match="lost one another"):
                solve()
        N.check(N.lib.lpg_fem_set_poll_limit(problem[0].handle, LIMIT))
        assert np.array_equal(solve(), before)


def test_one_block_waits_for_no_one():
    problem = _problem([mesh.make_box(3)], "f64")
    N.check(N.lib.lpg_fem_set_poll_limit(problem[0].handle, 0))
    newton, _, _ = _solves(problem)
    assert np.all(np.isfinite(newton()))
