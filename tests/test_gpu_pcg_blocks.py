"""The one-launch PCG at the lines of its block rule (chunks of 32 rows per system, exactly at a line and past it;
its two builds meet at 296 chunks), checked as in test_gpu_pcg.py; and a handle that solves in both precisions in
turn, each with a plan of its own."""

import numpy as np
import pytest

import test_gpu_pcg as base
from litepgo_b200 import _native as N
from litepgo_b200 import fem, mesh

pytestmark = pytest.mark.gpu

# Cube counts: 16, 18, 32, 35, 56, 59, 296, 318, 1184 and 1229 chunks.
BOXES = [(7, 7, 7), (7, 7, 8), (7, 7, 15), (9, 9, 10), (7, 7, 27), (11, 11, 12), (15, 15, 36), (21, 21, 20), (31, 31, 36),
         (33, 33, 33)]


@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("box", BOXES)
def test_lines_of_the_rule(monkeypatch, box, precision):
    monkeypatch.setitem(base.MESHES, "box", lambda: mesh.make_box(*box))
    base.test_residual_of_a_solve("box", precision)


def test_precisions_in_turn():
    X, tets = mesh.make_box(9, 8, 10)
    e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, np.array([1.4e4, 3.4e3]))
    fixed = (3 * np.flatnonzero(X[:, 2] == X[:, 2].min())[:, None] + np.arange(3)).ravel().astype(np.int32)
    w = np.random.default_rng(1).standard_normal(X.size)

    def solve(precision):
        lam = np.empty(X.size)
        N.check(N.lib.lpg_adjoint_solve_terms(e.handle, None, N.vptr(np.zeros(X.size)), N.vptr(w), N.iptr(fixed),
                                              int(fixed.size), N.MEM_HOST, precision, 1e-9, N.vptr(lam)))
        return lam

    first = [solve(p) for p in (N.PRECISION_F64, N.PRECISION_MIXED)]
    for _ in range(3):
        for lam, p in zip(first, (N.PRECISION_F64, N.PRECISION_MIXED)):
            assert np.array_equal(solve(p), lam)
    assert np.abs(first[0] - first[1]).max() <= 1e-5 * np.abs(first[0]).max()
