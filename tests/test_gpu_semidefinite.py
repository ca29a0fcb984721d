"""Hex and Hermite elements whose tangents are all semi-definite keep their Hessian bit by bit in the projected one
(FP64; rounded once in mixed precision), beside elements that are clamped; neo-Hookean and Python materials."""

import numpy as np
import pytest

from litepgo_b200 import dof, energy, fem, mesh
from test_gpu_projection import CORNERS, Prescribed, _cells, _check

pytestmark = pytest.mark.gpu
Exact, Projected = energy.HessianKind.Exact, energy.HessianKind.Projected
Q = np.linalg.qr(np.random.default_rng(1).standard_normal((3, 3)))[0]
KEPT = [np.eye(3), Q * np.sign(np.linalg.det(Q)), 1.1 * np.eye(3), np.diag([1.05, 1.02, 1.0])]
CLAMPED = [0.6 * np.eye(3), np.diag([1.0, 0.9, 0.5]), np.diag([0.8, 0.8, 1.0])]


def _kept_exactly(e, u, size, kept):
    H = e.eval(u, hessian=Exact)[2].toarray()
    for precision in ("f64", "mixed"):
        P = e.eval(u, hessian=Projected, precision=precision)[2].toarray()
        for k, keep in enumerate(kept):
            s = slice(size * k, size * (k + 1))
            want = H[s, s] if precision == "f64" else H[s, s].astype(np.float32)
            assert np.array_equal(P[s, s], want) == keep, (k, precision)
    _check(e, u, size)
    _check(e, u, size, "mixed", 1e-6)


@pytest.mark.parametrize("points", [2, 4])
@pytest.mark.parametrize("basis", ["hex", "hermite"])
def test_neo_hookean(basis, points):
    states = KEPT + CLAMPED + KEPT[:1]
    kept = [True] * len(KEPT) + [False] * len(CLAMPED) + [True]
    X, cells = _cells(len(states))
    theta = np.tile([1.5e4, 1e4], (len(states), 1))
    if basis == "hex":
        u = np.concatenate([CORNERS @ A.T - CORNERS for A in states]).ravel()
        cls = fem.VolumetricFemEnergy[fem.NeoHookean, fem.HexQ1Basis, fem.GaussLegendre3D[points]]
    else:
        u = np.zeros((len(states), 8, 8, 3))
        for k, A in enumerate(states):
            u[k, :, 0] = CORNERS @ (A - np.eye(3)).T
            u[k, :, 1:4] = (A - np.eye(3)).T
        u = u.ravel()
        cls = fem.VolumetricFemEnergy[fem.NeoHookean, fem.HexHermiteBasis, fem.GaussLegendre3D[points]]
    _kept_exactly(cls.from_arrays(X, cells, theta), u, 24 if basis == "hex" else 192, kept)


@pytest.mark.parametrize("least, kept", [(1.0, True), (0.0, True), (-0.5, False)])
def test_material(least, kept):
    R = np.linalg.qr(np.random.default_rng(2).standard_normal((9, 9)))[0]
    Prescribed.A = ((R * np.r_[least, np.arange(1.0, 9.0)]) @ R.T).reshape(3, 3, 3, 3)
    X, cells = _cells(5)
    cls = fem.VolumetricFemEnergy[Prescribed, fem.HexQ1Basis, fem.GaussLegendre3D[2]]
    e = cls(dof.VertexDofMap(mesh.HexTopology(X.shape[0], cells), 3), X, None, np.array([1.0, 1.0]))
    _kept_exactly(e, np.zeros(X.size), 24, [kept] * 5)
