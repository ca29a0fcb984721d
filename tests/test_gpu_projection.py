"""The PSD projections of hex and Hermite element Hessians against numpy's eigensolver, on meshes of
disjoint cells: the assembled Exact Hessian is then block diagonal and its blocks are the element
Hessians, so the Projected one must be each block's V max(L, 0) V^T. Both run on the same element pass, so
what differs is the eigen-decomposition's round-off, a modest multiple of N eps |H|: 1e-12 of the block's
largest entry. Cell counts around a block of warps (4) and of the element pass (7); spectra: semi-definite,
indefinite, with repeated eigenvalues (a cube under a uniform stretch), negative semi-definite, zero."""

import numpy as np
import pytest

from litepgo_b200 import dof, energy, fem, mesh

pytestmark = pytest.mark.gpu
Exact, Projected = energy.HessianKind.Exact, energy.HessianKind.Projected

CORNERS = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]], dtype=float)
SYM = {
    "rest": np.eye(3),
    "stretched": 1.4 * np.eye(3),
    "compressed": 0.55 * np.eye(3),
    "crushed": np.diag([0.2, 0.2, 0.2]),
    "uniaxial": np.diag([1.0, 1.0, 0.4]),
    "sheared": np.array([[1.0, 0.5, 0.0], [0.1, 0.8, 0.2], [0.0, -0.3, 0.7]]),
}


def _cells(count):
    X = np.concatenate([CORNERS + [3.0 * e, 0, 0] for e in range(count)])
    return X, np.arange(8 * count, dtype=np.int32).reshape(count, 8)


def _check(e, u, size, precision="f64", tol=1e-12):
    H = e.eval(u, hessian=Exact)[2].toarray()
    P = e.eval(u, hessian=Projected, precision=precision)[2].toarray()
    assert np.array_equal(P, P.T)
    for k in range(H.shape[0] // size):
        s = slice(size * k, size * (k + 1))
        L, Q = np.linalg.eigh(0.5 * (H[s, s] + H[s, s].T))
        ref = (Q * np.maximum(L, 0)) @ Q.T
        assert np.abs(P[s, s] - ref).max() <= tol * max(np.abs(H[s, s]).max(), 1e-300), (k, L[:3], L[-3:])
        P[s, s] = 0
    assert not P.any()


@pytest.mark.parametrize("points", [2, 4])
@pytest.mark.parametrize("count", [1, 3, 4, 5, 7, 8, 29])
def test_hex(count, points):
    X, cells = _cells(count)
    rng = np.random.default_rng(count)
    theta = np.stack([rng.uniform(1e3, 1e5, count), rng.uniform(1e3, 1e5, count)], axis=1)
    e = fem.VolumetricFemEnergy[fem.NeoHookean, fem.HexQ1Basis, fem.GaussLegendre3D[points]].from_arrays(X, cells, theta)
    states = list(SYM.values())
    u = np.concatenate([CORNERS @ states[k % len(states)].T - CORNERS for k in range(count)])
    _check(e, u.ravel(), 24)
    u += 0.02 * rng.standard_normal(u.shape)
    _check(e, u.ravel(), 24)
    _check(e, u.ravel(), 24, "mixed", 1e-6)


class Prescribed(fem.PyVolumetricMaterial):
    """W = 0, P = 0 and a given d2W/dF2 at every point."""

    num_parameters = 2
    A = None

    @staticmethod
    def eval(F, Fp, theta, *, outputs):
        import torch

        n = F.shape[0]
        make = lambda *shape: torch.zeros(*shape, dtype=torch.float64, device=F.device)  # noqa: E731
        given = {"W": make(n), "dW_dF": make(n, 3, 3),
                 "d2W_dF2": torch.as_tensor(Prescribed.A, device=F.device).expand(n, 3, 3, 3, 3).contiguous()}
        return {o: given[o] for o in outputs}


@pytest.mark.parametrize("kind", ["zero", "negative", "mostly negative", "mostly positive", "rank one", "random"])
def test_hex_tangents(kind):
    rng = np.random.default_rng(5)
    Q = np.linalg.qr(rng.standard_normal((9, 9)))[0]
    L = {"zero": np.zeros(9), "negative": -np.ones(9), "mostly negative": np.r_[-np.arange(1.0, 8.0), 0.5, 3.0],
         "mostly positive": np.r_[np.arange(1.0, 8.0), -0.5, -3.0], "rank one": np.r_[-2.0, np.zeros(8)],
         "random": rng.standard_normal(9)}[kind]
    Prescribed.A = ((Q * L) @ Q.T).reshape(3, 3, 3, 3)
    X, cells = _cells(5)
    cls = fem.VolumetricFemEnergy[Prescribed, fem.HexQ1Basis, fem.GaussLegendre3D[2]]
    e = cls(dof.VertexDofMap(mesh.HexTopology(X.shape[0], cells), 3), X, None, np.array([1.0, 1.0]))
    _check(e, np.zeros(X.size), 24)


@pytest.mark.parametrize("state", list(SYM))
@pytest.mark.parametrize("points", [2, 4])
def test_hermite(state, points):
    X, cells = _cells(3)
    theta = np.array([[1e4, 3e4], [2e5, 1e4], [7e3, 7e3]])
    e = fem.VolumetricFemEnergy[fem.NeoHookean, fem.HexHermiteBasis, fem.GaussLegendre3D[points]].from_arrays(X, cells, theta)
    u = np.zeros((24, 8, 3))
    A = SYM[state] - np.eye(3)
    u[:, 0] = np.tile(CORNERS, (3, 1)) @ A.T
    u[:, 1:4] = A.T
    _check(e, u.ravel(), 192)
    # A mixed second derivative does not move the corners: a different spectrum in each cell.
    u[:8, 4:7] += 0.02 * np.random.default_rng(2).standard_normal((8, 3, 3))
    _check(e, u.ravel(), 192)
    _check(e, u.ravel(), 192, "mixed", 1e-6)
