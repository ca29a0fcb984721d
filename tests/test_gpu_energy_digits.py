"""W of small strains keeps its digits: the FP64 energy against extended precision, for displacement
gradients from 1e-6 to well past the stretches that the correction of log J covers."""

import numpy as np
import pytest
import torch

from litepgo_b200 import energy, fem, mesh

pytestmark = pytest.mark.gpu


def _extended(X, tets, theta, u):
    """Sum of vol W in long double: J - 1 and |F|^2 - 3 from the invariants of the displacement gradient."""
    L = np.longdouble
    X, U = X.astype(L), u.reshape(-1, 3).astype(L)
    D = X[tets[:, 1:]] - X[tets[:, :1]]
    B = np.stack([np.cross(D[:, 1], D[:, 2]), np.cross(D[:, 2], D[:, 0]), np.cross(D[:, 0], D[:, 1])], axis=1)
    det = np.sum(D[:, 0] * B[:, 0], axis=1)
    E = U[tets[:, 1:]] - U[tets[:, :1]]
    H = np.einsum("eai,eaj->eij", E, B) / det[:, None, None]
    c1 = H[:, 0, 0] + H[:, 1, 1] + H[:, 2, 2]
    c2 = sum(H[:, i, i] * H[:, j, j] - H[:, i, j] * H[:, j, i] for i, j in ((0, 1), (0, 2), (1, 2)))
    c3 = np.sum(H[:, 0] * np.cross(H[:, 1], H[:, 2]), axis=1)
    logJ = np.log1p(c1 + c2 + c3)
    lam, mu = theta[:, 0].astype(L), theta[:, 1].astype(L)
    psi = mu / 2 * (2 * c1 + np.sum(H * H, axis=(1, 2))) - mu * logJ + lam / 2 * logJ * logJ
    return np.sum(det / 6 * psi)


# W sums terms of order mu strain that cancel to mu strain^2, each rounded a handful of times:
# 64 roundings of 1.1e-16 relative to W, over the strain where that is below one.
@pytest.mark.parametrize("strain", [1e-6, 1e-4, 1e-2, 0.2, 3.0])
def test_energy_digits_at_small_strain(strain):
    X, tets = mesh.make_box(3, 2, 2)
    rng = np.random.default_rng(5)
    theta = np.stack([rng.uniform(1e4, 1e5, len(tets)), rng.uniform(1e3, 1e5, len(tets))], axis=1)
    G = np.array([[1.0, 0.3, -0.2], [0.1, 0.8, 0.25], [-0.3, 0.2, 0.9]])
    u = strain * (X @ G.T + 0.02 * rng.standard_normal(X.shape)).ravel()
    e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, theta)
    ut = torch.as_tensor(u, device="cuda")
    want = _extended(X, tets, theta, u)
    tol = 64 * np.finfo(float).eps / 2 * max(1.0, 1.0 / strain)
    for hessian in (None, energy.HessianKind.Exact):
        got = e.eval_device(ut, gradient=True, **({} if hessian is None else {"hessian": hessian}))[0]
        assert abs(got - float(want)) <= tol * abs(float(want))
