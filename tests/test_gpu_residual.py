"""Energy with and without the gradient (the passes without a Hessian) against the oracle, FP64 to
1e-12 of the largest entry as the Hessian pass, and bitwise the gradient of the Hessian pass: one
cluster, a cluster boundary, more clusters than one wave of blocks, irregular valence, a vertex of no
element, and a plastic field."""

import numpy as np
import pytest
import torch

import oracle
from conftest import rel_err
from litepgo_b200 import energy, fem, mesh

pytestmark = pytest.mark.gpu

MESHES = {
    "one cube": lambda: mesh.make_box(1),
    "one cluster": lambda: mesh.make_box(3, 3, 2),
    "two clusters": lambda: mesh.make_box(4, 4, 3),
    "ragged": lambda: mesh.make_box(9, 7, 5),
    "waves": lambda: mesh.make_box(37, 31, 23),
    "ball": lambda: mesh.delaunay_ball(700, seed=4),
}


def _state(X):
    rng = np.random.default_rng(8)
    A = 0.08 * rng.standard_normal((3, 3))
    return (X @ A.T + 1e-4 * rng.standard_normal(X.shape)).ravel()


@pytest.mark.parametrize("plastic", [False, True])
@pytest.mark.parametrize("name", MESHES)
def test_energy_and_gradient_passes(name, plastic):
    X, tets = MESHES[name]()
    rng = np.random.default_rng(1)
    T = tets.shape[0]
    theta = np.stack([rng.uniform(1e4, 1e5, T), rng.uniform(1e3, 1e5, T)], axis=1)
    Fp = None
    if plastic:
        Fp = np.stack([(np.eye(3) + 0.02 * rng.standard_normal((3, 3))).T.ravel() for _ in range(T)])
    u = _state(X)
    e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, theta, Fp=Fp)
    orc = oracle.OracleMesh(X, tets, theta, Fp=Fp) if plastic else oracle.OracleMesh(X, tets, theta)
    Er, gr, _ = orc.eval(u, True, 0)
    ut = torch.as_tensor(u, device="cuda")
    E0, none, _ = e.eval_device(ut, gradient=False)
    E1, g1, _ = e.eval_device(ut, gradient=True)
    E2, g2, _ = e.eval_device(ut, gradient=True, hessian=energy.HessianKind.Exact)
    assert none is None
    for E in (E0, E1, E2):
        assert abs(E - Er) <= 1e-12 * abs(Er)
    assert rel_err(g1.cpu().numpy(), gr) <= 1e-12
    assert torch.equal(g1, g2)
    again = e.eval_device(ut, gradient=True)
    assert again[0] == E1 and torch.equal(again[1], g1)


def test_vertex_without_elements_and_bad_state():
    X, tets = mesh.make_box(3, 2, 2)
    X = np.vstack([X, [[5.0, 5.0, 5.0]]])
    e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, np.array([2.0, 3.0]))
    u = torch.as_tensor(_state(X), device="cuda")
    g = e.eval_device(u, gradient=True)[1]
    assert torch.all(g[-3:] == 0)
    bad = torch.as_tensor(-2.0 * X.ravel(), device="cuda")  # det F < 0 everywhere
    for gradient in (False, True):
        with pytest.raises(ValueError):
            e.eval_device(bad, gradient=gradient)
    assert np.isfinite(e.eval_device(u, gradient=False)[0])  # the status word was cleared
