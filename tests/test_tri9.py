"""The tet tangent's clamp by the few eigenpairs of one sign (litepgo_b200/csrc/lpg_tri9.h) on the host
against an eigensolver, over the families where it can go wrong, and the projected Hessian on the GPU against
the oracle at the warps' and the grid's edges."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest

import oracle
from conftest import ROOT, rel_err

_dp = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def clamp(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    out = tmp_path_factory.mktemp("tri9") / "libtri9.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(ROOT / "litepgo_b200" / "csrc"),
                    str(ROOT / "tests" / "tri9_host.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.tri9_host.argtypes = [ctypes.c_int, _dp, _dp]

    def run(M, fp32):
        P = np.empty((9, 9))
        how = lib.tri9_host(1 if fp32 else 0, np.ascontiguousarray(M).ctypes.data_as(_dp), P.ctypes.data_as(_dp))
        return how, P

    return run


def _with(rng, w):
    Q = np.linalg.qr(rng.standard_normal((9, 9)))[0]
    return (Q * w) @ Q.T


def _tangent(rng, strain):
    while True:
        F = np.eye(3) + strain * rng.standard_normal((3, 3))
        if np.linalg.det(F) > 0.05:
            break
    Rq, mu, lam = rng.standard_normal((3, 3)), 3.4e4, 1.4e5
    G = np.linalg.inv(F).T
    f, p = G @ Rq.T, lam * np.log(np.linalg.det(F)) - mu
    M = (mu * np.einsum("ik,jl->jilk", np.eye(3), Rq @ Rq.T) + lam * np.einsum("ij,kl->jilk", f, f)
         - p * np.einsum("il,kj->jilk", f, f))
    return M.reshape(9, 9)


FAMILIES = {
    "small strain": lambda r: _tangent(r, 0.05),
    "large strain": lambda r: _tangent(r, 0.3),
    "random": lambda r: r.standard_normal((9, 9)) * 10.0 ** r.integers(-9, 9),
    "graded": lambda r: _with(r, r.standard_normal(9) * 10.0 ** r.uniform(-12, 0, 9)),
    "near zero": lambda r: _with(r, np.r_[-1e-6, 0, 0, 0, 1, 1, 1, 2, 3]),
    "repeated": lambda r: _with(r, np.r_[-1, -1 - 1e-5, -1 + 1e-12, 2, 2, 2, 5, 6, 7]),
    "diagonal": lambda r: np.diag(r.standard_normal(9)),
    "blocks": lambda r: np.kron(np.eye(3), (lambda B: B + B.T)(r.standard_normal((3, 3)))),
    "definite": lambda r: r.choice([-1, 1]) * (lambda B: B @ B.T)(r.standard_normal((9, 9))),
    "zero": lambda r: np.zeros((9, 9)),
}


# Residuals end within 36 round-offs of the norm and eigenvalues within 24 of zero are left; at most four pairs:
# 128 round-offs of the Frobenius norm. Repeated eigenvalues may be given up on, the others hardly.
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("name", FAMILIES)
def test_clamp_by_few_pairs(clamp, name, fp32):
    rng = np.random.default_rng(7)
    given_up = 0
    for _ in range(300):
        M = FAMILIES[name](rng)
        M = (0.5 * (M + M.T)).astype(np.float32 if fp32 else np.float64).astype(np.float64)
        how, P = clamp(M, fp32)
        given_up += how == 0
        if how != 0:
            eps = np.finfo(np.float32 if fp32 else np.float64).eps
            assert np.linalg.norm(P - oracle.project_psd(M)) <= 128 * eps * np.linalg.norm(M)
    assert given_up <= (30 if name in ("repeated", "graded") else 3)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("f64", 1e-11), ("mixed", 1e-4)])
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 1), (13, 1, 1), (7, 5, 4), (24, 23, 22)])
def test_projected_hessian(dims, precision, tol):
    from litepgo_b200 import energy, fem, mesh

    X, tets = mesh.make_box(*dims)
    rng = np.random.default_rng(2)
    theta = np.stack([rng.uniform(1e4, 1e5, len(tets)), rng.uniform(1e3, 1e5, len(tets))], axis=1)
    h = np.ptp(X, axis=0).max() / max(dims)
    u = (X @ (0.1 * rng.standard_normal((3, 3))) + 0.08 * h * rng.standard_normal(X.shape)).ravel()
    e = fem.VolumetricFemEnergyTetP1.from_arrays(X, tets, theta)
    _, _, H = e.eval(u, hessian=energy.HessianKind.Projected, precision=precision)
    _, _, ref = oracle.OracleMesh(X, tets, theta).eval(u, False, 2)
    assert rel_err(H.data, ref) <= tol
