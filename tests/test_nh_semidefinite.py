"""The closed-form semi-definiteness test of the neo-Hookean tangent (litepgo_b200/csrc/lpg_psd.h), which lets hex
and Hermite elements keep their Hessian without an eigen-decomposition, against the eigenvalues of the 9x9 tangent.

Whenever it says yes, no eigenvalue may be below the allowance it is given, 64 eps of the largest diagonal entry,
plus the round-off of F and of the eigensolver (another 64 eps). It has to say yes wherever the least eigenvalue is
at least 4e-3 of s = mu (1 + (|a| + l) max g^2): the block's determinant is then above (4e-3 s)^3 and its margin,
1e-8 of at most 4 s^3, below that; without expansion (a <= 0) wherever no eigenvalue is negative at all."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

_dp, _ip = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def semidefinite(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    out = tmp_path_factory.mktemp("nh") / "libnh.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(ROOT / "litepgo_b200" / "csrc"),
                    str(ROOT / "tests" / "nh_point_host.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.nh_semidefinite_host.argtypes = [ctypes.c_int, _dp, _dp, _dp, _ip]

    def run(F, theta):
        n = F.shape[0]
        J, G = np.linalg.det(F), np.linalg.inv(F).transpose(0, 2, 1)
        out = np.empty(n, np.int32)
        args = [np.ascontiguousarray(x) for x in (G, J, theta)]
        lib.nh_semidefinite_host(n, *[x.ctypes.data_as(_dp) for x in args], out.ctypes.data_as(_ip))
        return out.astype(bool)

    return run


def _tangents(F, theta):
    n, lam, mu = F.shape[0], theta[:, 0], theta[:, 1]
    G = np.linalg.inv(F).transpose(0, 2, 1)
    p = lam * np.log(np.linalg.det(F)) - mu
    eye = np.eye(3)
    A = (mu[:, None, None, None, None] * np.einsum("ik,jl->ijkl", eye, eye) +
         lam[:, None, None, None, None] * np.einsum("nij,nkl->nijkl", G, G) -
         p[:, None, None, None, None] * np.einsum("nil,nkj->nijkl", G, G))
    return A.reshape(n, 9, 9), p / mu, np.abs(G).max(axis=(1, 2)) ** 2


def _rotations(rng, n):
    Q = np.linalg.qr(rng.standard_normal((n, 3, 3)))[0]
    return Q * np.sign(np.linalg.det(Q))[:, None, None]


STRETCHES = {
    "rest": lambda r, n: np.ones((n, 3)),
    "near rest": lambda r, n: 1 + 1e-7 * r.standard_normal((n, 3)),
    "small": lambda r, n: 1 + 0.05 * r.standard_normal((n, 3)),
    "large": lambda r, n: np.exp(0.4 * r.standard_normal((n, 3))),
    "expanded": lambda r, n: np.exp(0.15 * np.abs(r.standard_normal((n, 3)))),
    "uniform": lambda r, n: np.repeat(np.exp(0.3 * r.standard_normal((n, 1))), 3, axis=1),
    # Straddling the equality |a| s_k = J of the 2 x 2 blocks.
    "boundary": lambda r, n: np.stack([1 + r.choice([-1, 1], n) * 10.0 ** r.uniform(-15, -2, n), np.ones(n), np.ones(n)], 1),
}


@pytest.mark.parametrize("poisson", [0.0, 0.3, 0.45, 0.49])
@pytest.mark.parametrize("kind", list(STRETCHES))
def test_against_eigenvalues(semidefinite, kind, poisson):
    rng, n = np.random.default_rng([list(STRETCHES).index(kind), int(100 * poisson)]), 20000
    F = _rotations(rng, n) * STRETCHES[kind](rng, n)[:, None, :] @ _rotations(rng, n)
    mu = 10.0 ** rng.uniform(-6, 6, n)
    theta = np.stack([2 * mu * poisson / (1 - 2 * poisson), mu], axis=1)
    A, a, gmax = _tangents(F, theta)
    least = np.linalg.eigvalsh(A)[:, 0]
    allowance = 128 * EPS * np.abs(np.diagonal(A, axis1=1, axis2=2)).max(axis=1)
    said = semidefinite(F, theta)
    assert np.all(least[said] >= -allowance[said])
    gmax = 3 * gmax  # of the singular values
    clear = np.where(a <= 0, least > 0, least >= 4e-3 * mu * (1 + (np.abs(a) + theta[:, 0] / mu) * gmax))
    assert np.all(said[clear])
    if kind in ("rest", "uniform"):
        assert said.any()


def test_refuses_what_it_cannot_tell(semidefinite):
    F = np.stack([np.diag([np.nan, 1, 1]), np.diag([np.inf, 1, 1]), 1e200 * np.eye(3), np.diag([1e-200, 1, 1.0])])
    with np.errstate(all="ignore"):
        assert not semidefinite(F, np.tile([1.0, 1.0], (4, 1))).any()
