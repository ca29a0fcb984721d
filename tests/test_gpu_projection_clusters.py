"""The PSD projections of 24 x 24 and 192 x 192 element Hessians against numpy's eigensolver where eigenvalues
coincide or nearly so: vectors of one cluster come out of the inverse iteration almost parallel there, and what
Gram-Schmidt leaves of them has lost digits unless they are iterated again. Residuals are accepted up to 1e-13 of
the tridiagonal form's norm bound, at most three times |H|, so entries are within 1e-12 of |H|. With no rounds
allowed the Jacobi method takes every matrix, to the same bound (it stops at 1e-14 |H|)."""

import numpy as np
import pytest

from litepgo_b200 import _native as N

pytestmark = pytest.mark.gpu


def _spectrum(kind, n, rng):
    h, i = n // 2, np.arange(n)
    near = 10.0 ** rng.uniform(-16, -4, n) * rng.standard_normal(n)
    return {
        "two": np.where(i < h, -1.0, 1.0),
        "three": np.where(i < n // 3, -1.0, np.where(i < h, -0.5, rng.uniform(2, 3, n))),
        "pairs": np.where(i % 4 < 2, -1.0, 1.0) * (1 + 0.1 * (i // 4)),
        "near": np.where(i < h, -1 + near, 1 + 0.3 * rng.standard_normal(n)),
        "spaced": np.where(i < h, -1 - 1e-15 * i * i, 3.0),
        "graded": np.where(i < h, -10.0 ** rng.uniform(-16, 0, n), 1.0),
        "positive few": np.where(i < 5, 1.0, -1.0),
        "random": rng.standard_normal(n),
    }[kind]


KINDS = ["two", "three", "pairs", "near", "spaced", "graded", "positive few", "random"]


def _records(H, nodes):
    count = H.shape[0]
    blocks = H.reshape(count, nodes, 3, nodes, 3).transpose(0, 1, 3, 2, 4)
    a, b = np.triu_indices(nodes)
    return np.ascontiguousarray(blocks[:, a, b]).reshape(count, -1)


def _matrices(kind, nodes, count):
    n, rng = 3 * nodes, np.random.default_rng([nodes, KINDS.index(kind)])
    Q = np.linalg.qr(rng.standard_normal((count, n, n)))[0]
    L = np.stack([_spectrum(kind, n, rng) for _ in range(count)])
    L *= 10.0 ** rng.uniform(-8, 8, (count, 1))
    H = (Q * L[:, None]) @ Q.transpose(0, 2, 1)
    return 0.5 * (H + H.transpose(0, 2, 1))


@pytest.mark.parametrize("rounds", [-1, 0])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nodes, count", [(8, 2001), (64, 40)])
def test_projection(nodes, count, kind, rounds):
    if rounds == 0:
        count = count // 8
    H = _matrices(kind, nodes, count)
    w, V = np.linalg.eigh(H)
    ref = _records((V * np.maximum(w, 0)[:, None]) @ V.transpose(0, 2, 1), nodes)
    given, out = _records(H, nodes), np.empty_like(ref)
    N.check(N.lib.lpg_project_hessians(nodes, count, N.dptr(given), N.dptr(out), rounds))
    error = np.abs(out - ref).max(axis=1) / np.abs(w).max(axis=1)
    assert error.max() <= 1e-12, (int(np.argmax(error)), error.max(), int((error > 1e-12).sum()))


def test_invalid_arguments():
    H = np.zeros((1, 9 * 36))
    assert N.lib.lpg_project_hessians(4, 1, N.dptr(H), N.dptr(H), -1) != 0
    assert N.lib.lpg_project_hessians(8, -1, N.dptr(H), N.dptr(H), -1) != 0
    assert N.lib.lpg_project_hessians(8, 1, None, N.dptr(H), -1) != 0
    assert N.lib.lpg_project_hessians(8, 0, None, None, -1) == 0
