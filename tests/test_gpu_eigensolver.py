"""The symmetric eigensolver over sizes (one to sixteen CTAs' worth of rows, rows in shared memory and in
L2) and spectra: random, repeated, rank-deficient, graded over 16 decades, scaled far from one.

Bounds, as for any backward stable method: eigenvalues and residuals within 8 n 2^-53 of the largest
eigenvalue, eigenvectors orthonormal to 64 n 2^-53."""
import numpy as np
import pytest

from ttdft_public_gb300 import api, system

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def unit_op(k):
    n = 64
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n))
    return api.Operator(api.ProjectHamiltonianSparse(H), k)


def spectrum(kind, n, rng):
    if kind == "random":
        return rng.standard_normal(n)
    if kind == "repeated":
        return np.repeat([1.0, -2.0, 0.5], n)[:n] + 0.0
    if kind == "deficient":
        return np.concatenate([np.linspace(1, 2, (n + 1) // 2), np.zeros(n // 2)])
    if kind == "graded":
        return np.geomspace(1.0, 1e-16, n)
    if kind == "huge":
        return 1e150 * rng.standard_normal(n)
    return 1e-150 * rng.standard_normal(n)


def check(op, A):
    n = A.shape[0]
    w, V = np.zeros(n), np.zeros((n, n), order="F")
    api.EigenSolver(op).computeEigenPairsSeq(A, n, n, w, V)
    ref = np.linalg.eigvalsh(A)
    scale = max(np.abs(ref).max(), 1e-300)
    assert np.all(np.diff(w) >= 0)
    assert np.abs(w - ref).max() <= 8 * n * U * scale
    assert np.abs(A @ V - V * w).max() <= 8 * n * U * scale + 1e-300
    assert np.abs(V.T @ V - np.eye(n)).max() <= 64 * n * U
    return w, V


@pytest.mark.parametrize("n", [1, 2, 3, 5, 16, 31, 33, 97, 127, 128, 129, 160, 257, 360, 500])
def test_random_matrices(n):
    op = unit_op(512)
    try:
        A = np.random.default_rng(n).standard_normal((n, n))
        check(op, A + A.T)
    finally:
        op.close()


@pytest.mark.parametrize("kind", ["random", "repeated", "deficient", "graded", "huge", "tiny"])
@pytest.mark.parametrize("n", [7, 60, 200])
def test_spectra(kind, n):
    op = unit_op(512)
    try:
        rng = np.random.default_rng(n)
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        A = (Q * spectrum(kind, n, rng)) @ Q.T
        check(op, 0.5 * (A + A.T))
    finally:
        op.close()


@pytest.mark.parametrize("n", [60, 130])
def test_diagonal_and_zero_matrices(n):
    op = unit_op(512)
    try:
        check(op, np.diag(np.arange(n, dtype=float) - 5.0))
        check(op, np.zeros((n, n)))
        check(op, np.eye(n))
    finally:
        op.close()


def test_rows_beyond_shared_memory():
    n = 700
    op = unit_op(n)
    try:
        A = np.random.default_rng(1).standard_normal((n, n))
        check(op, A + A.T)
    finally:
        op.close()
