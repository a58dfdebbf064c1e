"""Cholesky-QR of blocks wider than 128: last diagonal blocks of 1 to 64 columns, and a pivot that fails in
the second block.

X has condition about 2, so Q^T Q - I and the part of Q^T X below the diagonal are a few k 2^-53 and the Gram
matrix' own 2^-44 of |X|^T |X|: 2^-40 is granted."""
import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


def plain_operator(n, k):
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n))
    return api.Operator(api.ProjectHamiltonianSparse(H), k)


@pytest.mark.parametrize("k", [129, 160, 191, 192, 193, 320])
def test_orthonormal_and_triangular(k):
    n = 4000
    X = np.random.default_rng(k).standard_normal((n, k)) / np.sqrt(n)
    op = plain_operator(n, k)
    try:
        Xm = api.Mat(op, k, X)
        api.MultTM().orth(Xm)
        Q = Xm.get()
        assert np.abs(Q.T @ Q - np.eye(k)).max() <= 2.0 ** -40
        assert np.abs(np.tril(Q.T @ X, -1)).max() <= 2.0 ** -40
    finally:
        op.close()


def test_failing_pivot_is_reported():
    n, k = 4000, 160
    X = np.random.default_rng(0).standard_normal((n, k))
    X[:, 100] = X[:, 7]
    op = plain_operator(n, k)
    try:
        with pytest.raises(_lib.TtgError, match="NOT_SPD"):
            api.MultTM().orth(api.Mat(op, k, X))
    finally:
        op.close()
