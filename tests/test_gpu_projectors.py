"""The projector products W = diag(D) C X at the edges of their split: rows of zero to many entries, around
the 16 loads in flight and the 128 entries of a part; widths around the 128 states of a block.

A sum of m products in any order is within (m + 1) 2^-53 sum |c x| of the exact one; C^T adds its own, and
the reference as much again."""
import numpy as np
import pytest

from ttdft_public_gb300 import api, system

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 15, 16, 17, 127, 128, 129, 143, 257, 2100]


@pytest.mark.parametrize("k", [1, 7, 127, 128, 130, 300])
def test_projector_rows_of_many_lengths(k):
    n, rng = 2200, np.random.default_rng(k)
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), rng.standard_normal(n))
    ptr = np.concatenate([[0], np.cumsum(LENGTHS)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(n, m, replace=False)) for m in LENGTHS]).astype(np.int32)
    C = system.Csr(len(LENGTHS), n, ptr, col, rng.standard_normal(ptr[-1]))
    D = rng.standard_normal(len(LENGTHS))
    X = rng.standard_normal((n, k))
    op = api.Operator(api.ProjectHamiltonianSparse(H, C, D), k)
    try:
        ax = api.AX(1, k)
        ax.op = op
        Xm, Ym = api.Mat(op, k, X), api.Mat(op, k)
        ax.perform_ax(Xm, Ym)
        S, A, X1 = C.to_scipy(), abs(C.to_scipy()), np.abs(X)
        ref = H.val[:, None] * X + S.T @ (D[:, None] * (S @ X))
        mag = np.abs(H.val)[:, None] * X1 + A.T @ (np.abs(D)[:, None] * (A @ X1))
        m = max(LENGTHS) + len(LENGTHS) + 4
        assert np.all(np.abs(Ym.get() - ref) <= 2.0 * m * 2.0 ** -53 * mag)
    finally:
        op.close()
