"""H X of the Rayleigh-Ritz step on the tensor cores, at the edges of its groups of 32 states, with several
tiles a CTA, rows of very different sizes and rows without entries; and again after new values.

Bound: a product's operands carry 2^-55 of the largest value of their row of H and column of X, and the sums
are double-FP32 (2^-48); the eigenvalues of X^T H X move by at most the Frobenius norm of that matrix' error, and the
eigensolver's own error is far below 2^-40 of its norm."""
import numpy as np
import pytest
import scipy.sparse as sp

from ttdft_public_gb300 import api, system

pytestmark = pytest.mark.gpu


# the last: about 380,000 chunks of H, more than are held at a time
@pytest.mark.parametrize("n, k, band", [(300, 32, 150), (1000, 33, 150), (1000, 64, 150), (1000, 97, 150),
                                        (20100, 160, 150), (20100, 40, 150), (260000, 32, 1500)])
def test_ritz_values(n, k, band):
    rng = np.random.default_rng(n + k)
    col = np.clip(np.arange(n)[:, None] + rng.integers(-band, band, (n, 15)), 0, n - 1)
    M = sp.csr_matrix((rng.standard_normal(n * 15), (np.repeat(np.arange(n), 15), col.ravel())), shape=(n, n))
    M = M + M.T
    d = 10.0 ** rng.uniform(-2, 2, n)
    d[5] = 0.0
    M = (sp.diags(d) @ M @ sp.diags(d)).tocsr()
    M.eliminate_zeros()
    M.sort_indices()
    C = sp.random(3, n, density=0.05, random_state=rng, format="csr")
    C.sort_indices()
    D = np.array([2.0, -1.0, 0.5])
    H = system.Csr(n, n, M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data)
    Cs = system.Csr(3, n, C.indptr.astype(np.int64), C.indices.astype(np.int32), C.data)
    X, _ = np.linalg.qr(rng.standard_normal((n, k)))
    op = api.Operator(api.ProjectHamiltonianSparse(H, Cs, D), k)
    try:
        w = api.rayleigh_ritz(op, api.Mat(op, k, X), rotate=False)
        W = D[:, None] * (C @ X)
        P = X.T @ (M @ X + C.T @ W)
        rows = np.maximum(np.asarray(abs(M).max(axis=1).todense()).ravel(),
                          np.asarray(abs(C).max(axis=0).todense()).ravel())
        count = np.diff(M.indptr) + 3
        cols = np.maximum(np.abs(X).max(axis=0), np.abs(W).max(axis=0))
        E = 2.0 ** -45 * (np.abs(X).T @ (rows * count))[:, None] * cols[None, :]
        assert np.abs(w - np.linalg.eigvalsh(0.5 * (P + P.T))).max() <= \
            np.linalg.norm(E) + 2.0 ** -40 * np.linalg.norm(P)
    finally:
        op.close()
