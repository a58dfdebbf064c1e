"""The native FP64 product at the edges of its lane layout: one to many states a lane, two and four
sets of lanes (k <= 16, k <= 8), odd widths, a last row group that is not full, rows without entries
and explicit zeros.

A row's sum of m products in any order is within (m + 1) 2^-53 sum |h x| of the exact value; the
reference (scipy's FP64 product) is too, so the two differ by at most twice that."""
import numpy as np
import pytest
import scipy.sparse as sp

from ttdft_public_gb300 import api, system

pytestmark = pytest.mark.gpu


def random_csr(n, seed):
    rng = np.random.default_rng(seed)
    M = sp.random(n, n, density=0.2, random_state=rng, format="lil")
    M[3, :] = 0.0
    M = M.tocsr()
    M.sort_indices()
    M.data[::7] = 0.0                      # explicit zeros stay stored
    return system.Csr(n, n, M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data)


@pytest.mark.parametrize("n", [125, 512])
@pytest.mark.parametrize("k", [2, 7, 8, 9, 16, 17, 32, 33, 95, 160, 161, 322])
def test_fp64_product_at_width_edges(n, k):
    H = random_csr(n, 5)
    X = np.random.default_rng(k).standard_normal((n, k))
    op = api.Operator(api.ProjectHamiltonianSparse(H), k)
    try:
        ax = api.AX(1, k)
        ax.op = op
        Xm, Ym = api.Mat(op, k, X), api.Mat(op, k)
        ax.perform_ax(Xm, Ym)
        A = H.to_scipy()
        m = np.diff(H.row_ptr)[:, None]
        bound = 2.0 * (m + 1) * 2.0 ** -53 * (abs(A) @ np.abs(X))
        assert np.all(np.abs(Ym.get() - A @ X) <= bound)
    finally:
        op.close()
