"""Filter degrees on tiles of few chunks: the last stage of a tile then has slots without one, for the same gathering
warps tile after tile, and the warps are on other tiles than the MMAs.  The rows of a tile use 60 of the 128 + 2 w
columns around it: 9, 10, 11 and 13 chunks of 16.  And very sparse operators, whose FP32 degrees run on the row groups.

Small whole numbers, whose sums every format holds, come out exact."""
import numpy as np
import pytest
import scipy.sparse as sp

from ttdft_public_gb300 import api, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec, k", [("fp32", 20), ("fp32", 160), ("fp32", 256), ("bf16", 48), ("bf16", 160)])
@pytest.mark.parametrize("w", [5, 12, 20, 36])
def test_exact_on_short_tiles(w, prec, k):
    n, rng = 152 * 128 * 2 + 77, np.random.default_rng(w + k)
    first = np.arange(n) // 128 * 128 - w
    col = first[:, None] + np.argsort(rng.random((n, 128 + 2 * w)), axis=1)[:, :60]
    ok = ((col >= 0) & (col < n)).ravel()
    row, val = np.repeat(np.arange(n), 60)[ok], rng.choice([-1.0, 1.0], n * 60)[ok]
    check(sp.csr_matrix((val, (row, col.ravel()[ok])), shape=(n, n)), prec, k)


@pytest.mark.parametrize("k", [4, 8, 36, 240])
@pytest.mark.parametrize("band", [0, 3])
def test_exact_on_sparse_rows(band, k):
    n, rng = 5000, np.random.default_rng(band + k)
    off = np.arange(-band, band + 1)
    check(sp.diags([rng.choice([-1.0, 1.0], n - abs(o)) for o in off], off, format="csr"), "fp32", k)


def check(M, prec, k):
    n, rng = M.shape[0], np.random.default_rng(k)
    M.sort_indices()
    H = system.Csr(n, n, M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data)
    X = rng.integers(-3, 4, (n, k)).astype(float)
    op = api.Operator(api.ProjectHamiltonianSparse(H), k)
    try:
        ax = api.AX(1, k)
        ax.op = op
        Xm = api.Mat(op, k, X)
        # interval [-1, 1], lowest -2: one degree is -0.5 H X, of at most 15
        api.ChebyShevFilter(api.sched(prec)).computeFilteredSubspace(None, ax, Xm, n, 1, -1.0, 1.0, -2.0)
        op.sync()
        assert np.array_equal(Xm.get(), -0.5 * (M @ X))
    finally:
        op.close()
