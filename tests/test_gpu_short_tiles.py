"""Filter degrees on tiles of few chunks: the last stage of a tile then has slots without one, for the same gathering
warps tile after tile, and the warps are on other tiles than the MMAs.  A band of +-w has 128 + 2 w columns a tile:
9, 10, 11 and 13 chunks of 16.

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
    off = np.array([-w, -w // 2, 0, 1, w])
    M = sp.diags([rng.integers(-2, 3, n - abs(o)).astype(float) for o in off], off, format="csr")
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
