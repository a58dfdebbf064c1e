"""The FP64 tensor-core GEMM at the edges of its exact groups (128 values of K, chunks of 16) and of its digits: Gram
matrices of whole numbers below 2^17 (three digits), whose sums stay below 2^45, must come out exact."""
import numpy as np
import pytest

from ttdft_public_gb300 import api, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 128, 129, 255, 257, 383, 385, 1025])
@pytest.mark.parametrize("k", [3, 33, 64, 129])
def test_exact_whole_numbers(n, k):
    rng = np.random.default_rng(n + 1000 * k)
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n))
    op = api.Operator(api.ProjectHamiltonianSparse(H), k)
    try:
        X, Y = (rng.integers(-(1 << 17) + 1, 1 << 17, (n, k)) for _ in range(2))
        S = api.MultTM().mult(api.Mat(op, k, X.astype(float)), api.Mat(op, k, Y.astype(float)))
        assert np.array_equal(S, (X.T @ Y).astype(float))
    finally:
        op.close()


@pytest.mark.parametrize("k", [334, 701, 1199, 1200])
def test_cholesky_qr_of_wide_blocks(k):
    """Odd widths update by the CUDA-core kernel, even ones on the tensor cores: orthonormal to 3001 2^-45."""
    op = api.Operator(api.ProjectHamiltonianSparse(system.Csr(3001, 3001, np.arange(3002, dtype=np.int64),
                                                              np.arange(3001, dtype=np.int32), np.ones(3001))), k)
    try:
        X = api.Mat(op, k, np.random.default_rng(k).standard_normal((3001, k)) * np.geomspace(1e3, 1e-3, k))
        api.MultTM().orth(X)
        Q = X.get()
        assert np.abs(Q.T @ Q - np.eye(k)).max() < 3001 * 2.0 ** -45
    finally:
        op.close()
