"""The FP64 tensor-core GEMM at the edges of its tiles (128 x 64, halves of 32 columns, chunks of 16 and
groups of 96 values of K), at odd widths and leading dimensions, and beyond its plane workspace, where
the operands are taken in slabs.

Bound (derived in csrc/ozgemm.cu): each value is rounded to 2^-41 of its row's 2^e <= 2 max|row| over 256
(2^-48 of the scale), digit products beyond level 5 are below 2^-47 of the two scales, so an entry is
within K 2^-45 max|x_m| max|y_n| of the exact product; the sums add 2^-46 of sum |x||y|."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


def unit_op(n, k):
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n))
    return api.Operator(api.ProjectHamiltonianSparse(H), k)


def bound(X, Y):
    K = X.shape[0]
    return (K * 2.0 ** -45 * np.outer(np.abs(X).max(0), np.abs(Y).max(0))
            + 2.0 ** -46 * (np.abs(X).T @ np.abs(Y)))


@pytest.mark.parametrize("n", [65, 1000, 1729])
@pytest.mark.parametrize("k", [1, 2, 16, 31, 33, 57, 64, 65, 127, 129, 200])
def test_gram_and_products_at_tile_edges(n, k):
    op = unit_op(n, max(k, 8))
    try:
        rng = np.random.default_rng(1000 * n + k)
        X = rng.standard_normal((n, k)) * np.geomspace(1.0, 1e-5, k)
        Y = rng.standard_normal((n, k))
        Xm, Ym = api.Mat(op, k, X), api.Mat(op, k, Y)
        L = X.astype(np.longdouble)
        S = api.MultTM().mult(Xm, Ym)
        assert np.all(np.abs(S - (L.T @ Y).astype(float)) <= bound(X, Y))
        S = api.MultTM().mult(Xm, Xm)
        assert np.all(np.abs(S - (L.T @ L).astype(float)) <= bound(X, X))
        Q = np.asfortranarray(rng.standard_normal((k, k)))
        assert _lib.ttg().ttg_rotate(op.h, Xm.h, ctypes.c_void_p(Q.ctypes.data)) == 0
        assert np.all(np.abs(Xm.get() - (L @ Q).astype(float)) <= bound(X.T, Q))
    finally:
        op.close()


@pytest.mark.parametrize("k", [33, 57, 130])
def test_cholesky_qr_of_odd_widths(k):
    """X L^-T with the triangular operand and its column scales: orthonormal to cond^2 2^-45."""
    op = unit_op(3001, k)
    try:
        X = np.random.default_rng(k).standard_normal((3001, k)) * np.geomspace(1e3, 1e-6, k)
        Xm = api.Mat(op, k, X)
        api.MultTM().orth(Xm)
        Q = Xm.get()
        assert np.abs(Q.T @ Q - np.eye(k)).max() < 3001 * 2.0 ** -45
    finally:
        op.close()


@pytest.mark.parametrize("n,k", [(400000, 300), (700001, 131)])
def test_operands_beyond_the_plane_workspace(n, k):
    import torch
    op = unit_op(n, k)
    try:
        g = torch.Generator(device="cuda").manual_seed(3)
        x = torch.randn(k, n, dtype=torch.float64, device="cuda", generator=g)
        X = api.Mat(op, k)
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        assert _lib.ttg().ttg_block_set_device(X.h, p(x), n) == 0
        ref = x @ x.T
        S = torch.from_numpy(api.MultTM().mult(X, X)).cuda()
        tol = (n * 2.0 ** -45 + 2.0 ** -40) * float(x.abs().max()) ** 2
        assert float((S - ref).abs().max()) <= tol
        Q = torch.linalg.qr(torch.randn(k, k, dtype=torch.float64, device="cuda", generator=g))[0]
        Qh = np.asfortranarray(Q.cpu().numpy())
        assert _lib.ttg().ttg_rotate(op.h, X.h, ctypes.c_void_p(Qh.ctypes.data)) == 0
        out = torch.empty_like(x)
        assert _lib.ttg().ttg_block_get_device(X.h, p(out), n) == 0
        op.sync()
        assert float((out - Q.T @ x).abs().max()) <= k * 2.0 ** -44 * float(x.abs().max())
    finally:
        op.close()
