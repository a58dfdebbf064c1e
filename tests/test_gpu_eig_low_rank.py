"""The symmetric eigensolver on matrices of low rank, whose Householder columns fall by 1e-16 at a time after the
last of the rank, and at scales whose squares leave the FP64 range; and a separable field's Tucker compression, whose
mode Grams are such matrices.

Bounds as for any backward stable method: eigenvalues and residuals within 8 n 2^-53 of the largest eigenvalue,
eigenvectors orthonormal to 64 n 2^-53; the compression and its factors, whose products are double-FP32 (2^-44), to 2^-40."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(scope="module")
def op():
    n = 64
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n))
    o = api.Operator(api.ProjectHamiltonianSparse(H), 512)
    yield o
    o.close()


def check(op, A):
    n = A.shape[0]
    w, V = np.zeros(n), np.zeros((n, n), order="F")
    api.EigenSolver(op).computeEigenPairsSeq(A, n, n, w, V)
    scale = 2.0 ** np.floor(np.log2(np.abs(A).max()))
    A, w = A / scale, w / scale
    ref = np.linalg.eigvalsh(A)
    top = np.abs(ref).max()
    assert np.abs(w - ref).max() <= 8 * n * U * top
    assert np.abs(A @ V - V * w).max() <= 8 * n * U * top
    assert np.abs(V.T @ V - np.eye(n)).max() <= 64 * n * U


@pytest.mark.parametrize("n", [3, 60, 100, 127, 128, 200, 255, 360, 500])
def test_ones(op, n):
    check(op, np.ones((n, n)))


@pytest.mark.parametrize("rank", [1, 2, 3])
@pytest.mark.parametrize("n", [50, 127, 200, 361])
def test_outer_products_of_smooth_vectors(op, n, rank):
    x = np.linspace(0.0, 1.0, n)
    V = np.stack([np.exp(-((x - 0.2 - 0.3 * i) / 0.2) ** 2) for i in range(rank)])
    check(op, V.T @ V)


@pytest.mark.parametrize("scale", [1e-160, 1e-140, 1e120, 1e150])
@pytest.mark.parametrize("n", [40, 130])
def test_far_scales(op, n, scale):
    A = np.random.default_rng(n).standard_normal((n, n))
    check(op, scale * (A + A.T))
    check(op, scale * np.ones((n, n)))


@pytest.mark.parametrize("dims", [(100, 127, 64), (150, 150, 150)])
def test_separable_field(op, dims):
    import torch
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    lib, f = _lib.ttg(), [np.exp(-np.linspace(-2, 2, d) ** 2) for d in dims]
    T = f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]
    field, out = torch.from_numpy(T.reshape(-1)).cuda(), torch.empty(T.size, dtype=torch.float64, device="cuda")
    core = torch.zeros(8 ** 3, dtype=torch.float64, device="cuda")
    F = [torch.zeros(d * 8, dtype=torch.float64, device="cuda") for d in dims]
    d3, caps, ranks = np.array(dims, np.int32), np.full(3, 8, np.int32), np.zeros(3, np.int32)
    assert lib.ttg_tucker_sthosvd(op.h, p(field), _lib.ptr(d3), 0.0, _lib.ptr(caps), _lib.ptr(ranks), p(core),
                                  *[p(u) for u in F]) == 0
    assert lib.ttg_tucker_reconstruct(p(core), _lib.ptr(ranks), *[p(u) for u in F], _lib.ptr(d3), p(out), None) == 0
    assert np.abs(out.cpu().numpy() - T.reshape(-1)).max() <= 2.0 ** -40 * T.max()
    for d, u in zip(dims, F):
        V = u.cpu().numpy().reshape(8, d)
        assert np.abs(V @ V.T - np.eye(8)).max() <= 2.0 ** -40
