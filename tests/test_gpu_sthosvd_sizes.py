"""STHOSVD of grids large enough for the tensor-core Gram matrices and mode products (every mode, odd
dimensions), against NumPy's.  The field is of Tucker rank 40 plus 1e-7 of noise, cut at rank 40: the kept
eigenvalues are above 1e-6 of the largest and the first discarded one is 1e-14 of it, so a Gram error of
2^-45 of its trace turns the kept subspace by at most 1e-13 / 1e-6, and the field moves by that share of
the components of size 1e-3 it holds: 1e-10 of its norm."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(203, 151, 97), (97, 203, 151), (90, 111, 240)])
def test_large_grids_match_numpy(dims):
    import torch
    rng = np.random.default_rng(sum(dims))
    r = 40
    U = [np.linalg.qr(rng.standard_normal((d, r)))[0] for d in dims]
    G = rng.standard_normal((r, r, r)) * np.exp(-0.08 * np.add.outer(np.add.outer(
        np.arange(r), np.arange(r)), np.arange(r)))
    T = np.einsum("abc,xa,yb,zc->xyz", G, *U, optimize=True)
    T += 1e-7 * np.linalg.norm(T) / np.sqrt(T.size) * rng.standard_normal(dims)
    ref = T
    for d in range(3):
        M = np.moveaxis(ref, d, 0).reshape(dims[d], -1)
        V = np.linalg.eigh(M @ M.T)[1][:, -r:]
        ref = np.moveaxis(np.tensordot(V @ V.T, np.moveaxis(ref, d, 0), 1), 0, d)
    n = 64
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n))
    op = api.Operator(api.ProjectHamiltonianSparse(H), 8)
    try:
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        t = torch.from_numpy(np.asfortranarray(T).reshape(-1, order="F")).cuda()
        core = torch.zeros(r ** 3, dtype=torch.float64, device="cuda")
        f = [torch.zeros(d * r, dtype=torch.float64, device="cuda") for d in dims]
        nd, caps, ranks = np.array(dims, np.int32), np.array([r] * 3, np.int32), np.zeros(3, np.int32)
        lib = _lib.ttg()
        assert lib.ttg_tucker_sthosvd(op.h, p(t), _lib.ptr(nd), 0.0, _lib.ptr(caps), _lib.ptr(ranks),
                                      p(core), *[p(u) for u in f]) == 0
        assert list(ranks) == [r] * 3
        out = torch.empty_like(t)
        assert lib.ttg_tucker_reconstruct(p(core), _lib.ptr(ranks), *[p(u) for u in f], _lib.ptr(nd),
                                          p(out), None) == 0
        got = out.cpu().numpy().reshape(dims, order="F")
        assert np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)
        for u, d in zip(f, dims):
            Q = u.cpu().numpy().reshape(r, d)
            assert np.abs(Q @ Q.T - np.eye(r)).max() < 1e-12
    finally:
        op.close()
