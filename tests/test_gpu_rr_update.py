"""A Rayleigh-Ritz step, new Hamiltonian values, a Rayleigh-Ritz step again, as in every iteration of an SCF: the
second step has to see the new values in every format that the product keeps.  Widths that end in a column block of
one group of 32 states after full ones (97, 160), on as few as one tile a CTA and on several.

Bound: new values are within 2^-43 of the sums of magnitudes of their three products
(test_gpu_h_update_sizes.py), H X within 2^-45 of the largest values of its rows and columns, summed over the
row's entries (test_gpu_rr_products.py); the eigensolver's error is far below 2^-40 of the matrix' norm."""
import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank, k", [(9, 33), (20, 97), (20, 160)])
def test_ritz_values_follow_the_update(rank, k):
    spec = system.small_spec(name="rru", n_atoms=4, box=0.8 * rank, n_el=2 * rank, rank=rank, n_states=k, degree=4,
                             seed=rank)
    s = system.build_system(spec)
    op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), k)
    lib, rng, r = _lib.ttg(), np.random.default_rng(rank + k), rank
    try:
        K = [np.ascontiguousarray(b.stiffness()) for b in s.basis]
        K += [np.ascontiguousarray(b.overlap()) for b in s.basis]
        assert lib.ttg_op_set_kinetic(op.h, *[_lib.ptr(m) for m in K]) == 0
        row = np.repeat(np.arange(s.N), np.diff(s.H.row_ptr))
        col = s.H.col.astype(np.int64)
        i = [row % r, row // r % r, row // (r * r)]
        j = [col % r, col // r % r, col // (r * r)]
        D, M = [K[d][i[d], j[d]] for d in range(3)], [K[3 + d][i[d], j[d]] for d in range(3)]
        kin = 0.5 * (D[0] * M[1] * M[2] + M[0] * D[1] * M[2] + M[0] * M[1] * D[2])
        X, _ = np.linalg.qr(rng.standard_normal((s.N, k)))
        C = s.C.to_scipy()
        W = s.D[:, None] * (C @ X)
        cols = np.maximum(np.abs(X).max(axis=0), np.abs(W).max(axis=0))
        count = np.diff(s.H.row_ptr) + s.C.n_rows

        def ritz(A, tol):
            w = api.rayleigh_ritz(op, api.Mat(op, k, X), rotate=False)
            P = X.T @ (A @ X + C.T @ W)
            rows = np.maximum(np.asarray(abs(A).max(axis=1).todense()).ravel(),
                              np.asarray(abs(C).max(axis=0).todense()).ravel())
            E = 2.0 ** -45 * (np.abs(X).T @ (rows * count))[:, None] * cols[None, :]
            E += np.abs(X).T @ (tol @ np.abs(X))
            assert np.abs(w - np.linalg.eigvalsh(0.5 * (P + P.T))).max() <= \
                np.linalg.norm(E) + 2.0 ** -40 * np.linalg.norm(P)

        A = s.H.to_scipy()
        ritz(A, 0 * abs(A))
        for ranks in ((3, 7, 4), (5, 2, 6)):
            G = rng.standard_normal(ranks[::-1])                    # z, y, x ranks
            P = [np.ascontiguousarray(rng.standard_normal((m, r, r))) for m in ranks]
            P = [0.5 * (p + p.transpose(0, 2, 1)) for p in P]       # a symmetric operator
            assert lib.ttg_op_update_potential(op.h, _lib.ptr(np.array(ranks, np.int32)), _lib.ptr(G),
                                               *[_lib.ptr(np.ascontiguousarray(p)) for p in P]) == 0
            Q = [P[d][:, i[d], j[d]] for d in range(3)]
            A = s.H.to_scipy()
            A.data = kin + np.einsum("cba,an,bn,cn->n", G, *Q, optimize=True)
            tol = A.copy()
            mag = np.einsum("cba,an,bn,cn->n", abs(G), *[abs(q) for q in Q], optimize=True)
            tol.data = np.full(col.size, 2.0 ** -43 * (np.abs(kin).max() + mag.max()))
            ritz(A, tol)
    finally:
        op.close()
