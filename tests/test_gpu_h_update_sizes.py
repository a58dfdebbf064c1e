"""New Hamiltonian values for random potentials in Tucker form, on ranks that are no multiples of the
update's tiles (8 rows, 128 pairs, 64 columns), twice on one operator with growing potential ranks, against
the sum over the pattern in NumPy.

Bound: T1, T2 and the sum over the z rank are three products whose operands carry 2^-48 of their rows'
largest values (at most 2^-43 of the product of the sums of magnitudes for ranks below 64), the kinetic
part a few FP64 roundings."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [5, 9, 11])
def test_values_on_the_pattern(rank):
    spec = system.small_spec(name="upd", n_atoms=2, box=8.0 + 0.3 * rank, n_el=2 * rank, rank=rank, n_states=8,
                             degree=4, seed=rank)
    s = system.build_system(spec)
    op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), 16)
    lib, rng, r = _lib.ttg(), np.random.default_rng(rank), rank
    try:
        K = [np.ascontiguousarray(b.stiffness()) for b in s.basis]
        K += [np.ascontiguousarray(b.overlap()) for b in s.basis]
        assert lib.ttg_op_set_kinetic(op.h, *[_lib.ptr(k) for k in K]) == 0
        row = np.repeat(np.arange(s.N), np.diff(s.H.row_ptr))
        col = s.H.col.astype(np.int64)
        i = [row % r, row // r % r, row // (r * r)]
        j = [col % r, col // r % r, col // (r * r)]
        D, M = [K[d][i[d], j[d]] for d in range(3)], [K[3 + d][i[d], j[d]] for d in range(3)]
        kin = 0.5 * (D[0] * M[1] * M[2] + M[0] * D[1] * M[2] + M[0] * M[1] * D[2])
        kmag = 0.5 * (abs(D[0] * M[1] * M[2]) + abs(M[0] * D[1] * M[2]) + abs(M[0] * M[1] * D[2]))
        for ranks in ((3, 7, 4), (8, 6, 17)):
            G = rng.standard_normal(ranks[::-1])                    # z, y, x ranks
            P = [np.ascontiguousarray(rng.standard_normal((m, r, r))) for m in ranks]
            assert lib.ttg_op_update_potential(op.h, _lib.ptr(np.array(ranks, np.int32)), _lib.ptr(G),
                                               *[_lib.ptr(p) for p in P]) == 0
            Q = [P[d][:, i[d], j[d]] for d in range(3)]
            pot = np.einsum("cba,an,bn,cn->n", G, *Q, optimize=True)
            mag = np.einsum("cba,an,bn,cn->n", abs(G), *[abs(q) for q in Q], optimize=True)
            A = s.H.to_scipy()
            A.data = kin + pot
            B = A.copy()
            B.data = kmag + mag.max() + 0 * mag                     # row scales: the largest magnitudes
            X = rng.standard_normal((s.N, 4))
            ax = api.AX(1, 4)
            ax.op = op
            Xm, Ym = api.Mat(op, 4, X), api.Mat(op, 4)
            ax.perform_ax(Xm, Ym)
            C = s.C.to_scipy()
            ref = A @ X + C.T @ (s.D[:, None] * (C @ X))
            nl = abs(C).T @ (abs(s.D)[:, None] * (abs(C) @ np.abs(X)))
            assert np.all(np.abs(Ym.get() - ref) <= 2.0 ** -43 * (B @ np.abs(X) + nl))
    finally:
        op.close()
