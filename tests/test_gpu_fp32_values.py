"""The entries of H as an FP32 degree holds them, one by one (the block is a set of unit vectors, so that each
result is a single product), as built and after updates that shrink every row by up to 400: an entry far below its
row's largest one keeps its bits.

Bound: FP32 rounding and the two FP16 terms, below 2^-20 of the entry; 2^-29 of its row's largest value, half of
FP16's smallest step of 2^-24 over a row scaled to at least 2^4; halved by the recurrence as the results are."""
import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


def test_small_entries_keep_their_bits():
    r, k = 9, 48
    s = system.build_system(system.small_spec(name="vals", n_atoms=2, box=7.0, n_el=18, rank=r, n_states=k, degree=4,
                                              seed=6, with_nonlocal=False))
    op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), k)
    lib = _lib.ttg()
    row = np.repeat(np.arange(s.N), np.diff(s.H.row_ptr))
    col = s.H.col.astype(np.int64)
    i, j = [row % r, row // r % r, row // (r * r)], [col % r, col // r % r, col // (r * r)]
    at = np.linspace(0, s.N - 1, k).astype(int)
    X = np.zeros((s.N, k))
    X[at, np.arange(k)] = 1.0
    ax = api.AX(1, k)
    ax.op = op

    def check(A):
        Xm = api.Mat(op, k, X)
        # interval [-1, 1], lowest -2: one degree is -0.5 H X
        api.ChebyShevFilter(api.sched("fp32")).computeFilteredSubspace(None, ax, Xm, s.N, 1, -1.0, 1.0, -2.0)
        op.sync()
        ref = A[:, at].toarray()
        top = np.asarray(abs(A).max(axis=1).todense())
        small = (np.abs(ref) < 2.0 ** -10 * top) & (ref != 0)
        assert small.sum() > 1000
        assert np.all(np.abs(-2.0 * Xm.get() - ref) <= 2.0 ** -20 * np.abs(ref) + 2.0 ** -29 * top)

    try:
        A = s.H.to_scipy().tocsr()
        check(A)
        G, P = np.zeros((1, 1, 1)), [np.zeros((1, r, r)) for _ in range(3)]
        for f in (1.0, 1 / 40.0, 1 / 60.0, 1 / 360.0, 1 / 400.0, 10.0):
            K = [np.ascontiguousarray(f * b.stiffness()) for b in s.basis]
            K += [np.ascontiguousarray(b.overlap()) for b in s.basis]
            assert lib.ttg_op_set_kinetic(op.h, *[_lib.ptr(m) for m in K]) == 0
            assert lib.ttg_op_update_potential(op.h, _lib.ptr(np.ones(3, np.int32)), _lib.ptr(G),
                                               *[_lib.ptr(p) for p in P]) == 0
            D, M = [K[d][i[d], j[d]] for d in range(3)], [K[3 + d][i[d], j[d]] for d in range(3)]
            A.data = 0.5 * (D[0] * M[1] * M[2] + M[0] * D[1] * M[2] + M[0] * M[1] * D[2])
            check(A)
    finally:
        op.close()
