"""FP32 filter degrees at the edges of the tcgen05 kernel: widths that are no multiple of 16 or that take
several column blocks, tiles shared by a cluster, columns and rows of very different sizes, zero columns,
and Hamiltonian values that leave the range of a row's scale.

Bound of one product, elementwise: an accumulation step of the tensor core is off by at most 2^-22 of the sum
of magnitudes so far, with three steps for each of a tile's 16-slot chunks (at most 1400 columns here); what the FP16 terms leave out
(3 x 2^-22) and the recurrence in FP32 fit into the 64 more that are granted; a value's terms also stop at
2^-23 of the largest one of its row.  Errors pass through the recurrence with |H|."""
import numpy as np
import pytest
import scipy.sparse as sp

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


def run(op, X, m, prec="fp32"):
    ax = api.AX(1, X.shape[1])
    ax.op = op
    Xm = api.Mat(op, X.shape[1], X)
    api.ChebyShevFilter(api.sched(prec)).computeFilteredSubspace(None, ax, Xm, X.shape[0], m, -1.0, 1.0, -2.0)
    op.sync()
    return Xm.get()


def check(op, A, C, D, X, m):
    """The recurrence for [-1, 1] and -2 in FP64, and the bound beside it."""
    n = A.shape[0]
    S, B = C.to_scipy(), abs(A)
    T = abs(S)
    floor = np.asarray(abs(A).max(axis=1).todense())
    pattern = (A != 0).astype(float)
    unit = (3.0 * (min(n, 1400) // 16 + 2) + 64.0) * 2.0 ** -22

    def h(Y):
        return A @ Y + S.T @ (D[:, None] * (S @ Y))

    def mag(Y):
        return B @ Y + T.T @ (np.abs(D)[:, None] * (T @ Y))

    def step(al, Y, E):
        a = abs(al)
        return al * h(Y), a * (mag(E) + unit * (mag(np.abs(Y)) + floor * (pattern @ np.abs(Y)) / 64.0))

    sigma, gamma = -0.5, -4.0
    x, ex = X, 2.0 ** -24 * np.abs(X)
    y, ey = step(sigma, x, ex)
    for _ in range(2, m + 1):
        s2 = 1.0 / (gamma - sigma)
        z, ez = step(2.0 * s2, y, ey)
        d = sigma * s2
        x, ex, y, ey = y, ey, z - d * x, ez + abs(d) * ex + 2.0 ** -22 * np.abs(d * x)
        sigma = s2
    assert np.all(np.abs(run(op, X, m) - y) <= ey)


def problem(n, seed, wide):
    rng = np.random.default_rng(seed)
    M = sp.random(n, n, density=0.15, random_state=rng, format="csr")
    M.data = rng.standard_normal(M.nnz)
    if wide:
        M = sp.diags(10.0 ** rng.uniform(-6, 6, n)) @ M
    M = M.tocsr()
    M.sort_indices()
    C = sp.random(5, n, density=0.3, random_state=rng, format="csr")
    C.sort_indices()
    H = system.Csr(n, n, M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data)
    Cs = system.Csr(5, n, C.indptr.astype(np.int64), C.indices.astype(np.int32), C.data)
    return M, H, Cs, 10.0 ** rng.uniform(-3, 3, 5)


@pytest.mark.parametrize("n", [90, 700, 1500])
@pytest.mark.parametrize("k", [4, 12, 24, 60, 240, 260, 528])
def test_widths_and_shared_tiles(n, k):
    M, H, C, D = problem(n, n + k, wide=False)
    X = np.random.default_rng(k).standard_normal((n, k))
    X[:, k // 2] = 0.0
    op = api.Operator(api.ProjectHamiltonianSparse(H, C, D), k)
    try:
        check(op, M, C, D, X, 3)
    finally:
        op.close()


def banded(n, seed):
    """Thirty entries a row within 300 columns: about 23 stages a tile, many of them odd."""
    rng = np.random.default_rng(seed)
    col = np.clip(np.arange(n)[:, None] + rng.integers(-300, 300, (n, 30)), 0, n - 1)
    M = sp.csr_matrix((rng.standard_normal(n * 30), (np.repeat(np.arange(n), 30), col.ravel())), shape=(n, n))
    M.sum_duplicates()
    C = sp.random(3, n, density=0.01, random_state=rng, format="csr")
    C.sort_indices()
    H = system.Csr(n, n, M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data)
    return M, H, system.Csr(3, n, C.indptr.astype(np.int64), C.indices.astype(np.int32), C.data), np.ones(3)


@pytest.mark.parametrize("n, k", [(10000, 300), (20100, 36), (20100, 520), (42000, 16)])
def test_several_tiles_and_blocks_a_cta(n, k):
    M, H, C, D = banded(n, n + k)
    X = np.random.default_rng(k).standard_normal((n, k))
    op = api.Operator(api.ProjectHamiltonianSparse(H, C, D), k)
    try:
        check(op, M, C, D, X, 3)
    finally:
        op.close()


@pytest.mark.parametrize("n, k", [(10000, 288), (42000, 16)])
def test_several_tiles_a_cta_in_bf16(n, k):
    """H, the block and the result are rounded to 8 bits: 3 x 2^-9 of the magnitudes, FP32 sums below that."""
    M, H, C, D = banded(n, n + k)
    X = np.random.default_rng(k).standard_normal((n, k))
    op = api.Operator(api.ProjectHamiltonianSparse(H, C, D), k)
    try:
        S = C.to_scipy()
        mag = abs(M) @ np.abs(X) + abs(S).T @ (abs(S) @ np.abs(X))
        ref = -0.5 * (M @ X + S.T @ (S @ X))
        assert np.all(np.abs(run(op, X, 1, "bf16") - ref) <= 0.5 * 5.0 * 2.0 ** -9 * mag)
    finally:
        op.close()


def test_rows_and_columns_of_many_sizes():
    M, H, C, D = problem(600, 9, wide=True)
    rng = np.random.default_rng(1)
    X = rng.standard_normal((600, 40)) * 10.0 ** rng.uniform(-12, 12, 40)
    op = api.Operator(api.ProjectHamiltonianSparse(H, C, D), 40)
    try:
        check(op, M, C, D, X, 1)
    finally:
        op.close()


def test_new_values_out_of_the_rows_range():
    r = 6
    s = system.build_system(system.small_spec(name="scale", n_atoms=2, box=9.0, n_el=16, rank=r, n_states=8,
                                              degree=4, seed=4))
    op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), 16)
    lib = _lib.ttg()
    row = np.repeat(np.arange(s.N), np.diff(s.H.row_ptr))
    col = s.H.col.astype(np.int64)
    i, j = [row % r, row // r % r, row // (r * r)], [col % r, col // r % r, col // (r * r)]
    X = np.random.default_rng(2).standard_normal((s.N, 16))
    G, P = np.zeros((1, 1, 1)), [np.zeros((1, r, r)) for _ in range(3)]
    try:
        for f in (1.0, 1e9, 1e-9, 1.0):
            K = [np.ascontiguousarray(f * b.stiffness()) for b in s.basis]
            K += [np.ascontiguousarray(b.overlap()) for b in s.basis]
            assert lib.ttg_op_set_kinetic(op.h, *[_lib.ptr(k) for k in K]) == 0
            assert lib.ttg_op_update_potential(op.h, _lib.ptr(np.ones(3, np.int32)), _lib.ptr(G),
                                               *[_lib.ptr(p) for p in P]) == 0
            D, M = [K[d][i[d], j[d]] for d in range(3)], [K[3 + d][i[d], j[d]] for d in range(3)]
            A = s.H.to_scipy().tocsr()
            A.data = 0.5 * (D[0] * M[1] * M[2] + M[0] * D[1] * M[2] + M[0] * M[1] * D[2])
            check(op, A, s.C, s.D, X, 1)
    finally:
        op.close()
