"""Hamiltonian updates in several slabs, on the per-entry sum, and where workspaces do not fit: the values are the
same in all of them, an update never ends half way, and one without room does not keep the next from the tensor cores.

Bound: that of test_gpu_h_update_sizes.py (the per-entry sum is nearer)."""
import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


class Problem:
    def __init__(self, rank=11):
        self.s = s = system.build_system(system.small_spec(name="upl", n_atoms=2, box=11.3, n_el=2 * rank, rank=rank,
                                                           n_states=8, degree=4, seed=rank))
        self.r = r = rank
        self.op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), 16)
        K = [np.ascontiguousarray(b.stiffness()) for b in s.basis]
        K += [np.ascontiguousarray(b.overlap()) for b in s.basis]
        assert _lib.ttg().ttg_op_set_kinetic(self.op.h, *[_lib.ptr(k) for k in K]) == 0
        row = np.repeat(np.arange(s.N), np.diff(s.H.row_ptr))
        col = s.H.col.astype(np.int64)
        self.i = i = [row % r, row // r % r, row // (r * r)]
        self.j = j = [col % r, col // r % r, col // (r * r)]
        D, M = [K[d][i[d], j[d]] for d in range(3)], [K[3 + d][i[d], j[d]] for d in range(3)]
        self.X = np.random.default_rng(1).standard_normal((s.N, 4))
        self.Xm, self.Ym = api.Mat(self.op, 4, self.X), api.Mat(self.op, 4)
        self.kin = 0.5 * (D[0] * M[1] * M[2] + M[0] * D[1] * M[2] + M[0] * M[1] * D[2])

    def update(self, ranks, seed):
        """A call with new inputs; its status and the kernels it launched."""
        rng, r, lib = np.random.default_rng(seed), self.r, _lib.ttg()
        self.G = rng.standard_normal(ranks[::-1])
        self.P = [np.ascontiguousarray(rng.standard_normal((m, r, r))) for m in ranks]
        before = lib.ttg_kernel_launches()
        rc = lib.ttg_op_update_potential(self.op.h, _lib.ptr(np.array(ranks, np.int32)), _lib.ptr(self.G),
                                         *[_lib.ptr(p) for p in self.P])
        return rc, lib.ttg_kernel_launches() - before

    def entries(self, G, P):
        """sum_abc G_abc PX_a PY_b PZ_c at the pattern's entries."""
        T = G
        for p in P:                                                  # x, y, z: the last axis goes first
            T = np.tensordot(p.reshape(len(p), -1), T, ([0], [2]))
        q = [self.i[d] * self.r + self.j[d] for d in range(3)]
        return T[q[2], q[1], q[0]]

    def check(self):
        s, X = self.s, self.X
        A, B = s.H.to_scipy(), s.H.to_scipy()
        A.data = self.kin + self.entries(self.G, self.P)
        B.data = np.full(A.nnz, np.abs(self.kin).max() + self.entries(abs(self.G), [abs(p) for p in self.P]).max())
        ax = api.AX(1, 4)
        ax.op = self.op
        ax.perform_ax(self.Xm, self.Ym)
        C = s.C.to_scipy()
        ref = A @ X + C.T @ (s.D[:, None] * (C @ X))
        nl = abs(C).T @ (abs(s.D)[:, None] * (abs(C) @ np.abs(X)))
        assert np.all(np.abs(self.Ym.get() - ref) <= 2.0 ** -43 * (B @ np.abs(X) + nl))


@pytest.fixture(params=[11])
def problem(request):
    p = Problem(request.param)
    yield p
    p.op.close()


@pytest.mark.parametrize("problem", [5, 9, 11], indirect=True)
def test_values_in_slabs_and_by_entry(problem, monkeypatch):
    assert problem.update((2, 3, 4), 8)[0] == 0                      # by entry: a small operator
    problem.check()
    for values in (200000, 100000000):                               # one y a slab (11 functions), one slab
        monkeypatch.setenv("TTG_UPDATE_SLAB_VALUES", str(values))
        for seed, ranks in enumerate(((8, 6, 17), (3, 7, 40))):
            rc, launches = problem.update(ranks, seed)
            assert rc == 0 and launches >= 12                        # scales, digits, product of three sums
            problem.check()
    monkeypatch.setenv("TTG_DISABLE_OZGEMM", "1")
    assert problem.update((8, 6, 17), 9)[0] == 0
    problem.check()


def test_every_limit_of_the_workspaces(problem, monkeypatch):
    """The first slab (y = 0) needs smaller planes than those in the middle: 1,217 and 1,327 pairs."""
    ranks = (8, 6, 17)
    monkeypatch.setenv("TTG_UPDATE_SLAB_VALUES", "200000")
    monkeypatch.setenv("TTG_DISABLE_OZGEMM", "1")
    assert problem.update(ranks, 0)[0] == 0                          # the intermediates of this rank
    monkeypatch.delenv("TTG_DISABLE_OZGEMM")
    assert problem.update((3, 7, 4), 1)[0] == 0                      # the plan and the slab's values
    for n, limit in enumerate(range(400000, 1200000, 20000)):
        monkeypatch.setenv("TTG_ALLOC_LIMIT", str(limit))
        assert problem.update(ranks, n)[0] == 0, limit
        problem.check()


def test_no_room_once_is_not_for_good(problem, monkeypatch):
    ranks = (8, 6, 17)
    monkeypatch.setenv("TTG_DISABLE_OZGEMM", "1")
    by_entry = problem.update(ranks, 0)
    monkeypatch.delenv("TTG_DISABLE_OZGEMM")
    monkeypatch.setenv("TTG_UPDATE_SLAB_VALUES", "100000000")        # the tensor cores for a small operator
    monkeypatch.setenv("TTG_ALLOC_LIMIT", "1000")
    assert problem.update(ranks, 1) == by_entry                      # nothing fits: the same kernels
    problem.check()
    monkeypatch.delenv("TTG_ALLOC_LIMIT")
    rc, launches = problem.update(ranks, 2)
    assert rc == 0 and launches >= by_entry[1] + 5                   # three products with scales and digits
    problem.check()
