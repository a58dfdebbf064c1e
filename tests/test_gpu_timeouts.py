"""A bounded wait that runs out in an FP64 tensor-core kernel: every call that hands results to the host has to
return TTG_TIMEOUT itself, not the next one.  TTG_FAKE_TIMEOUT sets the error word after a launch as such a kernel
does; no wait runs out here.  The call after it, without the switch, is sound again."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api

pytestmark = pytest.mark.gpu
TIMEOUT = 6


@pytest.fixture(scope="module")
def op(small_system):
    s, o = small_system, api.Operator(api.ProjectHamiltonianSparse.from_system(small_system), 24)
    K = [np.ascontiguousarray(b.stiffness()) for b in s.basis]
    K += [np.ascontiguousarray(b.overlap()) for b in s.basis]
    assert _lib.ttg().ttg_op_set_kinetic(o.h, *[_lib.ptr(m) for m in K]) == 0
    yield o
    o.close()


def block(op, k=24):
    return api.Mat(op, k, np.random.default_rng(k).standard_normal((op.n, k)))


def gram(op, lib):
    X, Y = block(op), block(op)
    return lib.ttg_gram(op.h, X.h, Y.h, _lib.ptr(np.zeros((24, 24))))


def chol_qr(op, lib):
    X = block(op)
    return lib.ttg_chol_qr(op.h, X.h)


def ritz(op, lib):
    X = block(op)
    return lib.ttg_rayleigh_ritz(op.h, X.h, 0, _lib.ptr(np.zeros(24)), None)


def ritz_on_the_device(op, lib):
    X = block(op)
    return lib.ttg_rayleigh_ritz(op.h, X.h, 0, None, None)


def rotate(op, lib):
    X = block(op)
    return lib.ttg_rotate(op.h, X.h, _lib.ptr(np.eye(24)))


def syev(op, lib):
    A = np.random.default_rng(3).standard_normal((400, 400))       # its own products are on the tensor cores
    return lib.ttg_syev(op.h, 400, _lib.ptr(A + A.T), _lib.ptr(np.zeros(400)), _lib.ptr(np.zeros((400, 400))))


def update(op, lib):
    P = [np.ones((2, 12, 12)) for _ in range(3)]
    return lib.ttg_op_update_potential(op.h, _lib.ptr(np.full(3, 2, np.int32)), _lib.ptr(np.ones((2, 2, 2))),
                                       *[_lib.ptr(p) for p in P])


def tucker(op, lib, back=False):
    import torch
    n, r = 160, 40
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    T = torch.rand(n ** 3, dtype=torch.float64, device="cuda")
    core = torch.rand(r ** 3, dtype=torch.float64, device="cuda")
    U = [torch.rand(n * r, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    dims, ranks, out = np.full(3, n, np.int32), np.full(3, r, np.int32), np.zeros(3, np.int32)
    if back:
        return lib.ttg_tucker_reconstruct(p(core), _lib.ptr(ranks), *[p(u) for u in U], _lib.ptr(dims), p(T), None)
    return lib.ttg_tucker_sthosvd(op.h, p(T), _lib.ptr(dims), 0.0, _lib.ptr(ranks), _lib.ptr(out), p(core),
                                  *[p(u) for u in U])


def reconstruct(op, lib):
    return tucker(op, lib, back=True)


@pytest.mark.parametrize("call", [gram, chol_qr, ritz, ritz_on_the_device, rotate, syev, update, tucker, reconstruct])
def test_the_call_itself_reports_it(op, call, monkeypatch):
    lib = _lib.ttg()
    monkeypatch.setenv("TTG_UPDATE_SLAB_VALUES", "100000000")        # the tensor cores for a small update
    assert call(op, lib) == 0
    monkeypatch.setenv("TTG_FAKE_TIMEOUT", "1")
    assert call(op, lib) == TIMEOUT
    monkeypatch.delenv("TTG_FAKE_TIMEOUT")
    assert call(op, lib) == 0
    op.sync()
