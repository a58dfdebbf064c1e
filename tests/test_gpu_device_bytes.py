"""device_bytes counts what an operator really holds: its growth over calls that make workspaces (digit planes, the
Hamiltonian update's slabs, the Hartree and density products, the STHOSVD) is the device memory that is gone, up
to the allocation granularity of 2 MiB a buffer."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


def test_growth_is_the_memory_taken():
    import torch
    r, k = 20, 96
    s = system.build_system(system.small_spec(name="bytes", n_atoms=4, box=16.0, n_el=40, rank=r, n_states=k, degree=4,
                                              seed=3))
    lib, p = _lib.ttg(), lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), k)
    try:
        K = [np.ascontiguousarray(b.stiffness()) for b in s.basis]
        K += [np.ascontiguousarray(b.overlap()) for b in s.basis]
        assert lib.ttg_op_set_kinetic(op.h, *[_lib.ptr(m) for m in K]) == 0
        X = api.Mat(op, k, np.random.default_rng(0).standard_normal((s.N, k)))
        n = 200
        T = torch.rand(n ** 3, dtype=torch.float64, device="cuda")
        core = torch.empty(50 ** 3, dtype=torch.float64, device="cuda")
        U = [torch.empty(n * 50, dtype=torch.float64, device="cuda") for _ in range(3)]
        u = torch.from_numpy(np.ascontiguousarray(s.basis[0].nodal.T)).cuda()
        nodes = s.basis[0].nodal.shape[0]
        rho = torch.empty(nodes ** 3, dtype=torch.float64, device="cuda")
        P = [np.ones((12, r, r)) for _ in range(3)]
        i3 = lambda v: _lib.ptr(np.full(3, v, np.int32))  # noqa: E731
        lib.ttg_kernel_launches()
        op.sync()
        free, held = torch.cuda.mem_get_info()[0], op.info()["device_bytes"]
        api.MultTM().orth(X)
        api.rayleigh_ritz(op, X, rotate=True)
        assert lib.ttg_op_update_potential(op.h, i3(12), _lib.ptr(np.ones((12, 12, 12))),
                                           *[_lib.ptr(m) for m in P]) == 0
        assert lib.ttg_tucker_sthosvd(op.h, p(T), i3(n), 0.0, i3(50), _lib.ptr(np.zeros(3, np.int32)), p(core),
                                      *[p(m) for m in U]) == 0
        assert lib.ttg_density_device(op.h, X.h, _lib.ptr(np.ones(k)), i3(r), i3(nodes), p(u), p(u), p(u), p(rho),
                                      0) == 0
        op.sync()
        taken = free - torch.cuda.mem_get_info()[0]
        grown = op.info()["device_bytes"] - held
        # kernels loaded on first use take some memory as well
        assert grown > 3e8 and abs(taken - grown) < 0.1 * grown + 64 * 2 ** 21
    finally:
        op.close()
