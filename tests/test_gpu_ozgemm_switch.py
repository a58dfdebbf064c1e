"""TTG_DISABLE_OZGEMM keeps the whole Rayleigh-Ritz step off the FP64 tensor-core kernels, H X included: its Ritz
values are the oracle's and the operator never makes the digits of H (28 KB per 16 slots of its tiles)."""
import numpy as np
import pytest

import oracle
from ttdft_public_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [False, True])
def test_rayleigh_ritz_without_the_digits(small_system, monkeypatch, off):
    s = small_system
    if off:
        monkeypatch.setenv("TTG_DISABLE_OZGEMM", "1")
    X, _ = oracle.cholqr(np.random.default_rng(23).standard_normal((s.N, 24)))
    op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), 24)
    try:
        held = op.info()["device_bytes"]
        w = api.rayleigh_ritz(op, api.Mat(op, 24, X), rotate=False)
        wr, _, _ = oracle.rayleigh_ritz(s, X, rotate_x=False)
        assert np.abs(w - wr).max() < 1e-11 * np.abs(wr).max()
        info = op.info()
        assert (info["device_bytes"] - held < info["umma_slots"] // 16 * 28672) == off
    finally:
        op.close()
