"""The Hartree and density contractions where the workspace of their operands' slices does not fit: they take smaller
slabs of rows and give the same bits.  The limits lie above every other buffer of these calls (the largest is the
last product's FP32 operand, 4 bytes a value) and below its slices (6 bytes, in whole tiles)."""
import numpy as np
import pytest

from ttdft_public_gb300 import _lib, api, system

pytestmark = pytest.mark.gpu


def test_hartree(monkeypatch):
    alpha, omega, G, quad, U, grids = system.hartree_blob_case(rank=16, n_blobs=12, seed=5, n_el=24, box=16.0)
    ref, _ = api.hartree(alpha, omega, G, quad, U, grids)
    points = grids[0].size
    rows = points * points * len(alpha) * 16 * 4
    monkeypatch.setenv("TTG_ALLOC_LIMIT", str(int(1.2 * rows)))
    V, _ = api.hartree(alpha, omega, G, quad, U, grids)
    assert np.array_equal(V, ref) and np.abs(ref).max() > 0


def test_density(small_system, monkeypatch):
    s, k = small_system, 24
    X = np.random.default_rng(2).standard_normal((s.N, k))
    out = []
    for limited in (False, True):
        op = api.Operator(api.ProjectHamiltonianSparse.from_system(s), k)
        try:
            Xm = api.Mat(op, k, X)
            if limited:
                nodes = s.basis[0].nodal.shape[0]
                monkeypatch.setenv("TTG_ALLOC_LIMIT", str(int(1.2 * k * nodes * nodes * 12 * 4)))
            out.append(api.density(op, Xm, np.linspace(1.0, 0.1, k), s.basis))
        finally:
            op.close()
    assert np.array_equal(*out) and out[0].max() > 0


def test_no_room_at_all(monkeypatch):
    alpha, omega, G, quad, U, grids = system.hartree_blob_case(rank=16, n_blobs=12, seed=5, n_el=24, box=16.0)
    monkeypatch.setenv("TTG_ALLOC_LIMIT", "1000")
    with pytest.raises(_lib.TtgError, match="OOM"):
        api.hartree(alpha, omega, G, quad, U, grids)
