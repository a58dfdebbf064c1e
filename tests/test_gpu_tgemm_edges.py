"""The tensor-core contraction at the edges of its tiles (128 x 64, warps of 16 columns, chunks of 16
values, groups up to 192): integer operands with every slice in use must come out exact, whatever the
shape; K beyond the operand and rows beyond the tile count as zero.

|a| < 2^24 on the slicing grid of its group: with integers below 2^16 two slices are used and a sum of k
products of a 16-bit and an 8-bit integer stays below 2^32, which the double-FP32 result holds."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib

pytestmark = pytest.mark.gpu


def tc_gemm(A, B, groups, pad=0):
    import torch
    (m, k), n = A.shape, B.shape[0]
    ld = (k + 3) // 4 * 4 + 4 * pad
    a = torch.full((m, ld), np.nan, dtype=torch.float32, device="cuda")
    b = torch.full((n, ld), np.nan, dtype=torch.float32, device="cuda")
    a[:, :k] = torch.from_numpy(A.astype(np.float32)).cuda()
    b[:, :k] = torch.from_numpy(B.astype(np.float32)).cuda()
    c = torch.full((m, n + 3), np.nan, dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert _lib.ttg().ttg_tc_gemm(m, n, k, p(a), ld, p(b), ld, groups, p(c), n + 3, None) == 0
    out = c.cpu().numpy()
    assert np.isnan(out[:, n:]).all()
    return out[:, :n]


@pytest.mark.parametrize("m,n", [(1, 1), (127, 15), (128, 64), (129, 65), (257, 127), (640, 193)])
@pytest.mark.parametrize("k,groups", [(1, 1), (15, 1), (16, 1), (17, 1), (40, 1), (192, 1), (100, 3),
                                      (1000, 7), (2240, 35)])
def test_exact_at_tile_edges(m, n, k, groups):
    rng = np.random.default_rng(m + 1000 * n + k)
    A = rng.integers(-65535, 65536, (m, k))
    B = rng.integers(-255, 256, (n, k))
    assert np.array_equal(tc_gemm(A, B, groups, pad=k % 3), (A @ B.T).astype(np.float64))


def test_rows_beyond_one_slab():
    """900,000 rows of 160 values: planes of 1.1 GB."""
    rng = np.random.default_rng(1)
    A = rng.integers(-255, 256, (900000, 160))
    B = rng.integers(-255, 256, (5, 160))
    assert np.array_equal(tc_gemm(A, B, 1), (A @ B.T).astype(np.float64))
