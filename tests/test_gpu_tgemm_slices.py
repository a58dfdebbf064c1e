"""The tensor-core contraction with every slice of both operands in use: integers of up to 24 bits are cut into three
slices of 8 bits, so A of 24 bits and B of 16 bits (and the other way round) have nonzero products in all four
levels but a2 b2, the one that is left out.  The levels' sums are exact and the double-FP32 result holds 48 bits:
sums below 2^47 come out exact.

Edges: a tile's rows and columns, a chunk of 16 values, groups of several chunks and several groups."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib

pytestmark = pytest.mark.gpu


def product(A, B, groups):
    import torch
    (m, k), n = A.shape, B.shape[0]
    ld = (k + 3) // 4 * 4
    a, b = (torch.zeros(x.shape[0], ld, dtype=torch.float32, device="cuda") for x in (A, B))
    a[:, :k] = torch.from_numpy(A.astype(np.float32)).cuda()
    b[:, :k] = torch.from_numpy(B.astype(np.float32)).cuda()
    c = torch.full((m, n), np.nan, dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert _lib.ttg().ttg_tc_gemm(m, n, k, p(a), ld, p(b), ld, groups, p(c), n, None) == 0
    return c.cpu().numpy()


@pytest.mark.parametrize("bits", [(24, 16), (16, 24)])
@pytest.mark.parametrize("m, n", [(1, 1), (128, 64), (131, 67), (300, 129)])
@pytest.mark.parametrize("k, groups", [(1, 1), (16, 1), (17, 1), (50, 1), (192, 1), (70, 2), (640, 5)])
def test_exact_in_all_levels(bits, m, n, k, groups):
    rng = np.random.default_rng(m + 7 * n + 31 * k)
    # sums of k products below 2^47: the operands' sizes shrink with k, their low bits stay
    wide = 47 - int(np.ceil(np.log2(k + 1)))
    ba, bb = bits
    cut = max(0, ba + bb - wide)
    A = rng.integers(-(1 << ba) + 1, 1 << ba, (m, k))
    B = rng.integers(-(1 << bb) + 1, 1 << bb, (n, k))
    if ba > bb:
        B >>= cut
    else:
        A >>= cut
    A.flat[0], B.flat[0] = (1 << ba) - 1 >> (cut if ba < bb else 0), (1 << bb) - 1 >> (cut if bb < ba else 0)
    assert np.array_equal(product(A, B, groups), (A @ B.T).astype(np.float64))
