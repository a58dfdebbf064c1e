"""ttg_grid_lincomb with a point a thread (up to 1.25 or 5 million points) and with four, in one pass or several,
up to the most fields: each point is a chain of fused steps over the fields, 2^-48 of the sum of magnitudes for 24
and the reference's own."""
import ctypes

import numpy as np
import pytest

from ttdft_public_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 100003, 1250000, 1250001, 2490369, 5000000, 5000001])
@pytest.mark.parametrize("fields", [1, 2, 7, 8, 9, 24])
@pytest.mark.parametrize("take_abs", [0, 1])
def test_sums(n, fields, take_abs):
    import torch
    rng = np.random.default_rng(n + fields)
    f, c = rng.standard_normal((fields, n)), rng.standard_normal(fields)
    d, out = torch.from_numpy(f).cuda(), torch.full((n + 1,), np.nan, dtype=torch.float64, device="cuda")
    ptrs = (ctypes.c_void_p * fields)(*[d[i].data_ptr() for i in range(fields)])
    assert _lib.ttg().ttg_grid_lincomb(fields, ptrs, _lib.ptr(c), n, ctypes.c_void_p(out.data_ptr()), take_abs,
                                       None) == 0
    got, ref = out.cpu().numpy(), c @ f
    assert np.isnan(got[n])
    assert np.all(np.abs(got[:n] - (np.abs(ref) if take_abs else ref)) <= 2.0 ** -48 * (np.abs(c) @ np.abs(f)))
