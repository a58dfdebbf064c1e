"""ttg_grid_integrate on grids of few or short lines: pieces of lines, remainders, a single point; against an exactly
rounded sum.  And its time: a grid of one line takes about as long as a cube of as many points.

Bound: a lane adds at most 2^13 terms of its piece, then 1024 x 8 partial sums in a tree and 32 steps: 2^-53 each
time, 2^-38 of the sum of magnitudes in all."""
import ctypes
import math
import time

import numpy as np
import pytest

from ttdft_public_gb300 import _lib

pytestmark = pytest.mark.gpu


def integrate(lib, f, g, dims, w):
    out = ctypes.c_double()
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.ttg_grid_integrate(p(f), p(g), _lib.ptr(np.array(dims, np.int32)), *[p(v) for v in w],
                                  ctypes.byref(out), None) == 0
    return out.value


@pytest.mark.parametrize("dims", [(100001, 1, 1), (262147, 2, 1), (1, 1, 100001), (1, 1, 1), (127, 3, 5), (128, 1, 9),
                                  (5000, 3, 2), (257, 63, 128), (3, 300, 7), (40, 33, 65)])
@pytest.mark.parametrize("two", [False, True])
def test_sum(dims, two):
    import torch
    rng, n = np.random.default_rng(sum(dims)), dims[0] * dims[1] * dims[2]
    f, g = rng.standard_normal(n), rng.standard_normal(n) if two else np.ones(n)
    w = [rng.uniform(0.5, 1.5, d) for d in dims]
    terms = f * g * (w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]).reshape(-1)
    dev = [torch.from_numpy(a).cuda() for a in (f, g, *w)]
    v = integrate(_lib.ttg(), dev[0], dev[1] if two else None, dims, dev[2:])
    assert abs(v - math.fsum(terms)) <= 2.0 ** -38 * np.abs(terms).sum()


def test_time_of_one_line():
    import torch
    lib, best = _lib.ttg(), {}
    f = torch.rand(1 << 24, dtype=torch.float64, device="cuda")
    for dims in ((256, 256, 256), (1 << 24, 1, 1), (1 << 20, 4, 4)):
        w = [torch.ones(d, dtype=torch.float64, device="cuda") for d in dims]
        times = []
        for _ in range(6):
            torch.cuda.synchronize()
            t = time.perf_counter()
            integrate(lib, f, f, dims, w)
            times.append(time.perf_counter() - t)
        best[dims] = min(times)
    assert max(best.values()) < 6 * best[(256, 256, 256)], best
