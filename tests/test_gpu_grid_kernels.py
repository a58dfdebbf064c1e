"""Grid kernels at the edges of their ranges: the LDA potential and energy over densities from zero to
infinity, weighted integrals of short and ragged lines, linear combinations of odd lengths in place.

Bounds.  LDA: rho^(1/3), rs and its roots are within 16 units of 2^-53 of the exact ones, the logarithm
then within 16 units absolute, and every term's coefficient is at most 1.2: 64 units of
|exchange| + |correlation| + 0.1.  Sums: a chain of m additions is within m 2^-53 of the sum of |terms|."""
import ctypes

import numpy as np
import pytest

from oracle import scf as oscf
from ttdft_public_gb300 import _lib

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def p(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def lda(rho, v0=None):
    import torch
    r, e = dev(rho), torch.zeros(rho.size, dtype=torch.float64, device="cuda")
    v = torch.zeros_like(e) if v0 is None else dev(v0)
    both_v, both_e = torch.zeros_like(e), torch.zeros_like(e)
    lib = _lib.ttg()
    assert lib.ttg_grid_lda(p(r), rho.size, p(v), None, 0 if v0 is None else 1, None) == 0
    assert lib.ttg_grid_lda(p(r), rho.size, None, p(e), 0, None) == 0
    assert lib.ttg_grid_lda(p(r), rho.size, p(both_v), p(both_e), 0, None) == 0
    torch.cuda.synchronize()
    if v0 is None:
        assert torch.equal(v.nan_to_num(), both_v.nan_to_num())
    assert torch.equal(e.nan_to_num(), both_e.nan_to_num())
    return v.cpu().numpy(), e.cpu().numpy()


def test_lda_over_the_range_of_densities():
    rho = np.concatenate([np.geomspace(1e-300, 1e20, 4001), np.geomspace(0.2, 0.3, 501),
                          [1e-30, 1.0000001e-30, 1e30]])
    v, e = lda(rho)
    vr, er = oscf.lda(rho)
    x = 0.75 * (3.0 / np.pi) ** (1.0 / 3.0) * np.cbrt(rho)
    bound = 64 * U * (4.0 / 3.0 * x + np.abs(vr) + 0.1)
    assert np.all(np.abs(v - vr) <= bound)
    assert np.all(np.abs(e - er) <= bound * rho + 1e-300)
    v0 = np.linspace(-3.0, 3.0, rho.size)
    va, _ = lda(rho, v0)
    assert np.all(np.abs(va - (v0 + vr)) <= bound + 4 * U * np.abs(v0))


def test_lda_of_values_that_are_no_densities():
    rho = np.array([0.0, -0.5, -1e-40, np.inf, np.nan, 1e-320, 1e300])
    with np.errstate(all="ignore"):
        vr, er = oscf.lda(rho)
    v, e = lda(rho)
    for got, ref in ((v, vr), (e, er)):
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        ok = np.isfinite(ref)
        np.testing.assert_array_equal(got[~ok & ~np.isnan(ref)], ref[~ok & ~np.isnan(ref)])
        np.testing.assert_allclose(got[ok], ref[ok], rtol=64 * U)


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 50, 7), (31, 5, 3), (33, 17, 65), (241, 9, 40)])
@pytest.mark.parametrize("two", [False, True])
def test_weighted_integral_of_ragged_lines(dims, two):
    rng = np.random.default_rng(sum(dims))
    f, g = rng.standard_normal(dims[::-1]), rng.standard_normal(dims[::-1])
    w = [rng.uniform(0.5, 1.5, d) for d in dims]
    terms = f * (g if two else 1.0) * w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]
    fd, gd, wd = dev(f), dev(g), [dev(x) for x in w]
    res = ctypes.c_double()
    d = np.array(dims, np.int32)
    assert _lib.ttg().ttg_grid_integrate(p(fd), p(gd) if two else None, _lib.ptr(d), *[p(x) for x in wd],
                                         ctypes.byref(res), None) == 0
    exact = float(np.sum(terms.astype(np.longdouble)))
    assert abs(res.value - exact) <= 400 * U * np.abs(terms).sum()


@pytest.mark.parametrize("n", [1, 5, 1027, 2490371])
@pytest.mark.parametrize("nt", [1, 2, 7, 24])
def test_linear_combination_in_place(n, nt):
    rng = np.random.default_rng(n + nt)
    base = rng.standard_normal(n + nt)
    F = [dev(base[i:i + n]) for i in range(nt)]
    c = rng.standard_normal(nt)
    ref = sum(c[i] * base[i:i + n] for i in range(nt))
    mag = sum(abs(c[i] * base[i:i + n]) for i in range(nt))
    arr = (ctypes.c_void_p * nt)(*[t.data_ptr() for t in F])
    assert _lib.ttg().ttg_grid_lincomb(nt, arr, _lib.ptr(c), n, p(F[0]), 1, None) == 0
    assert np.all(np.abs(F[0].cpu().numpy() - np.abs(ref)) <= 2 * (nt + 1) * U * mag)
