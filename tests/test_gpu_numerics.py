"""Device checks of the numerical helpers the kernels rely on.

``div_rcp(a, b, rb)`` replaces ``a / b`` for divisors with a precomputed
correctly rounded reciprocal (the flux stencils' 1/60 and 1/12, the upwind
fluxes' dx, dy and dz).  It must reproduce CUDA's IEEE division bit for bit,
so the kernels keep the reference's rounding.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from wrf_gpu_b200 import build

pytestmark = pytest.mark.gpu


def _selftest_lib():
    build.build()
    lib = ctypes.CDLL(str(build.SELFTEST_LIB))
    f = lib.wrfgpu_selftest_div_rcp
    f.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_long, ctypes.c_void_p]
    f.restype = ctypes.c_int
    return f


def _random_doubles(rng, n, emin, emax):
    mant = rng.integers(0, 1 << 52, size=n, dtype=np.uint64)
    exp = rng.integers(emin + 1023, emax + 1024, size=n, dtype=np.uint64)
    sign = rng.integers(0, 2, size=n, dtype=np.uint64)
    return ((sign << np.uint64(63)) | (exp << np.uint64(52)) | mant).view(np.float64)


def test_div_rcp_matches_cuda_division_bitwise(cuda_ready):
    f = _selftest_lib()
    rng = np.random.default_rng(7)
    n_per = 1 << 20
    divisors = [60.0, 12.0, 9.81, 6.0, 2.0 / 3.0, 1000.0, 1.0 / (1.0 / 3000.0), 1.0 / (1.0 / 333.3)]
    divisors += list(np.abs(_random_doubles(rng, 24, -30, 30)))
    for b in divisors:
        a = np.concatenate([_random_doubles(rng, n_per - 4, -600, 600), [0.0, 1.0, -1.0, 1.0e-20]])
        da = torch.as_tensor(a, device="cuda")
        db = torch.full_like(da, b)
        drb = torch.full_like(da, 1.0 / b)
        q1, q2 = torch.empty_like(da), torch.empty_like(da)
        rc = f(da.data_ptr(), db.data_ptr(), drb.data_ptr(), q1.data_ptr(), q2.data_ptr(), da.numel(),
               torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        x, y = q1.cpu().numpy(), q2.cpu().numpy()
        same = (x.view(np.uint64) == y.view(np.uint64)) | ((x == 0.0) & (y == 0.0))
        assert same.all(), f"b={b!r}: {int((~same).sum())} mismatches, e.g. a={a[~same][:3]}"


def test_div_batch_matches_cuda_division_bitwise(cuda_ready):
    """``div_batch`` (reciprocal iteration and Markstein correction, one special
    test per batch) against ``/`` bit for bit on drawn operands: ordinary ones up
    to the ends of its range (2^-500..2^500; numerators from 2^-400), all-ones and
    power-of-two mantissas, and batches with a zero, infinite, NaN or
    out-of-range operand, which take ``/`` for all three quotients.  (Operands
    that can differ are drawn for it below.)"""
    build.build()
    f = ctypes.CDLL(str(build.SELFTEST_LIB)).wrfgpu_selftest_div_batch
    f.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_long, ctypes.c_void_p]
    f.restype = ctypes.c_int
    rng = np.random.default_rng(11)
    n = 3 << 20
    a, b = _random_doubles(rng, n, -400, 499), _random_doubles(rng, n, -499, 499)
    near = _random_doubles(rng, n, 0, 0)  # quotients of neighbouring mantissas
    ones = np.full(n, np.nextafter(2.0, 0.0)) * 2.0 ** rng.integers(-20, 20, n)
    special = b.copy()
    special[::7] = np.resize([0.0, -0.0, np.inf, -np.inf, np.nan, 5.0e-324, 1.0e308, 2.0 ** 500, 2.0 ** -501], special[::7].size)
    odd = a.copy()
    odd[::5] = np.resize([0.0, np.inf, -np.inf, np.nan, 1.7e308, 2.0 ** 500], odd[::5].size)
    for x, y in ((a, b), (near, _random_doubles(rng, n, 0, 0)), (a, ones), (ones, b), (a, 2.0 ** rng.integers(-499, 499, n)),
                 (a, special), (odd, b), (odd, special)):
        da, db = torch.as_tensor(x, device="cuda"), torch.as_tensor(y, device="cuda")
        q1, q2 = torch.empty_like(da), torch.empty_like(da)
        assert f(da.data_ptr(), db.data_ptr(), q1.data_ptr(), q2.data_ptr(), n // 3,
                 torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        g, w = q1.cpu().numpy(), q2.cpu().numpy()
        same = (g.view(np.uint64) == w.view(np.uint64)) | ((g == 0.0) & (w == 0.0)) | (np.isnan(g) & np.isnan(w))
        # a zero divided by a zero inside the fast path's range does not occur: b = 0 is out of range
        assert same.all(), (x[~same][:3], y[~same][:3], g[~same][:3], w[~same][:3])


def _div_batch(x, y):
    """(div_batch, CUDA's ``/``) of the operands, in groups of three."""
    build.build()
    f = ctypes.CDLL(str(build.SELFTEST_LIB)).wrfgpu_selftest_div_batch
    f.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_long, ctypes.c_void_p]
    f.restype = ctypes.c_int
    n = x.size // 3
    da, db = torch.as_tensor(x[:3 * n], device="cuda"), torch.as_tensor(y[:3 * n], device="cuda")
    q1, q2 = torch.empty_like(da), torch.empty_like(da)
    assert f(da.data_ptr(), db.data_ptr(), q1.data_ptr(), q2.data_ptr(), n,
             torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return q1.cpu().numpy(), q2.cpu().numpy()


@pytest.mark.parametrize("emin,emax", [(-1074, -1022), (-1022, -1000), (-1000, -900), (-900, -500)])
def test_div_batch_tiny_numerators(cuda_ready, emin, emax):
    """Numerators down to the subnormals, alone and beside ordinary ones and
    zeros: from 2^-900 up ``/``'s bits; below, where the residual a - b q may be
    no double, within 2 ulp (the uncorrected quotient's 1.5 or the residual's
    rounding, and the last rounding)."""
    rng = np.random.default_rng(31)
    n = 3 << 18
    if emin < -1022:
        a = rng.integers(1, 1 << 52, size=n, dtype=np.uint64).view(np.float64)
    else:
        a = _random_doubles(rng, n, emin, emax)
    b = _random_doubles(rng, n, -2, 2)
    mixed = a.copy()
    mixed[::3] = _random_doubles(rng, a[::3].size, -3, 3)
    mixed[1::6] = np.resize([0.0, -0.0], a[1::6].size)
    for x, y in ((a, b), (a, _random_doubles(rng, n, -100, 499)), (a, _random_doubles(rng, n, -499, -100)), (mixed, b)):
        g, w = _div_batch(x, y)
        assert np.all(np.abs(g - w) <= 2.0 * np.spacing(np.abs(w))), (emin, emax)
        big = (np.abs(x) >= 2.0 ** -900) | (x == 0.0)
        assert np.array_equal(g[big], w[big]), (emin, emax)


@pytest.mark.parametrize("kind", ["random", "near_one", "near_two", "below_two"])
def test_div_batch_next_to_a_midpoint(cuda_ready, kind):
    """The hardest operands: for an odd 53-bit b the a with a 2^54 = b m + 1 or
    b m - 1, m odd, whose quotient lies 2^-53 / b of an ulp from the midpoint of
    two doubles, where the bound on ``div_batch``'s error (half an ulp and 2^-50 of
    one) allows the other neighbour for b > 2 (1 - 2^-6) and for no other b."""
    rng = np.random.default_rng(17)
    n = 90000
    b = {"random": rng.integers(1 << 51, 1 << 52, size=n) * 2 + 1, "near_one": (1 << 52) + 2 * np.arange(n) + 1,
         "near_two": (1 << 53) - 2 * np.arange(n) - 1,
         "below_two": (1 << 53) - 2 * (2.0 ** rng.uniform(1, 46, n)).astype(np.int64) - 1}[kind]
    a = np.empty(n)
    for i, x in enumerate(map(int, b)):
        inv = pow(x, -1, 1 << 54)
        m, one = (inv, -1) if inv >> 53 else ((1 << 54) - inv, 1)
        assert (x * m + one) % (1 << 54) == 0
        a[i] = float((x * m + one) >> 54)
    y = b.astype(np.float64)
    g, w = _div_batch(a, y)
    other = g != w
    assert not np.any(other & (y < 2.0 ** 53 * (1.0 - 2.0 ** -6)))
    assert np.all(np.abs(g - w)[other] == np.spacing(np.minimum(g, w))[other])


def test_reciprocal_seed_is_as_good_as_div_batch_needs(cuda_ready):
    """|1 - b y0| < 2^-19.9 of rcp.approx.ftz.f64, over every high word: e^3 is then
    less than 2^-6 of an ulp of 1/b."""
    build.build()
    f = ctypes.CDLL(str(build.SELFTEST_LIB)).wrfgpu_selftest_rcp_seed
    f.argtypes, f.restype = [ctypes.c_void_p, ctypes.c_void_p], ctypes.c_int
    e0 = torch.empty(1 << 20, dtype=torch.float64, device="cuda")
    assert f(e0.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert float(e0.max()) < 2.0 ** -19.9
