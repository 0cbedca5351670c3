"""The device code's own divisions against CUDA's, bit for bit.

A quotient by Markstein's correction is off only where the exact quotient lies
within 2^-50 units of a rounding boundary: fewer than 1e-7 expected among the 4e7
quotients below, so any difference fails.  The Newton reciprocal alone may miss
the correctly rounded one within 2^-27 units of a boundary, 2^-26 of the
arguments: 0.06 expected among 4e6, so three fail.
"""

import ctypes
import os
import subprocess

import numpy as np
import pytest

from montepath_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
F64 = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("arithmetic") / "arithmetic.so")
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler",
                    "-fPIC", "-shared", "-I", build.CSRC, os.path.join(HERE, "arithmetic.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def p(a):
    return a.ctypes.data_as(F64)


def same_quotients(lib, num, den):
    num, den = np.ascontiguousarray(num), np.ascontiguousarray(den)
    out = [np.zeros_like(num) for _ in range(4)]
    assert lib.quotients(p(num), p(den), ctypes.c_uint64(num.size), *(p(o) for o in out)) == 0
    ours, plain, ours_inv, plain_inv = out
    assert np.array_equal(ours, plain), int((ours != plain).sum())
    off = ours_inv != plain_inv
    assert off.sum() < 3 and np.all(np.abs(ours_inv - plain_inv)[off] <= np.spacing(plain_inv[off]))


def centre_rational(u):
    """Numerator and denominator of the inverse normal's centre, each operation rounded."""

    a = (-3.969683028665376e1, 2.209460984245205e2, -2.759285104469687e2, 1.38357751867269e2, -3.066479806614716e1,
         2.506628277459239)
    b = (-5.447609879822406e1, 1.615858368580409e2, -1.556989798598866e2, 6.680131188771972e1, -1.328068155288572e1, 1.0)
    q = u - 0.5
    r = q * q
    num, den = np.full_like(u, a[0]), np.full_like(u, b[0])
    for x, y in zip(a[1:], b[1:]):
        num, den = num * r + x, den * r + y
    return num * q, den


def test_inverse_normal_quotients(lib):
    m = np.arange(203_424, 1 << 22, dtype=np.float64)  # every 23-bit uniform of the centre below 1/2
    same_quotients(lib, *centre_rational((m + 0.5) / (1 << 23)))
    same_quotients(lib, *centre_rational(np.random.default_rng(5).uniform(0.02425, 0.97575, 1 << 22)))


def test_sixths(lib):
    n = ctypes.c_ulonglong()
    for exponent in (-40, -20, -1, 0, 1, 20):  # all 2^23 mantissas
        assert lib.sixths_f32(ctypes.c_uint32((exponent + 127) << 23), ctypes.c_uint32(1 << 23), ctypes.byref(n)) == 0
        assert n.value == 0
    rng = np.random.default_rng(7)
    x = rng.uniform(1.0, 2.0, 1 << 22) * np.exp2(rng.integers(-60, 20, 1 << 22))
    ours, plain = np.zeros_like(x), np.zeros_like(x)
    assert lib.sixths_f64(p(x), ctypes.c_uint64(x.size), p(ours), p(plain)) == 0
    assert np.array_equal(ours, plain), int((ours != plain).sum())


@pytest.mark.parametrize("dim", [2, 3, 4])
def test_lsm_normal_equations(lib, dim):
    """Regressions of a date with `dim` to 300 in-the-money paths: prices spread
    over the strike, or so close together that later pivots pass the 1e-12 limit."""

    rng = np.random.default_rng(dim)
    n = 1 << 17
    systems = np.zeros((3, n, 20))
    for k, (paths, spread) in enumerate([(dim, 0.5), (300, 0.4), (8, 1e-3)]):
        for lo in range(0, n, 1 << 14):
            x = 1.0 - spread * rng.random((1 << 14, paths))
            basis = np.stack([np.ones_like(x), 1 - x, 1 - 2 * x + 0.5 * x * x, 1 - 3 * x + 1.5 * x * x - x**3 / 6], -1)
            cash = 100.0 * rng.random((1 << 14, paths, 1))
            systems[k, lo:lo + (1 << 14), :16] = (basis.transpose(0, 2, 1) @ basis).reshape(-1, 16)
            systems[k, lo:lo + (1 << 14), 16:] = (basis.transpose(0, 2, 1) @ cash)[..., 0]
    systems = systems.reshape(-1, 20)
    ours, plain = np.zeros((3 * n, 5)), np.zeros((3 * n, 5))
    assert lib.solves(dim, p(systems), ctypes.c_uint64(3 * n), p(ours), p(plain)) == 0
    assert plain[:, 0].sum() > n
    assert np.array_equal(ours, plain), int((ours != plain).any(1).sum())
