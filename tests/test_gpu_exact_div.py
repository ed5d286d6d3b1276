"""The exact form's quotients by a shared denominator equal the correctly
rounded division bit for bit: ordinary operands, significands next to 2 and
next to 1, quotients next to a rounding boundary, and operands outside the
ranges of the fast path (zeros of both signs, subnormals, infinities, NaN)."""
import ctypes

import numpy as np
import pytest

from fvm3d import abi

pytestmark = pytest.mark.gpu


def gpu_div(x, y):
    lib = abi.load_library()
    lib.fvm_test_exact_div.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p]
    x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
    q = np.empty_like(x)
    assert lib.fvm_test_exact_div(x.ctypes.data, y.ctypes.data, x.size, q.ctypes.data) == 0
    return q


def same(x, y):
    with np.errstate(all="ignore"):
        ref = x / y
    got = gpu_div(x, y)
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.int64), ref[~nan].view(np.int64))  # signs of zeros too


@pytest.mark.parametrize("exps", [(0, 0), (20, 20), (300, 60), (700, 260), (1000, 1000)])
def test_random_operands(exps):
    rng = np.random.default_rng(exps[0])
    n = 1 << 20
    r = lambda e: rng.choice([-1.0, 1.0], n) * np.ldexp(rng.uniform(1, 2, n), rng.integers(-e, e + 1, n))  # noqa: E731
    same(r(exps[0]), r(exps[1]))


def test_significands_near_one_and_two():
    k = np.arange(0, 64, dtype=np.float64)
    y = np.concatenate([2.0 - np.ldexp(k + 1, -52), 1.0 + np.ldexp(k, -52), 1.5 + np.ldexp(k, -52)])
    x = np.concatenate([2.0 - np.ldexp(k + 1, -52), 1.0 + np.ldexp(k, -52), 1.25 + np.ldexp(k, -52), 1.0 - np.ldexp(k + 1, -53)])
    X, Y = np.meshgrid(x, y)
    for e in (-3, 0, 5):
        same(np.ldexp(X.ravel(), e), Y.ravel())
        same(X.ravel(), np.ldexp(Y.ravel(), e))


def test_quotients_near_rounding_boundaries():
    # x = RN(m y) for midpoints m of two neighbouring doubles: the quotient is
    # as close to the boundary as two doubles can make it
    rng = np.random.default_rng(5)
    n = 1 << 20
    y = rng.uniform(1, 2, n)
    q = rng.uniform(1, 2, n)
    hi = q * y
    for ulps in (-1, 0, 1):
        same(hi + ulps * np.spacing(hi), y)
    yl = rng.integers(1 << 26, 1 << 27, n).astype(np.float64)  # short factors: exact products and near ties
    ql = rng.integers(1 << 26, 1 << 27, n).astype(np.float64) + 0.5
    p = yl * ql
    for ulps in (-1, 0, 1):
        same(p + ulps * np.spacing(p), yl)


def test_special_operands():
    v = np.array([0.0, -0.0, 1.0, -1.0, 3.0, 5e-324, -5e-324, 2.2e-308, 1e-300, 1e-181, 1e-180, 1e-61, 1e-60, 1.6e60,
                  1.7e60, 1e180, 4e180, 1.7e308, -1.7e308, np.inf, -np.inf, np.nan, 0.1, 1 / 3])
    X, Y = np.meshgrid(v, v)
    same(X.ravel().copy(), Y.ravel().copy())
