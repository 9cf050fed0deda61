"""The plain form's functions on the device one at a time (sin and cos apart from sincos, exp, the
division through a reciprocal): correctly rounded, against 70-digit decimals and IEEE division."""
from decimal import Decimal, getcontext

import numpy as np
import pytest

from tests.test_crmath_midpoints import HARD
from tests.test_gpu_crmath import _reference

pytestmark = pytest.mark.gpu

SIN, COS, EXP, DIV = 1, 2, 3, 4


def _eval(lib, fn, x, y=None):
    x, out = np.ascontiguousarray(x), np.empty(len(x))
    y = None if y is None else np.ascontiguousarray(y)
    assert lib.cmpmc_gpu_math_eval(0, fn, len(x), x.ctypes.data, None if y is None else y.ctypes.data, out.ctypes.data) == 0
    return out


def test_sin_and_cos(lib):
    rng = np.random.default_rng(3)
    k = np.arange(1, 33) * (np.pi / 4)
    x = np.concatenate([HARD, k, np.nextafter(k, 0), np.nextafter(k, 1e3), rng.uniform(0, 2 * np.pi, 100),
                        2.0 ** -rng.uniform(1, 60, 50)])
    want = _reference(x)
    assert np.array_equal(_eval(lib, SIN, x), want[:, 1])
    assert np.array_equal(_eval(lib, COS, x), want[:, 2])


# the fast path's limits (|x| near 700), its reductions (multiples of ln 2 and their halves) and tiny x
def test_exp(lib):
    rng = np.random.default_rng(4)
    k = np.arange(-40, 41) * (0.5 * np.log(2.0))
    tiny = 2.0 ** -rng.uniform(1, 70, 100)
    x = np.concatenate([k, np.nextafter(k, 1e3), np.nextafter(k, -1e3), tiny, -tiny, rng.uniform(-699.9, 699.9, 200),
                        rng.uniform(-2, 2, 200), [0.0, -0.0, np.nextafter(700, 0), -np.nextafter(700, 0)]])
    getcontext().prec = 70
    want = np.array([float(Decimal(float(v)).exp()) for v in x])
    assert np.array_equal(_eval(lib, EXP, x), want)


def test_division(lib):
    rng = np.random.default_rng(5)
    n = 200000
    y = np.where(np.arange(n) % 2, rng.choice([1.588 / 0.12, 0.081 / 0.12, 1.0, 3.0], n), rng.uniform(1, 2, n) * 2.0 ** rng.integers(-20, 20, n))
    x = rng.uniform(-2, 2, n) * 2.0 ** rng.integers(-200, 200, n)
    x[:8] = [0.0, -0.0] * 4
    assert _eval(lib, DIV, x, y).tobytes() == (x / y).tobytes()


def test_refusals(lib):
    x = np.ones(2)
    for fn, px in ((-1, x.ctypes.data), (5, x.ctypes.data), (DIV, x.ctypes.data), (EXP, None)):
        assert lib.cmpmc_gpu_math_eval(0, fn, 2, px, None, x.ctypes.data) == 1
