"""The correctly rounded log, sin and cos of the plain form on the device against 70-digit
decimals, at the arguments that stress their reductions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(x):
    """log, sin and cos rounded from 60-digit decimals."""
    from decimal import Decimal, getcontext
    getcontext().prec = 70
    pi = Decimal("3.14159265358979323846264338327950288419716939937510582097494459230781640628620899862803")

    def sincos(d):
        d = d % (2 * pi)
        s, c, t, k = Decimal(0), Decimal(0), Decimal(1), 0
        while abs(t) > Decimal(10) ** -65:
            (c, s) = (c + (t if k % 4 == 0 else -t), s) if k % 2 == 0 else (c, s + (t if k % 4 == 1 else -t))
            k += 1
            t = t * d / k
        return float(s), float(c)
    out = np.empty((len(x), 3))
    for i, v in enumerate(x):
        d = Decimal(float(v))
        out[i, 0] = float(d.ln()) if v > 0 else np.nan
        out[i, 1:] = sincos(d)
    return out


# uniform draws near 1 and 0, the reduction points n/128 and their neighbours (residuals of zero and
# one unit), angles around the quadrants
@pytest.mark.parametrize("kind", ["uniform", "tiny", "nodes", "quadrants"])
def test_log_sin_cos_are_correctly_rounded(kind):
    from cmpmc_b200 import _ffi
    rng = np.random.default_rng(7)
    if kind == "uniform":
        x = rng.uniform(0, 1, 300)
    elif kind == "tiny":
        x = np.concatenate([2.0 ** -rng.uniform(1, 53, 150), 1.0 - 2.0 ** -rng.uniform(1, 53, 150)])
    elif kind == "nodes":
        n = np.arange(64, 256) / 128.0
        x = np.concatenate([n, np.nextafter(n, 0), np.nextafter(n, 4)])
    else:
        k = np.arange(1, 65) * (np.pi / 4)
        x = np.concatenate([k, np.nextafter(k, 0), np.nextafter(k, 1e3), rng.uniform(0, 2 * np.pi, 100)])
    x = np.ascontiguousarray(x)
    got = np.empty((len(x), 3))
    lib = _ffi.load()
    assert lib.cmpmc_gpu_math_check(0, len(x), x.ctypes.data, got.ctypes.data) == 0
    want = _reference(x)
    assert np.array_equal(got, want)
