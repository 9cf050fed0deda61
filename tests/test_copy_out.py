"""cmpmc_copy_out: every byte once, nothing beside it, at the sizes where the pieces change."""
import numpy as np
import pytest

MIB = 1 << 20


@pytest.mark.parametrize("n", [0, 1, 4 * MIB - 1, 4 * MIB, 4 * MIB + 1, 6 * MIB + 4097, 33 * MIB + 5])
@pytest.mark.parametrize("shift", [0, 3])
def test_copy_out(lib, n, shift):
    rng = np.random.default_rng(n)
    src = rng.integers(0, 256, n + 16, dtype=np.uint8)
    dst = np.full(n + 16, 0xAB, np.uint8)
    assert lib.cmpmc_copy_out(dst.ctypes.data + shift, src.ctypes.data + 5, n) == 0
    assert np.array_equal(dst[shift:shift + n], src[5:5 + n])
    assert (dst[:shift] == 0xAB).all() and (dst[shift + n:] == 0xAB).all()


def test_copy_out_refuses_null(lib):
    assert lib.cmpmc_copy_out(None, None, 8) != 0
    assert lib.cmpmc_copy_out(None, None, 0) == 0
