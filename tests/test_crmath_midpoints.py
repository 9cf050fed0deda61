"""sin and cos of the plain form next to the midpoint of two FP64 numbers, where an error of the fast
path above the margin of its rounding test gives the wrong neighbour: arguments near odd multiples
of pi/4, at which the cosine kernel did."""
import numpy as np
import pytest

from tests.test_gpu_crmath import _reference

HARD = [float.fromhex(h) for h in """
0x1.921fb84461609p-1 0x1.9db6f79d6eb4cp-1 0x1.9d36b36c0581p-1 0x1.92d70df0444d6p-1 0x1.96349e1c94ffap-1
0x1.940e71fc102bep-1 0x1.9d77c75b00e67p-1 0x1.9f610edf60538p-1 0x1.9cf941ba5245ep-1 0x1.98606057e32d2p-1
0x1.96167e0a66bf9p-1 0x1.ac5c28aa3fc19p-1 0x1.9380a8f900f7p-1 0x1.93ab44d8569f2p-1 0x1.96681711caeb4p-1
0x1.98a5161ab9541p-1 0x1.f70046d9c22e5p+1 0x1.96cce9517dc1ep-1 0x1.94e9aad6f9be4p-1 0x1.92ecc495734bbp-1
0x1.94fa5f6407434p-1 0x1.5ed17f9423037p+2""".split()]


def test_host(lib):
    want = _reference(np.array(HARD))
    for x, w in zip(HARD, want):
        assert (lib.cmpmc_cr_sin(x), lib.cmpmc_cr_cos(x)) == (w[1], w[2]), x.hex()


@pytest.mark.gpu
def test_device(lib):
    x = np.array(HARD)
    got = np.empty((len(x), 3))
    assert lib.cmpmc_gpu_math_check(0, len(x), x.ctypes.data, got.ctypes.data) == 0
    assert np.array_equal(got, _reference(x))
