"""charge_shortcuts.cuh, compiled on the host, against the full computation in FP32: a carrier that it
takes as clear of the walls has an exit distance over its step, and an electron whose |k| is outside
the band has its kinetic energy on that side of the threshold."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.test_charge_shortcuts import _exit_distance

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
f = np.float32

SRC = """
#include "charge_shortcuts.cuh"
using namespace cmpmc_gpu;
extern "C" void clear(float R, float H, int n, const float* p, const float* step, char* out) {
    for (int i = 0; i < n; ++i)
        out[i] = clear_of_walls(R, H, wall_edge(R, H), p[3 * i], p[3 * i + 1], p[3 * i + 2], step[i]);
}
extern "C" void band(double e_min, double m, float* out) {
    const KBand b = k_band(e_min, m);
    out[0] = b.lo;
    out[1] = b.hi;
}
"""


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    d = tmp_path_factory.mktemp("shortcuts")
    (d / "s.cpp").write_text(SRC)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-shared", "-fPIC", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "cmpmc_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    str(d / "s.cpp"), "-o", str(d / "s.so")], check=True)
    return ctypes.CDLL(str(d / "s.so"))


def _clear(lib, R, H, p, step):
    p, step, out = np.ascontiguousarray(p, f), np.ascontiguousarray(step, f), np.zeros(len(p), np.int8)
    lib.clear(ctypes.c_float(R), ctypes.c_float(H), len(p), p.ctypes.data_as(ctypes.c_void_p),
              step.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p))
    return out.astype(bool)


@pytest.mark.parametrize("R,H", [(0.0381, 0.0127), (0.0127, 0.0381), (1e-3, 1.0), (1.0, 1e-3)])
def test_a_clear_carrier_reaches_no_wall(built, R, H):
    rng = np.random.default_rng(8)
    n, R, H = 400000, f(R), f(H)
    gap = np.exp(rng.uniform(np.log(1e-9), 0.0, n))  # distances to a wall over nine decades
    rho = np.where(rng.random(n) < 0.5, 1.0 - gap, rng.random(n)).clip(0, 1) * R
    zed = np.where(rng.random(n) < 0.5, 1.0 - gap, rng.random(n)).clip(0, 1) * H * rng.choice([-1.0, 1.0], n)
    phi = rng.uniform(0, 2 * np.pi, n)
    p = np.stack([rho * np.cos(phi), rho * np.sin(phi), zed], 1).astype(f)
    v = rng.normal(size=(n, 3))
    q = n // 4
    v[:q, :2] *= 1e-8  # along the axis, across it, and radially outward
    v[q:2 * q, 2] *= 1e-8
    v[2 * q:3 * q] = np.stack([p[2 * q:3 * q, 0], p[2 * q:3 * q, 1], 0 * gap[:q]], 1) + 1e-3 * R * v[2 * q:3 * q]
    v = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(f)
    step = (np.exp(rng.uniform(np.log(1e-10), 0.0, n)) * min(R, H)).astype(f)
    clear = _clear(built, R, H, p, step)
    assert n // 100 < clear.sum() < n
    assert (_exit_distance(R, H, p, v)[clear] > step[clear]).all()


def test_what_is_not_finite_takes_the_test(built):
    p = np.array([[0, 0, 0], [np.nan, 0, 0], [0, np.nan, 0], [0, 0, np.nan], [np.inf, 0, 0], [0, 0, -np.inf], [0, 0, 0],
                  [0, 0, 0]], f)
    step = np.array([1e-6] * 6 + [np.nan, np.inf], f)
    assert list(_clear(built, 0.0381, 0.0127, p, step)) == [True] + [False] * 7


@pytest.mark.parametrize("e_min", [1e-6, 10.3e-3, 1.0, 1e3])
def test_k_outside_the_band_decides_as_the_energy(built, e_min):
    rng = np.random.default_rng(9)
    m = f(0.12 * 510998.95)
    hbarc = 6.582119569e-16 * 299792458.0
    band = np.empty(2, f)
    built.band(ctypes.c_double(e_min), ctypes.c_double(float(m)), band.ctypes.data_as(ctypes.c_void_p))
    inv = rng.uniform(0.3, 4.0, 3).astype(f)  # Herring-Vogt scaling of a valley
    u = rng.normal(size=(300000, 3))
    u /= np.linalg.norm(u * inv, axis=1, keepdims=True)
    e = e_min * (1.0 + rng.choice([-1, 1], len(u)) * np.exp(rng.uniform(np.log(1e-8), np.log(0.9), len(u))))
    p = (u * np.sqrt(e * e + 2.0 * e * np.float64(m))[:, None]).astype(f)

    def norm2(x):
        return x[:, 0] * x[:, 0] + x[:, 1] * x[:, 1] + x[:, 2] * x[:, 2]
    k = np.sqrt(norm2(p * f(1.0 / hbarc) * inv))
    p2 = norm2(p * inv)
    ekin = p2 / (np.sqrt(p2 + m * m) + m)
    assert (k < band[0]).any() and (k > band[1]).any()
    assert (ekin[k < band[0]] < f(e_min)).all() and (ekin[k > band[1]] >= f(e_min)).all()


@pytest.mark.parametrize("e_min", [0.0, -1.0, float("nan")])
def test_no_threshold_no_shortcut(built, e_min):
    band = np.empty(2, f)
    built.band(ctypes.c_double(e_min), ctypes.c_double(6e4), band.ctypes.data_as(ctypes.c_void_p))
    assert band[0] < 0.0 and band[1] == np.inf
