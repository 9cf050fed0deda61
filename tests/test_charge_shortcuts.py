"""The two shortcuts of the batched charge step (charges_batched.cu k_charges_fp32) against the
computation they stand for, in the same FP32 arithmetic on the CPU: a carrier taken as far from
every wall must have an exit distance over its step, and an electron whose |k| is outside the
band around the intervalley threshold must have its kinetic energy on the same side."""
import numpy as np
import pytest

f = np.float32
RNG = np.random.default_rng(3)


def _exit_distance(R, H, p, v):
    """fexit (fp32.cuh) without the normal."""
    with np.errstate(divide="ignore", invalid="ignore"):
        t = np.full(len(p), np.inf, f)
        tz = np.where(v[:, 2] > f(1e-15), (H - p[:, 2]) / v[:, 2],
                      np.where(v[:, 2] < f(-1e-15), (-H - p[:, 2]) / v[:, 2], f(np.inf)))
        t = np.where((tz >= 0) & (tz < t), tz, t)
        a = v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]
        b = p[:, 0] * v[:, 0] + p[:, 1] * v[:, 1]
        c = p[:, 0] * p[:, 0] + p[:, 1] * p[:, 1] - R * R
        tr = (-b + np.sqrt(np.maximum(f(0), b * b - a * c))) / a
        t = np.where((a > f(1e-18)) & (tr >= 0) & (tr < t), tr, t)
    return np.maximum(f(0), t)


@pytest.mark.parametrize("R,H", [(0.0381, 0.0127), (0.0127, 0.0381), (1e-3, 1.0), (1.0, 1e-3)])
def test_inside_carriers_cannot_reach_a_wall(R, H):
    R, H = f(R), f(H)
    n = 400000
    # distances to a wall from far below the edge to the whole solid, steps over as many decades
    gap = np.exp(RNG.uniform(np.log(1e-9), 0.0, n))
    rho = np.where(RNG.random(n) < 0.5, 1.0 - gap, RNG.random(n)).clip(0, 1) * R
    zed = np.where(RNG.random(n) < 0.5, 1.0 - gap, RNG.random(n)).clip(0, 1) * H * RNG.choice([-1.0, 1.0], n)
    phi = RNG.uniform(0, 2 * np.pi, n)
    p = np.stack([rho * np.cos(phi), rho * np.sin(phi), zed], 1).astype(f)
    v = RNG.normal(size=(n, 3))
    v[: n // 4, :2] *= 1e-8  # nearly along the axis: the quadratic's leading term vanishes
    v[n // 4: n // 2, 2] *= 1e-8
    v[n // 2: 3 * n // 4] = np.stack([p[n // 2: 3 * n // 4, 0], p[n // 2: 3 * n // 4, 1], 0 * phi[n // 2: 3 * n // 4]], 1) \
        + 1e-3 * R * v[n // 2: 3 * n // 4]  # radially outward
    v = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(f)
    step = (np.exp(RNG.uniform(np.log(1e-10), 0.0, n)) * min(R, H)).astype(f)
    reach = f(2.0) * step + f(1e-4) * (R + H)
    r_in = R - reach
    inside = (r_in > 0) & (np.abs(p[:, 2]) < H - reach) & (p[:, 0] * p[:, 0] + p[:, 1] * p[:, 1] < r_in * r_in)
    assert inside.sum() > n // 100
    d = _exit_distance(R, H, p, v)
    assert (d[inside] > step[inside]).all()


@pytest.mark.parametrize("e_min", [1e-6, 10.3e-3, 1.0, 1e3])
def test_k_outside_the_band_decides_as_the_energy(e_min):
    m = f(0.12 * 510998.95)  # an effective conduction mass (eV)
    hbarc = 6.582119569e-16 * 299792458.0
    lo, hi = (f(np.sqrt(e * e + 2.0 * e * np.float64(m)) / hbarc) for e in (e_min * 0.999, e_min * 1.001))
    inv = RNG.uniform(0.3, 4.0, 3).astype(f)  # Herring-Vogt scaling of a valley
    u = RNG.normal(size=(300000, 3))
    u /= np.linalg.norm(u * inv, axis=1, keepdims=True)
    e = e_min * (1.0 + RNG.choice([-1, 1], len(u)) * np.exp(RNG.uniform(np.log(1e-8), np.log(0.9), len(u))))
    p = (u * np.sqrt(e * e + 2.0 * e * np.float64(m))[:, None]).astype(f)

    def norm2(x):
        return x[:, 0] * x[:, 0] + x[:, 1] * x[:, 1] + x[:, 2] * x[:, 2]
    k = np.sqrt(norm2(p * f(1.0 / hbarc) * inv))
    p2 = norm2(p * inv)
    ekin = p2 / (np.sqrt(p2 + m * m) + m)
    assert (k < lo).any() and (k > hi).any()
    assert (ekin[k < lo] < f(e_min)).all()
    assert (ekin[k > hi] >= f(e_min)).all()
