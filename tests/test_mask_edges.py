"""find_channel's shortcuts (full rings, one angle per centre, sector edges by side) against the
plain test of every pad by its angle, over shapes, wrapped and degenerate sectors, angles outside
[0, 2 pi], off-centre pads, and points on the edges, the axes and the centre."""
import math

import numpy as np
import pytest

import cmpmc_b200 as cm


def _contains(p, x, y):
    dx, dy = x - p.cx, y - p.cy
    if p.shape == 2:
        return abs(dx) <= p.r_min and abs(dy) <= p.r_max
    r2 = dx * dx + dy * dy
    if p.shape == 0:
        return r2 <= p.r_max * p.r_max
    if r2 < p.r_min * p.r_min or r2 > p.r_max * p.r_max:
        return False
    phi = math.atan2(dy, dx)
    if phi < 0.0:
        phi += 2.0 * math.pi
    if p.phi_min <= p.phi_max:
        return p.phi_min <= phi <= p.phi_max
    return phi >= p.phi_min or phi <= p.phi_max


@pytest.mark.parametrize("angles", ["inside", "any", "special"])
def test_find_channel_matches_the_angle_test(angles):
    rng = np.random.default_rng({"inside": 1, "any": 2, "special": 3}[angles])
    two_pi = 2.0 * math.pi
    special = [0.0, 0.5 * math.pi, math.pi, 1.5 * math.pi, two_pi, 3.0, two_pi - 3.0, 1e-12, two_pi - 1e-12]
    for _ in range(400):
        pads = []
        for ch in range(int(rng.integers(1, 7))):
            if angles == "special":
                a, b = (special[int(rng.integers(len(special)))] for _ in range(2))
            else:
                a, b = rng.uniform(0, two_pi, 2) if angles == "inside" else rng.uniform(-4.0, 9.0, 2)
            c = (0.0, 0.0) if rng.random() < 0.7 else tuple(rng.uniform(-0.3, 0.3, 2))
            r = rng.uniform(0, 0.5)
            pads.append(cm.ElectrodePad(int(rng.choice([0, 1, 1, 1, 2])), ch, c[0], c[1], r, r + rng.uniform(0, 0.5),
                                        float(a), float(b), 1.0))
        mask = cm.ElectrodePatternMask(pads)
        gen = cm.Rng(1)
        for _ in range(60):
            x, y = rng.uniform(-1, 1, 2)
            kind = rng.random()
            if kind < 0.3:  # on, or next to, an edge of a pad
                p = pads[int(rng.integers(len(pads)))]
                phi = (p.phi_min if rng.random() < 0.5 else p.phi_max) + rng.choice([0.0, 1e-15, -1e-12, 1e-9, math.pi])
                rr = rng.uniform(p.r_min, p.r_max)
                x, y = p.cx + rr * math.cos(phi), p.cy + rr * math.sin(phi)
            elif kind < 0.4:
                x = float(rng.choice([0.0, -0.0]))
            elif kind < 0.5:
                y = float(rng.choice([0.0, -0.0]))
            want = next((p.channel_id for p in pads if _contains(p, x, y)), -1)
            assert mask.find_channel((x, y, 0.0), gen) == want, (x, y, pads)
