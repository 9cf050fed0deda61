"""div_by (transport.cuh), the plain form's division by a mass ratio with its reciprocal at hand,
against the division, compiled on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "transport.cuh"
using namespace cmpmc_gpu;
static int bad = 0;
static void check(double x, double m) {
    const double want = x / m, got = div_by(x, m, 1.0 / m);
    if (std::memcmp(&want, &got, 8) != 0 && bad++ < 10) std::printf("%a / %a: %a, not %a\n", x, m, got, want);
}
int main() {
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> u(1.0, 2.0);
    const double ratios[] = {1.588 / 0.12, 0.081 / 0.12, 1.0, 3.0, 1.0 / 3.0, 0x1.fffffffffffffp-1, 0x1.0000000000001p0};
    for (double m : ratios) {
        check(0.0, m);
        check(-0.0, m);
        check(m, m);
        check(-m, m);
    }
    for (int i = 0; i < 2000000; ++i) {
        const double m = (i & 1) ? ratios[i / 2 % 7] : std::ldexp(u(g), static_cast<int>(g() % 40) - 20);
        const double x = std::ldexp(u(g), static_cast<int>(g() % 400) - 200);
        check((i & 2) ? -x : x, m);
        // next to the midpoint of two quotients, where one correction would not do
        const double q = u(g);
        const double at = std::fma(q + std::nextafter(q, 3.0), 0.5 * m, 0.0);
        check(at, m);
        check(std::nextafter(at, 1e9), m);
    }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_div_by_is_the_division(tmp_path):
    src, exe = tmp_path / "div.cpp", tmp_path / "div"
    src.write_text(SRC)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O2", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "cmpmc_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
