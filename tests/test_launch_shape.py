"""The launch shapes of launch_shape.hpp, compiled on the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, body, args):
    """Compiles a program with `body` in main (x: the arguments as integers) and returns the rows it prints."""
    src, exe = tmp_path / "shape.cpp", tmp_path / "shape"
    src.write_text('#include <cstdio>\n#include <cstdlib>\n#include <vector>\n#include "launch_shape.hpp"\n'
                   "using namespace cmpmc_gpu;\nint main(int n, char** v) {\n    std::vector<unsigned long long> x;\n"
                   "    for (int i = 1; i < n; ++i) x.push_back(strtoull(v[i], nullptr, 10));\n" + body + "\n}\n")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", os.path.join(ROOT, "cmpmc_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True, text=True).stdout
    return [tuple(map(int, line.split())) for line in out.splitlines()]


@pytest.mark.parametrize("late", [0, 25])
@pytest.mark.parametrize("blocks,tpb", [(444, 128), (296, 128), (148, 32), (1, 32), (888, 64)])
def test_units_beyond_one_per_warp_start_at_once(tmp_path, blocks, tpb, late):
    warps = blocks * tpb // 32
    sizes = sorted({0, 1, 2, warps - 1, warps, warps + 1, warps * (100 + late) // 100, warps * (100 + late) // 100 + 1,
                    2 * warps, 2 * warps + 1, 3 * warps - 1, 6 * warps - 1, 31 * warps + 1, 32 * warps, 40 * warps})
    rows = _run(tmp_path, "for (auto u : x) { const Spread s = spread_units(u, %d, %d, %d); "
                          'printf("%%llu %%u\\n", (unsigned long long)s.grid, s.lanes); }' % (blocks, tpb, late), sizes)
    for units, (grid, lanes) in zip(sizes, rows):
        assert 1 <= grid <= blocks and 1 <= lanes <= 32
        if lanes == 1:
            assert units <= warps * (100 + late) // 100
        elif lanes < 32:
            assert grid * (tpb // 32) * lanes >= units
            assert warps * (lanes - 1) < units  # no more lanes than that takes
