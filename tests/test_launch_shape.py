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


# rows: the shape of each size, then what it becomes over four overflows of that size
_GROW = """
    for (auto u : x) {
        PoolRing r;
        for (int k = 0; k < 5; ++k) {
            const PoolShape s = pool_shape(r, u, 148, %d), one = pool_shape(r, 100, 148, %d);
            printf("%%llu %%u %%llu %%llu %%u\\n", (unsigned long long)s.grid, s.ring, (unsigned long long)s.per_block,
                   (unsigned long long)one.grid, one.ring);
            pool_grow(r, s, %d);
        }
    }"""


@pytest.mark.parametrize("threads", [512, 768])
def test_a_pool_overflow_reruns_with_more_room(tmp_path, threads):
    sizes = [1, 2, 147, 148, 149, 2368, 18900, 20300, 76000, 200000, 1000000, 4000000]
    rows = _run(tmp_path, _GROW % (threads, threads, threads), sizes)
    for i, units in enumerate(sizes):
        packed = max(1, min(148, -(-units // threads)))
        prev = None
        for grid, ring, per_block, one_grid, one_ring in rows[5 * i:5 * i + 5]:
            assert grid * per_block >= units and ring & (ring - 1) == 0 and 4096 <= ring <= 1 << 24
            assert packed <= grid <= min(148, units)
            assert grid * ring <= max(148 << 17, packed * ring)  # the memory of a full batch
            if prev is None:  # spread at first: a block on every SM, no less room per unit than packed ones
                assert grid == min(148, units) and ring >= min(1 << 17, (1 << 17) * per_block // threads)
            else:  # no rerun is the launch that overflowed
                assert ring > prev or ring == 1 << 24
            prev = ring
            # a small call afterwards: spread over the chip unless its own kind needs rings over 2^17
            assert one_grid == 100 or (per_block < threads and one_ring > 1 << 17)
