"""The untuned air sweeps' choice of a tile shape (csrc/weno_tiles.cuh, plain
C++) against a count of the faces and points that each shape's tiles compute,
over ragged extents on every axis."""
import math
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = """
#include <cstdio>
#include "weno_tiles.cuh"
int main() {
  for (int y = 0; y < 2; ++y)
    for (int v = 0; v < 3; ++v) printf("%d %d\\n", cfk::kAirTileNodes[y][v], cfk::kAirTileColumns[y][v]);
  int ext, across, outer, dir, order, sm;
  while (scanf("%d %d %d %d %d %d", &ext, &across, &outer, &dir, &order, &sm) == 6)
    printf("%d\\n", cfk::weno_air_tile(ext, across, outer, dir, order, sm));
}
"""


def _work(ext, across, outer, n, c, order):
    """Faces, and points at a tenth each, of a sweep's tiles, tile by tile."""
    total = 0
    for _ in range(0, ext, n):
        for _ in range(0, across, c):
            total += c * (10 * (n + 1) + n + (8 if order == 7 else 6))
    return total * outer


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_the_choice_computes_least(tmp_path):
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-x", "c++", "-I", os.path.join(ROOT, "corefl-cpc_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    rng = random.Random(4)
    asked = [(ext, across, outer, d, order, 148) for d in (0, 1, 2) for order in (5, 7) for outer in (1, 40)
             for ext, across in [(1, 1), (7, 9), (9, 7), (33, 9), (9, 33), (65, 17), (161, 113), (257, 257), (400, 7)]]
    asked += [(*(int(math.exp(rng.uniform(0, 6.3))) for _ in range(3)), rng.randrange(3), rng.choice((5, 7)),
               rng.choice((80, 148))) for _ in range(400)]
    out = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, a)) for a in asked), capture_output=True,
                         text=True, check=True).stdout.split()
    shapes = [(int(out[2 * q]), int(out[2 * q + 1])) for q in range(6)]
    one_wave = 0
    for a, got in zip(asked, map(int, out[12:]), strict=True):
        ext, across, outer, d, order, sm = a
        if d and math.ceil(across / 16) * math.ceil(ext / 15) * outer <= 4 * sm:
            one_wave += 1
            assert got == 2, a
            continue
        works = [_work(ext, across, outer, *shapes[3 * (d > 0) + v], order) for v in range(2 if d else 3)]
        assert got == works.index(min(works)), a
    assert 50 < one_wave < len(asked) - 100  # both sides of the line
