"""Runs of more (turn, tile) items than a launch may have go out in several:
the cut (tcstencil_gb300/csrc/tile_walk.h, compiled as host C++) covers the run,
keeps every launch's items and a CTA's walk past them inside an int, and cuts
nothing that fits.  On the GPU, the launches that plans report."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import normalized_coeffs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER_DIR = os.path.join(ROOT, "tcstencil_gb300", "csrc")
MAX_ITEMS = 1 << 27
PROGRAM = r"""
#include <cstdio>
#include "tile_walk.h"
int main() {
    int steps, depth;
    long long tiles;
    while (std::scanf("%d %d %lld", &steps, &depth, &tiles) == 3) {
        for (int left = steps; left > 0;) {
            const tcs::Launch l = tcs::next_launch(left, (left - 1) / depth + 1, depth, tiles);
            std::printf("%d %d\n", l.turns, l.steps);
            left -= l.steps;
        }
        std::printf("end\n");
    }
}
"""
CASES = [(10, 8, 24), (343_000, 3, 18769), (572_001, 5, 18769), (2_400_000, 2, 4290), (706_000, 1, 3040),
         (2**31 - 1, 4, 330), (2**31 - 1, 9, 1), (MAX_ITEMS // 7 * 5, 5, 7), (MAX_ITEMS // 7 * 5 + 1, 5, 7),
         (1, 1, 16641), (3, 1, MAX_ITEMS + 5)]


def test_launches_cover_the_run_within_an_int(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    (tmp_path / "cut.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "cut")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", HEADER_DIR, str(tmp_path / "cut.cpp"), "-o", exe], check=True,
                   timeout=120)
    out = subprocess.run([exe], input="".join(f"{s} {d} {t}\n" for s, d, t in CASES), capture_output=True, text=True,
                         check=True, timeout=120).stdout.split("end\n")
    for (steps, depth, tiles), block in zip(CASES, out):
        cuts = [tuple(map(int, line.split())) for line in block.strip().splitlines()]
        assert sum(s for _, s in cuts) == steps
        for turns, s in cuts:
            assert turns == -(-s // depth)  # the shape's depth holds, no turn empty
            assert turns * tiles <= MAX_ITEMS or turns == 1
        fits = -(-steps // depth) * tiles <= MAX_ITEMS
        assert (len(cuts) == 1) == (fits or steps <= depth), (steps, depth, tiles, cuts[:3])


@pytest.mark.gpu
@pytest.mark.parametrize("engine,precision,shape", [("tensor", "f16", (700, 900)), ("cudacore", "f16", (700, 900)),
                                                    ("cudacore", "f32", (700, 900)), ("tensor", "split", (2300, 2100))])
def test_plans_cut_runs_of_too_many_items(tcs, torch_cuda, engine, precision, shape):
    p = tcs.Plan(*shape, "star2d1r", normalized_coeffs(np.random.default_rng(0), "star2d1r"), engine=engine,
                 precision=precision, temporal_depth=1)
    assert p.launches(1000) == 1
    assert p.launches(2_000_000_000) > 1
    p.close()
