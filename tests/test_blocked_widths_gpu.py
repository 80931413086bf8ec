"""Two-step split launches at every tile width the size rule takes (32, 80 and
128 columns) against single steps: the same bits, at the tiles' edges (columns
32, 80, 128; rows 124, 128), with update rectangles, odd step counts and values
that change the scale."""
import zlib

import numpy as np
import pytest

from conftest import STENCILS
from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu


def _run(tcs, A, B, stencil, depth, runs, rect):
    p = tcs.Plan(*A.shape, stencil, B, engine="tensor", precision="split", rect=rect, temporal_depth=depth)
    if depth == 1:
        p.set_multistep(0)
    p.upload(A)
    for steps in runs:
        p.run(steps, use_graph=steps % 2 == 0)
    out = np.empty_like(A)
    p.download(out)
    p.close()
    assert tcs.device_error() == 0
    return out


@pytest.mark.parametrize("stencil", STENCILS)
@pytest.mark.parametrize("shape,rect", [
    ((40, 31), None), ((128, 33), None), ((129, 64), None), ((252, 65), None), ((253, 97), (120, 131, 30, 36)),  # 32
    ((500, 700), None), ((877, 801), None), ((124, 5000), (3, 119, 77, 2403)), ((1024, 161), None),  # 32 or 80
    ((1100, 1281), None), ((640, 4100), (5, 601, 80, 4000)), ((1733, 2049), (60, 1700, 127, 1920)),  # 80 or 128
])
def test_pairs_of_every_width_equal_single_steps(tcs, torch_cuda, stencil, shape, rect):
    rng = np.random.default_rng(zlib.crc32(repr((stencil, shape)).encode()))
    A, B = grid(rng, *shape) * np.float32(3.0), normalized_coeffs(rng, stencil)
    B = B * np.float32(0.6)  # values fall by 2^-0.7 a step: the scale moves
    for runs in ((2,), (6, 5, 18)):
        np.testing.assert_array_equal(_run(tcs, A, B, stencil, 2, runs, rect), _run(tcs, A, B, stencil, 1, runs, rect))
