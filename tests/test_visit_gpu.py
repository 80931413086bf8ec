"""Plain FP16 steps taken several per tile visit (a plan's one-launch form)
against one launch per step: the same windows in the same order, so the same
bits, at the edges of its tiles (row tiles overlap and start at multiples of
112, 120 or 124, column tiles at multiples of 32 to 128), for step counts that
divide into full and shorter visits, with update rectangles that cut panels,
and again after the launch has reset its own counters."""
import zlib

import numpy as np
import pytest

from conftest import STENCILS
from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu


def _run(tcs, A, B, stencil, runs, mode, rect=None, tile_w=128, use_graph=True):
    p = tcs.Plan(*A.shape, stencil, B, engine="tensor", precision="f16", rect=rect)
    p.set_multistep(mode)
    p.set_tile_width(tile_w)
    p.upload(A)
    for steps in runs:
        p.run(steps, use_graph=use_graph)
    out = np.empty_like(A)
    p.download(out)
    p.close()
    assert tcs.device_error() == 0
    return out


def _case(stencil, shape, runs):
    rng = np.random.default_rng(zlib.crc32(repr((stencil, shape, runs)).encode()))
    return grid(rng, *shape), normalized_coeffs(rng, stencil)


@pytest.mark.parametrize("stencil", STENCILS)
@pytest.mark.parametrize("shape", [(5, 9), (128, 32), (129, 33), (240, 64), (249, 95), (241, 129), (361, 257)])
@pytest.mark.parametrize("runs", [(2,), (17,), (8, 9, 8)])
def test_visits_equal_single_steps(tcs, torch_cuda, stencil, shape, runs):
    A, B = _case(stencil, shape, runs)
    ref = _run(tcs, A, B, stencil, runs, 0)
    for w in (128, 96, 64):
        np.testing.assert_array_equal(_run(tcs, A, B, stencil, runs, 1, tile_w=w), ref, err_msg=f"width {w}")
    np.testing.assert_array_equal(_run(tcs, A, B, stencil, runs, 1, use_graph=False), ref)


@pytest.mark.parametrize("stencil", ["star2d1r", "box2d2r"])
@pytest.mark.parametrize("rect", [(2, 298, 2, 268), (3, 4, 5, 6), (117, 131, 60, 67), (100, 290, 33, 200), (2, 298, 127, 130)])
def test_visits_with_rectangles(tcs, torch_cuda, stencil, rect):
    A, B = _case(stencil, (300, 270), rect)
    ref = _run(tcs, A, B, stencil, (13,), 0, rect)
    for w in (128, 64):
        np.testing.assert_array_equal(_run(tcs, A, B, stencil, (13,), 1, rect, w), ref)


@pytest.mark.parametrize("stencil,shape", [("box2d2r", (4099, 3001)), ("star2d1r", (2600, 4500)), ("box2d1r", (124 * 9 + 4, 9000))])
def test_visits_with_many_tiles_per_sm(tcs, torch_cuda, stencil, shape):
    A, B = _case(stencil, shape, 0)
    np.testing.assert_array_equal(_run(tcs, A, B, stencil, (9,), 1), _run(tcs, A, B, stencil, (9,), 0))


@pytest.mark.parametrize("stencil", ["star2d1r", "box2d2r"])
def test_an_infinite_cell_stays_within_its_windows_reach(tcs, torch_cuda, stencil):
    """An infinity makes its windows' outputs NaN (32 columns a step), in one
    launch as in single steps: what gold's reach covers is not finite, and
    nothing beyond the windows' reach differs."""
    A, B = _case(stencil, (200, 600), 1)
    A[90, 300] = np.inf
    steps, r = 5, 1 if stencil.endswith("1r") else 2
    one, ref = (_run(tcs, A, B, stencil, (steps,), m) for m in (1, 0))
    far = np.ones(A.shape, bool)
    far[90 - r * steps:91 + r * steps, 300 - 32 * steps:301 + 32 * steps] = False
    np.testing.assert_array_equal(one[far], ref[far])
    assert np.isfinite(one[far]).all()
    assert not np.isfinite(one[90, 300 - r * steps:301 + r * steps]).any()
