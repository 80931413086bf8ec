"""Blocked split pairs at the edges of their tiles (row tiles start at
multiples of 124, column tiles at multiples of 128, 16-column blocks), with
many tiles per SM, and on fields whose step scale moves, against single steps:
the same bits, and the same scale exponent."""
import zlib

import numpy as np
import pytest

from conftest import STENCILS
from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu


def _run(tcs, A, c, stencil, runs, depth, rect=None, use_graph=True):
    p = tcs.Plan(*A.shape, stencil, c, engine="tensor", precision="split", rect=rect, temporal_depth=depth)
    if depth == 1:
        p.set_multistep(0)
    p.upload(A)
    for steps in runs:
        p.run(steps, use_graph=use_graph)
    out = np.empty_like(A)
    p.download(out)
    e = p.scale_exp()
    p.close()
    assert tcs.device_error() == 0
    return out, e


def _same(tcs, A, c, stencil, runs, rect=None):
    ref, e = _run(tcs, A, c, stencil, runs, 1, rect)
    for use_graph in (True, False):
        got, e2 = _run(tcs, A, c, stencil, runs, 2, rect, use_graph)
        np.testing.assert_array_equal(got, ref)
        assert e2 == e


@pytest.mark.parametrize("stencil", STENCILS)
@pytest.mark.parametrize("shape", [(5, 5), (124, 128), (126, 129), (128, 16), (129, 17), (252, 256), (253, 257), (377, 144)])
def test_pairs_at_tile_edges(tcs, torch_cuda, stencil, shape):
    rng = np.random.default_rng(zlib.crc32(repr((stencil, shape)).encode()))
    _same(tcs, grid(rng, *shape), normalized_coeffs(rng, stencil), stencil, (2, 7))


@pytest.mark.parametrize("stencil", ["star2d1r", "box2d2r"])
@pytest.mark.parametrize("rect", [None, (120, 140, 100, 150), (3, 380, 127, 130), (200, 201, 5, 290)])
def test_pairs_while_the_scale_moves(tcs, torch_cuda, stencil, rect):
    """A zero-sum field decays fast, so E moves on most steps and cells that
    are only copied are re-split; nonzero everywhere outside the rectangle."""
    rng = np.random.default_rng(17)
    A = (rng.uniform(-1, 1, (390, 300)) * 300).astype(np.float32)
    if rect is None:
        A[:2] = A[-2:] = 0
        A[:, :2] = A[:, -2:] = 0
    _same(tcs, A, normalized_coeffs(rng, stencil) * np.float32(0.4), stencil, (8, 5), rect)


@pytest.mark.parametrize("stencil,shape", [("box2d1r", (3000, 2050)), ("box2d2r", (2100, 3000))])
def test_pairs_with_many_tiles_per_sm(tcs, torch_cuda, stencil, shape):
    rng = np.random.default_rng(5)
    _same(tcs, grid(rng, *shape), normalized_coeffs(rng, stencil), stencil, (9,))


def test_the_one_call_form_takes_pairs(tcs, torch_cuda):
    """tcs_sweep_host runs split grids at depth 2: the bits of single steps."""
    rng = np.random.default_rng(9)
    A, c = grid(rng, 259, 300), normalized_coeffs(rng, "star2d2r")
    ref, _ = _run(tcs, A, c, "star2d2r", (7,), 1)
    np.testing.assert_array_equal(tcs.sweep_host(A, 7, "star2d2r", c, precision="split"), ref)
