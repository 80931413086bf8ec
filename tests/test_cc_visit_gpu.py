"""CUDA-core steps taken several per tile visit (the one-launch form of larger
grids) against one launch per step: each cell is computed by itself in the same
order, so the same bits, also with infinities and NaN, in every form the size
rule takes (few, some and many tiles per SM of 32, 64 and 128 rows, FP16 and
FP32), at tile edges (rows 16, 24, 48, 56, 112, 120, 128; columns 112, 240 FP16
and 56, 120 FP32), with update
rectangles and over repeated runs; FP32 storage also against gold."""
import zlib

import numpy as np
import pytest

import oracle
from conftest import STENCILS
from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu


def _run(tcs, A, B, stencil, prec, runs, one_launch, rect=None, use_graph=True):
    p = tcs.Plan(*A.shape, stencil, B, engine="cudacore", precision=prec, rect=rect)
    if not one_launch:
        p.set_multistep(0)
    assert (p.launches(max(runs)) == 1) == one_launch
    p.upload(A)
    for steps in runs:
        p.run(steps, use_graph=use_graph)
    out = np.empty_like(A)
    p.download(out)
    p.close()
    assert tcs.device_error() == 0
    return out


def _same(tcs, A, B, stencil, prec, runs, rect=None):
    ref = _run(tcs, A, B, stencil, prec, runs, False, rect)
    for use_graph in (True, False):
        np.testing.assert_array_equal(_run(tcs, A, B, stencil, prec, runs, True, rect, use_graph), ref)


def _case(stencil, shape):
    rng = np.random.default_rng(zlib.crc32(repr((stencil, shape)).encode()))
    return grid(rng, *shape), normalized_coeffs(rng, stencil)


@pytest.mark.parametrize("prec", ["f16", "f32"])
@pytest.mark.parametrize("stencil", STENCILS)
@pytest.mark.parametrize("shape", [(129, 800), (241, 649), (361, 561), (8, 1300), (1400, 9), (249, 728), (505, 513), (64, 70),
                                   (33, 129), (49, 241), (177, 340), (225, 121), (529, 700), (611, 130), (729, 64)])
@pytest.mark.parametrize("runs", [(2, 11), (11, 4, 12)])
def test_visits_equal_single_steps(tcs, torch_cuda, stencil, prec, shape, runs):
    A, B = _case(stencil, shape)
    _same(tcs, A, B, stencil, prec, runs)


@pytest.mark.parametrize("prec,shape", [("f16", (1900, 2300)), ("f32", (1300, 1500)), ("f16", (4200, 3900)), ("f32", (2300, 2500)), ("f32", (3100, 2700))])
@pytest.mark.parametrize("stencil", STENCILS)
def test_forms_for_more_tiles_per_sm(tcs, torch_cuda, stencil, prec, shape):
    A, B = _case(stencil, shape)
    if stencil == "box2d2r" and shape[0] > 3000:
        p = tcs.Plan(*shape, stencil, B, engine="cudacore", precision=prec)
        assert p.launches(5) == 5  # many tiles: its FMAs bound it
        p.close()
        return
    _same(tcs, A, B, stencil, prec, (7,))


@pytest.mark.parametrize("prec", ["f16", "f32"])
@pytest.mark.parametrize("stencil", ["star2d1r", "box2d2r"])
@pytest.mark.parametrize("rect", [(3, 4, 5, 6), (115, 130, 50, 64), (2, 598, 110, 114), (200, 520, 3, 590)])
def test_visits_with_rectangles_infinities_and_nan(tcs, torch_cuda, stencil, prec, rect):
    A, B = _case(stencil, (600, 598))
    A[90, 300], A[300, 111], A[301, 480] = np.inf, -np.inf, np.nan
    with np.errstate(all="ignore"):
        _same(tcs, A, B, stencil, prec, (9,), rect)


@pytest.mark.parametrize("stencil", STENCILS)
def test_f32_visits_equal_gold(tcs, torch_cuda, stencil):
    A, B = _case(stencil, (470, 531))
    got = _run(tcs, A, B, stencil, "f32", (8,), True)
    np.testing.assert_array_equal(got, oracle.sweep_f32(A, B, stencil, 8))
