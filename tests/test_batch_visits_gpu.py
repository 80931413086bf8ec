"""FP16 grids of a batch take several steps per turn (visits): the bits of the
same grids alone in single steps, at tile edges (rows 120, 128; columns 64, 128),
with update rectangles, every step count around a turn's five or three, grids of
different turns together, and over repeated runs."""
import numpy as np
import pytest

from conftest import STENCILS
from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu

SHAPES = [(5, 7), (120, 64), (128, 65), (129, 129), (240, 190), (248, 257), (249, 383), (369, 130), (61, 900), (1000, 33)]


def _solo(tcs, A, stencil, c, steps, runs, rect):
    p = tcs.Plan(*A.shape, stencil, c, engine="tensor", precision="f16", rect=rect)
    p.set_multistep(0)
    p.upload(A)
    for _ in range(runs):
        p.run(steps)
    out = np.empty_like(A)
    p.download(out)
    p.close()
    return out


@pytest.mark.parametrize("stencil", STENCILS)
@pytest.mark.parametrize("runs", [1, 3])
def test_turns_of_several_steps(tcs, torch_cuda, stencil, runs):
    rng = np.random.default_rng(len(stencil) + runs)
    b = tcs.Batch()
    work = []
    for k, shape in enumerate(SHAPES * 2):
        steps = (0, 1, 2, 3, 4, 5, 6, 7, 10, 11, 16)[(3 * k + k // len(SHAPES)) % 11]
        rect = (2, max(3, shape[0] // 2), 2, shape[1] - 2) if k >= len(SHAPES) else None
        A, c = grid(rng, *shape), normalized_coeffs(rng, stencil)
        b.add(*shape, stencil, c, steps, "f16", rect=rect)
        work.append((A, c, steps, rect))
    for k, (A, *_) in enumerate(work):
        b.upload(k, A)
    for run in range(runs):
        b.run(use_graph=run % 2 == 1)
    for k, (A, c, steps, rect) in enumerate(work):
        out = np.empty_like(A)
        b.download(k, out)
        np.testing.assert_array_equal(out, _solo(tcs, A, stencil, c, steps, runs, rect), err_msg=f"{A.shape} {steps} {rect}")
    assert tcs.device_error() == 0
    b.close()
