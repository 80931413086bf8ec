"""Solves one after another on a stream with nothing between them: each kernel's
launch may start beside its predecessors (programmatic launches), so every
result is compared with the same solve made alone."""
import numpy as np
import pytest

from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine,precision", [("tensor", "f16"), ("cudacore", "f16"), ("cudacore", "f32"), ("tensor", "split")])
@pytest.mark.parametrize("shape", [(64, 64), (257, 190), (552, 664), (1026, 1026), (2500, 91)])
@pytest.mark.parametrize("steps", [0, 1, 2])
def test_solves_in_a_row(tcs, torch_cuda, engine, precision, shape, steps):
    torch = torch_cuda
    rng = np.random.default_rng(shape[0])
    p = tcs.Plan(*shape, "box2d2r", normalized_coeffs(rng, "box2d2r"), engine=engine, precision=precision)
    grids = [torch.from_numpy(grid(rng, *shape)).cuda() for _ in range(6)]
    alone, row = ([torch.zeros_like(g) for g in grids] for _ in range(2))
    for outs, wait in ((alone, True), (row, False)):
        for _ in range(1 if wait else 3):
            for g, o in zip(grids, outs):
                p.upload(g)
                p.run(steps)
                p.download(o)
                if wait:
                    torch.cuda.synchronize()
    torch.cuda.synchronize()
    for a, b in zip(alone, row):
        assert torch.equal(a, b)
    p.close()
    assert tcs.device_error() == 0
