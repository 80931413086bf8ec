"""Several plans at once, each on a stream of its own, in the one-launch forms:
launches that share the GPU (and, for small FP16 grids, an SM's TMEM) with one
another and with launches of one step.  Every result is the plan's alone."""
import numpy as np
import pytest

from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu

PLANS = [("tensor", "f16", "star2d1r", (512, 500), -1), ("tensor", "f16", "box2d2r", (260, 300), -1),
         ("tensor", "f16", "box2d1r", (512, 500), 0), ("tensor", "f16", "star2d2r", (600, 500), -1),
         ("tensor", "f16", "star2d1r", (1026, 1026), -1), ("tensor", "split", "box2d1r", (400, 380), -1),
         ("cudacore", "f16", "star2d2r", (512, 500), -1), ("cudacore", "f32", "box2d2r", (700, 650), -1)]


@pytest.mark.parametrize("picked", [(0, 1), (0, 3, 0, 1), (0, 2, 1, 5), tuple(range(8)), (0,) * 8])
def test_plans_on_streams_of_their_own(tcs, torch_cuda, picked):
    torch = torch_cuda
    jobs = []
    for k in picked:
        engine, precision, stencil, shape, mode = PLANS[k]
        rng = np.random.default_rng(k)
        A = torch.from_numpy(grid(rng, *shape)).cuda()
        p = tcs.Plan(*shape, stencil, normalized_coeffs(rng, stencil), engine=engine, precision=precision)
        p.set_multistep(mode)
        jobs.append((p, A, torch.empty_like(A), torch.cuda.Stream()))
    torch.cuda.synchronize()

    def solve(p, A, out, stream, turns):
        p.upload(A, stream=stream)
        for _ in range(turns):
            p.run(20, stream=stream)
        p.download(out, stream=stream)

    refs = []
    for p, A, out, stream in jobs:
        solve(p, A, out, stream, 5)
        torch.cuda.synchronize()
        refs.append(out.clone())
    for _ in range(5):
        for _, _, out, _ in jobs:
            out.zero_()
        torch.cuda.synchronize()
        for job in jobs:
            solve(*job, 5)
        torch.cuda.synchronize()
        assert tcs.device_error() == 0
        for (_, _, out, _), ref in zip(jobs, refs):
            assert torch.equal(out, ref)
    for p, *_ in jobs:
        p.close()
