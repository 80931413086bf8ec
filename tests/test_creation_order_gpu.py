"""Plans and batches made while the default stream is busy and first used on a
stream that it does not order (torch's streams are non-blocking): what creation
zeroes and builds has to be in place by then.  The memory they get held other
values before."""
import numpy as np
import pytest

from helpers import grid, normalized_coeffs

pytestmark = pytest.mark.gpu

BUSY_CYCLES = 300_000_000  # 0.15 s at 2 GHz


def _plan(tcs, torch, engine, precision, depth):
    rng = np.random.default_rng(11)
    A = torch.from_numpy(grid(rng, 700, 900)).cuda()
    B = normalized_coeffs(rng, "box2d1r")
    torch.cuda.synchronize()

    def go(stream):
        out = torch.empty_like(A)
        p = tcs.Plan(700, 900, "box2d1r", B, engine=engine, precision=precision, temporal_depth=depth)
        p.upload(A, stream=stream)
        p.run(30, stream=stream)
        p.download(out, stream=stream)
        return p, [out]
    return go


def _batch(tcs, torch):
    rng = np.random.default_rng(12)
    specs = [((300, 411), "box2d2r", "f16", 9), ((257, 190), "star2d1r", "split", 7), ((64, 500), "star2d1r", "f16", 12)]
    grids = [torch.from_numpy(grid(rng, *s[0])).cuda() for s in specs]
    taps = [normalized_coeffs(rng, s[1]) for s in specs]
    torch.cuda.synchronize()

    def go(stream):
        b = tcs.Batch()
        outs = [torch.empty_like(g) for g in grids]
        for (shape, st, prec, steps), c in zip(specs, taps):
            b.add(*shape, st, c, steps, prec)
        for i, g in enumerate(grids):
            b.upload(i, g, stream=stream)
        b.run(stream=stream)
        for i, o in enumerate(outs):
            b.download(i, o, stream=stream)
        return b, outs
    return go


@pytest.mark.parametrize("what", [("tensor", "f16", 1), ("tensor", "split", 1), ("tensor", "split", 2),
                                  ("cudacore", "f16", 1), ("cudacore", "f32", 1), "batch"])
def test_first_use_beside_a_busy_default_stream(tcs, torch_cuda, what):
    torch = torch_cuda
    side = torch.cuda.Stream()
    go = _batch(tcs, torch) if what == "batch" else _plan(tcs, torch, *what)
    obj, ref = go(side.cuda_stream)
    torch.cuda.synchronize()
    obj.close()
    dirty = torch.full((256 << 20,), 255, dtype=torch.uint8, device="cuda")
    del dirty
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    torch.cuda._sleep(BUSY_CYCLES)
    assert not torch.cuda.default_stream().query()
    obj, out = go(side.cuda_stream)
    side.synchronize()
    got = [o.cpu().numpy() for o in out]
    obj.close()
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b.cpu().numpy())
    assert tcs.device_error() == 0
