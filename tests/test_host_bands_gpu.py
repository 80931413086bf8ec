"""One-call sweeps of large host grids, cut into row bands whose copies and
sweeps overlap: the bits of one resident plan, for every band count, engine and
storage the rule takes, ragged rows, step counts up to the halo's power of two,
in place, and with the grid as a whole where the rule says so."""
import numpy as np
import pytest

from helpers import normalized_coeffs

pytestmark = pytest.mark.gpu


def _plan(tcs, A, stencil, c, steps, engine, precision, rect=None):
    p = tcs.Plan(*A.shape, stencil, c, engine=engine, precision=precision, rect=rect)
    p.set_multistep(0)
    p.upload(A)
    p.run(steps)
    out = np.empty_like(A)
    p.download(out)
    p.close()
    return out


@pytest.mark.parametrize("engine,precision", [("tensor", "f16"), ("cudacore", "f16"), ("cudacore", "f32"), ("tensor", "split")])
@pytest.mark.parametrize("stencil,shape,steps", [
    ("box2d1r", (2051, 2101), 16), ("star2d2r", (1537, 2900), 8),  # four bands, halo 16
    ("star2d1r", (2999, 1500), 33), ("box2d2r", (4099, 1111), 17),  # four, halo 64
    ("box2d2r", (1600, 2702), 31),  # three, halo 64
    ("star2d1r", (1100, 4000), 60), ("star2d2r", (900, 5000), 120),  # two or one
    ("box2d1r", (2051, 2101), 1),
])
def test_banded_calls_equal_one_plan(tcs, torch_cuda, engine, precision, stencil, shape, steps):
    rng = np.random.default_rng(shape[0] + steps)
    A = rng.uniform(-1, 1, shape).astype(np.float32)
    c = normalized_coeffs(rng, stencil)
    ref = _plan(tcs, A, stencil, c, steps, engine, precision)
    np.testing.assert_array_equal(tcs.sweep_host(A, steps, stencil, c, engine=engine, precision=precision), ref)
    h = torch_cuda.from_numpy(A.copy()).pin_memory().numpy()
    tcs.sweep_host(h, steps, stencil, c, engine=engine, precision=precision, h_out=h)  # pinned, in place
    np.testing.assert_array_equal(h, ref)


def test_other_calls_between_and_rectangles(tcs, torch_cuda):
    """Step counts that change the halo, coefficients that change, and a
    rectangle (the grid as a whole) on one shape."""
    rng = np.random.default_rng(5)
    A = rng.uniform(-1, 1, (2200, 2100)).astype(np.float32)
    for steps, rect in ((9, None), (40, None), (5, (30, 1900, 7, 2000)), (9, None), (7, (1, 2199, 300, 900))):
        c = normalized_coeffs(rng, "star2d1r")
        np.testing.assert_array_equal(tcs.sweep_host(A, steps, "star2d1r", c, rect=rect),
                                      _plan(tcs, A, "star2d1r", c, steps, "tensor", "f16", rect))
    tcs.lib().tcs_release_cache()
    assert tcs.device_error() == 0
