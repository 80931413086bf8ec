"""Split planes bit for bit where hi rounds to zero: a negative value below
2^-12 of the scale keeps its sign in hi (a -0), as the oracle's split and
tcs_pack_split store it.  A step whose only tap is the centre's 1 gives back
the values it got, so the planes have to be the oracle's split of them."""
import numpy as np
import pytest

import oracle
from helpers import grid16, plane16

pytestmark = pytest.mark.gpu


def _values(shape):
    """Values that a split holds exactly, most of them of hi = -0 or +0."""
    rng = np.random.default_rng(17)
    x = rng.integers(1, 2 ** 10, shape) * rng.choice([-1.0, 1.0], shape) * 2.0 ** -22
    x[rng.random(shape) < 0.2] *= 2.0 ** 11
    x.flat[0] = 1.0  # scale exponent 1 ([1, 2) for an upload)
    return x


def _identity(stencil):
    n = 3 if stencil.endswith("1r") else 5
    c = np.zeros((n, n), np.float32)
    c[n // 2, n // 2] = 1.0
    return c


class _Plane:  # a plan's plane as a torch tensor
    def __init__(self, ptr, nbytes):
        self.__cuda_array_interface__ = dict(shape=(nbytes // 2,), typestr="<i2", data=(ptr, False), version=3)


@pytest.mark.parametrize("stencil", ["star2d1r", "box2d2r"])
@pytest.mark.parametrize("shape", [(5, 9), (129, 131), (300, 411)])
def test_hi_keeps_the_sign_of_small_values(tcs, torch_cuda, stencil, shape):
    torch = torch_cuda
    x = _values(shape)
    hi, lo = oracle.split(x, 0)
    assert (hi == 0x8000).any()
    c = _identity(stencil)
    d_hi, d_lo = plane16(torch, hi), plane16(torch, lo)
    o_hi, o_lo = torch.zeros_like(d_hi), torch.zeros_like(d_lo)
    tcs.sweep_step(d_hi, o_hi, *shape, stencil, c, precision="split", d_in_lo=d_lo, d_out_lo=o_lo)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(grid16(o_hi, *shape), hi)
    np.testing.assert_array_equal(grid16(o_lo, *shape), lo)

    up = torch.from_numpy(x.astype(np.float32)).cuda()
    for depth, mode in ((1, 0), (1, 1), (2, -1)):
        p = tcs.Plan(*shape, stencil, c, precision="split", temporal_depth=depth)
        p.set_multistep(mode)
        p.upload(up)
        p.run(2)
        torch.cuda.synchronize()
        want = oracle.split(x, p.scale_exp())
        a, b, n = p.state()
        for ptr, w in zip((a, b), want):
            np.testing.assert_array_equal(grid16(torch.as_tensor(_Plane(ptr, n), device="cuda"), *shape), w)
        p.close()
    assert tcs.device_error() == 0
