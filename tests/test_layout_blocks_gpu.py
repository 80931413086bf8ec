"""Pack and unpack at the edges of their blocks (32 plane rows by 32 panels)
and on grids that start at any float, bit for bit against the oracle's panel
layout; and a split plan's scale record against its grid's maximum and border."""
import numpy as np
import pytest

import oracle
from helpers import grid, normalized_coeffs, to_plane

pytestmark = pytest.mark.gpu


def _offset(torch, a, shift):
    """`a` on the device, `shift` floats past an aligned address."""
    t = torch.empty(a.size + 4, dtype=torch.float32, device="cuda")
    v = t[shift:shift + a.size].view(a.shape)
    v.copy_(torch.from_numpy(a))
    return v


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("ny,nx,pad", [(1, 1, 0), (28, 247, 0), (29, 248, 0), (60, 249, 2), (33, 124, 16), (200, 505, 0)])
def test_pack_and_unpack_at_block_edges(tcs, torch_cuda, ny, nx, pad, shift):
    torch, L = torch_cuda, tcs.lib()
    rng = np.random.default_rng(1000 * ny + nx)
    A = rng.uniform(-1, 1, (ny, nx)).astype(np.float32)
    d_A = _offset(torch, A, shift)
    d_o = _offset(torch, np.full_like(A, 7.0), shift)
    padded = np.full((ny + 2 * pad, nx + 2 * pad), 0.5, np.float32)
    padded[pad:pad + ny, pad:pad + nx] = A
    n16, n32 = (tcs.plane_elems(*padded.shape, p) for p in ("f16", "f32"))
    h, lo = (torch.full((n16,), 12345, dtype=torch.int16, device="cuda") for _ in range(2))
    f = torch.full((n32,), 9.0, dtype=torch.float32, device="cuda")
    assert L.tcs_pack_f16(d_A.data_ptr(), ny, nx, pad, 0.5, h.data_ptr(), None) == 0
    np.testing.assert_array_equal(h.cpu().numpy().view(np.uint16), to_plane(oracle.f32_to_f16(padded)))
    assert L.tcs_unpack_f16(h.data_ptr(), ny, nx, pad, d_o.data_ptr(), None) == 0
    np.testing.assert_array_equal(d_o.cpu().numpy(), oracle.f16_to_f32(oracle.f32_to_f16(A)))
    assert L.tcs_pack_f32(d_A.data_ptr(), ny, nx, pad, 0.5, f.data_ptr(), None) == 0
    np.testing.assert_array_equal(f.cpu().numpy(), to_plane(padded, cpp=4))
    assert L.tcs_unpack_f32(f.data_ptr(), ny, nx, pad, d_o.data_ptr(), None) == 0
    np.testing.assert_array_equal(d_o.cpu().numpy(), A)
    assert L.tcs_pack_split(d_A.data_ptr(), ny, nx, pad, 0.5, 0, h.data_ptr(), lo.data_ptr(), None) == 0
    hi_ref, lo_ref = oracle.split(padded.astype(np.float64), 0)
    np.testing.assert_array_equal(h.cpu().numpy().view(np.uint16), to_plane(hi_ref))
    np.testing.assert_array_equal(lo.cpu().numpy().view(np.uint16), to_plane(lo_ref))
    assert L.tcs_unpack_split(h.data_ptr(), lo.data_ptr(), ny, nx, pad, 0, d_o.data_ptr(), None) == 0
    assert np.max(np.abs(d_o.cpu().numpy().astype(np.float64) - A)) <= 2.0 ** -23


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("shape", [(7, 9), (130, 517), (1025, 300)])
@pytest.mark.parametrize("at,scale", [((0, 0), 40.0), ((-1, -1), 3e-5), ((3, 4), 900.0)])
def test_split_upload_scale_of_any_grid(tcs, torch_cuda, shape, shift, at, scale):
    """The exponent comes from the largest |x| wherever it is (first and last
    cell, interior), and a second upload starts from a clean record."""
    torch = torch_cuda
    rng = np.random.default_rng(shape[0] + shift)
    c = normalized_coeffs(rng, "box2d1r")
    p = tcs.Plan(*shape, "box2d1r", c, engine="tensor", precision="split")
    out = torch.empty(shape, dtype=torch.float32, device="cuda")
    for mul in (1.0, 1.0 / 1024):
        A = (grid(rng, *shape) * 1e-6 * mul).astype(np.float32)
        A[at] = -scale * mul
        p.upload(_offset(torch, A, shift))
        assert p.scale_exp() == oracle.split_scale_exp(A)
        p.download(out)
        assert np.max(np.abs(out.cpu().numpy().astype(np.float64) - A)) <= 2.0 ** (p.scale_exp() - 23)
    p.close()
    assert tcs.device_error() == 0
