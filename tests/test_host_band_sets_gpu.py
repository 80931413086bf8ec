"""The band sets of one-call sweeps: how many bands the rule takes (seen by the
planes that a first call allocates), that calls of changing step counts settle
on what they have and allocate no more, and that threads keep sets apart."""
import threading

import numpy as np
import pytest

from helpers import normalized_coeffs

pytestmark = pytest.mark.gpu


@pytest.fixture
def allocations(tcs, torch_cuda):
    """The names of the library's allocations since the last clear()."""
    names = []
    tcs.lib().tcs_release_cache()
    tcs.set_alloc_hook(lambda n, what: bool(names.append(what)))
    yield names
    tcs.set_alloc_hook(None)
    tcs.lib().tcs_release_cache()


def _plan(tcs, A, stencil, c, steps, engine, precision):
    p = tcs.Plan(*A.shape, stencil, c, engine=engine, precision=precision)
    p.set_multistep(0)
    p.upload(A)
    p.run(steps)
    out = np.empty_like(A)
    p.download(out)
    p.close()
    return out


def _case(stencil, shape):
    rng = np.random.default_rng(shape[1])
    return rng.uniform(-1, 1, shape).astype(np.float32), normalized_coeffs(rng, stencil)


# the largest steps a halo of 16 or 32 serves among them
@pytest.mark.parametrize("stencil,engine,precision,shape,steps,bands", [
    ("box2d1r", "tensor", "f16", (2051, 2101), 16, 2), ("box2d1r", "tensor", "f16", (2200, 2100), 16, 3),
    ("box2d1r", "tensor", "f16", (2200, 2100), 12, 4), ("star2d2r", "tensor", "f16", (1537, 2900), 8, 4),
    ("star2d1r", "cudacore", "f32", (3001, 2900), 32, 3), ("box2d2r", "cudacore", "f16", (2601, 2304), 8, 3),
    ("star2d1r", "tensor", "f16", (3001, 2900), 128, 1),
])
def test_band_counts(tcs, allocations, stencil, engine, precision, shape, steps, bands):
    A, c = _case(stencil, shape)
    allocations.clear()
    got = tcs.sweep_host(A, steps, stencil, c, engine=engine, precision=precision)
    assert allocations.count("plane") == 2 * bands  # two of each band's plan
    np.testing.assert_array_equal(got, _plan(tcs, A, stencil, c, steps, engine, precision))


def test_changing_step_counts_settle(tcs, allocations):
    A, c = _case("box2d1r", (2200, 2100))
    counts = (12, 17, 16, 60, 3, 33, 1)
    ref = {n: _plan(tcs, A, "box2d1r", c, n, "tensor", "f16") for n in counts}
    for turn in range(3):
        if turn == 1:
            allocations.clear()
        for n in counts:
            np.testing.assert_array_equal(tcs.sweep_host(A, n, "box2d1r", c), ref[n])
    assert allocations == []


def test_bands_give_way_to_the_whole_grid(tcs, torch_cuda):
    """Where the device has no room for the grid as a whole beside its cached
    bands (a hook refuses what would pass a budget), the bands go; later calls
    that could take bands again go as a whole."""
    A, c = _case("box2d1r", (2200, 2100))
    ref = {n: _plan(tcs, A, "box2d1r", c, n, "tensor", "f16") for n in (16, 600)}
    tcs.lib().tcs_release_cache()
    base = tcs.alloc_stats()[1]
    np.testing.assert_array_equal(tcs.sweep_host(A, 16, "box2d1r", c), ref[16])  # three bands
    budget = tcs.alloc_stats()[1] + (16 << 20)  # room for less than a whole plan
    assert tcs.alloc_stats()[1] - base > 2 * A.nbytes
    tcs.set_alloc_hook(lambda n, what: tcs.alloc_stats()[1] + n > budget)
    try:
        np.testing.assert_array_equal(tcs.sweep_host(A, 600, "box2d1r", c), ref[600])  # above 512: as a whole
        np.testing.assert_array_equal(tcs.sweep_host(A, 16, "box2d1r", c), ref[16])
    finally:
        tcs.set_alloc_hook(None)
        tcs.lib().tcs_release_cache()
    assert tcs.alloc_stats()[1] == base


def test_two_threads_band_their_own_grids(tcs, torch_cuda):
    cases = [_case("star2d1r", (2300, 2000)), _case("box2d2r", (2400, 2100))]
    names, steps = ("star2d1r", "box2d2r"), (15, 7)
    ref = [_plan(tcs, A, s, c, n, "tensor", "f16") for (A, c), s, n in zip(cases, names, steps)]
    wrong = []

    def work(k):
        A, c = cases[k]
        for _ in range(6):
            if not np.array_equal(tcs.sweep_host(A, steps[k], names[k], c), ref[k]):
                wrong.append(k)
        tcs.lib().tcs_release_cache()

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == []
