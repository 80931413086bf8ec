"""Plan(engine="auto") leaves the tile width of one-launch FP16 runs to the
library's choice by grid and steps, takes a class's tuned width with one launch
per step, and a width that the caller gives always."""
import json

import numpy as np
import pytest

from conftest import STENCILS
from helpers import normalized_coeffs
from tcstencil_gb300 import autotune

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stencil", STENCILS)
@pytest.mark.parametrize("side", [256, 1026, 1500, 2048, 5800, 6500])
def test_one_launch_runs_keep_their_free_width(tcs, torch_cuda, stencil, side):
    c = normalized_coeffs(np.random.default_rng(0), stencil)
    p = tcs.Plan(side, side, stencil, c, engine="auto")
    assert p.launches(50) == 1 and p.tile_width() == 128
    p.close()
    p = tcs.Plan(side, side, stencil, c, engine="auto", tile_w=96)
    assert p.tile_width() == 96
    p.close()


def test_single_step_classes_take_their_width(tcs, torch_cuda, tmp_path, monkeypatch):
    path = tmp_path / "t.json"
    path.write_text(json.dumps({autotune.device_key(): {"sweep": {"star2d1r/f16/9x9": {
        "engine": "tensor", "temporal_depth": 1, "multistep": 0, "tile_w": 64}}}}))
    monkeypatch.setenv("TCS_AUTOTUNE_CACHE", str(path))
    p = tcs.Plan(500, 500, "star2d1r", normalized_coeffs(np.random.default_rng(0), "star2d1r"), engine="auto")
    assert p.launches(50) == 50 and p.tile_width() == 64
    p.close()
