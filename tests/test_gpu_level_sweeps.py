"""The level sweeps (incision, the belts' cut) at their extremes, against the oracle bit for bit: worlds of
hundreds of levels of a few cells each (one CTA's levels alone), of a few levels of more cells than two of
a CTA's passes, and grids narrower than a warp."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import ErosionConfig, ErosionStage, synthetic
from test_gpu_belt import check, run_both

pytestmark = pytest.mark.gpu


def world(kind, W, H, seed):
    y, x = np.mgrid[0:H, 0:W].astype(np.float32)
    noise = np.random.default_rng(seed).normal(0.0, 1e-3, (H, W)).astype(np.float32)
    if kind == "valley":    # one river along the map: as many levels as columns
        return (0.75 - 0.2 * x / W + 0.1 * np.abs(y - H / 2) / H).astype(np.float32) + noise * np.float32(0.1)
    if kind == "ramp":      # every row drains on its own: a few levels' steps, thousands of cells each
        return (0.4 + 0.3 * ((x % 8) / 8)).astype(np.float32) + noise
    return synthetic.world(W, H, seed)[0]


@pytest.mark.parametrize("kind,W,H", [("valley", 1024, 16), ("ramp", 512, 256), ("noise", 8, 64), ("noise", 1024, 512)])
def test_incision(kind, W, H):
    h = world(kind, W, H, 3)
    options = dict(sea_level=0.3, profile=0, hydraulic_rounds=2)
    got = ErosionStage.apply(ErosionConfig(W, H, 3, **options), h, None, None, want=("receivers", "area"))
    want = oracle.erode_stage(oracle.default_params(W, H, 3, **options), h, None, None, want=("receivers", "area"))
    assert np.array_equal(got.height.view(np.uint32), want["height"].view(np.uint32))
    assert np.array_equal(got.area.view(np.uint32), want["area"].view(np.uint32))


@pytest.mark.parametrize("W,H,seed", [(16, 32, 4), (64, 32, 9), (1024, 256, 6)])
def test_belt_cut(W, H, seed):
    check(*run_both(W, H, seed)[:5])
