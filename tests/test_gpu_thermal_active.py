"""The thermal sweeps where few, all or none of the cells give, against the oracle bit for bit: single
spikes and pits on every column and row of a tile's edge and at the poles (x wraps, y stops), fields in
which every cell gives, fields at rest, grids narrower and lower than a tile, negative zeros, and limits
of zero and below."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300.api import GpuErosionAccelerator, ThermalLimits

pytestmark = pytest.mark.gpu


def check(h, limits, passes, rate=0.25):
    H, W = h.shape
    got = GpuErosionAccelerator().erode(W, H, h, ThermalLimits(*limits), passes, rate)
    want = oracle.thermal_sweep(h, ThermalLimits(*limits), passes, rate, skip=False)
    # A settled share below 0 divides 0 by 0 where nothing falls; a NaN's own bits are the machine's.
    diff = np.flatnonzero((got.view(np.uint32) != want.view(np.uint32)) & ~(np.isnan(got) & np.isnan(want)))
    assert diff.size == 0, f"{diff.size} cells differ, first {diff[:5]}"


LIMITS = (0.01, 0.012, 0.0156)


@pytest.mark.parametrize("W,H", [(2, 2), (8, 64), (16, 8), (64, 32), (128, 64), (256, 128), (512, 32)])
@pytest.mark.parametrize("passes", [1, 2, 3, 6])
def test_rough_everywhere(W, H, passes):
    rng = np.random.default_rng(W * H + passes)
    check(rng.random((H, W)).astype(np.float32), LIMITS, passes)


@pytest.mark.parametrize("passes", [1, 2, 5])
def test_spikes_across_a_tile(passes):
    """One spike or pit a 9 x 9 neighbourhood, at every offset to the tiles' edges, rows at both poles included."""
    W, H = 256, 128
    h = np.full((H, W), 0.5, np.float32)
    k = 0
    for r in range(0, H, 9):
        for c in range((r * 5) % 9, W - 8, 9):
            h[r, c] += 0.3 if k % 2 else -0.3
            k += 1
    h[H - 1, ::7] += 0.2
    h[:, 0] += 0.05
    check(h, LIMITS, passes)


@pytest.mark.parametrize("passes", [1, 2, 9])
def test_at_rest_but_for_one_cell(passes):
    W, H = 256, 128
    rng = np.random.default_rng(1)
    h = (0.5 + 0.001 * rng.random((H, W))).astype(np.float32)
    h[64, 64] = 0.9
    check(h, LIMITS, passes)
    h[64, 64] = 0.5
    check(h, LIMITS, passes)


def test_negative_zeros():
    h = np.zeros((64, 128), np.float32)
    h[::3] = -0.0
    h[20, 30:40] = 0.2
    check(h, LIMITS, 3)


@pytest.mark.parametrize("limits", [(0.0, 0.0, 0.0), (0.01, 0.0, 0.02), (-0.001, 0.01, 0.01), (0.01, -0.002, -0.003)])
@pytest.mark.parametrize("passes", [1, 2, 3])
def test_limits_of_zero_and_below(limits, passes):
    rng = np.random.default_rng(9)
    check(rng.random((64, 128)).astype(np.float32), limits, passes, 0.1)
