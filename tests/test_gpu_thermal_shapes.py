"""The thermal sweeps on both sides of the grid size where the tile changes, and where a tile's region is
wider or taller than the map, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import ErosionConfig, GpuErosionAccelerator, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2, 64), (64, 2), (32, 16), (128, 8), (64, 1024), (512, 512), (4096, 64), (1024, 512),
                                 (4096, 128)])
@pytest.mark.parametrize("passes", [1, 2, 9])
def test_tile_shapes(W, H, passes):
    h = np.random.default_rng(W + H).uniform(0.0, 1.0, (H, W)).astype(np.float32)
    if W >= 32 and H >= 16:
        h = (synthetic.heights_field(W, H, seed=passes) + 0.02 * h).astype(np.float32)
    lim, _ = ErosionConfig(W, H, 5).thermal_limits()
    got = GpuErosionAccelerator().erode(W, H, h, lim, passes, 0.25)
    want = oracle.thermal_sweep(h, oracle.thermal_limits(oracle.default_params(W, H, 5))[0], passes, 0.25, skip=True)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
