"""The drowned basins' outlets (SeaLevelStage.drained_cut's passes) where many basins share channels, on
small rough grids of both cell shapes, against the oracle bit for bit: the notch runs 32 basins at a
time and must cut as if one after another."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import ErosionConfig, SeaLevelStage, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,seed,sea_level,rough", [(64, 32, 1, 0.5, 0.0), (64, 64, 2, 0.6, 0.05), (128, 64, 3, 0.7, 0.1),
                                                      (256, 256, 4, 0.6, 0.1), (512, 256, 5, 0.8, 0.05)])
def test_drained_cut_of_a_rough_world(W, H, seed, sea_level, rough):
    rng = np.random.default_rng(seed)
    h = synthetic.heights_field(W, H, seed) + (rough * rng.random((H, W))).astype(np.float32)
    cfg = ErosionConfig(W, H, seed, sea_level=sea_level)
    s1, l1, r1, n1, p1 = SeaLevelStage.drained_cut(cfg, h)
    s0, l0, r0, n0, p0 = oracle.sea_level_drained_cut(oracle.default_params(W, H, seed, sea_level=sea_level), h)
    assert np.float32(s0).view(np.uint32) == np.float32(s1).view(np.uint32)
    assert (n0, p0) == (n1, p1)
    assert np.array_equal(l0, l1) and np.array_equal(r0.view(np.uint32), r1.view(np.uint32))
