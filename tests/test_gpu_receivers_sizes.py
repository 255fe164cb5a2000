"""Receivers on both sides of the grid sizes where a lane goes on to four cells at a time, on the smallest
grids and on rows of one and two cells, of square and other cells, by facet and by the steepest neighbour,
with and without the flats' potential, against the oracle."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import FlowRouting

pytestmark = pytest.mark.gpu

SIZES = [(1, 64), (2, 32), (4, 2), (8, 16), (256, 128), (256, 256), (512, 256), (512, 512), (2, 1 << 17)]


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("r", [1.0, 2.0])
@pytest.mark.parametrize("by_facet", [True, False])
@pytest.mark.parametrize("over_potential", [True, False])
def test_receivers(W, H, r, by_facet, over_potential):
    rng = np.random.default_rng(W + 3 * H)
    y, x = np.mgrid[0:H, 0:W]
    rel = (0.3 * np.sin(2 * np.pi * x / W + 1.0) + 0.2 * np.sin(5 * np.pi * y / H) + 0.2 * rng.random((H, W))).astype(np.float32)
    land = (rel > 0.0).astype(np.uint8)
    filled = oracle.fill_depressions(land, rel)
    want, _ = oracle.flow_directions(land, rel, filled, 9, r, 214, by_facet, over_potential)
    got, _ = FlowRouting.flow_directions(land, rel, filled, 9, r, 214, by_facet, over_potential)
    assert np.array_equal(got, want)
