"""The fill's tile relaxation at its edges, against the oracle bit for bit: grids narrower, shorter and just
as wide as a tile, basins that wrap around the map or span many tiles, and quantised ground whose ties pin
cells to their parents."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import FlowRouting

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(2, 8), (4, 64), (16, 64), (32, 32), (64, 8), (128, 64), (512, 256)])
@pytest.mark.parametrize("kind", ["noise", "basins", "quantised"])
def test_fill(W, H, kind):
    rng = np.random.default_rng(W * H)
    y, x = np.mgrid[0:H, 0:W]
    rel = rng.uniform(0.1, 0.9, (H, W))
    if kind == "basins":     # two basins with walls, across the seam and across every tile between
        rel = 0.2 + 0.3 * np.abs(np.sin(2 * np.pi * x / W)) + 0.4 * np.abs(y - H / 2) / H + 1e-4 * rel
    if kind == "quantised":
        rel = np.round(rel * 12) / 16
    rel = rel.astype(np.float32)
    land = (rng.random((H, W)) > 0.01).astype(np.uint8)
    land[H // 2, W // 2] = 0
    want = oracle.fill_depressions(land, rel)
    got = FlowRouting.fill_depressions(land, rel)
    got = got[0] if isinstance(got, tuple) else got
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
