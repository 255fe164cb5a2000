"""The fill where the ground holds a NaN or an infinity: in the sea, on land that drains, on a polar row, in
the first and last column of a tile and of the map. Such a cell is settled from the start, so the fill gives
the oracle's levels around it, and the calls over the fill go through."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import ErosionConfig, FlowRouting

pytestmark = pytest.mark.gpu


def basins(W, H):
    """Land with many pits in every tile, an ocean over a third of the map; heights relative to the shore."""
    rng = np.random.default_rng(W + H)
    y, x = np.mgrid[0:H, 0:W]
    rel = 0.3 * np.sin(2 * np.pi * x / W) + 0.2 * np.sin(3 * np.pi * y / H) + 0.1 * rng.random((H, W)) + 0.1
    land = rel > 0.0
    return land.astype(np.uint8), rel.astype(np.float32)


def same(got, want):
    return np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.nan_to_num(got), np.nan_to_num(want))


def drained_land(land, rel):
    """A cell one step above an outlet on land, away from every pit: it drains whatever it holds."""
    H, W = land.shape
    filled = oracle.fill_depressions(land, rel)
    for y in range(2, H - 2):
        for x in range(2, W - 2):
            block = (slice(y - 1, y + 2), slice(x - 1, x + 2))
            if land[y, x] and not land[block].all() and np.array_equal(filled[block], rel[block]):
                return y, x
    raise AssertionError("no such cell")


@pytest.mark.parametrize("W,H", [(32, 32), (64, 64), (256, 128), (16, 64)])
@pytest.mark.parametrize("value", [np.nan, -np.inf])
@pytest.mark.parametrize("where", ["sea", "tile corner", "seam", "pole", "land"])
def test_fill(W, H, value, where):
    land, rel = basins(W, H)
    assert (oracle.fill_depressions(land, rel) > rel).any()
    if where == "land":
        at = drained_land(land, rel)
    else:
        at = {"sea": (H // 2, W * 3 // 4), "tile corner": (H // 2 - 1, W // 2 - 1), "seam": (H // 2, W - 1),
              "pole": (0, W // 2)}[where]
        land[at] = 0
    rel[at] = value
    want = oracle.fill_depressions(land, rel)
    got, _, unresolved = FlowRouting.fill_depressions(land, rel, with_ties=True)
    assert unresolved == 0
    assert same(got, want)


def test_route_cut():
    W, H = 256, 128
    land, rel = basins(W, H)
    at = (H // 2, W * 3 // 4)
    land[at] = 0
    rel[at] = np.nan
    filled, recv, area, order = FlowRouting.route_cut(ErosionConfig(W, H, 1), land, rel, int(land.sum()))
    assert same(filled, oracle.fill_depressions(land, rel))
    assert np.array_equal(np.sort(order), np.flatnonzero(land))
