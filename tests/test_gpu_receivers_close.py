"""The facet rule on square cells where its single-precision slopes cannot tell the facets apart or do not
apply: planes whose facets tie on slope, slopes a few units in the last place apart, falls below 2^-60 and
above 2^60, shares next to 0 and 1, and grids two and four cells wide, against the oracle."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import FlowRouting

pytestmark = pytest.mark.gpu


def relief(kind, W, H, rng):
    y, x = np.mgrid[0:H, 0:W].astype(np.float64)
    if kind == "planes":      # 3:4 gradients: an inside facet's slope ties with 5, diagonals with 1:1
        return np.where((x // 16 + y // 16) % 2 == 0, 3 * x + 4 * y, np.where(y < H / 2, x + y, 4 * y - x)) / 1024 + 1.0
    if kind == "nearly":      # a cone: every share, slopes nearly the same all around, in steps of 2^-24
        return 2.0 - np.round(np.hypot(x - W / 2, y - H / 2) / 64 * 2**20) / 2**20 + rng.integers(0, 3, (H, W)) * 2.0**-23
    if kind == "terraces":    # outward falls of a last place beside falls of a terrace
        return 1.0 + np.floor(y / 2) / 8 + rng.integers(0, 2, (H, W)) * 2.0**-23
    return rng.integers(1, 6, (H, W)).astype(np.float64)   # "steps": small whole numbers, ties everywhere


@pytest.mark.parametrize("W,H", [(2, 16), (4, 8), (128, 64)])
@pytest.mark.parametrize("kind", ["planes", "nearly", "terraces", "steps"])
@pytest.mark.parametrize("scale", [1.0, 2.0**-75, 2.0**75])
def test_close_facets(W, H, kind, scale):
    rel = (relief(kind, W, H, np.random.default_rng(W + H)) * scale).astype(np.float32)
    land = np.ones((H, W), np.uint8)
    land[0] = land[H // 3] = 0
    want, _ = oracle.flow_directions(land, rel, rel, 9, 1.0, 214, True, False)
    got, _ = FlowRouting.flow_directions(land, rel, rel, 9, 1.0, 214, True, False)
    assert np.array_equal(got, want)
