"""One filled pit of each size at which the flat solvers change form or a warp's or a CTA's share of the
members is just full (segments of 4 to 32 lanes, a CTA of 128 threads, a cluster of eight CTAs), as a
square, a wall one cell wide down a column and one along a row, on square cells (every weight exactly 1)
and on cells half as tall, against the oracle: receivers exact, the routing surface to 1e-12."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300.api import FlowRouting

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 64, 96, 97, 128, 129, 256, 257, 511, 512, 513, 1500]


def pit(cells, shape, rng):
    """Land sloping to a sea on the north, with a pit of `cells` cells behind a sill."""
    W, H = 256, 1024
    land = np.ones((H, W), np.uint8)
    land[:4] = 0
    y = np.arange(H)[:, None]
    rel = (0.05 + 0.0004 * y + 1e-5 * rng.random((H, W))).astype(np.float32)
    rel[:4] = -0.1
    w = {"square": int(np.ceil(np.sqrt(cells))), "column": 1, "row": min(cells, 200)}[shape]
    k = np.arange(cells)
    rows, cols = 40 + (k // w if shape != "column" else k % 900), 30 + (k % w if shape != "column" else k // 900)
    rel[rows, cols] = np.float32(0.05) + np.float32(1e-4) * rng.random(cells).astype(np.float32)
    return land, rel


@pytest.mark.parametrize("shape", ["square", "column", "row"])
@pytest.mark.parametrize("r", [1.0, 0.5])
def test_flat_of_each_size(shape, r):
    rng = np.random.default_rng(5)
    for cells in SIZES:
        land, rel = pit(cells, shape, rng)
        filled = oracle.fill_depressions(land, rel)
        want, wsurf, wc = oracle.flow_directions(land, rel, filled, 7, r, 214, want_surface=True)
        got, gsurf, gc = FlowRouting.flow_directions(land, rel, filled, 7, r, 214, want_surface=True)
        assert list(wc) == list(gc), cells
        np.testing.assert_allclose(gsurf, wsurf, rtol=1e-12, atol=0, err_msg=str(cells))
        assert np.array_equal(got, want), cells
