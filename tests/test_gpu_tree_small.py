"""The drainage tree on the smallest grids: two cells, four, a column and a row, every cell's donors beside it,
against the oracle."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import FlowRouting

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1, 1), (1, 2), (2, 1), (2, 2), (1, 4), (4, 1), (2, 4), (4, 4)])
@pytest.mark.parametrize("last_is_land", [False, True])
def test_one_chain(W, H, last_is_land):
    """The cells in reading order, each draining into the next, the last the sea or an outlet."""
    N = W * H
    land = np.ones((H, W), np.uint8)
    recv = np.arange(1, N + 1, dtype=np.int32).reshape(H, W)
    if H > 1 and W > 2:   # from a row's end to the next row's start, across the seam
        assert recv[0, -1] == W
    recv[-1, -1] = -1
    if not last_is_land:
        land[-1, -1] = 0
    cells = int(land.sum())
    weights = np.linspace(0.1, 1.7, N).astype(np.float32).reshape(H, W)
    got = FlowRouting.accumulate(land, recv, cells, weights)
    assert np.array_equal(got.view(np.uint32), oracle.accumulate(land, recv, cells, weights).view(np.uint32))
    assert np.array_equal(FlowRouting.drainage_order(land, recv, cells), oracle.drainage_order(land, recv, cells))
