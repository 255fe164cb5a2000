"""The fill's chains to an outlet at their longest and shortest, against the oracle bit for bit: a
serpentine channel descending through the whole map to one outlet, the same channel ending in a pit, a
plain slope, and grids a cell or two tall."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import FlowRouting

pytestmark = pytest.mark.gpu


def serpentine(W, H, into_pit):
    """Corridors every other row, joined at alternating ends, walls between them; the sea is one cell."""
    rel = np.full((H, W), 0.9, np.float32)
    land = np.ones((H, W), np.uint8)
    path = []
    for k, row in enumerate(range(2, H - 2, 2)):
        cols = range(1, W - 1) if k % 2 == 0 else range(W - 2, 0, -1)
        path += [(row, c) for c in cols]
        if row + 2 < H - 2:
            path.append((row + 1, path[-1][1]))
    falls = np.linspace(0.8, 0.1, len(path)).astype(np.float32)
    for (r, c), z in zip(path, falls):
        rel[r, c] = z
    if not into_pit:
        land[path[-1]] = 0
        rel[path[-1]] = 0.0
    return land, rel


@pytest.mark.parametrize("W,H", [(64, 64), (512, 128), (2048, 16)])
@pytest.mark.parametrize("into_pit", [False, True])
def test_long_chains(W, H, into_pit):
    land, rel = serpentine(W, H, into_pit)
    want = oracle.fill_depressions(land, rel)
    got = FlowRouting.fill_depressions(land, rel)
    got = got[0] if isinstance(got, tuple) else got
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("W,H", [(64, 1), (64, 2), (8, 4), (1024, 512)])
def test_slopes(W, H):
    y, x = np.mgrid[0:H, 0:W]
    rel = (0.2 + 0.5 * np.abs(x - W / 2) / W + 0.1 * y / H).astype(np.float32)
    land = np.ones((H, W), np.uint8)
    land[:, W // 2] = 0
    want = oracle.fill_depressions(land, rel)
    got = FlowRouting.fill_depressions(land, rel)
    got = got[0] if isinstance(got, tuple) else got
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
