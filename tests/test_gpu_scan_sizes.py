"""The prefix sum over the grid's cells, seen through the basins' labels (every ponded cell alone, so a basin's
label is the number of ponded cells before it), on both sides of a tile and of the number of tiles whose sums
each CTA adds up itself, with the sums scanned on their own beyond."""
import numpy as np
import pytest

from cartogenesis_gb300 import FlowRouting

pytestmark = pytest.mark.gpu

SIZES = [(2, 4), (64, 32), (64, 64), (128, 64), (1024, 512), (4096, 4096), (8192, 4096), (8192, 8192)]


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("share", [0.02, 0.9])
def test_labels(W, H, share):
    rng = np.random.default_rng(W * 3 + H)
    ponded = np.zeros((H, W), bool)
    ponded[::2, ::2] = rng.random((H // 2, W // 2)) < share   # apart from one another
    rel = np.zeros((H, W), np.float32)
    filled = ponded.astype(np.float32)
    out = FlowRouting.spillways(np.ones((H, W), np.uint8), rel, filled, np.full((H, W), -1, np.int32), 0.5)
    want = np.where(ponded, np.cumsum(ponded, dtype=np.int32).reshape(H, W) - 1, -1)
    assert out["count"] == ponded.sum()
    assert np.array_equal(out["labels"], want)
    assert (out["cells"] == 1).all()
