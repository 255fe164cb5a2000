"""The sea-level cut's bracket (the cells of the histogram bin that holds the answer) at the sizes where
its sort changes form, and its histogram walk where the answer lies at an end of the histogram, against
the oracle: shoreline, land and relative field bit for bit."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import SeaLevelStage

pytestmark = pytest.mark.gpu

W, H = 512, 256


def check(h, sea_level):
    s0, l0, r0, n0 = oracle.percentile_cut(h, sea_level, 0.0)
    s1, l1, r1, n1 = SeaLevelStage.percentile_cut(h, sea_level, 0.0)
    assert np.float32(s0).view(np.uint32) == np.float32(s1).view(np.uint32)
    assert n0 == n1 and np.array_equal(l0, l1) and np.array_equal(r0.view(np.uint32), r1.view(np.uint32))


@pytest.mark.parametrize("cells", [1, 2, 3, 4, 5, 31, 33, 4097, 16383, 16384, 16385, 40000])
def test_bracket_of(cells):
    """Half the planet below one bin's cells and half above, so the answer is among them; equal heights too."""
    rng = np.random.default_rng(cells)
    n = W * H
    h = np.where(rng.random(n) < 0.5, rng.uniform(0.0, 0.49, n), rng.uniform(0.51, 1.0, n))
    h[0], h[1] = 0.0, 1.0
    at = 2 + rng.permutation(n - 2)[:cells]
    h[at] = 0.5001 + 1e-5 * rng.integers(0, 12, cells) / 12.0
    check(h.astype(np.float32).reshape(H, W), 0.5)


@pytest.mark.parametrize("sea_level", [1e-6, 1e-4, 0.5, 0.9999, 1.0])
def test_steep_histogram(sea_level):
    """Bins that each hold more than all before them, and empty bins between them."""
    rng = np.random.default_rng(3)
    h = (2.0 ** rng.uniform(-14.0, 0.0, W * H)).astype(np.float32).reshape(H, W)
    check(h, sea_level)
