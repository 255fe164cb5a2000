"""The sequential sums on both sides of the size where one CTA stops taking them whole (three blocks of 8192
values): the runs that leave a binade often, and the belts' five totals side by side, whose lengths differ (a
belt at that size, and a frontier of none, one or two cells beside it), against numpy and the oracle."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import BeltErosion, BeltWindow, ErosionConfig, synthetic
from cartogenesis_gb300.api import sequential_sum, sequential_sum_f64
from test_gpu_belt import check
from test_gpu_seqsum_runs import BLOCK, KINDS, running, series

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [3 * BLOCK - 1, 3 * BLOCK, 3 * BLOCK + 1, 4 * BLOCK + 77])
def test_values_and_terms(kind, n):
    x = series(kind, n, np.random.default_rng(n))
    f = x.astype(np.float32)
    assert np.float64(sequential_sum(f)[0]).view(np.uint64) == running(f).view(np.uint64)
    if kind == "overflow":
        x = np.where(x > 1e38, 1.7e308, x)
    with np.errstate(over="ignore"):
        assert np.float64(sequential_sum_f64(x)).view(np.uint64) == running(x).view(np.uint64)


@pytest.mark.parametrize("cells", [3 * BLOCK - 1, 3 * BLOCK, 3 * BLOCK + 1, 256 * 128 - 2, 256 * 128 - 1, 256 * 128])
@pytest.mark.parametrize("travel_km", [0.0, 1875.0])
def test_the_belts_totals(cells, travel_km):
    W, H, seed = 256, 128, 5
    h, up, rk = synthetic.world(W, H, seed)
    belt = (np.arange(W * H) < cells).reshape(H, W)
    tectonic = np.where(belt, 4.0 + 30.0 * up, 0.0).astype(np.float32)
    wear = (0.3 * tectonic).astype(np.float32)
    onset = np.where(belt, 5.0, -1.0).astype(np.float32)
    scale = dict(sea_level=0.4, critical_fall_metres_per_km=2.0, debris_travel_km=travel_km)
    surface = h.copy()
    got = BeltErosion.replay(ErosionConfig(W, H, seed, **scale), surface, BeltWindow(tectonic, wear, onset, 6.0), up, None, None,
                             rk)
    want_h, want_e, want = oracle.belt_replay(oracle.default_params(W, H, seed, **scale), h, tectonic, wear, onset, 6.0,
                                              uplift=up, rock=rk)
    assert got.belt_cells == cells and got.rounds > 1
    check(surface, got, want_h, want_e, want)
