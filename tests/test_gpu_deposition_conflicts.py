"""Worlds whose deposition has conflicted mouths (a lake fan laid on a ponded cell of its own level ranked
after it), refitted at their turn, and grids whose sea lobes wrap around or span the map, against the
oracle's stage bit for bit."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import ErosionConfig, ErosionStage, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,seed,conflicts", [(2048, 1024, 3, True), (2048, 1024, 8, True), (64, 256, 5, False),
                                                (16, 64, 2, False), (8, 32, 2, False)])
def test_conflicted_mouths_match_the_oracle(W, H, seed, conflicts):
    h, up, rk = synthetic.world(W, H, seed, uplift="ridges")
    options = dict(sea_level=0.6, profile=2, hydraulic_rounds=2)
    got = ErosionStage.apply(ErosionConfig(W, H, seed, **options), h, up, rk, want=("receivers",))
    want = oracle.erode_stage(oracle.default_params(W, H, seed, **options), h, up, rk, want=("receivers",))
    assert np.array_equal(got.height.view(np.uint32), want["height"].view(np.uint32))
    assert np.array_equal(got.receivers, want["receivers"])
    assert not conflicts or sum(s["deposit_redone"] for s in got.stats) > 0
