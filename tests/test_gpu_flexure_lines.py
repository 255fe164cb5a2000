"""The plate flexure's line transform at its edges, against the oracle bit for bit: lines too short for
the register stages, line lengths with an odd and an even number of later stages, several short lines in
a CTA with the last CTA partly empty, exact and signed zeros, and loads that are not finite."""
import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import ErosionConfig, Isostasy

pytestmark = pytest.mark.gpu


def both(W, H, load):
    got = Isostasy.Flexure(ErosionConfig(W, H, 1)).deflection_metres(load)
    return got, oracle.flexure_deflection(oracle.default_params(W, H, 1), load)[0]


@pytest.mark.parametrize("W,H", [(2, 1), (2, 2), (4, 8), (8, 8), (16, 4), (32, 16), (64, 128), (512, 32), (128, 1024), (4096, 4)])
@pytest.mark.parametrize("kind", ["rough", "spikes", "flat", "minus zero"])
def test_lines_match_the_oracle(W, H, kind):
    rng = np.random.default_rng(W * 31 + H)
    load = np.zeros((H, W), np.float32)
    if kind == "rough":
        load = rng.normal(1e8, 3e7, (H, W)).astype(np.float32)
    elif kind == "spikes":   # antisymmetric about a mean of exactly 0
        load.flat[:: max(2, W * H // 8)] = 2.5e7
        load.flat[1:: max(2, W * H // 8)] = -2.5e7
    elif kind == "minus zero":
        load = -load
    got, want = both(W, H, load)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_a_load_that_is_not_finite(bad):
    load = np.random.default_rng(1).normal(1e8, 3e7, (32, 64)).astype(np.float32)
    load[7, 9] = bad
    got, want = both(64, 32, load)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isnan(got).all()
