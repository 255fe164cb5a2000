"""The fill's chains where a thread reaches their cells long before it reaches the cells they run through: a
channel through the whole of a map larger than the GPU's threads, planes that fall down and up the map, and
chains just about as long as one cell's share of steps. The levels are the oracle's, and the long chains take
no more than a few times a short one's time."""
import time

import numpy as np
import pytest

import oracle
from cartogenesis_gb300 import FlowRouting
from test_gpu_fill_chains import serpentine

pytestmark = pytest.mark.gpu


def bits(a):
    return a.view(np.uint32)


def plane(W, H, length):
    """Slopes of `length` rows down the map, one below the other, each to its own row of sea."""
    y = np.mgrid[0:H, 0:W][0]
    rel = (0.8 - 0.5 * (y % length) / length).astype(np.float32)
    land = np.ones((H, W), np.uint8)
    land[length - 1::length] = 0
    land[-1] = 0
    return land, rel


@pytest.mark.parametrize("length", [2, 31, 33, 34, 35, 543, 561, 600, 1024])
@pytest.mark.parametrize("W,H", [(64, 1024), (1024, 1024)])
@pytest.mark.parametrize("up", [False, True])
def test_chain_lengths(W, H, length, up):
    land, rel = plane(W, H, length)
    if up:
        land, rel = np.ascontiguousarray(land[::-1]), np.ascontiguousarray(rel[::-1])
    rel[H // 2, W // 3] -= np.float32(0.05)   # and a pit on the way
    assert np.array_equal(bits(FlowRouting.fill_depressions(land, rel)), bits(oracle.fill_depressions(land, rel)))


def least_ms(land, rel):
    FlowRouting.fill_depressions(land, rel)
    took = []
    for _ in range(3):
        t = time.perf_counter()
        FlowRouting.fill_depressions(land, rel)
        took.append(time.perf_counter() - t)
    return 1e3 * min(took)


@pytest.mark.parametrize("into_pit", [False, True])
def test_a_channel_through_the_map(into_pit):
    W, H = 2048, 1024
    land, rel = serpentine(W, H, into_pit)
    got = FlowRouting.fill_depressions(land, rel)
    assert np.array_equal(bits(got), bits(oracle.fill_depressions(land, rel)))
    short = least_ms(*plane(W, H, 64))
    assert least_ms(land, rel) < 20.0 * short   # half a million cells a step each take over a thousand times
