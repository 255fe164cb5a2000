"""Sums told apart by predicted binades, bit for bit against numpy's running sum: around the sizes where one
CTA stops taking them whole, blocks with a few, hundreds and too many values to take alone, sums that sit on
powers of two, that cancel far below the magnitudes before them, and unaligned and masked fields."""
import numpy as np
import pytest

from cartogenesis_gb300.api import sequential_sum, sequential_sum_f64

pytestmark = pytest.mark.gpu

BLOCK = 8192
SIZES = [3 * BLOCK - 1, 3 * BLOCK, 3 * BLOCK + 1, 7 * BLOCK + 5, 33 * BLOCK, 40 * BLOCK + 4095]


def running(x):
    return np.float64(np.cumsum(np.concatenate([[0.0], x.astype(np.float64)]))[-1])


def series(kind, n, rng):
    if kind == "walk":          # a random walk: hundreds of crossings near zero, few far from it
        return rng.normal(0.0, 1e7, n)
    if kind == "flips":         # back and forth across zero at every value
        return np.where(np.arange(n) % 2 == 0, 1.0, -1.0) * rng.uniform(0.9, 1.1, n) * 3.0
    if kind == "powers":        # ones: the sum stands on every power of two
        return np.ones(n)
    if kind == "cancel":        # up by whole blocks and down again to almost nothing
        return np.where((np.arange(n) // (2 * BLOCK)) % 2 == 0, 1.0, -1.0) * rng.uniform(1.0, 1.0 + 1e-6, n)
    return np.concatenate([[2.0 ** 40], rng.normal(0.0, 2.0 ** -13, n)])[:n]   # "small": far below the sum's last places


KINDS = ["walk", "flips", "powers", "cancel", "small"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", SIZES)
def test_floats_with_and_without_a_mask(kind, n):
    rng = np.random.default_rng(n)
    x = series(kind, n, rng).astype(np.float32)
    mask = (rng.random(n) < 0.5).astype(np.uint8)
    got, _ = sequential_sum(x)
    assert np.float64(got).view(np.uint64) == running(x).view(np.uint64)
    got, _ = sequential_sum(x, mask)
    assert np.float64(got).view(np.uint64) == running(x[mask != 0]).view(np.uint64)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", SIZES)
def test_doubles(kind, n):
    x = series(kind, n, np.random.default_rng(n + 1))
    assert np.float64(sequential_sum_f64(x)).view(np.uint64) == running(x).view(np.uint64)
