"""The sequential double sums at the sizes where their form changes (one CTA from the first value up to
ten blocks of 8192 values, blocks reduced in parallel and chained beyond) and on runs that leave a
binade often, bit for bit against numpy's running sum: a sum that wanders around zero, whole blocks of
zeros, powers of two left by terms below half an ulp, ties in double terms, and sums that reach
infinity."""
import numpy as np
import pytest

from cartogenesis_gb300.api import sequential_sum, sequential_sum_f64

pytestmark = pytest.mark.gpu

BLOCK = 8192
SIZES = [1, 31, 33, BLOCK - 1, BLOCK + 1, 10 * BLOCK - 1, 10 * BLOCK, 10 * BLOCK + 1, 43 * BLOCK + 17]


def running(x):
    """s = 0.0, then s += v in order (so a first -0 leaves +0)."""
    return np.float64(np.cumsum(np.concatenate([[0.0], x.astype(np.float64)]))[-1])


def series(kind, n, rng):
    if kind == "wander":        # changes sign and binade all along
        return rng.choice([1.0, -1.0], n) * rng.uniform(0.5, 2.0, n)
    if kind == "sparse":        # mostly zeros of both signs, as the belts' exports are
        x = np.where(rng.random(n) < 0.01, rng.exponential(1e7, n), 0.0)
        return np.where(rng.random(n) < 0.5, x, np.where(x == 0.0, -0.0, x))
    if kind == "quiet":         # nothing for blocks on end, then a few values
        x = np.zeros(n)
        x[n // 2:: max(n // 7, 1)] = -3.0
        return x
    if kind == "powers":        # a power of two, then steps down of less than its ulp and back
        return np.concatenate([[2.0 ** 30], np.tile([-(2.0 ** -24), 2.0 ** -24, -(2.0 ** -22)], n // 3 + 1)])[:n]
    if kind == "ties":
        return np.concatenate([[2.0 ** 53 - 3.0], rng.choice([0.5, -0.5, 1.5, -1.5, 1.0], n)])[:n]
    if kind == "growing":       # from nothing, every term above all before it for a while
        return 2.0 ** np.minimum(np.arange(n) * 0.7, 100.0) * rng.uniform(0.9, 1.1, n)
    x = rng.normal(0.0, 1.0, n)   # "overflow": leaves the finite range and stays there
    x[n // 2] = 3e38
    x[n // 2 + n // 4:] = 3e38
    return x


KINDS = ["wander", "sparse", "quiet", "powers", "ties", "growing", "overflow"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", SIZES)
def test_float_values(kind, n):
    x = series(kind, n, np.random.default_rng(n)).astype(np.float32)
    got, _ = sequential_sum(x)
    assert np.float64(got).view(np.uint64) == running(x).view(np.uint64)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", SIZES)
def test_double_terms(kind, n):
    x = series(kind, n, np.random.default_rng(n + 1))
    if kind == "overflow":
        x = np.where(x > 1e38, 1.7e308, x)
    got = sequential_sum_f64(x)
    with np.errstate(over="ignore"):
        assert np.float64(got).view(np.uint64) == running(x).view(np.uint64)
