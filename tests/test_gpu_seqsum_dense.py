"""Sums that leave their binade at nearly every value, as a load of alternating sign makes them: whole fields of
them, runs of them between quiet stretches, masked and in double terms, bit for bit against numpy's running
sum, in a time of the order of one addition after another."""
import time

import numpy as np
import pytest

from cartogenesis_gb300.api import sequential_sum, sequential_sum_f64

pytestmark = pytest.mark.gpu

BLOCK = 8192
SIZES = [7, 129, 1023, BLOCK - 1, 3 * BLOCK, 3 * BLOCK + 130, 9 * BLOCK + 77]


def running(x):
    return np.float64(np.cumsum(np.concatenate([[0.0], x.astype(np.float64)]))[-1])


def series(kind, n, rng):
    sign = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    if kind == "alternating":    # back to zero at every second value
        return sign * 1e7
    if kind == "noisy":
        return sign * rng.uniform(0.9, 1.1, n)
    if kind == "teeth":          # four up, four down
        return np.where(np.arange(n) % 8 < 4, 1.0, -1.0) * rng.uniform(1.0, 1.0 + 1e-6, n)
    if kind == "bursts":         # runs of 50 to 300 alternating values from a sum near zero, ones far from it between
        x = np.zeros(n)
        i = 0
        while i < n:
            k = int(rng.integers(50, 300))
            x[i:i + k] = sign[i:i + k] * rng.uniform(0.5, 2.0, len(x[i:i + k]))
            i += k
            k = int(rng.integers(1, 400))
            x[i:i + k] = rng.choice([0.0, 1e-3, 1.0], len(x[i:i + k]))
            x[i + k - 1:i + k] = -x[:i + k - 1].sum()
            i += k
        return x
    x = sign * rng.uniform(0.5, 2.0, n)   # "ends": to infinity and to NaN on the way
    x[n // 2:] = np.where(np.arange(n - n // 2) % 2 == 0, 3e38, -3e38)
    x[n - n // 4:] = np.inf
    x[n - n // 8:] = -np.inf
    return x


KINDS = ["alternating", "noisy", "teeth", "bursts", "ends"]


def same(got, want):
    return np.float64(got).view(np.uint64) == want.view(np.uint64) or (np.isnan(got) and np.isnan(want))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", SIZES)
def test_sums(kind, n):
    rng = np.random.default_rng(n)
    x = series(kind, n, rng)
    f = x.astype(np.float32)
    mask = (rng.random(n) < 0.7).astype(np.uint8)
    with np.errstate(invalid="ignore", over="ignore"):
        assert same(sequential_sum(f)[0], running(f))
        assert same(sequential_sum(f, mask)[0], running(f[mask != 0]))
        assert same(sequential_sum_f64(x), running(x))


def test_a_field_of_alternating_sign():
    n = 1 << 19
    x = series("alternating", n, None).astype(np.float32)
    assert sequential_sum(x)[0] == 0.0
    took = []
    for _ in range(3):
        t = time.perf_counter()
        sequential_sum(x)
        took.append(time.perf_counter() - t)
    assert min(took) < n * 150e-9   # an addition takes some 40 ns, a window for every value 500
