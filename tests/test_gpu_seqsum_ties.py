"""Long sums whose values tie (half-way between two sums), bit for bit against numpy's running sum: every
value a tie, ties now and then, ties from an odd and an even start, and ties between crossings."""
import numpy as np
import pytest

from cartogenesis_gb300.api import sequential_sum, sequential_sum_f64

pytestmark = pytest.mark.gpu

BLOCK = 8192


def series(kind, n, rng):
    half = 2.0 ** -13                         # half a last place of 2^40
    odd = 2.0 * rng.integers(0, 400, n) + 1.0
    if kind == "every":
        x = odd * half
    elif kind == "some":
        x = np.where(rng.random(n) < 0.01, odd, 2.0 * odd) * half
    elif kind == "signs":
        x = odd * half * rng.choice([1.0, -1.0], n)
    else:                                     # "crossings": down to the next binade and back, again and again
        x = odd * half * np.where((np.arange(n) // 700) % 2 == 0, -1.0, 1.0)
    x[0] = 2.0 ** 40 + (2.0 ** 17 if kind != "crossings" else 0.0)
    return x


@pytest.mark.parametrize("kind", ["every", "some", "signs", "crossings"])
@pytest.mark.parametrize("n", [3 * BLOCK, 5 * BLOCK + 77, 70 * BLOCK + 1])
def test_ties(kind, n):
    x = series(kind, n, np.random.default_rng(n))
    for first in (0.0, 2.0 ** -12):           # from an even and an odd sum
        y = np.concatenate([[first], x])
        want = np.float64(np.cumsum(np.concatenate([[0.0], y]))[-1])
        assert np.float64(sequential_sum_f64(y)).view(np.uint64) == want.view(np.uint64)
        f = y.astype(np.float32)
        want = np.float64(np.cumsum(np.concatenate([[0.0], f.astype(np.float64)]))[-1])
        assert np.float64(sequential_sum(f)[0]).view(np.uint64) == want.view(np.uint64)
