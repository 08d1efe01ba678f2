"""A sweep's statistics are the slices' values summed in row order."""
import numpy as np
import pytest

from internals import f64, internals, ptr  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rows", [1, 2, 31, 32, 33, 64, 257, 1000])
def test_statistics_in_row_order(internals, n_rows):
    """Values whose sums need more than 53 bits: the order of the additions shows."""
    rng = np.random.default_rng(n_rows)
    x = np.round(rng.uniform(0, 2.0 ** 24, (n_rows, 4)) * 2.0 ** 32) / 2.0 ** 32
    out = f64(4)
    assert internals.t_reduce_stats(ptr(x), n_rows, 4, ptr(out)) == 0
    want = np.zeros(4)
    for row in x:
        want = want + row
    assert np.array_equal(out, want)


@pytest.mark.parametrize("n_rows", [1, 33, 256])
def test_small_statistics(internals, n_rows):
    """Sums below 2^21, which are exact in any order, and just above it."""
    rng = np.random.default_rng(n_rows)
    x = np.round(rng.uniform(0, 2.0 ** 20 / n_rows, (n_rows, 4)) * 2.0 ** 32) / 2.0 ** 32
    x[:, 1] *= 4
    x[:, 2] = rng.integers(0, 8192, n_rows)
    x[0, 3] = 2.0 ** 21 - 2.0 ** -32
    out = f64(4)
    assert internals.t_reduce_stats(ptr(x), n_rows, 4, ptr(out)) == 0
    want = np.zeros(4)
    for row in x:
        want = want + row
    assert np.array_equal(out, want)
