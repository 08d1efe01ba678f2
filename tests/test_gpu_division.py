"""The division of the gain/offset sums against numpy's (IEEE, correctly rounded): the same bits."""
import numpy as np
import pytest

from internals import internals, ptr  # noqa: F401

pytestmark = pytest.mark.gpu

N = 1 << 20


def divide(internals, x, g):
    q = np.empty_like(x)
    assert internals.t_div_by(ptr(x), ptr(g), ptr(q), x.size) == 0
    with np.errstate(all="ignore"):
        want = x / g
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(q))
    assert np.array_equal(q[~nan].view(np.uint64), want[~nan].view(np.uint64))


def mantissas(rng, n):
    """Random ones, and the neighbourhoods of 1, 2 and the midpoint, where rounding is closest."""
    m = 1.0 + rng.random(n)
    near = rng.integers(0, 4, n)
    k = rng.integers(0, 4, n).astype(np.float64) * 2.0 ** -52
    return np.where(near == 0, m, np.where(near == 1, 1.0 + k, np.where(near == 2, 2.0 - 2.0 ** -52
                                                                        - k, 1.5 + k)))


# measurements and gains as they come; whole exponent range; its ends on either or both sides
@pytest.mark.parametrize("ex,eg", [
    ((-30, 30), (-10, 10)), ((-1074, 1023), (-1074, 1023)), ((590, 625), (-625, -590)),
    ((-625, -590), (590, 625)), ((395, 405), (-405, -395)), ((-405, -395), (395, 405)),
    ((-1074, -1000), (-30, 30)), ((1000, 1023), (-30, 30))])
def test_quotients_are_correctly_rounded(internals, ex, eg):
    rng = np.random.default_rng(abs(ex[0]) + abs(eg[0]))
    x = np.ldexp(mantissas(rng, N), rng.integers(ex[0], ex[1], N).astype(np.int32))
    g = np.ldexp(mantissas(rng, N), rng.integers(eg[0], eg[1], N).astype(np.int32))
    divide(internals, x * rng.choice([-1.0, 1.0], N), g * rng.choice([-1.0, 1.0], N))


def test_special_values(internals):
    v = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -3.0, 5e-324, 1.7e308, 2.0 - 2.0 ** -52])
    x, g = (a.ravel().copy() for a in np.meshgrid(v, v))
    divide(internals, x, g)
