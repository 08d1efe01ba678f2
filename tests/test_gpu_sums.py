"""The bright-field sums of the FP32 engine against exact rational arithmetic."""
from ctypes import c_double
from fractions import Fraction

import numpy as np
import pytest

from internals import f64, internals, ptr  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_theta,n_r,n_t", [(1, 1, 1), (1, 2, 1), (2, 5, 1), (3, 33, 2)])
@pytest.mark.parametrize("kind", ["variance", "cost"])
def test_selected_terms_keep_fp64_precision(internals, kind, n_theta, n_r, n_t):
    """Every term e^2 w is held to more than the 53 bits of an FP64 product: what the sum of n
    selected entries is off by is the rounding of one FP64 value per thread and one FP64 addition
    per further entry, at most (n + 1) 2^-53 of the sum of magnitudes."""
    rng = np.random.default_rng(n_r)
    shape = (n_t, n_theta, n_r)
    worst = 0.0
    for _ in range(64):
        e = (rng.standard_normal(shape) * 3).astype(np.float32)
        w = rng.uniform(0.5, 2.0, shape).astype(np.float32)
        sel = np.ones(shape, np.uint8)
        alpha = np.ones(n_theta)
        out = f64(2)
        rc = internals.t_bf_sums(0 if kind == "variance" else 1, ptr(e), ptr(w), ptr(sel),
                                 ptr(alpha), c_double(3.0), c_double(0.5), n_theta, n_r, n_t,
                                 ptr(out))
        assert rc == 0
        exact = sum(Fraction(float(a)) ** 2 * Fraction(float(b))
                    for a, b in zip(e.ravel(), w.ravel()))
        worst = max(worst, float(abs(Fraction(float(out[0])) - exact) / exact))
    assert worst <= (e.size + 1) * 2.0 ** -53
