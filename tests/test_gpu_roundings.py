"""The FP32 engine's elementwise sinogram passes give the bits of their FP64 expressions: against the
FP64 kernels that a slab's passes use, and against numpy."""
from ctypes import c_double

import numpy as np
import pytest

from internals import internals, ptr  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPE = (3, 5, 1027)  # t, theta, r


def draws(seed, e_scale, w_scale):
    rng = np.random.default_rng(seed)
    e = (rng.standard_normal(SHAPE) * e_scale).astype(np.float32)
    w = (10.0 ** rng.uniform(-1, 1, SHAPE) * w_scale).astype(np.float32)
    return rng, e, w


# ordinary magnitudes; thresholds among the values; errors whose squares are subnormal in FP32
@pytest.mark.parametrize("e_scale,w_scale,step,T", [
    (1.0, 1.0, 0.01, 1.0), (1e-3, 1e6, 1e-5, 3.0), (1e4, 1e-8, 7.0, 1.0),
    (1e-21, 1e24, 1e-23, 1e-9), (1e-22, 1e26, 0.0, 1e-9), (1e-30, 1.0, 1e-30, 1.0),
    (1e19, 1.0, 1e18, 1e19), (1e15, 1e-20, 1e10, 1e5)])
def test_offset_step_bits(internals, e_scale, w_scale, step, T):
    _, e, w = draws(1, e_scale, w_scale)
    nt, nth, nr = SHAPE
    sums = np.stack([step * np.linspace(-1, 1.3, nth), np.ones(nth)], 1).copy()
    got = []
    for fused in (1, 0):
        ee, ss = e.copy(), np.zeros(SHAPE, np.uint8)
        assert internals.t_offset_step(fused, ptr(ee), ptr(w), ptr(ss), ptr(sums), c_double(T), nth,
                                       nr, nt) == 0
        got.append((ee, ss))
    assert np.array_equal(got[0][0].view(np.uint32), got[1][0].view(np.uint32))
    assert np.array_equal(got[0][1], got[1][1])
    st = (sums[:, 0] / sums[:, 1])[None, :, None]
    want = (e.astype(np.float64) - st).astype(np.float32)
    assert np.array_equal(got[0][0].view(np.uint32), want.view(np.uint32))
    e64 = want.astype(np.float64)
    assert np.array_equal(got[0][1] != 0, e64 * e64 * w.astype(np.float64) < T * T)


# variances and their inverses at both ends of FP32, weights at the other end
@pytest.mark.parametrize("alpha,upd,w_scale", [
    (1.0, 1.3, 1.0), (0.37, 0.21, 1e3), (1e-34, 1e-30, 1e20), (3e-38, 1e-20, 1e25),
    (1e-40, 1e-3, 1e30), (1e30, 1e33, 1e-5), (1.0, 7e37, 1e20), (1e38, 1e3, 1e-30),
    (0.0, 1.0, 1.0)])
def test_new_weights_bits(internals, alpha, upd, w_scale):
    rng, e, w = draws(2, 1.0, w_scale)
    nt, nth, nr = SHAPE
    a = alpha * rng.uniform(0.5, 2.0, nth)
    sums, count, dT, T = np.array([0.75 * upd, 0.25 * upd]), 1.0, 1.0, 1.0
    got = []
    for fused in (1, 0):
        ww, ss = w.copy(), np.zeros(SHAPE, np.uint8)
        assert internals.t_new_weights(fused, ptr(e), ptr(ww), ptr(ss), ptr(a), ptr(sums),
                                       c_double(dT), c_double(count), c_double(T), nth, nr, nt) == 0
        got.append((ww, ss))
    u = (sums[0] + dT * sums[1]) / count
    with np.errstate(over="ignore"):
        w1 = (w.astype(np.float64) * a[None, :, None]).astype(np.float32)
        want = (w1.astype(np.float64) / u).astype(np.float32)
    for ww, ss in got:
        assert np.array_equal(ww.view(np.uint32), want.view(np.uint32))
        e64 = e.astype(np.float64)
        assert np.array_equal(ss != 0, e64 * e64 * want.astype(np.float64) < T * T)


@pytest.mark.parametrize("scale,gain,gain_ratio", [
    (1.0, 1.0, 1.01), (1e4, 3.7, 0.98), (1e-3, 0.2, 1.0), (1.0, 1e-36, 1e3), (1.0, 1e20, 1e-33)])
def test_rebuild_error_bits(internals, scale, gain, gain_ratio):
    rng, e, _ = draws(3, 0.1 * scale, 1.0)
    nt, nth, nr = SHAPE
    y = (rng.uniform(0, 2, SHAPE) * scale).astype(np.float32)
    mo = rng.standard_normal(nth) * 0.1 * scale
    mn = mo * rng.uniform(0.9, 1.1, nth)
    go = gain * rng.uniform(0.5, 2.0, nth)
    gn = go * gain_ratio * rng.uniform(0.99, 1.01, nth)
    got = e.copy()
    assert internals.t_rebuild_error(ptr(y), ptr(got), ptr(mo), ptr(go), ptr(mn), ptr(gn), nth, nr,
                                     nt) == 0
    c = lambda v: v[None, :, None]
    y64 = y.astype(np.float64)
    yh = (y64 - e.astype(np.float64) - c(mo)) / c(go)
    want = (y64 - c(mn) - c(gn) * yh).astype(np.float32)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
