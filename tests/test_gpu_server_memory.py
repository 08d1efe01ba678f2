"""A server's memory account with the requests' optional A-column tables."""
import time

import numpy as np
import pytest

from conftest import bf_case, bf_params, haadf_params
from test_gpu_table import series

pytestmark = pytest.mark.gpu


def haadf(mbir, n_r=40, n_t=64, views=41, **kw):
    y, ang, th = series(n_r, n_t, 12, views)
    return haadf_params(mbir, th, **kw), y, ang


def bright_field(mbir, **kw):
    y, ang, th = bf_case(n_r=48, n_t=40)
    return bf_params(mbir, th, **kw), y, ang


def dims(mbir, req):
    p, y, ang = req
    with mbir.Engine(p) as e:
        e.set_sinogram(y, ang)
        return e.dims()[:3]


def own_bytes(mbir, req):
    """The footprint without the table: the peak of a server whose budget has no room for one."""
    lo, hi = 1 << 20, 1 << 30
    p, y, ang = req
    while hi - lo > 1:  # the smallest budget that takes the request
        mid = (lo + hi) // 2
        with mbir.Server(0, mid, 1) as s:
            try:
                s.wait(s.submit(p, y, ang, max_outer=1, tol=0.0))
                hi = mid
            except mbir.MbirError:
                lo = mid
    return hi


def peak(mbir, req, budget):
    p, y, ang = req
    with mbir.Server(0, budget, 1) as s:
        s.wait(s.submit(p, y, ang, max_outer=1, tol=0.0))
        return s.stats().peak_bytes


@pytest.mark.parametrize("kind", ["haadf", "bf-no-nhicd", "bf-row-walk", "bf-scheduled", "coarse"])
def test_peak_counts_the_table(lib_built, kind):
    """peak_bytes is the largest estimated footprint resident at one time: the request's own arrays
    and its table, where it has one."""
    mbir = lib_built
    req = {"haadf": haadf, "bf-no-nhicd": lambda m: bright_field(m, nhicd=0),
           "bf-row-walk": lambda m: bright_field(m, call_schedule=1),
           "bf-scheduled": bright_field,
           "coarse": lambda m: haadf(m, num_resolutions=2, level=0)}[kind](mbir)
    nz, nx, _ = dims(mbir, req)
    table = 0 if kind in ("bf-scheduled", "coarse") else nz * nx * len(req[2]) * 16
    own = own_bytes(mbir, req)
    assert peak(mbir, req, own) == own  # no room for a table
    assert peak(mbir, req, 2 * (own + table) - 1) == (own if table else own)
    assert peak(mbir, req, 2 * (own + table)) == own + table
    assert peak(mbir, req, 0) == own + table


@pytest.mark.parametrize("n_t", [15, 16])
def test_thin_requests_take_none(lib_built, n_t):
    """Series of fewer than 16 slices build no table in a server."""
    mbir = lib_built
    req = haadf(mbir, n_r=128, n_t=n_t, views=61)
    nz, nx, ny = dims(mbir, req)
    assert ny == n_t
    own = own_bytes(mbir, req)
    assert peak(mbir, req, 0) == own + (nz * nx * 61 * 16 if n_t >= 16 else 0)


def test_tables_make_way_for_an_arrival(lib_built):
    """A request whose own arrays fit beside those of an active one joins it: the active one's table,
    which takes the room, goes back, and its result keeps every bit."""
    mbir = lib_built
    first, second = haadf(mbir), haadf(mbir, n_t=96)
    nz, nx, _ = dims(mbir, first)
    table = nz * nx * len(first[2]) * 16
    own1, own2 = own_bytes(mbir, first), own_bytes(mbir, second)
    budget = own1 + own2 + table // 2
    assert own1 + table <= budget // 2  # the first is granted its table
    outers = 1500
    with mbir.Server(0, own1, 1) as s:
        rid = s.submit(*first, max_outer=outers, tol=0.0)
        s.wait(rid)
        want = s.result(rid)
    with mbir.Server(0, budget, 2) as s:
        r1 = s.submit(*first, max_outer=outers, tol=0.0)
        t0 = time.monotonic()
        while s.poll(r1)[0] == 0 and time.monotonic() - t0 < 60:
            time.sleep(0.001)
        assert s.stats().peak_bytes == own1 + table
        r2 = s.submit(*second, max_outer=2, tol=0.0)
        s.wait(r2)
        assert s.poll(r1)[0] == 1  # the first still runs
        st = s.stats()
        assert st.peak_active == 2 and st.peak_bytes <= budget
        s.wait(r1)
        assert np.array_equal(s.result(r1), want)
