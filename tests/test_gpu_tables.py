"""The optional A-column table of an engine: built where there is room, used by the sweeps, given back
when the device runs out of memory, with the same bits after it is gone."""
import ctypes as C
import threading

import numpy as np
import pytest

from conftest import bf_case, bf_params, haadf_params
from internals import internals  # noqa: F401
from test_gpu_table import series

pytestmark = pytest.mark.gpu


@pytest.fixture
def hooks(internals):
    internals.t_optional_table_bytes.restype = C.c_long
    internals.t_optional_table_bytes.argtypes = [C.c_void_p]
    return internals


def held(hooks, e):
    return hooks.t_optional_table_bytes(e._h)


def haadf(mbir, n_r=40, n_t=6, views=41, **kw):
    y, ang, th = series(n_r, n_t, 12, views)
    e = mbir.Engine(haadf_params(mbir, th, **kw))
    e.set_sinogram(y, ang)
    e.prepare()
    return e


def run_steps(e, n=3):
    for k in range(n):
        e.sweep(k, 0)
        e.joint_estimation()
    return e.volume()


def test_which_engines_hold_one(lib_built, hooks):
    """FP32 levels whose voxels are detector pixels, in parallel order: 16 bytes per line and view."""
    mbir = lib_built
    with haadf(mbir) as e:
        nz, nx = e.dims()[:2]
        assert held(hooks, e) == nz * nx * 41 * 16
    for kw in ({"precision": mbir.FP64}, {"order_mode": mbir.ORDER_REFERENCE},
               {"num_resolutions": 2, "level": 0}):
        with haadf(mbir, **kw) as e:
            assert held(hooks, e) == 0
    y, ang, th = bf_case()
    for nhicd, schedule in ((1, 0), (1, 1), (0, 0)):
        with mbir.Engine(bf_params(mbir, th, nhicd=nhicd, call_schedule=schedule)) as e:
            e.set_sinogram(y, ang)
            e.prepare()
            nz, nx = e.dims()[:2]
            # a scheduled call cannot do without it
            want = 0 if nhicd and schedule == 0 else nz * nx * len(ang) * 16
            assert held(hooks, e) == want


def test_given_back_when_memory_runs_out(lib_built, hooks):
    mbir = lib_built
    with haadf(mbir) as e:
        want = run_steps(e)
    with haadf(mbir) as e, haadf(mbir, views=75, lane_shape=3) as other:
        e.sweep(0, 0)
        e.joint_estimation()
        assert held(hooks, e) > 0 and held(hooks, other) > 0
        assert hooks.t_huge_allocation_fails(0) == 1
        assert held(hooks, e) == 0 and held(hooks, other) == 0
        for k in (1, 2):
            e.sweep(k, 0)
            e.joint_estimation()
        assert np.array_equal(e.volume(), want)
        e.forward_project()


def test_given_back_between_the_colours_of_a_slab_call(lib_built, hooks):
    """A bright-field call that walks the rows, opened with the table and run without it."""
    mbir = lib_built
    y, ang, th = bf_case(n_r=48, n_t=6)
    volumes = []
    for reclaim in (False, True):
        with mbir.Engine(bf_params(mbir, th, nhicd=1, call_schedule=1)) as e:
            e.set_sinogram(y, ang)
            e.prepare()
            for k in range(3):
                e.bf_call_begin(0, k)
                e.sweep_colour(0, 0, k)
                if reclaim:
                    hooks.t_reclaim_tables(0)
                    assert held(hooks, e) == 0
                e.sweep_colour(1, 0, k)
                e.bf_call_end(e.bf_call_magnitudes())
            volumes.append(e.volume())
    assert np.array_equal(*volumes) and volumes[0].any()


def test_given_back_while_others_run(lib_built, hooks):
    """Engines on their own threads and a batch, the tables taken away again and again: the bits of
    undisturbed runs."""
    mbir = lib_built
    shapes = [(40, 6, 41, 1), (64, 5, 75, 3), (33, 4, 121, 4)]

    def make(c):
        return haadf(mbir, c[0], c[1], c[2], lane_shape=c[3])

    def all_runs():
        out, errors = {}, []

        def alone(c):
            try:
                for k in range(6):
                    with make(c) as e:
                        out[c, k] = run_steps(e, 4)
            except Exception as ex:  # noqa: BLE001
                errors.append(ex)

        def batched():
            try:
                engines = [make(c) for c in shapes]
                with mbir.Batch() as b:
                    for e in engines:
                        b.add(e)
                    for k in range(8):
                        b.sweep(k)
                    for c, e in zip(shapes, engines):
                        out["batch", c] = e.volume()
                for e in engines:
                    e.close()
            except Exception as ex:  # noqa: BLE001
                errors.append(ex)

        threads = [threading.Thread(target=alone, args=(c,)) for c in shapes]
        threads.append(threading.Thread(target=batched))
        for t in threads:
            t.start()
        return threads, out, errors

    threads, want, errors = all_runs()
    for t in threads:
        t.join()
    assert not errors
    threads, got, errors = all_runs()
    while any(t.is_alive() for t in threads):
        hooks.t_reclaim_tables(0)
    for t in threads:
        t.join()
    assert not errors
    assert set(got) == set(want)
    for k in want:
        assert np.array_equal(got[k], want[k])
