"""Rows so long that the table-driven row walk's shared memory does not fit its kernel while the
general kernel's does (few views): sweeps, shape trials and batches run, as they do at other widths."""
import numpy as np
import pytest

from conftest import bf_case, bf_params, haadf_params
from test_gpu_bf import sync_oracle
from test_gpu_table import rel, series

pytestmark = pytest.mark.gpu


# slices in HBM: 21 and 31 views; staged: 9 and 15 views (below and above the windows too)
@pytest.mark.parametrize("n_r,n_t,views", [
    (3740, 2, 21), (3800, 2, 21), (3860, 1, 21), (3790, 2, 31), (2350, 2, 9), (2400, 3, 9),
    (2430, 2, 9), (1908, 2, 15)])
def test_long_rows_match_oracle(lib_built, oracle_mod, n_r, n_t, views):
    """Tolerance as for the sweeps of other widths (test_sweep_and_projection_match_oracle)."""
    mbir = lib_built
    y, ang, th = series(n_r, n_t, 4, views)
    p = haadf_params(mbir, th, use_default_offset=1, lane_shape=0)
    o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
    with mbir.Engine(p) as e:
        e.set_sinogram(y, ang)
        e.prepare()
        o.prepare()
        rows, stride = e.schedule(0)
        sg = e.sweep(0, 0)
        so = o.sweep_slices(rows, stride, 0, 0)
        assert sg[3] == so[3]
        assert rel(e.volume(), o.volume()) <= 1e-5
        assert np.linalg.norm(e.error_sinogram() - o.error()) <= 1e-5 * np.linalg.norm(y)
        e.sweep(1, 0)
        assert np.isfinite(e.volume()).all()


@pytest.mark.parametrize("nhicd", [1, 0])
def test_long_rows_bright_field(lib_built, oracle_mod, nhicd):
    """The default lane shape: its trials walk the rows.  Tolerance as for the calls of other widths
    (test_rejected_entries_match_oracle)."""
    mbir = lib_built
    y, ang, th = bf_case(n_r=3800, n_t=2, step=6.0, thickness=4.0)
    p = bf_params(mbir, th, lane_shape=0, nhicd=nhicd, bragg_threshold=1e9)
    with mbir.Engine(p) as e:
        e.set_sinogram(y, ang)
        e.prepare()
        assert np.isfinite(e.volume()).all()
        if not nhicd:
            e.sweep(0, 0)
            assert e.volume().any()
            return
        o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
        o.prepare()
        e.sweep(0, 0)
        sync_oracle(e, o)
        before = e.volume().astype(np.float64)
        sg = e.sweep(0, 1)
        so = o.bf_sweep_slices_order(e.call_lines(), 0, 1)
        assert sg[3] == so[3]
        assert rel(e.volume() - before, o.volume() - before) <= 3e-3


def test_long_rows_in_a_batch(lib_built):
    """Series inside and outside the windows advanced together: the same bits as alone, whichever
    threads per CTA the batch takes."""
    mbir = lib_built
    cases = [(3800, 2, 21), (2400, 2, 9), (64, 3, 41), (2000, 2, 9)]
    alone = []
    for c in cases:
        y, ang, th = series(c[0], c[1], 4, c[2])
        with mbir.Engine(haadf_params(mbir, th, use_default_offset=1)) as e:
            e.set_sinogram(y, ang)
            e.prepare()
            for k in range(2):
                e.sweep(k, 0)
            alone.append(e.volume())
    for threads in (512, 256):
        engines = []
        with mbir.Batch() as b:
            b.set_threads(threads)
            for c in cases:
                y, ang, th = series(c[0], c[1], 4, c[2])
                e = mbir.Engine(haadf_params(mbir, th, use_default_offset=1))
                e.set_sinogram(y, ang)
                e.prepare()
                b.add(e)
                engines.append(e)
            for k in range(2):
                b.sweep(k)
            for e, want in zip(engines, alone):
                assert np.array_equal(e.volume(), want)
        for e in engines:
            e.close()
