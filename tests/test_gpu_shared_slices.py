"""Slices shared by a cluster of CTAs (FP64), with zero-skipped voxels, merged steps and bright field,
and slices of two detector rows (coarse levels) beyond the first sweep."""
import numpy as np
import pytest

from conftest import bf_case, bf_params, haadf_params
from test_gpu_bf import sync_oracle
from test_gpu_table import rel, series

pytestmark = pytest.mark.gpu

N_T = 320  # 160 slices per colour: one CTA each
SLABS = [(0, 38), (38, 114), (114, 266), (266, 320)]  # 8, 4, 2 and 4 CTAs per slice


def sparse(shape, seed):
    """Half of the rows empty, the others mostly so: zero-skipped voxels, sparse classes."""
    rng = np.random.default_rng(seed)
    v = rng.random(shape) * (rng.random(shape) < 0.08)
    v[rng.random(shape[0]) < 0.4] = 0.0
    return v


@pytest.mark.parametrize("zero_skipping", [0, 1])
@pytest.mark.parametrize("kind", ["haadf", "bf", "bf-lines"])
def test_clusters_give_the_bits_of_single_ctas(lib_built, kind, zero_skipping):
    """The colour-0 slices of a sweep or call over the whole volume, and the same in slabs."""
    mbir = lib_built
    if kind == "haadf":
        y, ang, th = series(26, N_T, 8, 19)
        p = haadf_params(mbir, th, precision=mbir.FP64, use_default_offset=1,
                         zero_skipping=zero_skipping)
    else:
        y, ang, th = bf_case(n_r=26, n_t=N_T, step=7.0, thickness=8.0)
        p = bf_params(mbir, th, precision=mbir.FP64, zero_skipping=zero_skipping,
                      nhicd=1 if kind == "bf-lines" else 0)

    def colour0(slab):
        with mbir.Engine(p) as e:
            e.set_sinogram(y, ang)
            e.set_initial_volume(sparse(e.dims()[:3], 4))
            e.prepare()
            if slab:
                e.set_slab(*slab)
            if kind != "haadf":
                e.bf_call_begin(1, 0)
            st = e.sweep_colour(0, 1, 0)
            sel = e.bf_state()[0] if kind != "haadf" else np.zeros(0)
            return st, e.volume64(), e.error_sinogram(), sel

    st, vol, err, sel = colour0(None)
    assert st[3] > 0 and (st[2] > 0) == bool(zero_skipping)
    assert kind == "haadf" or (sel == 0).any()
    counts = np.zeros(2)
    for a, b in SLABS:
        s, v, e, q = colour0((a, b))
        counts += s[2:4]
        assert np.array_equal(v[..., a:b:2], vol[..., a:b:2])
        assert np.array_equal(e[..., a:b:2], err[..., a:b:2])
        if kind != "haadf":
            assert np.array_equal(q[..., a:b:2], sel[..., a:b:2])
    assert np.array_equal(counts, st[2:4])


@pytest.mark.parametrize("n_r,n_t,n_z,views", [(64, 6, 12, 64), (48, 4, 8, 75), (40, 4, 8, 121)])
@pytest.mark.parametrize("staging", [0, 1])
def test_two_row_sweep_from_equal_state(lib_built, oracle_mod, n_r, n_t, n_z, views, staging):
    """The third sweep of a coarse level, zero skipping on, from equal state.  Tolerance: an update
    of a tenth of the voxel's value or more carries the FP32 rounding of the value (1e-5 of the
    update); a voxel at the edge of positivity may be skipped on one side and moved by its own
    (small) value on the other."""
    mbir = lib_built
    y, ang, th = series(n_r, n_t, n_z, views)
    p = haadf_params(mbir, th, use_default_offset=1, num_resolutions=2, level=0,
                     slice_staging=staging)
    with mbir.Engine(p) as e:
        o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
        e.set_sinogram(y, ang)
        e.prepare()
        o.prepare()
        assert e.status().t_rows == 2
        for k in range(2):
            e.sweep(k, 0)
        o.volume()[...] = before = e.volume().astype(np.float64)
        o.error()[...] = e.error_sinogram()
        rows, stride = e.schedule(2)
        sg = e.sweep(2, 0)
        so = o.sweep_slices(rows, stride, 2, 0)
        assert abs(sg[3] - so[3]) <= 1e-2 * so[3]
        assert rel(e.volume() - before, o.volume() - before) <= 1e-3


@pytest.mark.parametrize("step,shape,schedule,staging", [
    (2.0, 1, 0, 0), (2.0, 1, 0, 1), (2.0, 1, 1, 0), (1.6, 3, 0, 1), (1.6, 3, 1, 0), (1.0, 4, 0, 0)])
def test_two_row_bright_field_call(lib_built, oracle_mod, step, shape, schedule, staging):
    """A call of a coarse level whose footprints hold rejected entries, scheduled and walking the
    rows, from equal state.  Tolerance as for the fine level's (test_rejected_entries_match_oracle)."""
    mbir = lib_built
    y, ang, th = bf_case(n_r=64, n_t=6, step=step)
    p = bf_params(mbir, th, lane_shape=shape, slice_staging=staging, call_schedule=schedule,
                  num_resolutions=2, level=0)
    with mbir.Engine(p) as e:
        o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
        e.set_sinogram(y, ang)
        e.prepare()
        o.prepare()
        assert e.status().t_rows == 2
        for k in range(4):
            e.sweep(0, k)
        sync_oracle(e, o)
        o.offset()[...] = e.nuisance()[1]
        o.variance()[...] = e.nuisance()[2]
        before = e.volume().astype(np.float64)
        assert np.mean(e.bf_state()[0] == 0) > 1e-3
        rows, stride = e.schedule(4)
        sg = e.sweep(0, 4)
        if schedule:
            active = np.zeros(int(np.prod(e.dims()[:2])), np.uint8)
            active[e.call_lines()] = 1
            so = o.bf_sweep_slices(active, rows, stride, 0, 4)
        else:
            so = o.bf_sweep_slices_order(e.call_lines(), 0, 4)
        assert sg[2] == so[2] and sg[3] == so[3]
        assert rel(e.volume() - before, o.volume() - before) <= 3e-3
