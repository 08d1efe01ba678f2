"""Edges of the calls' device-built lists, the sinogram passes, the row walk and the weighting of
rejected bright-field entries."""
import numpy as np
import pytest

from conftest import bf_case, bf_params, haadf_params
from test_gpu_bf import sync_oracle
from test_gpu_table import rel, series

pytestmark = pytest.mark.gpu


# fewer lines than the last step of the selection ranks at once, and more; most magnitudes of the first calls are zeros, so that the order statistic lies among ties
@pytest.mark.parametrize("n_r,n_t,thickness", [(12, 2, 6.0), (64, 2, 16.0), (65, 3, 16.0),
                                               (96, 2, 24.0)])
def test_nonhomogeneous_lists(lib_built, n_r, n_t, thickness):
    """The call's lines are those whose filtered magnitude exceeds the order statistic at
    n - n / 20 (whole numbers: no tolerance)."""
    mbir = lib_built
    y, ang, th = bf_case(n_r=n_r, n_t=n_t, step=8.0, thickness=thickness)
    with mbir.Engine(bf_params(mbir, th)) as e:
        e.set_sinogram(y, ang)
        e.prepare()
        for k in range(6):
            e.sweep(0, k)
            if k % 2 == 0:
                continue
            filt = e.bf_state()[3].ravel()
            n = filt.size
            thr = np.sort(filt)[min(n - n // 20, n - 1)]
            np.testing.assert_array_equal(np.sort(e.call_lines()), np.flatnonzero(filt > thr))


@pytest.mark.parametrize("n_r,n_t,step", [(12, 1, 40.0), (33, 5, 7.5), (130, 3, 2.0)])
def test_bright_field_estimates(lib_built, oracle_mod, n_r, n_t, step):
    """Offset and variance updates from equal state, the widths around the passes' groups of four
    and of 128 bins.  Tolerance: both sides sum the same FP32 values, here to about 2^-48 of the
    sum of magnitudes; a thousandfold cancellation leaves 1e-11."""
    mbir = lib_built
    y, ang, th = bf_case(n_r=n_r, n_t=n_t, step=step, thickness=min(16.0, n_r / 2.0))
    p = bf_params(mbir, th)
    with mbir.Engine(p) as e:
        o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
        e.set_sinogram(y, ang)
        e.prepare()
        o.prepare()
        for k in range(3):
            e.sweep(0, k)
        sync_oracle(e, o)
        o.offset()[...] = e.nuisance()[1]
        o.variance()[...] = e.nuisance()[2]
        e.joint_estimation()
        o.bf_joint_estimation()
        np.testing.assert_allclose(e.nuisance()[1], o.offset(), rtol=1e-9)
        assert np.linalg.norm(e.error_sinogram() - o.error()) <= 1e-6 * np.linalg.norm(o.measured())
        sync_oracle(e, o)
        o.offset()[...] = e.nuisance()[1]
        e.update_weights()
        o.bf_update_weights()
        np.testing.assert_allclose(e.nuisance()[2], o.variance(), rtol=1e-9)
        assert rel(e.bf_state()[1], o.weight()) <= 1e-6


@pytest.mark.parametrize("step,shape,staging", [
    (2.0, 1, 0), (2.0, 1, 1), (2.0, 2, 1), (1.6, 3, 0), (1.6, 3, 1), (1.0, 4, 0), (1.0, 4, 1),
    (0.75, 5, 0)])
def test_rejected_entries_match_oracle(lib_built, oracle_mod, step, shape, staging):
    """A call whose footprints hold rejected entries, from equal state.  Tolerance: the selector
    is a threshold, and FP32 turns about one in 1e5 of its decisions around; each moves one
    voxel's update by up to its own size, 3e-3 of the call's updates in the root mean square."""
    mbir = lib_built
    y, ang, th = bf_case(n_r=48, n_t=3, step=step)
    p = bf_params(mbir, th, lane_shape=shape, slice_staging=staging)
    with mbir.Engine(p) as e:
        o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
        e.set_sinogram(y, ang)
        e.prepare()
        o.prepare()
        for k in range(4):
            e.sweep(0, k)
        sync_oracle(e, o)
        o.offset()[...] = e.nuisance()[1]
        o.variance()[...] = e.nuisance()[2]
        before = e.volume().astype(np.float64)
        assert np.mean(e.bf_state()[0] == 0) > 1e-3
        sg = e.sweep(0, 4)
        so = o.bf_sweep_slices_order(e.call_lines(), 0, 4)
        assert sg[2] == so[2] and sg[3] == so[3]
        assert rel(e.volume() - before, o.volume() - before) <= 3e-3
        assert np.mean(e.bf_state()[0] != o.selector()) <= 1e-4


# class strides above one word of candidates, rows longer than the voxels seen (empty columns), a
# row whose two caches do not fit behind the staged slice, widths off the copies' four values
@pytest.mark.parametrize("n_r,n_t,n_z,views,max_deg,kw", [
    (150, 2, 6, 5, 86.0, {}), (43, 2, 12, 21, 60.0, {"extend_object": 1}),
    (1200, 1, 4, 30, 60.0, {}), (1203, 2, 4, 30, 60.0, {"slice_staging": 0})])
def test_row_walk_edges(lib_built, n_r, n_t, n_z, views, max_deg, kw):
    """Sweeps with and without zero-skipped voxels: the same bits as the kernels that compute the
    columns."""
    mbir = lib_built
    y, ang, th = series(n_r, n_t, n_z, views, max_deg)
    y = np.where(np.arange(n_r)[None, :, None] < n_r // 2, y, y.min()).astype(np.float32)
    p = haadf_params(mbir, th, outer_iterations=3, use_default_offset=1, **kw)
    with mbir.Engine(p) as e:
        e.set_sinogram(y, ang)
        e.prepare()
        shape = e.dims()[:3]
        assert max_deg < 80 or e.status().stride > 31
        for k in range(3):
            e.sweep(k, 0)
            if p.joint_estimation:
                e.joint_estimation()
            if p.noise_model:
                e.update_weights()
        alone = e.volume()
    vox, sino = int(np.prod(shape)), n_t * views * ((n_r + 3) // 4 * 4)
    own = 4 * (3 * sino + vox) + 4 * max(y.size, vox) + (1 << 20)
    results = []
    for budget in (own + 64, 0):
        with mbir.Server(0, budget, 1) as s:
            rid = s.submit(p, y, ang, max_outer=3, tol=0.0)
            s.wait(rid, 120.0)
            results.append(s.result(rid))
    assert np.isfinite(alone).all() and alone.any()
    assert np.array_equal(results[0], alone) and np.array_equal(results[1], alone)
