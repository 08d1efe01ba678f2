"""The table-driven sweep and projection (A-column from the engine's table): against the FP64
oracle in the same visit order at the edges of the lane shapes, and bit for bit against the
kernels that compute the columns."""
import numpy as np
import pytest

from conftest import haadf_params

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def series(n_r, n_t, n_z, views, max_deg=60.0, seed=3):
    import synthetic
    ang = np.linspace(-max_deg, max_deg, views) if views > 1 else np.zeros(1)
    a = min(n_r, n_z) / 3.0
    proj = synthetic.ellipsoid_projection(ang, n_r, n_t,
                                          [(0.0, 0.0, 0.0, a, max(n_t, 2) / 1.5, a, 1.0)])
    y, _ = synthetic.haadf_measurements(proj + 0.05, seed=seed)
    return y, ang.astype(np.float32), n_z / 2.0


# detector widths around the padded row strides, view counts on both sides of each lane shape
# (16 x 4 to 64, 32 x 3 to 96, 32 x 5 to 160, 32 x 8 above), one slice and odd slice counts
@pytest.mark.parametrize("n_r,n_t,n_z,views", [
    (4, 1, 4, 2), (5, 2, 4, 16), (32, 3, 8, 17), (33, 1, 6, 63), (31, 2, 6, 64),
    (36, 3, 8, 65), (29, 2, 6, 96), (30, 2, 4, 97), (64, 1, 4, 160), (34, 2, 4, 161)])
def test_sweep_and_projection_match_oracle(lib_built, oracle_mod, n_r, n_t, n_z, views):
    """Tolerance: FP32 sums of at most ~500 terms with relative rounding 2^-24 each (root sum
    square 1.3e-6) and a few fast powers (1e-6 each); errors of the sinogram are relative to the
    measurements that it is a difference of."""
    mbir = lib_built
    y, ang, th = series(n_r, n_t, n_z, views)
    volumes = []
    for staging in (0, 1) if views <= 160 else (0,):
        p = haadf_params(mbir, th, slice_staging=staging, use_default_offset=1)
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
            volumes.append(e.volume())
            vol = np.random.default_rng(1).random(e.dims()[:3]).astype(np.float32)
        with mbir.Engine(p) as e:
            e.set_sinogram(y, ang)
            e.set_initial_volume(vol)
            e.prepare()
            o.prepare(vol.astype(np.float64))
            assert np.abs(e.projection() - o.yest()).max() / np.abs(o.yest()).max() <= 1e-5
    if len(volumes) == 2:  # staged and in place: the same bits
        assert np.array_equal(volumes[0], volumes[1])


@pytest.mark.parametrize("views", [41, 75, 121])
def test_bits_equal_without_the_table(lib_built, views):
    """A server whose budget has no room for the table runs the kernels that compute the
    columns: the same bits as an engine of its own."""
    mbir = lib_built
    y, ang, th = series(40, 6, 12, views)
    p = haadf_params(mbir, th, lane_shape={41: 1, 75: 3, 121: 4}[views], outer_iterations=3)
    batch_p = mbir.MbirParams.from_buffer_copy(p)
    with mbir.Engine(p) as e:
        e.set_sinogram(y, ang)
        e.prepare()
        for k in range(3):
            e.sweep(k, 0)
            if p.joint_estimation:
                e.joint_estimation()
            if p.noise_model:
                e.update_weights()
        alone = e.volume()
    sino, vox = y.size, int(np.prod(alone.shape))
    own = 4 * (3 * sino + vox) + 4 * max(sino, vox) + (1 << 20)
    for budget in (own + 1, 0):
        with mbir.Server(0, budget, 1) as s:
            rid = s.submit(batch_p, y, ang, max_outer=3, tol=0.0)
            s.wait(rid, 120.0)
            assert np.array_equal(s.result(rid), alone)
