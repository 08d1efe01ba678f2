"""The FP64 sweep with a slice shared by the CTAs of a cluster (few slices per colour) and with one
CTA per slice, against the FP64 oracle in the same visit order; and levels whose slices meet two
detector rows."""
import numpy as np
import pytest

from conftest import haadf_params
from test_gpu_table import rel, series

pytestmark = pytest.mark.gpu


# slices per colour 1, 2, 19 | 20, 38 | 39, 76 | 77: the ends of the 8-, 4-, 2- and 1-CTA ranges
@pytest.mark.parametrize("n_t", [1, 3, 38, 40, 76, 78, 152, 154])
def test_fp64_sweep_matches_oracle(lib_built, oracle_mod, n_t):
    """Tolerance: the engine's footprint constants are rounded to FP32 (6e-8), which moves the
    second sweep's updates by about as much; zero skipping is off (its decisions are exact tests)."""
    mbir = lib_built
    y, ang, th = series(24, n_t, 6, 19)
    p = haadf_params(mbir, th, precision=mbir.FP64, use_default_offset=1, zero_skipping=0)
    with mbir.Engine(p) as e:
        o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
        e.set_sinogram(y, ang)
        e.prepare()
        o.prepare()
        for k in range(2):
            rows, stride = e.schedule(k)
            sg = e.sweep(k, 0)
            so = o.sweep_slices(rows, stride, k, 0)
            assert sg[3] == so[3]
            np.testing.assert_allclose(sg[:2], so[:2], rtol=1e-6)
        assert rel(e.volume64(), o.volume()) <= 1e-6


@pytest.mark.parametrize("n_r,n_t,n_z,views,precision", [
    (32, 4, 8, 17, 0), (64, 6, 12, 64, 0), (48, 4, 8, 75, 0), (40, 4, 8, 121, 0),
    (32, 4, 8, 17, 1)])
def test_two_row_level_matches_oracle(lib_built, oracle_mod, n_r, n_t, n_z, views, precision):
    """The coarse one of two levels (five-bin footprints, two detector rows per slice).  Tolerance
    as for the fine level's sweeps."""
    mbir = lib_built
    y, ang, th = series(n_r, n_t, n_z, views)
    p = haadf_params(mbir, th, use_default_offset=1, num_resolutions=2, level=0,
                     precision=precision)
    with mbir.Engine(p) as e:
        o = oracle_mod.Oracle(oracle_mod.params_from_mbir(p), y, ang)
        e.set_sinogram(y, ang)
        e.prepare()
        o.prepare()
        assert e.status().t_rows == 2
        rows, stride = e.schedule(0)
        sg = e.sweep(0, 0)
        so = o.sweep_slices(rows, stride, 0, 0)
        assert sg[3] == so[3]
        assert rel(e.volume(), o.volume()) <= 1e-5
        assert np.linalg.norm(e.error_sinogram() - o.error()) <= 1e-5 * np.linalg.norm(y)
