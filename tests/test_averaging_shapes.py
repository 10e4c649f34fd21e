"""SpatialAveraging over the forms its kernels take: whole and ragged lane vectors, one and several chunks of lanes, strips
shorter and longer than the grid, near, far and mixed bins in one group, ranges of rows. Against the CPU oracle at the
tolerances of a lone averaging (tests/test_spatial_averaging.py): rel-L2 1e-14 (FP64), 1e-6 (FP32)."""
import numpy as np
import pytest

import ripple_b200 as rp
from ripple_b200 import _lib
from test_spatial_averaging import rel_l2, still_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-14), ("fp32", 1e-6)])
@pytest.mark.parametrize("Nk", [1, 2, 3, 4, 8, 25, 32, 36, 100, 130])
@pytest.mark.parametrize("dt", [60.0, 400.0, 1500.0])
def test_averaging_matches_oracle(oracle_mod, Nk, dt, precision, tol):
    w = still_field(Nx=41, Ny=30, kappa=np.geomspace(0.01, 0.3, Nk) if Nk > 1 else [0.02], alpha=(0.9, 0.7), dt=dt)
    m = w.model(precision)
    rp.time_step(m, w.dt, 1)
    assert rel_l2(m.action.interior(), oracle_mod.Oracle(w).spatial_averaging(w.N0, w.dt)) <= tol


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("Nk", [7, 8])
def test_row_ranges_and_changing_steps(precision, Nk):
    """A step's averaging in ranges of rows gives the bits of the whole; a change of dt changes what is far."""
    w = still_field(Nx=41, Ny=30, kappa=np.geomspace(0.01, 0.3, Nk), alpha=(0.9, 0.7))
    whole, parts = w.model(precision), w.model(precision)
    lib = parts._lib
    for dt in (60.0, 1500.0, 60.0, 400.0):
        rp.time_step(whole, dt, 1)
        for stage in (1, 2, 3):
            _lib.check(lib.rpl_stage_rows_async(parts.handle, dt, stage, 0, 30, 1 | 2 | (4 if stage == 3 else 0)))
        for a, b in ((0, 1), (1, 17), (17, 30)):
            _lib.check(lib.rpl_smooth_rows_async(parts.handle, dt, a, b - a, 0))
        _lib.check(lib.rpl_sync(parts.handle))
        assert np.array_equal(parts.action.interior(), whole.action.interior())
