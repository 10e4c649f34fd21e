"""The pseudomomentum velocity in its two forms, lane vectors (whole vectors that fill the warp, 8192 columns and more) and a
warp per column (everything else), with one and with per-column overlap tables. Against the CPU FP64 oracle over two
steps: rel-L2 1e-12 (FP64) and 1e-5 (FP32), as tests/test_pseudomomentum.py."""
import numpy as np
import pytest

import ripple_b200 as rp
from test_two_pass_stage import TOL, rel_l2, run, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape,depth_field",
                         [(s, False) for s in [(96, 90, 8, 3), (91, 91, 4, 5), (96, 90, 7, 3), (90, 91, 8, 13), (96, 86, 64, 3),
                                               (96, 86, 36, 3), (40, 30, 8, 5), (40, 30, 100, 3), (64, 64, 128, 3), (9, 7, 1, 4)]]
                         + [(s, True) for s in [(96, 90, 8, 3), (96, 90, 7, 3), (40, 30, 8, 5)]])
def test_self_coupled_steps_match_oracle(oracle_mod, shape, precision, depth_field):
    w = workload(shape, 0.3)
    w.velocities = rp.PseudomomentumVelocities()
    w.N0 = np.asfortranarray(0.05 * w.N0)
    if depth_field:
        x, y = np.meshgrid(np.arange(shape[0]), np.arange(shape[1]), indexing="ij")
        w.depth = np.asfortranarray(2.0 + 0.5 * np.sin(2 * np.pi * x / shape[0]) * np.cos(2 * np.pi * y / shape[1]))
    assert rel_l2(run(w, precision, 2), oracle_mod.Oracle(w).step(w.N0, w.dt, 2)[0]) <= TOL[precision]
