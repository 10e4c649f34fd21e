"""The stage kernels at the limits of what their tables, planes and ranges hold. Tolerances against the CPU FP64
oracle as in tests/test_two_pass_stage.py: rel-L2 1e-12 (FP64) and 1e-5 (FP32) over a few steps.
"""
import ctypes
import math

import numpy as np
import pytest

import ripple_b200 as rp
from ripple_b200 import _lib
from test_two_pass_stage import TOL, bundle, rel_l2, run, terms, workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(3, 5, 4, 1028), (4, 3, 32, 1025), (5, 3, 6, 1040), (3, 3, 8, 6200)])
@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
@pytest.mark.parametrize("sources", [None, bundle, terms])
def test_more_directions_than_a_table_holds(oracle_mod, shape, precision, transport, sources):
    """Above 1024 directions: the ring walk's and the source pass's direction tables hold part of the ring only. The
    time step shrinks with the direction spacing."""
    w = workload(shape, 0.3, sources() if sources else None, transport)
    w.dt = 0.02 * 8 / shape[3]
    assert rel_l2(run(w, precision), oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL[precision]


def test_ring_split_for_its_table_alone(monkeypatch):
    """A grid that fills the GPU without a split ring, 1025 directions: the table's limit alone splits it. Same bits as
    the pair kernel, which walks the whole ring."""
    import torch
    Nx, Ny, Nk, Np = 400, 380, 4, 1025
    rng = np.random.default_rng(3)
    g = rp.RectilinearGrid(size=(Nx, Ny, 1), x=(0.0, 800.0), y=(0.0, 760.0), z=(-3.0, 0.0))
    sg = rp.PolarWaveVectorGrid(κ=np.linspace(0.3, 0.9, Nk), φ=np.arange(Np) * 2 * math.pi / Np)
    u, v = (np.asfortranarray(rng.uniform(-0.3, 0.3, (Nx, Ny, 1))) for _ in range(2))
    torch.manual_seed(5)
    N = 0.5 + torch.rand(Nx * Ny * Nk * Np, device="cuda")
    out, lib = {}, _lib.load()
    torch.cuda.synchronize()
    for form in ("", "pairs"):
        monkeypatch.setenv("RPL_PASS_B", form)
        m = rp.SpectralWaveModel(g, sg, depth=2.0, velocities={"u": u, "v": v}, precision="fp32")
        _lib.check(lib.rpl_set_action_device(m.handle, ctypes.c_void_p(N.data_ptr()), _lib.RPL_F32, 0))
        rp.time_step(m, 1e-4, 1)
        out[form] = torch.empty_like(N)
        torch.cuda.synchronize()
        _lib.check(lib.rpl_get_action_device(m.handle, ctypes.c_void_p(out[form].data_ptr()), _lib.RPL_F32, 0))
        m.close()
    assert not torch.equal(out[""], N)
    assert torch.equal(out[""], out["pairs"])
