"""The two-pass stage (x/y pass as a y-walk, then the walk of the phi ring) at the sizes where it can go wrong:
wavenumber counts that are not whole lane vectors (4 FP32 or 2 FP64 bins), one to many lanes per cell, one
and several x tiles and row segments, split phi rings, the smallest grids, uniform and mixed upwind signs.

Tolerances against the CPU FP64 oracle are those of the FP64 path and the FP32 form over a few steps: rel-L2
1e-12 and 1e-5 (tests/test_gpu_parity.py).
"""
import math

import numpy as np
import pytest

import ripple_b200 as rp
from ripple_b200 import workloads

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32": 1e-5}
SHAPES = [(3, 5, 1, 3), (9, 7, 2, 5), (5, 4, 3, 3), (37, 29, 5, 7), (40, 9, 25, 7), (13, 140, 30, 6), (70, 33, 27, 8),
          (9, 6, 33, 4), (11, 8, 40, 5), (6, 5, 64, 4), (300, 4, 4, 3), (258, 3, 3, 4), (4, 3, 66, 3), (5, 4, 128, 3)]


def rel_l2(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b)))


def workload(shape, current=0.3, sources=None, transport="refraction"):
    Nx, Ny, Nk, Np = shape
    rng = np.random.default_rng(sum(shape))
    g = rp.RectilinearGrid(size=(Nx, Ny, 4), x=(0.0, Nx * 2.0), y=(0.0, Ny * 2.0), z=(-3.0, 0.0))
    κ = np.linspace(0.3, 0.9, Nk) if Nk > 1 else np.array([0.5])
    sg = rp.PolarWaveVectorGrid(κ=κ, φ=np.arange(Np) * 2 * math.pi / Np)
    velocities = None
    if transport == "refraction":
        u = np.asfortranarray(rng.uniform(-current, current, (Nx, Ny, 4)))
        v = np.asfortranarray(rng.uniform(-current, current, (Nx, Ny, 4)))
        velocities = {"u": u, "v": v}
    N0 = np.asfortranarray(rng.uniform(0.5, 1.0, shape))
    return workloads.Workload("two_pass", g, sg, 2.0, N0, 0.02, 3, velocities=velocities, sources=sources)


def bundle():
    return rp.PrecomputedSources(
        wind_input=rp.PressureCorrelationInput(drag=rp.BulkWindDrag("linear"), wind=18.0, direction=0.7),
        dissipation=rp.LocalSaturationDissipation(B_r=1.05e-2, σ_power=1.5))


def terms():
    return rp.SourceTermSet(rp.ExponentialWindInput(rate=2e-3, direction=0.6, spreading_power=2),
                            rp.WhitecappingDissipation(rate=1e-3, saturation_threshold=0.05))


def run(w, precision, steps=3, **kw):
    m = w.model(precision, **kw)
    rp.time_step(m, w.dt, steps)
    out = m.action.interior()
    m.close()
    return out


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_refraction_matches_oracle(oracle_mod, shape, precision):
    for current in (0.05, 3.0):
        w = workload(shape, current)
        assert rel_l2(run(w, precision), oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(3, 5, 1, 3), (40, 9, 25, 7), (13, 140, 30, 6), (11, 8, 40, 5), (9, 5, 32, 12)])
@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
@pytest.mark.parametrize("sources", [None, bundle, terms])
def test_sources_match_oracle(oracle_mod, shape, precision, transport, sources):
    w = workload(shape, 0.3, sources() if sources else None, transport)
    assert rel_l2(run(w, precision), oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL[precision]


@pytest.mark.parametrize("shape", [(3, 5, 4, 3), (31, 6, 32, 4), (64, 130, 8, 5), (40, 9, 64, 3), (255, 5, 4, 4)])
@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
def test_whole_vectors_fp32_match_oracle_and_repeat(oracle_mod, shape, transport):
    """Rows handed on without a CTA barrier (whole FP32 lane vectors): one to eight warps per CTA, segments of one row
    upwards, uniform and mixed signs; the oracle's result, and the same bits on every run."""
    for current in (0.05, 3.0):
        w = workload(shape, current, transport=transport)
        first = run(w, "fp32")
        assert rel_l2(first, oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL["fp32"]
        for _ in range(3):
            assert np.array_equal(run(w, "fp32"), first)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_model_without_room_for_the_planes_takes_the_column_kernel(precision):
    """A memory limit that holds the model but not the two-pass stage's c_g plane: same result."""
    Nx, Ny, Nk, Np = shape = (24, 20, 25, 8)
    w = workload(shape, transport="intrinsic")
    e, cells, bins = 8 if precision == "fp64" else 4, Nx * Ny, Nk * Np
    need = 3 * cells * bins * e + 16 * cells * Nk * 8 + (4 * cells + 2 * (Nx + Ny)) * 8 + 6 * cells * 8 + 8 * bins * 8
    with pytest.raises(rp.RplError):
        w.model(precision, memory_limit_bytes=need - 1)
    full, small = w.model(precision), w.model(precision, memory_limit_bytes=need)
    assert small.device_bytes() <= full.device_bytes() - cells * Nk * e
    rp.time_step(full, w.dt, 2)
    rp.time_step(small, w.dt, 2)
    assert rel_l2(small.action.interior(), full.action.interior()) <= (1e-13 if precision == "fp64" else 1e-6)
