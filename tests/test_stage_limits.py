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


REFRACTION = ("currents", "pseudomomentum", "refraction_terms", "averaging")


def bare_model(kind, precision, Nk, **kw):
    """A model of 24 x 20 cells and the call that asks for more device memory after its creation."""
    w = workload((24, 20, Nk, 48), 0.3, None, "refraction" if kind in REFRACTION else "intrinsic")
    w.dt = 0.02 * 8 / 48
    if kind == "pseudomomentum":
        w.velocities = rp.PseudomomentumVelocities()
    if kind in ("terms", "refraction_terms"):
        w.sources = terms()
    if kind == "averaging":
        w.propagation_smoothing = rp.SpatialAveraging()
    m = w.model(precision, **kw)
    if kind == "snapshot":
        from ripple_b200 import output
        output.snapshot_async(m)
        output.snapshot_wait(m)
    return w, m


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("Nk", [8, 25])
@pytest.mark.parametrize("kind", ["currents", "pseudomomentum", "terms", "refraction_terms", "averaging", "snapshot"])
def test_planes_are_given_up_for_what_a_later_call_needs(kind, precision, Nk):
    """A memory limit that holds the model and the planes, or the model and what a later call asks for, but not all
    three: the call is accepted, the planes go, and the other stage kernels give the same result (rounding apart).
    Without room for the call itself it is refused."""
    w, full = bare_model(kind, precision, Nk)
    total, cells, e = full.device_bytes(), 480, 8 if precision == "fp64" else 4
    planes = cells * Nk * e * (3 if kind in REFRACTION else 1)
    _, small = bare_model(kind, precision, Nk, memory_limit_bytes=total - 1)
    assert small.device_bytes() <= total - planes
    with pytest.raises(rp.RplError):
        bare_model(kind, precision, Nk, memory_limit_bytes=small.device_bytes() - 1)
    rp.time_step(full, w.dt, 2)
    rp.time_step(small, w.dt, 2)
    assert rel_l2(small.action.interior(), full.action.interior()) <= (1e-13 if precision == "fp64" else 1e-6)


def test_captured_planes_stay():
    """Steps recorded in a CUDA graph hold the planes' addresses: a later call over the limit is refused, and the graph
    still gives the steps' result."""
    import torch
    w = workload((24, 20, 25, 48), 0.3, None, "intrinsic")
    ref = w.model("fp64")
    m = w.model("fp64", memory_limit_bytes=ref.device_bytes() + 8 * w.units - 1)
    s = torch.cuda.Stream()
    _lib.check(m._lib.rpl_set_stream(m.handle, ctypes.c_void_p(s.cuda_stream)))
    rp.time_step(m, w.dt, 1)                       # kernels loaded before the capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        _lib.check(m._lib.rpl_step_async(m.handle, w.dt, 1))
    before = m.device_bytes()
    out = np.empty(w.N0.shape, order="F")
    assert m._lib.rpl_snapshot_async(m.handle, out.ctypes.data_as(ctypes.c_void_p), _lib.RPL_F64) == _lib.RPL_ERR_OOM
    assert m.device_bytes() == before
    graph.replay()
    torch.cuda.synchronize()
    rp.time_step(ref, w.dt, 2)
    assert np.array_equal(m.action.interior(), ref.action.interior())


@pytest.mark.parametrize("kind", ["diagnostics", "terms", "pseudomomentum"])
def test_models_of_different_sizes_launch_from_two_threads(kind):
    """Kernels whose shared-memory tables differ with the spectrum, launched by two threads at once: no launch is refused."""
    import threading
    import torch

    def make(Np):
        w = workload((8, 8, 32, Np), 0.1, terms() if kind == "terms" else None,
                     "refraction" if kind == "pseudomomentum" else "intrinsic")
        if kind == "pseudomomentum":
            w.velocities = rp.PseudomomentumVelocities()
        return w.model("fp64")

    def calls(m, out):
        lib, total = m._lib, torch.empty(1, dtype=torch.float64, device="cuda")
        field = torch.empty(4, 64, dtype=torch.float64, device="cuda")
        ptrs = [ctypes.c_void_p(field[k].data_ptr()) for k in range(4)] + [ctypes.c_void_p(total.data_ptr())]
        go.wait()
        for _ in range(1500):
            st = (lib.rpl_diagnostics_device(m.handle, *ptrs) if kind == "diagnostics"
                  else lib.rpl_stage_rows_async(m.handle, 1e-6, 1, 0, 0, 1))   # the stage's preparation alone
            if st != _lib.RPL_OK:
                out.append(lib.rpl_last_error().decode())
                break
        _lib.check(lib.rpl_sync(m.handle))

    models, errors, go = [make(16), make(120)], [], threading.Barrier(2)
    threads = [threading.Thread(target=calls, args=(m, errors)) for m in models]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == []


def uneven_depth(shape):
    x, y = np.meshgrid(np.arange(shape[0]), np.arange(shape[1]), indexing="ij")
    return np.asfortranarray(2.0 + 0.7 * np.sin(2 * np.pi * x / shape[0]) * np.cos(2 * np.pi * y / shape[1]))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(3, 5, 4, 3), (31, 6, 32, 4), (64, 130, 8, 5), (90, 40, 24, 3), (13, 9, 25, 5), (9, 7, 3, 4),
                                   (21, 6, 36, 3)])
@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
def test_uneven_depth_and_row_ranges(oracle_mod, shape, precision, transport):
    """c_g per cell, whole and ragged lane vectors, one and several x tiles and segments: the oracle's result, the same
    bits on every run, and the same bits from stages launched in ranges of one row upwards (the last row of a range is
    the last its CTA prepares for)."""
    w = workload(shape, 0.3, None, transport)
    w.depth = uneven_depth(shape)
    first = run(w, precision)
    assert rel_l2(first, oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL[precision]
    for _ in range(3):
        assert np.array_equal(run(w, precision), first)
    m, Ny = w.model(precision), shape[1]
    cuts = sorted({0, 1, 2, Ny // 2, Ny - 1, Ny})
    for _ in range(3):
        for stage in (1, 2, 3):
            for a, b in zip(cuts[:-1], cuts[1:]):
                flags = (1 if a == 0 else 0) | (2 if b == Ny else 0)
                _lib.check(m._lib.rpl_stage_rows_async(m.handle, w.dt, stage, a, b - a, flags))
    _lib.check(m._lib.rpl_sync(m.handle))
    assert np.array_equal(m.action.interior(), first)


@pytest.mark.parametrize("Nk", [7, 8])
@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
def test_large_fp32_action(oracle_mod, Nk, transport):
    w = workload((11, 8, Nk, 6), 0.3, None, transport)
    w.N0 = np.asfortranarray(1e8 * w.N0)
    assert rel_l2(run(w, "fp32"), oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL["fp32"]


@pytest.mark.parametrize("scale", [1e20, 1e31, 1e36, 1e38, 1e60, 1e75])
@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
@pytest.mark.parametrize("sources", ["none", "wind", "linear"])
def test_large_fp64_action(oracle_mod, scale, transport, sources):
    """WENO5 weights of large actions (the action enters the smoothness indicators squared and the weights to the fourth
    power): the oracle's result up to where its own weights end, from everywhere large and from single large cells."""
    src = {"none": None, "wind": rp.PrecomputedSources(wind_input=rp.PressureCorrelationInput(drag=rp.BulkWindDrag("linear"), wind=18.0,
                                                                                direction=0.7)),
           "linear": rp.SourceTermSet(rp.ExponentialWindInput(rate=2e-3, direction=0.6, spreading_power=2))}[sources]
    for shape in [(11, 8, 7, 6), (9, 12, 8, 5)]:
        w = workload(shape, 0.3, src, transport)
        for cells in (1.0, 0.05):
            large = np.random.default_rng(7).uniform(size=shape) < cells
            w.N0 = np.asfortranarray(np.where(large, scale, 1.0) * workload(shape).N0)
            assert rel_l2(run(w, "fp64"), oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL["fp64"]


@pytest.mark.parametrize("precision,Nk", [("fp64", 7), ("fp64", 8), ("fp32", 7)])
@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
@pytest.mark.parametrize("parameters", [dict(beta_max=-1.2e3), dict(rho_air=-1.225e3)])
def test_negative_growth_rates_are_left_out(oracle_mod, precision, Nk, transport, parameters):
    """Only a positive raw growth rate acts (precomputed_sources.jl:396-439), and only such rates enter the stress."""
    src = rp.PrecomputedSources(
        wind_input=rp.PressureCorrelationInput(drag=rp.BulkWindDrag("linear"), wind=18.0, direction=0.7, **parameters),
        dissipation=rp.LocalSaturationDissipation(B_r=1.05e-2))
    w = workload((9, 6, Nk, 12), 0.3, src, transport)
    assert rel_l2(run(w, precision), oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]) <= TOL[precision]


@pytest.mark.parametrize("transport", ["refraction", "intrinsic"])
def test_growth_beside_a_negative_inverse_wave_age(oracle_mod, transport):
    """z_alpha below -u* / C and a rough surface: log(k z1) > 0, so a bin grows only where cos(theta - theta_u) is small."""
    src = rp.PrecomputedSources(wind_input=rp.PressureCorrelationInput(
        drag=rp.BulkWindDrag("linear"), wind=18.0, direction=0.7, z_alpha=-1.0, alpha0=1e4, beta_max=1e4))
    w = workload((9, 6, 8, 96), 0.3, src, transport)
    w.dt = 5e-3
    ref = oracle_mod.Oracle(w).step(w.N0, w.dt, 3)[0]
    still = workload((9, 6, 8, 96), 0.3, None, transport)
    still.dt = w.dt
    assert rel_l2(oracle_mod.Oracle(still).step(w.N0, w.dt, 3)[0], ref) > 10 * TOL["fp32"]     # something grows
    assert rel_l2(run(w, "fp32"), ref) <= TOL["fp32"]


@pytest.mark.parametrize("scale", [3e31, 1e33, 3e33, 1e34, 1e35, 1e37, 3e37])
def test_large_fp64_action_where_neighbouring_bins_upwind_apart(oracle_mod, scale):
    """Currents as fast as the waves: the two bins of a lane take their faces from different sides. Large cells in every
    other bin alone (four bins have no kappa stencil that would join them), so that one bin's face leaves the range on the
    side its neighbour does not use."""
    for shape in [(24, 20, 16, 9), (60, 50, 4, 12), (60, 50, 3, 11)]:
        w = workload(shape, 3.0)
        rng = np.random.default_rng(11)
        large = rng.uniform(size=shape) < 0.04
        if shape[2] < 5:
            large[:, :, 0::2] = False
        w.N0 = np.asfortranarray(np.where(large, scale * 10.0 ** rng.uniform(-3, 0, shape), 1.0) * workload(shape).N0)
        out, ref = run(w, "fp64", 1), oracle_mod.Oracle(w).step(w.N0, w.dt, 1)[0]
        assert rel_l2(out, ref) <= TOL["fp64"]
        assert np.array_equal(out == 0.0, ref == 0.0)
