"""Timing cases of ripple_b200: what a user of the framework has it do, through its public entry points.

A case is one pass of a wave run: give the model its initial action (device memory, the caller's x-fastest
layout), advance it, read the action back into device memory. The sizes come from the package's workloads
(`ripple_b200/workloads.py`, `bench.py`), reduced in the horizontal where the full grid would only repeat
the same work, and from the spectral grids in common use (24 to 36 wavenumbers, 24 to 36 directions).

`prepare` builds the grids, the model with its currents, depth and sources, and the initial action; the
model is what a user's program keeps. `exact` restates the model's mathematics in 64-bit torch.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ripple.jl_b200"))

import ripple_b200 as rp  # noqa: E402

G = 9.81
F64, F32, XFAST = 0, 1, 0          # dtype and layout codes of include/rpl.h


# ---------------------------------------------------------------------------------------- the cases
def _case(name, kind, Nx, Ny, Nk, Np, precision, steps, depth="field", Nz=16, smooth=False):
    c = dict(kind=kind, Nx=Nx, Ny=Ny, Nk=Nk, Np=Np, precision=precision, steps=steps, depth=depth, Nz=Nz,
             smooth=smooth)
    if name:
        c = dict(name=name, **c)
    return c


def listed():
    return [
        # The README's vortex-refraction example in the default precision, one output interval of 20 steps:
        # a small grid, where launches and latency count.
        _case("vortex_64_f64", "currents", 64, 64, 4, 16, "fp64", 20, depth="infinite"),
        # The smallest call: a single FP32 step of that example (interactive use, callbacks every step).
        _case("vortex_64_f32_one_step", "currents", 64, 64, 4, 16, "fp32", 1, depth="infinite"),
        # The benchmark's seamount-eddies configuration at full size.
        _case("eddies_1024_f32", "currents", 1024, 1024, 32, 36, "fp32", 2, Nz=32),
        # The same physics in the default precision on a regional grid.
        _case("eddies_320_f64", "currents", 320, 320, 32, 36, "fp64", 2, Nz=32),
        # A regional grid of odd size with a 25 x 24 spectrum (25 wavenumbers are not a multiple of four).
        _case("eddies_389x251_k25_f32", "currents", 389, 251, 25, 24, "fp32", 3, Nz=24),
        # The benchmark's translating hurricane at full size: wind input with the stress cap, whitecapping.
        _case("hurricane_768_f32", "hurricane", 768, 768, 32, 36, "fp32", 2, depth="constant"),
        # The hurricane in the default precision.
        _case("hurricane_192_f64", "hurricane", 192, 192, 32, 36, "fp64", 2, depth="constant"),
        # Swell propagation over a sloping shelf with SpatialAveraging after every step, ragged size.
        _case("swell_601x417_smooth_f32", "swell", 601, 417, 24, 24, "fp32", 3, smooth=True),
        # A SourceTermSet of four terms (wind input, wave-age input, two whitecapping terms).
        _case("terms_384_f32", "terms", 384, 384, 32, 36, "fp32", 2, depth="constant"),
        # PseudomomentumVelocities: the coupling is recomputed from the action at every stage.
        _case("selfcoupled_384_f32", "selfcoupled", 384, 384, 32, 36, "fp32", 2, depth="constant"),
        # Time-varying currents: per pass the diagnostics of the state, new currents, then one step.
        _case("tides_448_f32", "tides", 448, 448, 32, 36, "fp32", 1, Nz=32),
        # The learned source's network forward (BF16 tensor cores) on one row per cell of a 320 x 320 grid.
        dict(name="network_forward_102400", kind="network", rows=102400, nbins=1152, hidden=512),
    ]


# Cost of a cell-bin stage relative to FP32 refraction, an upper estimate over the paths a draw can take.
def _cost(c):
    if c["kind"] == "network":
        return c["rows"] * 1e3
    w = 1.0
    if c["precision"] == "fp64":
        w *= 16.0 if c["kind"] == "hurricane" else 6.0
    elif c["Nk"] % 4 or c["Nk"] > 32:
        w *= 8.0
    if c["kind"] in ("terms", "hurricane"):
        w *= 3.0
    return w * c["Nx"] * c["Ny"] * c["Nk"] * c["Np"] * c["steps"]


def draw(rng):
    limit = 0.45 * 1024 * 1024 * 32 * 36 * 2
    if rng.random() < 0.07:
        return dict(kind="network", rows=128 * int(round(math.exp(rng.uniform(math.log(2), math.log(1000))))),
                    nbins=1152, hidden=512)
    while True:
        kind = rng.choice(["currents", "currents", "currents", "hurricane", "swell", "terms", "selfcoupled", "tides"])
        c = _case(None, kind, int(round(math.exp(rng.uniform(math.log(16), math.log(900))))), 0,
                  rng.choice([4, 8, 12, 16, 20, 24, 25, 27, 30, 32, 32, 36, 40]),
                  rng.choice([12, 16, 24, 25, 30, 36, 36, 40]), rng.choice(["fp64", "fp32", "fp32"]),
                  1 if kind == "tides" else rng.choice([1, 2, 3, 5]))
        c["Ny"] = max(12, int(round(c["Nx"] * math.exp(rng.uniform(-0.7, 0.7)))))
        c["Nz"] = rng.choice([8, 16, 24, 32])
        c["depth"] = {"selfcoupled": "constant", "terms": "constant", "hurricane": "constant"}.get(
            kind, rng.choice(["field", "field", "constant", "infinite"]))
        c["smooth"] = kind == "swell" and rng.random() < 0.5
        if _cost(c) <= limit and c["Nx"] * c["Ny"] * c["Nk"] * c["Np"] >= 60000:
            return c


# --------------------------------------------------------------------- inputs, made from the seed alone
def _wrapped(a, b, L):
    d = a - b
    return d - L * np.round(d / L)


def _inputs(case, seed):
    """The physical inputs of a case as plain numpy arrays and numbers (x is the first index)."""
    rng = np.random.default_rng(1000003 * seed + 17)
    Nx, Ny, Nk, Np, Nz = (case[k] for k in ("Nx", "Ny", "Nk", "Np", "Nz"))
    kind = case["kind"]
    vortex = kind == "currents" and case["depth"] == "infinite"
    swell = kind == "selfcoupled"
    dx = 1.25 * 64 / Nx if vortex else (2000.0 if swell else 5.12e6 / max(Nx, Ny))
    Lx, Ly = Nx * dx, Ny * dx
    x, y = (np.arange(Nx) + 0.5) * dx, (np.arange(Ny) + 0.5) * dx
    X, Y = np.meshgrid(x, y, indexing="ij")
    if vortex:
        kappa = np.linspace(0.3, 0.5, Nk)
    elif swell:
        kappa = np.geomspace(0.01, 0.3, Nk)
    else:
        kappa = np.geomspace(0.003, 0.4, Nk)
    phi = np.arange(Np) * (2.0 * math.pi / Np)
    kf = np.empty(Nk + 1)
    kf[1:-1] = (kappa[:-1] + kappa[1:]) / 2.0
    kf[0] = max(kappa[0] - (kf[1] - kappa[0]), 0.0)
    kf[-1] = kappa[-1] + (kappa[-1] - kf[-2])
    dphi = 2.0 * math.pi / Np
    pf = np.array([phi[0] - dphi / 2.0 + i * dphi for i in range(Np + 1)])
    d = dict(dx=dx, Lx=Lx, Ly=Ly, x=x, y=y, kappa=kappa, phi=phi, kf=kf, pf=pf, depth=None, u=None, v=None)

    # depth
    if case["depth"] == "constant":
        d["depth"] = 50.0 if swell else 4000.0
    elif case["depth"] == "field":
        h = np.full((Nx, Ny), 4000.0)
        for _ in range(3):
            w = rng.uniform(0.02, 0.05) * Lx
            r2 = _wrapped(X, rng.uniform(0, Lx), Lx) ** 2 + _wrapped(Y, rng.uniform(0, Ly), Ly) ** 2
            h -= rng.uniform(3000.0, 3900.0) * np.exp(-r2 / (2 * w * w))
        d["depth"] = np.asfortranarray(np.maximum(h, 100.0))

    # currents on the levels of the Q grid
    grad = umax = 0.0
    if kind in ("currents", "tides"):
        zf = np.linspace(-1.0, 0.0, Nz + 1) if vortex else -4000.0 * (1.0 - np.arange(Nz + 1) / Nz)
        z = 0.5 * (zf[:-1] + zf[1:])
        us, vs = np.zeros((Nx, Ny)), np.zeros((Nx, Ny))
        if vortex:
            a, U0 = Lx / 8.0, rng.uniform(0.3, 0.45)
            ex, ey = X - Lx / 2, Y - Ly / 2
            r = np.maximum(np.hypot(ex, ey), 1e-9)
            ut = U0 * (r / a) * np.exp(0.5 - 0.5 * (r / a) ** 2)
            us, vs = -ut * ey / r, ut * ex / r
            decay = np.ones(Nz)
        else:
            for _ in range(8):
                R = rng.uniform(0.008, 0.024) * Lx
                A = (1.0 if rng.uniform() < 0.5 else -1.0) * 0.5 * R * math.exp(0.5) / math.sqrt(2.0)
                ex, ey = _wrapped(X, rng.uniform(0, Lx), Lx), _wrapped(Y, rng.uniform(0, Ly), Ly)
                e = A * 2.0 / R ** 2 * np.exp(-(ex ** 2 + ey ** 2) / R ** 2)
                us += ey * e
                vs -= ex * e
            decay = np.exp(z / 200.0)
        d["zf"] = zf
        u, v = np.empty((Nx, Ny, Nz), order="F"), np.empty((Nx, Ny, Nz), order="F")
        for k in range(Nz):
            u[:, :, k] = us * decay[k]
            v[:, :, k] = vs * decay[k]
        d["u"], d["v"] = u, v
        umax = float(np.max(np.hypot(us, vs)))
        grad = max(float(np.max(np.abs(f - np.roll(f, 1, a)))) for f in (us, vs) for a in (0, 1)) / dx
    if swell:
        grad, umax = 2.0 * 0.3 / (Lx / 6), 0.3
    # time step from the CFL sum
    H = float(np.max(d["depth"])) if d["depth"] is not None else None
    cg = 0.5 * math.sqrt(G / kappa[0]) * (1.0 if H is None else 1.2) + umax
    rate = 2 * cg / dx + kappa[-1] * 2 * grad / (kf[1] - kf[0]) + 2 * grad / dphi
    d["dt"] = 0.4 / rate

    # spectrum and envelope of the initial action
    K, P = np.meshgrid(kappa, phi, indexing="ij")
    if vortex:
        spec = np.exp(-((K - 0.4) / 0.05) ** 2 - np.sin(P / 2.0) ** 2 / 0.3 ** 2)
    else:
        kp, phi0 = rng.uniform(0.02, 0.05), rng.uniform(0, 2 * math.pi)
        sig, sp = np.sqrt(G * kappa), math.sqrt(G * kp)
        w = np.where(sig <= sp, 0.07, 0.09)
        E = sig ** -5.0 * np.exp(-1.25 * (sp / sig) ** 4) * 3.3 ** np.exp(-((sig - sp) ** 2) / (2 * w * w * sp * sp))
        spec = np.outer(E / E.max(), np.cos((phi - phi0) / 2.0) ** 20)
    if swell:
        env = np.exp(-(_wrapped(X, rng.uniform(0, Lx), Lx) ** 2 + _wrapped(Y, rng.uniform(0, Ly), Ly) ** 2)
                     / (2 * (Lx / 6) ** 2))
        spec, floor = 4e4 * spec, 1e-3
    else:
        a, b = rng.uniform(0, 2 * math.pi, 2)
        env = 1.0 + 0.3 * np.sin(2 * math.pi * X / Lx + a) * np.cos(4 * math.pi * Y / Ly + b)
        # a storm starts from a calm sea under a weak swell
        spec, floor = (0.02 * spec, 1e-6) if kind == "hurricane" else (spec, 1e-5 if kind == "terms" else 0.0)
    d["spec"], d["env"], d["floor"] = spec, env, floor

    if kind == "hurricane":
        c0 = (rng.uniform(0.3, 0.7) * Lx, rng.uniform(0.2, 0.4) * Ly)
        d["storm"] = dict(t0=0.0, t1=1e6, c0=c0, c1=(c0[0], c0[1] + 5.0e6), vmax=rng.uniform(40.0, 55.0),
                          rmax=30e3, radius=500e3, B=1.5, inflow=math.radians(20.0))
    if kind == "terms":
        d["terms"] = dict(
            rate=np.asfortranarray(1e-5 * (1.0 + 0.5 * np.sin(2 * math.pi * X / Lx))), dir1=rng.uniform(0, 6.0),
            dir2=rng.uniform(0, 6.0), speed=rng.uniform(8.0, 15.0))
    return d


def _initial(case, d):
    """The initial action on the device in the caller's layout: (Np, Nk, Ny, Nx), x fastest."""
    dt = torch.float64 if case["precision"] == "fp64" else torch.float32
    spec = torch.from_numpy(np.ascontiguousarray(d["spec"].T)).cuda()
    env = torch.from_numpy(np.ascontiguousarray(d["env"].T)).cuda()
    N = torch.empty((case["Np"], case["Nk"], case["Ny"], case["Nx"]), dtype=dt, device="cuda")
    for n in range(case["Np"]):
        N[n] = spec[n][:, None, None] * env + d["floor"]
    return N


def _network(case, seed):
    g = np.random.default_rng(seed)
    B, H = case["nbins"], case["hidden"]
    parts = []
    for shape, scale in (((H, B), B ** -0.5), ((H, 4), 0.5), ((H,), 0.1), ((H, H), H ** -0.5), ((H,), 0.1),
                         ((H, H), H ** -0.5), ((H,), 0.1), ((B, H), H ** -0.5), ((B,), 0.1)):
        parts.append((scale * g.standard_normal(shape)).astype(np.float32).ravel())
    t = torch.Generator(device="cuda")
    t.manual_seed(seed)
    X = torch.randn((case["rows"], B), generator=t, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    E = torch.rand((case["rows"], 4), generator=t, device="cuda", dtype=torch.float32)
    return np.concatenate(parts), X, E


# ------------------------------------------------------------------------------------ prepare and run
class _State:
    pass


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    s = _State()
    s.case = case
    if case["kind"] == "network":
        params, s.X, s.E = _network(case, seed)
        s.net = rp.learned.SourceNetwork(nbins=case["nbins"], hidden=case["hidden"], rows=16384)
        s.net.set_params(params)
        torch.cuda.synchronize()
        return s
    d = _inputs(case, seed)
    Nx, Ny, Nz, kind = case["Nx"], case["Ny"], case["Nz"], case["kind"]
    x, y = (0.0, d["Lx"]), (0.0, d["Ly"])
    if d["u"] is not None:
        grid = rp.RectilinearGrid(size=(Nx, Ny, Nz), x=x, y=y, z=list(d["zf"]),
                                  topology=("Periodic", "Periodic", "Bounded"))
    else:
        grid = rp.RectilinearGrid(size=(Nx, Ny), x=x, y=y, topology=("Periodic", "Periodic", "Flat"))
    sg = rp.PolarWaveVectorGrid(κ=d["kappa"], φ=d["phi"])
    depth = rp.InfiniteDepth() if d["depth"] is None else d["depth"]
    velocities = sources = None
    if kind in ("currents", "tides"):
        velocities = {"u": d["u"], "v": d["v"]}
    elif kind == "selfcoupled":
        velocities = rp.PseudomomentumVelocities()
    if kind == "hurricane":
        st = d["storm"]
        wind = rp.HollandHurricaneWind(center=rp.LinearStormTrack([st["t0"], st["t1"]], [st["c0"], st["c1"]]),
                                       vmax=st["vmax"], rmax=st["rmax"], radius=st["radius"],
                                       shape_parameter=st["B"], inflow_angle=st["inflow"])
        sources = rp.PrecomputedSources(
            wind_input=rp.PressureCorrelationInput(drag=rp.BulkWindDrag("linear"), wind=wind),
            dissipation=rp.LocalSaturationDissipation(B_r=1.05e-2, σ_power=1.0))
    elif kind == "terms":
        t = d["terms"]
        sources = rp.SourceTermSet(
            rp.ExponentialWindInput(rate=t["rate"], direction=t["dir1"], spreading_power=2.0),
            rp.WaveAgeWindInput(rate=2e-6, speed=t["speed"], direction=t["dir2"]),
            rp.WhitecappingDissipation(rate=1e-6, saturation_threshold=1e-4, wavenumber_power=2.0,
                                       reference_wavenumber=0.1),
            rp.MeanSpectrumWhitecapping())
    s.model = rp.SpectralWaveModel(grid, sg, depth=depth, velocities=velocities, sources=sources,
                                   propagation_smoothing=rp.SpatialAveraging() if case["smooth"] else None,
                                   precision=case["precision"])
    s.lib = rp.load_library()
    s.dt = d["dt"]
    s.code = F64 if case["precision"] == "fp64" else F32
    s.N0 = _initial(case, d)
    s.out = torch.empty_like(s.N0)
    if kind == "tides":
        # the next currents, as a circulation model hands them over: float64, x fastest
        def cur(a, f):
            return torch.from_numpy(np.ascontiguousarray((f * a).T)).cuda().permute(2, 1, 0)
        s.u, s.v = cur(d["u"], 0.8), cur(d["v"], 1.1)
        s.fields = torch.empty((4, Ny, Nx), dtype=torch.float64, device="cuda")
        s.total = torch.empty(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return s


def _check(status):
    if status:
        raise RuntimeError(rp.load_library().rpl_last_error().decode())


def run(s):
    if s.case["kind"] == "network":
        return s.net.forward(s.X, s.E)
    m = s.model
    m.clock.time, m.clock.iteration = 0.0, 0
    _check(s.lib.rpl_set_action_device(m.handle, _ptr(s.N0), s.code, XFAST))
    if s.case["kind"] == "tides":
        rp.diagnostics_device(m, m0=s.fields[0], hs=s.fields[1], kappa_rms=s.fields[2], mean_direction=s.fields[3],
                              total_action=s.total)
        m.update_currents(s.u, s.v)
    rp.time_step(m, s.dt, nsteps=s.case["steps"])
    _check(s.lib.rpl_get_action_device(m.handle, _ptr(s.out), s.code, XFAST))
    return (s.out, s.fields, s.total) if s.case["kind"] == "tides" else s.out


# ---------------------------------------------------------------------------------------- bytes and flops
def work(case):
    """Bytes: the initial action in and the final one out (caller's layout, to and from the state), and per
    step the three stages' reads and writes of the state (N0 -> N1; N1, N0 -> N2; N2, N0 -> N3) with the
    per-(i, j, kappa) coupling; flops: four WENO5 faces per cell-bin and stage at 60, plus sources."""
    if case["kind"] == "network":
        r, B, H = case["rows"], case["nbins"], case["hidden"]
        return {"bytes": r * (2 * B + 16 + 4 * B) + 2 * (2 * B * H + 2 * H * H),
                "flops": 2.0 * r * (2 * B * H + 2 * H * H)}
    w = 8 if case["precision"] == "fp64" else 4
    cells = case["Nx"] * case["Ny"]
    units = cells * case["Nk"] * case["Np"]
    kind, steps = case["kind"], case["steps"]
    refract = kind in ("currents", "tides", "selfcoupled")
    per_step = 8 * w * units + (3 * cells * case["Nk"] * 6 * w if refract else 0)
    if case["smooth"]:
        per_step += 2 * w * units
    if kind in ("hurricane", "terms", "selfcoupled"):
        per_step += 3 * w * units          # a column's integrals come before its bins' tendencies
    total = 4 * w * units + steps * per_step
    if kind == "tides":
        total += w * units + 2 * cells * case["Nz"] * 8 + 4 * cells * 8
    flops = steps * 3 * units * (4 * 60 if refract else 2 * 60)
    if kind in ("hurricane", "terms"):
        flops += steps * 3 * units * 30
    return {"bytes": float(total), "flops": float(flops)}


# ------------------------------------------------------------------------- the same in 64-bit torch
EPS = 1e4 * 2.0 ** -52


def _weno(a, b, c, d, e):
    """Jiang-Shu WENO5 value at the face between c and d, upwind side first."""
    v0 = a / 3.0 - 7.0 / 6.0 * b + 11.0 / 6.0 * c
    v1 = -b / 6.0 + 5.0 / 6.0 * c + d / 3.0
    v2 = c / 3.0 + 5.0 / 6.0 * d - e / 6.0
    w0 = 0.1 / (EPS + 13.0 / 12.0 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2) ** 2
    w1 = 0.6 / (EPS + 13.0 / 12.0 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2) ** 2
    w2 = 0.3 / (EPS + 13.0 / 12.0 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2) ** 2
    return (w0 * v0 + w1 * v1 + w2 * v2) / (w0 + w1 + w2)


def _both(at, vel):
    """N(+1/2) - N(-1/2) times vel; at(k) is the field shifted by k cells. Each cell's faces upwind by vel."""
    s = [at(k) for k in range(-3, 4)]
    left, right = _weno(*s[0:5]), _weno(*s[1:6])                  # faces -1/2 and +1/2 from the left
    diff = torch.where(vel >= 0, right - left, _weno(s[6], s[5], s[4], s[3], s[2]) - _weno(s[5], s[4], s[3], s[2], s[1]))
    return vel * diff


def _kappa_flux(N, vel):
    """vel * (F(m+1/2) - F(m-1/2)) along kappa (dim 0): first-order upwind near the ends, no flux through them."""
    Nk = N.shape[0]
    m = torch.arange(Nk, device=N.device)

    def at(k):
        return N[(m + k).clamp(0, Nk - 1)]

    pos = vel >= 0
    full_hi = ((m - 2 >= 0) & (m + 3 <= Nk - 1))[:, None, None]
    full_lo = ((m - 3 >= 0) & (m + 2 <= Nk - 1))[:, None, None]
    s = {k: at(k) for k in range(-3, 4)}
    hi = torch.where(pos, _weno(s[-2], s[-1], s[0], s[1], s[2]), _weno(s[3], s[2], s[1], s[0], s[-1]))
    lo = torch.where(pos, _weno(s[-3], s[-2], s[-1], s[0], s[1]), _weno(s[2], s[1], s[0], s[-1], s[-2]))
    hi = torch.where(full_hi, hi, torch.where(pos, s[0], s[1])) * vel
    lo = torch.where(full_lo, lo, torch.where(pos, s[-1], s[0])) * vel
    hi[Nk - 1] = 0.0
    lo[0] = 0.0
    return hi - lo


def _q_cdf(kappa, z, d):
    """CDF over depth of the transform's kernel at z, per (kappa) x (cells); d a number or a (Ny, Nx) field."""
    mu = kappa * d
    s = torch.as_tensor((z + d) / d, dtype=torch.float64, device="cuda").clamp(0.0, 1.0)
    return (torch.exp(2 * mu * (s - 1)) - torch.exp(-2 * mu * (s + 1))) / (1 - torch.exp(-4 * mu))


class _Exact:
    def __init__(self, case, d):
        def f(a):
            return torch.from_numpy(np.ascontiguousarray(a)).cuda().to(torch.float64)
        self.case, self.d = case, d
        self.kap, self.phi, self.kf, self.pf = f(d["kappa"]), f(d["phi"]), f(d["kf"]), f(d["pf"])
        self.cos, self.sin = torch.cos(self.phi), torch.sin(self.phi)
        k1, k2, p1, p2 = self.kf[:-1], self.kf[1:], self.pf[:-1], self.pf[1:]
        self.w = ((p2 - p1)[:, None] * (k2 ** 2 - k1 ** 2)[None] / 2)              # (Np, Nk) measures
        r1, r2 = (k2 ** 3 - k1 ** 3) / 3, (k2 ** 4 - k1 ** 4) / 4
        ds, dc = torch.sin(p2) - torch.sin(p1), torch.cos(p1) - torch.cos(p2)
        self.mx, self.my = ds[:, None] * r1, dc[:, None] * r1
        self.tr = (p2 - p1)[:, None] * r2
        H = d["depth"]
        self.H = f(H.T) if isinstance(H, np.ndarray) else H
        K = self.kap[:, None, None]
        if H is None:
            radial = (k2 ** 1.5 - k1 ** 1.5) / 1.5
            scale = math.sqrt(G) / (2 * self.w)
            self.gx, self.gy = scale * radial * ds[:, None], scale * radial * dc[:, None]
            self.cg = torch.ones((), dtype=torch.float64, device="cuda")
        else:
            mu = K * self.H
            self.cg = (1 + 2 * mu / torch.sinh(2 * mu)) / 2 * torch.sqrt(G * torch.tanh(mu) / K)
            self.gx, self.gy = self.cos[:, None].expand_as(self.w), self.sin[:, None].expand_as(self.w)
        self.refract = case["kind"] in ("currents", "tides", "selfcoupled")
        self.F = f
        self.t = 0.0

    def currents(self, u, v, zf, depth):
        u, v = self.F(u.T), self.F(v.T)                                              # (Nz, Ny, Nx)
        K = self.kap[:, None, None]
        Ux = Uy = 0.0
        lo = _q_cdf(K, zf[0], depth)
        for k in range(u.shape[0]):
            hi = _q_cdf(K, zf[k + 1], depth)
            Ux, Uy = Ux + u[k] * (hi - lo), Uy + v[k] * (hi - lo)
            lo = hi
        self.velocity(Ux, Uy)

    def velocity(self, Ux, Uy):
        h = 0.5 / self.d["dx"]

        def ddx(a, dim):
            return (torch.roll(a, -1, dim) - torch.roll(a, 1, dim)) * h
        self.U = (Ux, Uy, ddx(Ux, 2), ddx(Ux, 1), ddx(Uy, 2), ddx(Uy, 1))

    def overlap(self):
        """Pseudomomentum coupling of rings t and s on the automatic stretched vertical grid."""
        H, kmax = self.H, float(self.kap[-1])
        Nz = max(16, math.ceil((H / (1.0 / (20.0 * kmax))) ** 0.5))
        z = [-H * (1.0 - k / Nz) ** 2 for k in range(Nz + 1)]
        F = torch.stack([_q_cdf(self.kap, zk, H) for zk in z])
        Q = F[1:] - F[:-1]
        dz = torch.tensor([z[k + 1] - z[k] for k in range(Nz)], dtype=torch.float64, device="cuda")
        self.O = torch.einsum("kt,ks->ts", Q / dz[:, None], Q)

    def self_velocity(self, N):
        Mx = sum(N[n] * self.mx[n][:, None, None] for n in range(N.shape[0]))
        My = sum(N[n] * self.my[n][:, None, None] for n in range(N.shape[0]))
        self.velocity(torch.einsum("ts,syx->tyx", self.O, Mx), torch.einsum("ts,syx->tyx", self.O, My))

    def wind(self):
        st = self.d["storm"]
        w = (self.t - st["t0"]) / (st["t1"] - st["t0"])
        cx, cy = (st["c0"][i] * (1 - w) + st["c1"][i] * w for i in (0, 1))
        dx, dy = self.F(self.d["x"])[None, :] - cx, self.F(self.d["y"])[:, None] - cy
        r = torch.hypot(dx, dy)
        shape = (st["rmax"] / r) ** st["B"]
        speed = st["vmax"] * torch.sqrt(shape * torch.exp(1 - shape))
        speed = torch.where(r > st["radius"], speed * torch.exp(-(r - st["radius"]) / (st["radius"] - st["rmax"])), speed)
        ci, si = math.cos(st["inflow"]), math.sin(st["inflow"])
        vx, vy = speed * (-ci * dy - si * dx) / r, speed * (ci * dx - si * dy) / r
        self.U10, self.th = torch.hypot(vx, vy), torch.atan2(vy, vx)
        self.us = self.U10 * torch.sqrt((0.8 + 0.065 * self.U10) * 1e-3)

    def growth(self, n):
        """Janssen growth rate of direction n before the cap: beta_max 1.2, z_alpha 0.011, alpha0 0.0095."""
        k = self.kap[:, None, None]
        sig = torch.sqrt(G * k)
        ct = torch.cos(self.phi[n] - self.th)
        age = self.us * k / sig + 0.011
        Z = torch.log(k * 0.0095 * self.us ** 2 / G) + 0.4 / (age * ct)
        ok = (ct > 0) & (Z < 0) & (self.us > 0)
        Z = torch.where(ok, Z, torch.zeros_like(Z))
        r = (1.225 / 1025.0) * 1.2 / 0.16 * torch.exp(Z) * Z ** 4 * age ** 2 * ct ** 2 * sig
        return torch.where(ok, r, torch.zeros_like(r))

    def stress(self, N):
        tx = ty = 0.0
        slow = torch.sqrt(self.kap / G)[:, None, None]                                # k / sigma
        for n in range(N.shape[0]):
            f = (self.growth(n) * N[n].clamp(min=0) * slow * self.w[n][:, None, None]).sum(0) * 1025.0 * G
            tx, ty = tx + f * self.cos[n], ty + f * self.sin[n]
        par = (tx * torch.cos(self.th) + ty * torch.sin(self.th)).clamp(min=0)
        top = 0.4 * 1.225 * self.us ** 2
        self.factor = torch.where(par > top, top / par, torch.ones_like(par))

    def term_values(self, N):
        """Column integrals of the SourceTermSet: m0, and the mean wavenumber and frequency at p = 1/2."""
        m0 = sk = ss = sd = 0.0
        k = self.kap
        for n in range(N.shape[0]):
            a = N[n] * self.w[n][:, None, None]
            b = a.clamp(min=0)
            m0, sd = m0 + a.sum(0), sd + b.sum(0)
            sk = sk + (b * (k ** 0.5)[:, None, None]).sum(0)
            ss = ss + (b * (torch.sqrt(G * k) ** 0.5)[:, None, None]).sum(0)
        self.m0, self.kbar, self.sbar = m0, (sk / sd) ** 2, (ss / sd) ** 2

    def term_rate(self, n):
        t = self.d["terms"]
        k = self.kap[:, None, None]

        def cos2(a, b):                # integral of max(cos, 0)^2 over [a, b]
            s = 0.0
            for q in range(-2, 3):
                lo, hi = max(a, q * 2 * math.pi - math.pi / 2), min(b, q * 2 * math.pi + math.pi / 2)
                if hi > lo:
                    s += 0.5 * (hi - lo) + 0.25 * (math.sin(2 * hi) - math.sin(2 * lo))
            return s
        p1, p2 = float(self.pf[n]), float(self.pf[n + 1])
        r = self.F(t["rate"].T) * (cos2(p1 - t["dir1"], p2 - t["dir1"]) / (p2 - p1))
        al = max(math.cos(float(self.phi[n]) - t["dir2"]), 0.0)
        r = r + 2e-6 * (t["speed"] * al / torch.sqrt(G / k) - 0.83).clamp(min=0) * al
        k1, k2 = self.kf[:-1], self.kf[1:]
        k2avg = ((k2 ** 4 - k1 ** 4) / 4 / ((k2 ** 2 - k1 ** 2) / 2) / 0.1 ** 2)[:, None, None]
        r = r - 1e-6 * (self.m0 / 1e-4 - 1).clamp(min=0) * k2avg
        q = k / self.kbar
        return r - 2.1 * (self.m0 * self.kbar ** 2) ** 2 * self.sbar * (0.4 * q + 0.6 * q * q)

    def tendency(self, N):
        """Yields dN/dt of one direction at a time."""
        kind = self.case["kind"]
        if kind == "selfcoupled":
            self.self_velocity(N)
        if kind == "hurricane":
            self.stress(N)
        if kind == "terms":
            self.term_values(N)
        Np, dxi = N.shape[0], 1.0 / self.d["dx"]
        dki, dpi = 1.0 / float(self.kf[1] - self.kf[0]), 1.0 / float(self.pf[1] - self.pf[0])
        K = self.kap[:, None, None]
        for n in range(Np):
            a = N[n]
            ux, uy = self.cg * self.gx[n][:, None, None], self.cg * self.gy[n][:, None, None]
            if self.refract:
                Ux, Uy, Uxx, Uxy, Uyx, Uyy = self.U
                ux, uy = ux + Ux, uy + Uy
            g = -_both(lambda k: torch.roll(a, -k, 2), ux) * dxi
            g -= _both(lambda k: torch.roll(a, -k, 1), uy) * dxi
            if self.refract:
                c, s = float(self.cos[n]), float(self.sin[n])
                g -= _kappa_flux(a, -K * (c * c * Uxx + c * s * (Uyx + Uxy) + s * s * Uyy)) * dki
                g -= _both(lambda k: N[(n + k) % Np], c * s * (Uxx - Uyy) + s * s * Uyx - c * c * Uxy) * dpi
            if kind == "hurricane":
                g += self.growth(n) * self.factor * a
                sig = torch.sqrt(G * K)
                over = (a * sig * K ** 3 / 1.05e-2 - 1).clamp(0, 1e6)
                g -= torch.where(a > 0, 2.2e-5 * sig * over ** 2 * a, torch.zeros_like(a))
            if kind == "terms":
                g += self.term_rate(n) * a
            yield n, g

    def smooth(self, N):
        """Mean of four bilinear samples around each cell: half-widths 0.5 dcg dt along, 0.5 cg dphi dt across."""
        out = torch.empty_like(N)
        c = 0.5 * np.sqrt(G / self.d["kappa"])
        dc = np.abs(np.concatenate([c[:1], c[:-1]]) - np.concatenate([c[1:], c[-1:]])) / 2
        dphi = float(self.pf[1] - self.pf[0])
        for n in range(N.shape[0]):
            cs, sn = float(self.cos[n]), float(self.sin[n])
            for m in range(N.shape[1]):
                ls, ln = (0.5 * v * self.dt / self.d["dx"] for v in (dc[m], c[m] * dphi))
                acc = 0.0
                for s1 in (-1, 1):
                    for s2 in (-1, 1):
                        di, dj = s1 * ls * cs - s2 * ln * sn, s1 * ls * sn + s2 * ln * cs
                        fi, fj = math.floor(di), math.floor(dj)
                        wi, wj = di - fi, dj - fj
                        for a, wa in ((fi, 1 - wi), (fi + 1, wi)):
                            for b, wb in ((fj, 1 - wj), (fj + 1, wj)):
                                acc = acc + wa * wb / 4 * torch.roll(N[n, m], (-b, -a), (0, 1))
                out[n, m] = acc
        return out

    def step(self, N0, dt):
        self.dt = dt
        if self.case["kind"] == "hurricane":
            self.wind()
        N = N0
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            new = torch.empty_like(N)
            for n, g in self.tendency(N):
                new[n] = (a * N0[n] + b * (N[n] + dt * g).clamp(min=0)).clamp(min=0)
            N = new
        self.t += dt
        return self.smooth(N) if self.case["smooth"] else N


def _exact_network(case, seed):
    params, X, E = _network(case, seed)
    B, H = case["nbins"], case["hidden"]
    p, at = [], 0
    for shape in ((H, B), (H, 4), (H,), (H, H), (H,), (H, H), (H,), (B, H), (B,)):
        size = int(np.prod(shape))
        p.append(torch.from_numpy(params[at:at + size].reshape(shape)).cuda().double())
        at += size
    W1, W1e, b1, W2, b2, W3, b3, W4, b4 = p

    def act(z):
        return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))
    Y = torch.empty((case["rows"], B), dtype=torch.float64, device="cuda")
    for r in range(0, case["rows"], 16384):
        x, e = X[r:r + 16384].double(), E[r:r + 16384].double()
        h = act(x @ W1.T + e @ W1e.T + b1)
        Y[r:r + 16384] = act(act(h @ W2.T + b2) @ W3.T + b3) @ W4.T + b4
    return Y


def exact(case, seed):
    if case["kind"] == "network":
        return _exact_network(case, seed)
    if case["Nx"] * case["Ny"] * case["Nk"] * case["Np"] * case["steps"] > 1.6e9:
        return None
    d = _inputs(case, seed)
    N = _initial(case, d).double()
    e = _Exact(case, d)
    fields = total = None
    if case["kind"] == "tides":
        def sums(w):
            return sum(torch.einsum("m,myx->yx", w[n], N[n]) for n in range(case["Np"]))
        m0 = sums(e.w)
        fields = torch.stack([m0, 4 * torch.sqrt(m0), torch.sqrt(sums(e.tr) / m0),
                              torch.atan2(sums(e.my), sums(e.mx))])
        total = (m0.sum() * d["dx"] ** 2).reshape(1)
        e.currents(0.8 * d["u"], 1.1 * d["v"], d["zf"], e.H if e.H is not None else -d["zf"][0])
    elif case["kind"] == "currents":
        e.currents(d["u"], d["v"], d["zf"], e.H if e.H is not None else -d["zf"][0])
    elif case["kind"] == "selfcoupled":
        e.overlap()
    for _ in range(case["steps"]):
        N = e.step(N, d["dt"])
    return (N, fields, total) if case["kind"] == "tides" else N
