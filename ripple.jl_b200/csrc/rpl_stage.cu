// rpl_stage.cu -- fused SSP-RK3 stage kernels: tendency (Doppler transport + refraction, or intrinsic
// transport) + sources + stage combination + max(0, .) clamp, one pass over the state per stage.
//
// Reference: src/Coupling/wave_current_refraction.jl:74-151 (tendency),
// src/Models/intrinsic_transport.jl:14-68, src/Models/tendencies.jl:28-41,82-101 (dispatch, sources),
// src/Models/time_step.jl:67-74,98-105,138-152 (stage update with clamp).
//
// Device layout of the state: kappa fastest, (i,j,m,n) at ((n*Ny + j)*Nx + i)*Nk + m.
//
// column_kernel (Nk <= 32): one warp segment of SEG lanes (SEG = Nk rounded up to a power of two)
// owns one horizontal cell (i,j) and walks the periodic phi ring n = 0 .. Np-1, lane m holding
// kappa bin m. Every face is reconstructed once where it can be:
//   kappa faces: the + face of lane m is the - face of lane m+1 (warp shuffle); the clamped kappa
//     stencil of the reference is a shuffle from the clamped lane;
//   phi faces: a 7-deep register window along the ring; the + face of step n is the - face of
//     step n+1;
//   x, y faces: both faces of the cell from one 7-point stencil, sharing its differences.
// A face is recomputed only where the two cells on its sides upwind in different directions
// (the reference upwinds each cell's two faces by that cell's own centre velocity).
// The per-(i,j,kappa) coupling record is read once per ring, i.e. once per Np cell-bins.
//
// generic_kernel (any Nk): one thread per cell-bin, same arithmetic, all neighbours from memory.
#include <cuda_runtime.h>

#include <type_traits>

#include "rpl_device.cuh"
#include "rpl_flux.cuh"
#include "rpl_internal.h"
#include "rpl_walk.h"

namespace rpl {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int BLOCK = 256;


// FP32 copy of a coefficient record, made once per ring so the per-cell-bin work stays in FP32.
struct CoefF {
    float k, Uxx, Uxy, Uyx, Uyy, Ux, Uy, cg;
};

__device__ __forceinline__ CoefF to_f32(const Coef& q) {
    return CoefF{(float)q.kap, (float)q.Uxx, (float)q.Uxy, (float)q.Uyx, (float)q.Uyy,
                 (float)q.Ux,  (float)q.Uy,  (float)q.cg};
}

// FP32 velocities from the FP32 direction and group-velocity tables (same expression order).
__device__ __forceinline__ void velocities_f32(const CoefF& q, float4 tg, float2 g, bool per_cell, bool refract,
                                               float& ux, float& uy, float& ck, float& cp) {
    const float gx = per_cell ? q.cg * g.x : g.x;
    const float gy = per_cell ? q.cg * g.y : g.y;
    if (!refract) {
        ux = gx;
        uy = gy;
        ck = cp = 0.0f;
        return;
    }
    ck = -q.k * (tg.x * q.Uxx + tg.y * (q.Uyx + q.Uxy) + tg.z * q.Uyy);
    cp = tg.y * (q.Uxx - q.Uyy) + tg.z * q.Uyx - tg.x * q.Uxy;
    ux = gx + q.Ux;
    uy = gy + q.Uy;
}

__device__ __forceinline__ int wrapi(int i, int N) { return i < 0 ? i + N : (i >= N ? i - N : i); }

// Stage epilogue: clamp, combine with N0, error word (time_step.jl:67-74,98-105).
template <typename T>
__device__ __forceinline__ T stage_out(const StageParams& p, T a, T G, T n0) {
    const T st = relu(a + T(p.dt) * G);
    return p.stage == 1 ? st : relu(T(p.a) * n0 + T(p.b) * st);
}

template <typename T, int SEG, bool REFRACT, bool TENDENCY>
__global__ void __launch_bounds__(BLOCK) column_kernel(const T* __restrict__ Nin, const T* N0, T* Nout,
                                                       double* __restrict__ Gout, StageParams p) {
    constexpr int CPW = 32 / SEG;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = lane & (SEG - 1);
    const int base = lane - m;
    const int Nx = (int)p.Nx, Ny = (int)p.Ny, Nk = (int)p.Nk, Np = (int)p.Np;
    const int64_t P = (int64_t)Nx * Ny, Pr = (int64_t)Nx * (p.j_hi - p.j_lo);  // Pr: cells of the updated rows
    const int64_t col = ((int64_t)blockIdx.x * (BLOCK / 32) + warp) * CPW + lane / SEG;
    const bool live = col < Pr && m < Nk;
    const int64_t cc = (col < Pr ? col : Pr - 1) + (int64_t)Nx * p.j_lo;
    const int mm = m < Nk ? m : Nk - 1;
    const int i = (int)(cc % Nx), j = (int)(cc / Nx);
    const Coef q = load_coef(p.coef + 8 * (cc * Nk + mm));
    const CoefF qf = to_f32(q);
    // offsets of the x and y neighbours (periodic)
    const int64_t xs = Nk, ys = (int64_t)Nx * Nk;
    const int64_t xo1 = (wrapi(i + 1, Nx) - i) * xs, xo2 = (wrapi(i + 2, Nx) - i) * xs, xo3 = (wrapi(i + 3, Nx) - i) * xs;
    const int64_t xn1 = (wrapi(i - 1, Nx) - i) * xs, xn2 = (wrapi(i - 2, Nx) - i) * xs, xn3 = (wrapi(i - 3, Nx) - i) * xs;
    const int64_t yo1 = (wrapi(j + 1, Ny) - j) * ys, yo2 = (wrapi(j + 2, Ny) - j) * ys, yo3 = (wrapi(j + 3, Ny) - j) * ys;
    const int64_t yn1 = (wrapi(j - 1, Ny) - j) * ys, yn2 = (wrapi(j - 2, Ny) - j) * ys, yn3 = (wrapi(j - 3, Ny) - j) * ys;
    const int64_t slice = P * Nk;
    const int64_t home = cc * Nk + mm;  // offset within a slice
    // phi window: bins n-3 .. n+3 of this lane's (i,j,m); refraction needs Np >= 3, so one wrap suffices
    T w0 = T(0), w1 = T(0), w2 = T(0), w3 = T(0), w4 = T(0), w5 = T(0), w6 = T(0);
    if constexpr (REFRACT) {
        w0 = Nin[home + slice * wrapi(-3, Np)];
        w1 = Nin[home + slice * wrapi(-2, Np)];
        w2 = Nin[home + slice * wrapi(-1, Np)];
        w3 = Nin[home];
        w4 = Nin[home + slice * wrapi(1, Np)];
        w5 = Nin[home + slice * wrapi(2, Np)];
        w6 = Nin[home + slice * wrapi(3, Np)];
    }
    const T dx_inv = T(p.dx_inv), dy_inv = T(p.dy_inv), dk_inv = T(p.dk_inv), dp_inv = T(p.dp_inv);
    const bool hp = (m - 2 >= 0) && (m + 3 <= Nk - 1);   // kappa + face has its WENO stencil
    const bool hm = (m - 3 >= 0) && (m + 2 <= Nk - 1);   // kappa - face
    T prevF = T(0);
    bool prevPos = false, havePrev = false;
    for (int n = 0; n < Np; ++n) {
        const int64_t at = home + slice * n;
        T nxt = T(0);
        if constexpr (REFRACT) nxt = Nin[home + slice * ((n + 4) % Np)];  // next window entry
        else w3 = Nin[at];
        const T c0 = w3;
        T ux, uy, ck, cp;
        if constexpr (std::is_same<T, float>::value) {
            velocities_f32(qf, __ldg(p.trig32 + n), __ldg(p.cg32 + mm + Nk * n), p.cg_per_cell, REFRACT, ux, uy,
                           ck, cp);
        } else {
            const double cph = __ldg(p.cosp + n), sph = __ldg(p.sinp + n);
            const double cgx = __ldg(p.cg_x + mm + Nk * n), cgy = __ldg(p.cg_y + mm + Nk * n);
            velocities<T>(q, cph, sph, cgx, cgy, p.cg_per_cell, REFRACT, ux, uy, ck, cp);
        }
        // x and y
        const T* row = Nin + at;
        const T fx = flux_diff(row[xn3], row[xn2], row[xn1], c0, row[xo1], row[xo2], row[xo3], ux) * dx_inv;
        const T fy = flux_diff(row[yn3], row[yn2], row[yn1], c0, row[yo1], row[yo2], row[yo3], uy) * dy_inv;
        T G;
        if constexpr (REFRACT) {
            // kappa: neighbours from the lanes of this segment, clamped at the ends
            const T km3 = __shfl_sync(FULL, c0, base + max(m - 3, 0));
            const T km2 = __shfl_sync(FULL, c0, base + max(m - 2, 0));
            const T km1 = __shfl_sync(FULL, c0, base + max(m - 1, 0));
            const T kp1 = __shfl_sync(FULL, c0, base + min(m + 1, Nk - 1));
            const T kp2 = __shfl_sync(FULL, c0, base + min(m + 2, Nk - 1));
            const T kp3 = __shfl_sync(FULL, c0, base + min(m + 3, Nk - 1));
            const bool pk = ck >= T(0);
            T Fkp;
            {
                const T w = pk ? weno5d(km2, km1, c0, kp1, kp2) : weno5d(kp3, kp2, kp1, c0, km1);
                Fkp = hp ? w : (pk ? c0 : kp1);
            }
            const T upF = __shfl_up_sync(FULL, Fkp, 1, SEG);
            const bool upPos = __shfl_up_sync(FULL, (int)pk, 1, SEG) != 0;
            T Fkm = upF;
            if (m >= 1 && upPos != pk) {
                const T w = pk ? weno5d(km3, km2, km1, c0, kp1) : weno5d(kp2, kp1, c0, km1, km2);
                Fkm = hm ? w : (pk ? km1 : c0);
            }
            const T fkp = (m == Nk - 1) ? T(0) : ck * Fkp;
            const T fkm = (m == 0) ? T(0) : ck * Fkm;
            const T fk = (fkp - fkm) * dk_inv;
            // phi: window
            const bool pp = cp >= T(0);
            const T Fpp = pp ? weno5d(w1, w2, w3, w4, w5) : weno5d(w6, w5, w4, w3, w2);
            T Fpm = prevF;
            if (!havePrev || prevPos != pp) Fpm = pp ? weno5d(w0, w1, w2, w3, w4) : weno5d(w5, w4, w3, w2, w1);
            prevF = Fpp;
            prevPos = pp;
            havePrev = true;
            const T fp = cp * (Fpp - Fpm) * dp_inv;
            G = -(fx + fy + fk + fp);
        } else {
            G = -(fx + fy);
        }
        if (p.has_wind || p.has_diss) G = G + T(source_term(p, cc, mm, n, (double)c0));
        if (p.lin_rates) G = fma(static_cast<const T*>(p.lin_rates)[at], c0, G);
        if constexpr (TENDENCY) {
            if (live) Gout[at] = (double)G;
        } else {
            const T out = stage_out(p, c0, G, p.stage == 1 ? T(0) : N0[at]);
            if (live) {
                if (!isfinite(out)) atomicOr(p.err, 1u);
                Nout[at] = out;
            }
        }
        w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; w5 = w6; w6 = nxt;
    }
}

// One thread per cell-bin, for any Nk.
template <typename T, bool REFRACT, bool TENDENCY>
__global__ void __launch_bounds__(BLOCK) generic_kernel(const T* __restrict__ Nin, const T* N0, T* Nout,
                                                        double* __restrict__ Gout, StageParams p) {
    const int64_t t = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
    const int Nx = (int)p.Nx, Ny = (int)p.Ny, Nk = (int)p.Nk, Np = (int)p.Np;
    const int64_t P = (int64_t)Nx * Ny, slice = P * Nk;
    if (t >= slice * Np) return;
    const int m = (int)(t % Nk);
    const int64_t cn = t / Nk;
    const int64_t c = cn % P;
    const int n = (int)(cn / P);
    const int i = (int)(c % Nx), j = (int)(c / Nx);
    if (j < p.j_lo || j >= p.j_hi) return;
    const BinArgs<T> b{Nin, p.coef, p.cosp, p.sinp, p.cg_x, p.cg_y, Nx, Ny, Nk, Np, p.cg_per_cell,
                       T(p.dx_inv), T(p.dy_inv), T(p.dk_inv), T(p.dp_inv)};
    const T c0 = Nin[t];
    T G = bin_tendency<T, REFRACT>(b, c, i, j, m, n, c0);
    if (p.has_wind || p.has_diss) G = G + T(source_term(p, c, m, n, (double)c0));
    if (p.lin_rates) G = fma(static_cast<const T*>(p.lin_rates)[t], c0, G);
    if constexpr (TENDENCY) {
        Gout[t] = (double)G;
    } else {
        const T out = stage_out(p, c0, G, p.stage == 1 ? T(0) : N0[t]);
        if (!isfinite(out)) atomicOr(p.err, 1u);
        Nout[t] = out;
    }
}

// No transport (horizontal_advection = nothing, no currents): G = sources only
// (tendencies.jl:230-246 with transport_tendency(::Nothing) = 0). Touches no neighbour.
template <typename T, bool TENDENCY>
__global__ void __launch_bounds__(BLOCK) source_only_kernel(const T* __restrict__ Nin, const T* N0, T* Nout,
                                                            double* __restrict__ Gout, StageParams p) {
    const int64_t t = (int64_t)blockIdx.x * BLOCK + threadIdx.x;
    const int64_t P = p.Nx * p.Ny, slice = P * p.Nk;
    if (t >= slice * p.Np) return;
    const int m = (int)(t % p.Nk);
    const int64_t cn = t / p.Nk;
    const int64_t jr = (cn % P) / p.Nx;
    if (jr < p.j_lo || jr >= p.j_hi) return;
    const T a = Nin[t];
    T G = T(0);
    if (p.has_wind || p.has_diss) G = T(source_term(p, cn % P, m, (int)(cn / P), (double)a));
    if (p.lin_rates) G = fma(static_cast<const T*>(p.lin_rates)[t], a, G);
    if constexpr (TENDENCY) {
        Gout[t] = (double)G;
    } else {
        const T out = stage_out(p, a, G, p.stage == 1 ? T(0) : N0[t]);
        if (!isfinite(out)) atomicOr(p.err, 1u);
        Nout[t] = out;
    }
}

template <typename T, bool TEND>
cudaError_t launch_impl(const Handle& h, const StageParams& p, const void* Nin, const void* N0, void* Nout, double* G,
                        cudaStream_t s) {
    const int64_t Nk = h.desc.Nk;
    const bool refract = p.transport == RPL_TRANSPORT_REFRACTION;
    const T* in = (const T*)Nin;
    const T* n0 = (const T*)N0;
    T* out = (T*)Nout;
    if (p.transport == RPL_TRANSPORT_NONE) {
        const dim3 grid((unsigned)((h.units + BLOCK - 1) / BLOCK));
        source_only_kernel<T, TEND><<<grid, BLOCK, 0, s>>>(in, n0, out, G, p);
    } else if (Nk <= 32) {
        const int seg = Nk <= 4 ? 4 : Nk <= 8 ? 8 : Nk <= 16 ? 16 : 32;
        const int64_t cols_per_block = (BLOCK / 32) * (32 / seg);
        const int64_t Pr = h.desc.Nx * (p.j_hi - p.j_lo);
        const dim3 grid((unsigned)((Pr + cols_per_block - 1) / cols_per_block));
#define RPL_COL(SEGV)                                                                                        \
    if (seg == SEGV) {                                                                                       \
        if (refract) column_kernel<T, SEGV, true, TEND><<<grid, BLOCK, 0, s>>>(in, n0, out, G, p);          \
        else column_kernel<T, SEGV, false, TEND><<<grid, BLOCK, 0, s>>>(in, n0, out, G, p);                 \
    }
        RPL_COL(4) RPL_COL(8) RPL_COL(16) RPL_COL(32)
#undef RPL_COL
    } else {
        const dim3 grid((unsigned)((h.units + BLOCK - 1) / BLOCK));
        if (refract) generic_kernel<T, true, TEND><<<grid, BLOCK, 0, s>>>(in, n0, out, G, p);
        else generic_kernel<T, false, TEND><<<grid, BLOCK, 0, s>>>(in, n0, out, G, p);
    }
    return cudaGetLastError();
}

}  // namespace

StageParams make_params(const Handle& h, double dt, int stage) {
    StageParams p{};
    const rpl_desc& d = h.desc;
    p.Nx = d.Nx; p.Ny = d.Ny; p.Nk = d.Nk; p.Np = d.Np;
    p.dx_inv = 1.0 / d.dx;
    p.dy_inv = 1.0 / d.dy;
    p.dk_inv = 1.0 / (h.kappa_faces[1] - h.kappa_faces[0]);
    p.dp_inv = 1.0 / (h.phi_faces[1] - h.phi_faces[0]);
    p.dt = dt;
    p.stage = stage;
    p.a = stage == 2 ? 0.75 : (stage == 3 ? 1.0 / 3.0 : 0.0);
    p.b = stage == 2 ? 0.25 : (stage == 3 ? 2.0 / 3.0 : 1.0);
    p.transport = d.transport;
    p.cg_per_cell = h.d_cgmag != nullptr;
    p.kappa = h.d_kappa; p.phi = h.d_phi; p.weights = h.d_weights;
    p.cosp = h.d_cos; p.sinp = h.d_sin;
    p.cg_x = h.d_cgx; p.cg_y = h.d_cgy; p.cg_mag = h.d_cgmag;
    p.coef = h.d_coef;
    p.trig32 = reinterpret_cast<const float4*>(h.d_tab32);
    p.cg32 = reinterpret_cast<const float2*>(h.d_tab32 + 4 * d.Np);
    p.cs32 = reinterpret_cast<const float2*>(h.d_tab32 + 4 * d.Np + 2 * d.Nk * d.Np);
    p.w32 = h.d_tab32 + 6 * d.Np + 2 * d.Nk * d.Np;
    p.cell32 = h.d_cell32;
    p.bin32 = h.d_bin32;
    p.learned = h.learned != nullptr;
    p.lrate = h.d_lr;
    p.lflag = h.d_lflag;
    p.lscale = h.learned ? mlp_desc(h.learned).target_scale : 0.0f;
    p.has_wind = h.has_sources && h.src.wind_kind != RPL_WIND_NONE;
    p.stress_cap = h.has_sources && h.src.stress_cap;
    p.has_diss = h.has_sources && h.src.has_dissipation;
    if (h.d_wind) {
        const int64_t c2 = d.Nx * d.Ny;
        p.wind_U10 = h.d_wind; p.wind_theta = h.d_wind + c2; p.wind_ustar = h.d_wind + 2 * c2;
        p.stress_factor = h.d_wind + 3 * c2;
    }
    p.rho_ratio = h.src.rho_air / h.src.rho_water;
    p.beta_max = h.src.beta_max; p.z_alpha = h.src.z_alpha; p.p_in = h.src.p_in;
    p.alpha0 = h.src.alpha0; p.von_karman = h.src.von_karman; p.wind_g = h.src.wind_gravity;
    p.C_ds = h.src.C_ds; p.B_r = h.src.B_r; p.ds_p = h.src.ds_p; p.sigma_power = h.src.sigma_power;
    p.ds_g = h.src.ds_gravity;
    p.wind_K32 = p.has_wind ? (float)(p.rho_ratio * (p.beta_max / (p.von_karman * p.von_karman))) : 0.0f;
    p.von_karman32 = (float)p.von_karman;
    p.z_alpha32 = (float)p.z_alpha;
    p.err = h.d_err;
    p.lin_rates = h.n_terms ? h.d_lin_rates : nullptr;
    p.j_lo = 0;
    p.j_hi = d.Ny;
    return p;
}

namespace {

// The two-pass stage (rpl_xyw.cu, rpl_ring.cu); intrinsic transport without the bundle is one pass.
template <typename T>
cudaError_t launch_walk(const Handle& h, const StageParams& p, const void* Nin, const void* N0, void* Nout,
                        cudaStream_t s) {
    const bool refract = p.transport == RPL_TRANSPORT_REFRACTION, bundle = p.has_wind || p.has_diss;
    const WalkArgs<T> a = make_walk_args<T>(h, p, Nin, N0, Nout);
    if (!refract && !bundle) return launch_xy_stage<T>(a, h.walk, s);
    cudaError_t e = launch_xy_pass<T>(a, h.walk, s);
    return e == cudaSuccess ? launch_ring<T>(a, p, refract, bundle, s) : e;
}

}  // namespace

cudaError_t launch_stage(const Handle& h, const StageParams& p, const void* Nin, const void* N0, void* Nout,
                         cudaStream_t s) {
    pin_planes(h, s);
    if (h.precision == RPL_FP64) {
        if (h.d_vel) return launch_walk<double>(h, p, Nin, N0, Nout, s);
        return launch_impl<double, false>(h, p, Nin, N0, Nout, nullptr, s);
    }
    // the tile kernel takes the SourceTermSet rates alone, not together with the bundle or the network
    const bool mixed = p.lin_rates && (p.has_wind || p.has_diss || p.learned);
    if (tile32_supported(h) && !h.force_column_kernel && !mixed) return launch_tile32(h, p, Nin, N0, Nout, s);
    if (h.d_vel) return launch_walk<float>(h, p, Nin, N0, Nout, s);
    return launch_impl<float, false>(h, p, Nin, N0, Nout, nullptr, s);
}

cudaError_t launch_tendency(const Handle& h, const StageParams& p, const void* Nin, double* G, cudaStream_t s) {
    if (h.precision == RPL_FP64) return launch_impl<double, true>(h, p, Nin, nullptr, nullptr, G, s);
    return launch_impl<float, true>(h, p, Nin, nullptr, nullptr, G, s);
}

}  // namespace rpl
