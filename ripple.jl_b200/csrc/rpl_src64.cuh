// rpl_src64.cuh -- FP64 evaluation of the source bundle split like rpl_src32.cuh into per-cell constants
// (wind), per-kappa constants and a cheap per-cell-bin part: wind input with the wave-supported stress cap
// (pressure_correlation.jl:109-151, precomputed_sources.jl:269-326) and local-saturation whitecapping
// (local_saturation.jl:30-47). jp_rate and source_term (rpl_device.cuh) evaluate every transcendental per
// cell-bin in the reference's order; here log(k z1) = log k + log z1 and cos(theta - theta_u) =
// cos cos + sin sin leave one exponential and one division per cell-bin on the growing side of the wind.
#pragma once

#include <cuda_runtime.h>

#include "rpl_device.cuh"

namespace rpl {

struct Cell64 {
    double ustar, logz1, cu, su, factor;
    bool on;
};

struct Bin64 {
    double logk, invC, sigma, skB, dsK;   // log k, k / sigma, sigma, sigma_ds k^3 / B_r, -C_ds sigma_ds^q
};

__device__ __forceinline__ Cell64 make_cell64(const StageParams& p, int64_t cell) {
    Cell64 c{0., 0., 1., 0., 1., false};
    if (!p.has_wind) return c;
    const double U = p.wind_U10[cell], us = p.wind_ustar[cell];
    const double z1 = p.alpha0 * (us * us) / p.wind_g;
    c.on = U > 0.0 && us > 0.0 && z1 > 0.0;
    if (!c.on) return c;
    c.ustar = us;
    c.logz1 = log(z1);
    sincos(p.wind_theta[cell], &c.su, &c.cu);
    if (p.stress_cap) c.factor = p.stress_factor[cell];
    return c;
}

__device__ __forceinline__ Bin64 make_bin64(const StageParams& p, int m) {
    Bin64 b{0., 0., 0., 0., 0.};
    const double k = p.kappa[m];
    if (p.has_wind) {
        b.sigma = sqrt(p.wind_g * k);
        b.logk = log(k);
        b.invC = k / b.sigma;
    }
    if (p.has_diss) {
        const double sd = sqrt(p.ds_g * k);
        b.skB = sd * (k * k * k) / p.B_r;
        b.dsK = -p.C_ds * (p.sigma_power == 1.0 ? sd : pow(sd, p.sigma_power));
    }
    return b;
}

// Janssen growth rate before the cap; 0 outside the growth window and where the parameters make it negative (the
// reference takes positive rates only).
__device__ __forceinline__ double wind_rate64(const StageParams& p, const Cell64& c, const Bin64& b, double cth,
                                              double sth) {
    const double cos_tu = fma(cth, c.cu, sth * c.su);
    if (!(c.on && cos_tu > 0.0)) return 0.0;
    const double inv_age = fma(c.ustar, b.invC, p.z_alpha);
    const double Z = (b.logk + c.logz1) + p.von_karman / (inv_age * cos_tu);
    if (!(Z < 0.0)) return 0.0;
    const double Z2 = Z * Z;
    const double cp = (p.p_in == 2.0) ? cos_tu * cos_tu : pow(cos_tu, p.p_in);
    const double rate = p.rho_ratio * (p.beta_max / (p.von_karman * p.von_karman)) * exp(Z) * (Z2 * Z2) *
                        (inv_age * inv_age) * cp * b.sigma;
    return rate > 0.0 ? rate : 0.0;
}

// Source tendency of one cell-bin with action a.
__device__ __forceinline__ double source64(const StageParams& p, const Cell64& c, const Bin64& b, double cth, double sth,
                                           double a) {
    double g = 0.0;
    if (p.has_wind) g = wind_rate64(p, c, b, cth, sth) * c.factor * a;
    if (p.has_diss) {
        const double ov = fma(a, b.skB, -1.0);
        if (a > 0.0 && ov > 0.0) {
            const double o = fmin(ov, 1e6);
            g -= b.dsK * ((p.ds_p == 2.0) ? o * o : pow(o, p.ds_p)) * a;
        }
    }
    return g;
}

}  // namespace rpl
