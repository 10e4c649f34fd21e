// rpl_flux.cuh -- difference forms of the WENO5 face, the velocities of one cell-bin and its transport tendency with
// every neighbour read from memory: the arithmetic of the column and generic kernels (rpl_stage.cu), and what the
// two-pass FP64 kernels fall back on for a cell-bin whose faces leave their range (rpl_vec.cuh, weno_face).
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "rpl_device.cuh"
#include "rpl_walk.h"

namespace rpl {

template <typename T> __device__ __forceinline__ T rcp_w(T x);
template <> __device__ __forceinline__ float rcp_w<float>(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
template <> __device__ __forceinline__ double rcp_w<double>(double x) { return 1.0 / x; }

// Jiang-Shu WENO5 value at the face between s2 and s3 from (s0, s1, s2, s3, s4), upwind side first
// (wave_current_refraction.jl:41-55), in difference form: with d_k the first differences and D_k the
// second differences of the stencil, beta_0 = 13/12 D1^2 + (D1/2 + d2)^2, beta_1 = 13/12 D2^2 +
// ((d2+d3)/2)^2, beta_2 = 13/12 D3^2 + (D3/2 - d3)^2 (exactly the reference's indicators), and the
// candidates enter as offsets from s2.
template <typename T>
__device__ __forceinline__ T weno5d(T s0, T s1, T s2, T s3, T s4) {
    const T eps = T(RPL_WENO_EPS);
    const T d1 = s1 - s0, d2 = s2 - s1, d3 = s3 - s2, d4 = s4 - s3;
    const T D1 = d2 - d1, D2 = d3 - d2, D3 = d4 - d3;
    const T g0 = fma(T(0.5), D1, d2);
    const T g1 = T(0.5) * (d2 + d3);
    const T g2 = fma(T(0.5), D3, -d3);
    const T t0 = fma(g0, g0, fma(T(13.0 / 12.0) * D1, D1, eps));
    const T t1 = fma(g1, g1, fma(T(13.0 / 12.0) * D2, D2, eps));
    const T t2 = fma(g2, g2, fma(T(13.0 / 12.0) * D3, D3, eps));
    const T r0 = rcp_w(t0), r1 = rcp_w(t1), r2 = rcp_w(t2);
    const T a0 = (T(0.1) * r0) * r0, a1 = (T(0.6) * r1) * r1, a2 = (T(0.3) * r2) * r2;
    const T w0 = fma(T(5.0 / 6.0), d2, T(-1.0 / 3.0) * d1);
    const T w1 = fma(T(1.0 / 3.0), d3, T(1.0 / 6.0) * d2);
    const T w2 = fma(T(2.0 / 3.0), d3, T(-1.0 / 6.0) * d4);
    const T num = fma(a2, w2, fma(a1, w1, a0 * w0));
    const T den = (a0 + a1) + a2;
    return fma(num, rcp_w(den), s2);
}

// Both faces of a cell from its 7-point stencil oriented upwind -> downwind (s3 is the cell):
// lo = value at the upwind face (from s0..s4), hi = value at the downwind face (from s1..s5).
template <typename T>
__device__ __forceinline__ void weno5_pair(T s0, T s1, T s2, T s3, T s4, T s5, T& lo, T& hi) {
    const T eps = T(RPL_WENO_EPS);
    const T d1 = s1 - s0, d2 = s2 - s1, d3 = s3 - s2, d4 = s4 - s3, d5 = s5 - s4;
    const T D1 = d2 - d1, D2 = d3 - d2, D3 = d4 - d3, D4 = d5 - d4;
    const T A1 = fma(T(13.0 / 12.0) * D1, D1, eps), A2 = fma(T(13.0 / 12.0) * D2, D2, eps);
    const T A3 = fma(T(13.0 / 12.0) * D3, D3, eps), A4 = fma(T(13.0 / 12.0) * D4, D4, eps);
    {   // upwind face: stencil s0..s4 (cells centred at s1, s2, s3)
        const T g0 = fma(T(0.5), D1, d2), g1 = T(0.5) * (d2 + d3), g2 = fma(T(0.5), D3, -d3);
        const T r0 = rcp_w(fma(g0, g0, A1)), r1 = rcp_w(fma(g1, g1, A2)), r2 = rcp_w(fma(g2, g2, A3));
        const T a0 = (T(0.1) * r0) * r0, a1 = (T(0.6) * r1) * r1, a2 = (T(0.3) * r2) * r2;
        const T w0 = fma(T(5.0 / 6.0), d2, T(-1.0 / 3.0) * d1);
        const T w1 = fma(T(1.0 / 3.0), d3, T(1.0 / 6.0) * d2);
        const T w2 = fma(T(2.0 / 3.0), d3, T(-1.0 / 6.0) * d4);
        lo = fma(fma(a2, w2, fma(a1, w1, a0 * w0)), rcp_w((a0 + a1) + a2), s2);
    }
    {   // downwind face: stencil s1..s5 (cells centred at s2, s3, s4)
        const T g0 = fma(T(0.5), D2, d3), g1 = T(0.5) * (d3 + d4), g2 = fma(T(0.5), D4, -d4);
        const T r0 = rcp_w(fma(g0, g0, A2)), r1 = rcp_w(fma(g1, g1, A3)), r2 = rcp_w(fma(g2, g2, A4));
        const T a0 = (T(0.1) * r0) * r0, a1 = (T(0.6) * r1) * r1, a2 = (T(0.3) * r2) * r2;
        const T w0 = fma(T(5.0 / 6.0), d3, T(-1.0 / 3.0) * d2);
        const T w1 = fma(T(1.0 / 3.0), d4, T(1.0 / 6.0) * d3);
        const T w2 = fma(T(2.0 / 3.0), d4, T(-1.0 / 6.0) * d5);
        hi = fma(fma(a2, w2, fma(a1, w1, a0 * w0)), rcp_w((a0 + a1) + a2), s3);
    }
}

// Flux difference u*(N_{+1/2} - N_{-1/2}) of a periodic direction from the 7-point stencil
// (m3 .. p3 around the cell), upwinded by the sign of u (wave_current_refraction.jl:104-123).
template <typename T>
__device__ __forceinline__ T flux_diff(T m3, T m2, T m1, T c, T p1, T p2, T p3, T u) {
    const bool pos = u >= T(0);
    T lo, hi;
    if (pos) weno5_pair(m3, m2, m1, c, p1, p2, lo, hi);      // lo = N(-1/2), hi = N(+1/2)
    else weno5_pair(p3, p2, p1, c, m1, m2, lo, hi);          // lo = N(+1/2), hi = N(-1/2)
    return pos ? u * (hi - lo) : u * (lo - hi);
}

struct Coef {
    double Ux, Uy, Uxx, Uxy, Uyx, Uyy, cg, kap;
};

__device__ __forceinline__ Coef load_coef(const double* __restrict__ rec) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(rec));
    const double2 b = __ldg(reinterpret_cast<const double2*>(rec) + 1);
    const double2 c = __ldg(reinterpret_cast<const double2*>(rec) + 2);
    const double2 d = __ldg(reinterpret_cast<const double2*>(rec) + 3);
    return Coef{a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
}

// Velocities of one cell-bin. FP64 keeps the reference's evaluation order
// (wave_current_refraction.jl:94-98); FP32 uses the same products regrouped.
template <typename T>
__device__ __forceinline__ void velocities(const Coef& q, double cph, double sph, double cgx, double cgy,
                                           bool per_cell, bool refract, T& ux, T& uy, T& ck, T& cp) {
    const double gx = per_cell ? q.cg * cgx : cgx;
    const double gy = per_cell ? q.cg * cgy : cgy;
    if (!refract) {
        ux = T(gx);
        uy = T(gy);
        ck = cp = T(0);
        return;
    }
    if constexpr (std::is_same<T, double>::value) {
        ck = -q.kap * (cph * cph * q.Uxx + cph * sph * (q.Uyx + q.Uxy) + sph * sph * q.Uyy);
        cp = cph * sph * (q.Uxx - q.Uyy) + sph * sph * q.Uyx - cph * cph * q.Uxy;
        ux = gx + q.Ux;
        uy = gy + q.Uy;
    } else {
        const float c = (float)cph, s = (float)sph, k = (float)q.kap;
        const float Uxx = (float)q.Uxx, Uxy = (float)q.Uxy, Uyx = (float)q.Uyx, Uyy = (float)q.Uyy;
        ck = -k * (c * c * Uxx + c * s * (Uyx + Uxy) + s * s * Uyy);
        cp = c * s * (Uxx - Uyy) + s * s * Uyx - c * c * Uxy;
        ux = (float)gx + (float)q.Ux;
        uy = (float)gy + (float)q.Uy;
    }
}

template <typename T>
struct BinArgs {
    const T* N;
    const double *coef, *cosp, *sinp, *cgx, *cgy;
    int Nx, Ny, Nk, Np, cg_per_cell;
    T dx_inv, dy_inv, dk_inv, dp_inv;
};

// Transport tendency of bin (m, n) of cell c = i + Nx j, whose action is c0.
template <typename T, bool REFRACT>
__device__ __forceinline__ T bin_tendency(const BinArgs<T>& p, int64_t c, int i, int j, int m, int n, T c0) {
    const int Nx = p.Nx, Ny = p.Ny, Nk = p.Nk, Np = p.Np;
    const int64_t slice = (int64_t)Nx * Ny * Nk;
    const Coef q = load_coef(p.coef + 8 * (c * Nk + m));
    const int b = m + Nk * n;
    T ux, uy, ck, cp;
    velocities<T>(q, p.cosp[n], p.sinp[n], p.cgx[b], p.cgy[b], p.cg_per_cell, REFRACT, ux, uy, ck, cp);
    const T* row = p.N + (int64_t)n * slice;
    auto X = [&](int ii) { return row[((int64_t)j * Nx + wrap(ii, Nx)) * Nk + m]; };
    auto Y = [&](int jj) { return row[((int64_t)wrap(jj, Ny) * Nx + i) * Nk + m]; };
    const T fx = flux_diff(X(i - 3), X(i - 2), X(i - 1), c0, X(i + 1), X(i + 2), X(i + 3), ux) * p.dx_inv;
    const T fy = flux_diff(Y(j - 3), Y(j - 2), Y(j - 1), c0, Y(j + 1), Y(j + 2), Y(j + 3), uy) * p.dy_inv;
    if constexpr (!REFRACT) return -(fx + fy);
    auto K = [&](int mk) { return row[c * Nk + clampi(mk, Nk)]; };
    auto F = [&](int nk) { return p.N[(int64_t)wrap(nk, Np) * slice + c * Nk + m]; };
    const bool hp = (m - 2 >= 0) && (m + 3 <= Nk - 1), hm = (m - 3 >= 0) && (m + 2 <= Nk - 1);
    const bool pk = ck >= T(0);
    const T Fkp = hp ? (pk ? weno5d(K(m - 2), K(m - 1), c0, K(m + 1), K(m + 2))
                           : weno5d(K(m + 3), K(m + 2), K(m + 1), c0, K(m - 1)))
                     : (pk ? c0 : K(m + 1));
    const T Fkm = hm ? (pk ? weno5d(K(m - 3), K(m - 2), K(m - 1), c0, K(m + 1))
                           : weno5d(K(m + 2), K(m + 1), c0, K(m - 1), K(m - 2)))
                     : (pk ? K(m - 1) : c0);
    const T fkp = (m == Nk - 1) ? T(0) : ck * Fkp;
    const T fkm = (m == 0) ? T(0) : ck * Fkm;
    const T fk = (fkp - fkm) * p.dk_inv;
    const T fp = flux_diff(F(n - 3), F(n - 2), F(n - 1), c0, F(n + 1), F(n + 2), F(n + 3), cp) * p.dp_inv;
    return -(fx + fy + fk + fp);
}

// The same for the two-pass FP64 kernels, outside their main flow.
template <bool REFRACT>
static __device__ __noinline__ double bin_tendency_wide(const WalkArgs<double>& p, int64_t c, int m, int n) {
    const BinArgs<double> b{p.Nin, p.coef, p.cosp, p.sinp, p.cgx, p.cgy, p.Nx, p.Ny, p.Nk, p.Np, p.cg_per_cell,
                            p.dx_inv, p.dy_inv, p.dk_inv, p.dp_inv};
    return bin_tendency<double, REFRACT>(b, c, (int)(c % p.Nx), (int)(c / p.Nx), m, n,
                                         p.Nin[((int64_t)p.Nx * p.Ny * n + c) * p.Nk + m]);
}

}  // namespace rpl
