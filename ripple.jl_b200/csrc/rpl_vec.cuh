// rpl_vec.cuh -- the 16-byte lane vector of the two-pass stage kernels (rpl_xyw.cu, rpl_ring.cu): four
// adjacent kappa bins of an FP32 model as two packed pairs (Q, rpl_weno32.cuh) or two adjacent kappa bins
// of an FP64 model (D), with the same operations on both, so one kernel body serves the two precisions.
#pragma once
#include <cuda_runtime.h>

#include "rpl_weno32.cuh"

namespace rpl {
namespace w32 {

struct D {                            // two adjacent kappa bins, FP64
    double a, b;
};

// explicitly rounded, so that no kernel body contracts a product and a sum that another one does not
__device__ __forceinline__ D qadd(D x, D y) { return {__dadd_rn(x.a, y.a), __dadd_rn(x.b, y.b)}; }
__device__ __forceinline__ D qsub(D x, D y) { return {__dsub_rn(x.a, y.a), __dsub_rn(x.b, y.b)}; }
__device__ __forceinline__ D qmul(D x, D y) { return {__dmul_rn(x.a, y.a), __dmul_rn(x.b, y.b)}; }
__device__ __forceinline__ D qmuls(D x, double s) { return {__dmul_rn(x.a, s), __dmul_rn(x.b, s)}; }
__device__ __forceinline__ D qfma(D x, D y, D z) { return {fma(x.a, y.a, z.a), fma(x.b, y.b, z.b)}; }
__device__ __forceinline__ Q qfma(Q x, Q y, Q z) { return {fma2(x.a, y.a, z.a), fma2(x.b, y.b, z.b)}; }
__device__ __forceinline__ D qneg(D x) { return {-x.a, -x.b}; }
__device__ __forceinline__ Q qneg(Q x) { return {mul2(f2(-1.f), x.a), mul2(f2(-1.f), x.b)}; }

// Reciprocal of a positive normal x below 2^1022: the hardware approximation (about 20 bits) and one step of
// Householder's iteration of order two for 1/x (A. S. Householder, The Numerical Treatment of a Single Nonlinear Equation,
// 1970; for a simple zero also called Chebyshev's iteration), r (1 + e + e^2) with e = 1 - x r, which leaves e^3
// (below 2^-58) before the roundings. Within one unit in the last place of the correctly rounded quotient.
__device__ __forceinline__ double rcpd(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// Nonlinear part of one FP64 WENO5 face, the form of weno_face2 (rpl_weno32.cuh: t_k = 4 (eps + beta_k),
// linear weights times 10) with the three 1/t_k^2 brought to a common denominator: u_0 : u_1 : u_2 =
// (t1 t2)^2 : (t0 t2)^2 : (t0 t1)^2. One reciprocal per face instead of four. den grows as t^4 (at least (4 eps)^4 =
// 6e-45) and num as t^4.5, t ~ 30 N^2: where den reaches 2^850 (N from about 1e31; below it num stays under 2^960) the face
// is a NaN, and the cell-bin's tendency is computed again by bin_tendency (rpl_flux.cuh), whose weights have the
// range of 1/t^2 (N to about 1e76), by the kernel that finds its result not finite.
__device__ __forceinline__ double weno_face(double d1, double d2, double d3, double d4, double D1, double D2,
                                            double D3, double A1, double A2, double A3, double s2, int& den_hi) {
    const double G0 = fma(2.0, d2, D1), G1 = d2 + d3, G2 = fma(-2.0, d3, D3);
    const double t0 = fma(G0, G0, A1), t1 = fma(G1, G1, A2), t2 = fma(G2, G2, A3);
    const double p0 = t1 * t2, p1 = t0 * t2, p2 = t0 * t1;
    const double u0 = p0 * p0, u1 = p1 * p1, u2 = p2 * p2;
    const double den = fma(3.0, u2, fma(6.0, u1, u0));
    const double w0 = fma(5.0 / 6.0, d2, (-1.0 / 3.0) * d1), e3 = d3 + d3, w1 = e3 + d2, w2 = fma(-0.5, d4, e3);
    const double num = fma(w2, u2, fma(w1, u1, w0 * u0));
    den_hi = __double2hiint(den);
    return fma(num, rcpd(den), s2);
}
__device__ __forceinline__ double in_range(double f, int den_hi) {
    return __hiloint2double(den_hi < (1023 + 850) << 20 ? __double2hiint(f) : 0x7ff80000, __double2loint(f));
}
__device__ __forceinline__ double weno_face(double d1, double d2, double d3, double d4, double D1, double D2,
                                            double D3, double A1, double A2, double A3, double s2) {
    int hi;
    const double f = weno_face(d1, d2, d3, d4, D1, D2, D3, A1, A2, A3, s2, hi);
    return in_range(f, hi);
}
__device__ __forceinline__ double areg(double D) { return fma((13.0 / 3.0) * D, D, 4.0 * RPL_WENO_EPS); }

__device__ __forceinline__ double weno5_1(double s0, double s1, double s2, double s3, double s4, int& den_hi) {
    const double d1 = s1 - s0, d2 = s2 - s1, d3 = s3 - s2, d4 = s4 - s3;
    const double D1 = d2 - d1, D2 = d3 - d2, D3 = d4 - d3;
    return weno_face(d1, d2, d3, d4, D1, D2, D3, areg(D1), areg(D2), areg(D3), s2, den_hi);
}
__device__ __forceinline__ double weno5_1(double s0, double s1, double s2, double s3, double s4) {
    int hi;
    const double f = weno5_1(s0, s1, s2, s3, s4, hi);
    return in_range(f, hi);
}

// A'_c of a second difference, and the face from first differences d, second differences E, regularised
// squares A and the base value (the two halves of qweno, for stencils that slide by one).
__device__ __forceinline__ D qareg(D x) { return {areg(x.a), areg(x.b)}; }
__device__ __forceinline__ Q qareg(Q x) { return {areg(x.a), areg(x.b)}; }
// (D: one NaN marks the vector, whose results are made again together.)
__device__ __forceinline__ D qface(D d1, D d2, D d3, D d4, D D1, D D2, D D3, D A1, D A2, D A3, D s2) {
    int ha, hb;
    const double fa = weno_face(d1.a, d2.a, d3.a, d4.a, D1.a, D2.a, D3.a, A1.a, A2.a, A3.a, s2.a, ha);
    const double fb = weno_face(d1.b, d2.b, d3.b, d4.b, D1.b, D2.b, D3.b, A1.b, A2.b, A3.b, s2.b, hb);
    return {in_range(fa, max(ha, hb)), fb};
}
__device__ __forceinline__ D qweno(D s0, D s1, D s2, D s3, D s4) {
    int ha, hb;
    const double fa = weno5_1(s0.a, s1.a, s2.a, s3.a, s4.a, ha), fb = weno5_1(s0.b, s1.b, s2.b, s3.b, s4.b, hb);
    return {in_range(fa, max(ha, hb)), fb};
}
// A candidate from which elements are selected one by one: each element marks itself.
__device__ __forceinline__ D qweno_each(D s0, D s1, D s2, D s3, D s4) {
    return {weno5_1(s0.a, s1.a, s2.a, s3.a, s4.a), weno5_1(s0.b, s1.b, s2.b, s3.b, s4.b)};
}
__device__ __forceinline__ Q qface(Q d1, Q d2, Q d3, Q d4, Q D1, Q D2, Q D3, Q A1, Q A2, Q A3, Q s2) {
    return {weno_face2(d1.a, d2.a, d3.a, d4.a, D1.a, D2.a, D3.a, A1.a, A2.a, A3.a, s2.a),
            weno_face2(d1.b, d2.b, d3.b, d4.b, D1.b, D2.b, D3.b, A1.b, A2.b, A3.b, s2.b)};
}

// bit 0: some element >= 0; bit 1: some element < 0
__device__ __forceinline__ int code2(float2 u) {
    return ((u.x >= 0.f || u.y >= 0.f) ? 1 : 0) | ((u.x < 0.f || u.y < 0.f) ? 2 : 0);
}
__device__ __forceinline__ int codeq(Q u) { return code2(u.a) | code2(u.b); }
__device__ __forceinline__ int codeq(D u) {
    return ((u.a >= 0. || u.b >= 0.) ? 1 : 0) | ((u.a < 0. || u.b < 0.) ? 2 : 0);
}
__device__ __forceinline__ float2 selp(float2 u, float2 a, float2 b) {  // per element: u >= 0 ? a : b
    return make_float2(u.x >= 0.f ? a.x : b.x, u.y >= 0.f ? a.y : b.y);
}
__device__ __forceinline__ Q selq(Q u, Q x, Q y) { return {selp(u.a, x.a, y.a), selp(u.b, x.b, y.b)}; }
__device__ __forceinline__ D selq(D u, D x, D y) { return {u.a >= 0. ? x.a : y.a, u.b >= 0. ? x.b : y.b}; }

__device__ __forceinline__ bool qfinite(Q o) {
    return isfinite(o.a.x) && isfinite(o.a.y) && isfinite(o.b.x) && isfinite(o.b.y);
}
__device__ __forceinline__ bool finite1(double x) { return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u; }
__device__ __forceinline__ bool qfinite(D o) { return finite1(o.a) && finite1(o.b); }

template <class T> struct LaneVec;
template <> struct LaneVec<float> {
    using V = Q;
    static constexpr int N = 4;
    __device__ static __forceinline__ V zero() { return qz(); }
    __device__ static __forceinline__ V all(float s) { return {f2(s), f2(s)}; }
    __device__ static __forceinline__ V make(float a, float b, float c, float d) {
        return {make_float2(a, b), make_float2(c, d)};
    }
};
template <> struct LaneVec<double> {
    using V = D;
    static constexpr int N = 2;
    __device__ static __forceinline__ V zero() { return {0., 0.}; }
    __device__ static __forceinline__ V all(double s) { return {s, s}; }
};

__device__ __forceinline__ D lds(const D* p) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ Q lds(const Q* p) { return ldq(reinterpret_cast<const float*>(p)); }
__device__ __forceinline__ void sts(D* p, D v) { *reinterpret_cast<double2*>(p) = make_double2(v.a, v.b); }
__device__ __forceinline__ void sts(Q* p, Q v) { stq(reinterpret_cast<float*>(p), v); }

// Bins m0 .. m0+N-1 of a kappa column at p (p points at bin m0). ALIGNED (Nk a multiple of N): one 16-byte
// access. Otherwise element by element: bins past the last take the value of bin Nk-1, `left` = Nk-1-m0
// (>= 0) being the last one in range, and are never stored.
template <bool ALIGNED>
__device__ __forceinline__ Q ldv(const float* p, int left) {
    if constexpr (ALIGNED) return ldq(p);
    else return {make_float2(p[0], p[min(1, left)]), make_float2(p[min(2, left)], p[min(3, left)])};
}
template <bool ALIGNED>
__device__ __forceinline__ D ldv(const double* p, int left) {
    if constexpr (ALIGNED) {
        const double2 v = *reinterpret_cast<const double2*>(p);
        return {v.x, v.y};
    } else {
        return {p[0], p[min(1, left)]};
    }
}
template <bool ALIGNED>
__device__ __forceinline__ Q ldgv(const float* p, int left) {
    if constexpr (ALIGNED) return ldgq(p);
    else
        return {make_float2(__ldg(p), __ldg(p + min(1, left))), make_float2(__ldg(p + min(2, left)), __ldg(p + min(3, left)))};
}
template <bool ALIGNED>
__device__ __forceinline__ D ldgv(const double* p, int left) {
    if constexpr (ALIGNED) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(p));
        return {v.x, v.y};
    } else {
        return {__ldg(p), __ldg(p + min(1, left))};
    }
}
template <bool ALIGNED>
__device__ __forceinline__ void stv(float* p, Q v, int left) {
    if constexpr (ALIGNED) stq(p, v);
    else {
        p[0] = v.a.x;
        if (left >= 1) p[1] = v.a.y;
        if (left >= 2) p[2] = v.b.x;
        if (left >= 3) p[3] = v.b.y;
    }
}
template <bool ALIGNED>
__device__ __forceinline__ void stv(double* p, D v, int left) {
    if constexpr (ALIGNED) *reinterpret_cast<double2*>(p) = make_double2(v.a, v.b);
    else {
        p[0] = v.a;
        if (left >= 1) p[1] = v.b;
    }
}

// max(0, x) with NaN propagation and -0 -> +0, as relu (rpl_device.cuh) in one instruction (FP32) or on the
// integer pipe (FP64: a negative number that is not a NaN becomes 0).
__device__ __forceinline__ float relu1(float x) {
    float r;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double relu1(double x) {
    const int hi = __double2hiint(x);
    return hi < 0 && (unsigned)hi << 1 <= 0xffe00000u ? 0.0 : x;
}
__device__ __forceinline__ Q qrelu(Q x) {
    return {make_float2(relu1(x.a.x), relu1(x.a.y)), make_float2(relu1(x.b.x), relu1(x.b.y))};
}
__device__ __forceinline__ D qrelu(D x) { return {relu1(x.a), relu1(x.b)}; }

// SSP-RK3 stage update with the clamps (time_step.jl:67-74,98-105): relu(c + dt g), combined with N0.
template <class T, class V>
__device__ __forceinline__ V stage_update(V g, V c, V n0, int stage, T dt, T a, T b) {
    using LV = LaneVec<T>;
    const V st = qrelu(qfma(LV::all(dt), g, c));
    if (stage == 1) return st;
    return qrelu(qfma(LV::all(a), n0, qmuls(st, b)));
}

// Sign tests on the sign bits: the vector's elements all clear (pos) or all set (neg). A velocity of -0 counts
// as negative; its flux is zero in either orientation.
__device__ __forceinline__ bool pos1(float x) { return __float_as_int(x) >= 0; }
__device__ __forceinline__ bool pos1(double x) { return __double2hiint(x) >= 0; }
__device__ __forceinline__ bool all_pos(Q u) {
    return (__float_as_int(u.a.x) | __float_as_int(u.a.y) | __float_as_int(u.b.x) | __float_as_int(u.b.y)) >= 0;
}
__device__ __forceinline__ bool all_neg(Q u) {
    return (__float_as_int(u.a.x) & __float_as_int(u.a.y) & __float_as_int(u.b.x) & __float_as_int(u.b.y)) < 0;
}
__device__ __forceinline__ bool all_pos(D u) { return (__double2hiint(u.a) | __double2hiint(u.b)) >= 0; }
__device__ __forceinline__ bool all_neg(D u) { return (__double2hiint(u.a) & __double2hiint(u.b)) < 0; }

// Copies the lane's vector from global to shared memory without passing through registers. Elements past the
// column's last repeat it, as in ldv.
template <bool AL, typename T>
__device__ __forceinline__ void copy_async(void* dst, const T* src, int left) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (AL) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(src) : "memory");
    } else if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a + 4 * q), "l"(src + min(q, left)) : "memory");
    } else {
#pragma unroll
        for (int q = 0; q < 2; ++q)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a + 8 * q), "l"(src + min(q, left)) : "memory");
    }
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

}  // namespace w32
}  // namespace rpl
