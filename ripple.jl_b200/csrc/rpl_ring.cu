// rpl_ring.cu -- the second pass of a stage after the y-walk x/y pass (rpl_xyw.cu) left S = fx + fy: the
// kappa and phi fluxes (wave_current_refraction.jl:88-147), SourceTermSet rates or the FP64 source bundle,
// and the SSP-RK3 stage update, FP32 and FP64.
//
// One lane holds one 16-byte vector of adjacent kappa bins of one cell (four FP32 or two FP64 bins) and
// walks a range of the periodic phi ring. A warp holds floor(32 / L) cells of L = ceil(Nk / bins per lane)
// lanes each, so every Nk up to 32 vectors takes this path; lanes past the last whole cell repeat live ones
// and store nothing.
//  * the phi window (directions n-3 .. n+3) is a ring of eight slices in shared memory, private to the
//    thread and filled by cp.async one step ahead (each slice twice, slots s and s+8, so the window sits at
//    constant offsets from one slot); S and N0 of the next step come the same way. Nothing waits in
//    registers: L1 returns a warp's loads in order, and with the loads in registers one DRAM latency per
//    step was exposed (1.95 long-scoreboard stalls per issue);
//  * kappa stencils come from the neighbouring lanes by shuffle, with the reference's clamped indices: bins
//    past the last hold the value of bin Nk-1 (ldv), so only a cell's end lanes clamp;
//  * where a warp's velocities share a sign the faces are read in upwind order without selects; the + face
//    of phi step n is then the - face of step n+1. Other warps reconstruct every face of a cell for itself;
//  * a grid too small to fill the GPU splits the ring over blockIdx.y; each range starts with its own
//    lower face.
// The pass is bound by instruction issue (FP32: 70% of the issue slots; FP64: 63% of the FP64 pipe).
// S and Nout may be the same buffer: every element is read and written by one thread, in that order.
// The order of additions, G = -(((S + fk) + fp)) + sources, is the fused kernels'.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "rpl_flux.cuh"
#include "rpl_src64.cuh"
#include "rpl_vec.cuh"
#include "rpl_walk.h"

namespace rpl {

namespace {

using namespace w32;

constexpr int RTHREADS = 128;

// Which of a lane's kappa faces have the five-point stencil; `top` marks bins whose upper face is the last.
struct Edges {
    int m0, Nk;
    __device__ __forceinline__ bool full(int q) const { return q - 2 >= 0 && q + 3 <= Nk - 1; }   // face q|q+1
};

__device__ __forceinline__ float2 zero_top(float2 F, int m, int Nk) {   // no flux through the last bin's upper face
    return make_float2(m == Nk - 1 ? 0.f : F.x, m + 1 == Nk - 1 ? 0.f : F.y);
}

// kappa flux differences ck (F(m+1/2) - F(m-1/2)) of the lane's bins before 1/dkappa, products and difference
// rounded separately (kflux, rpl_weno32.cuh). FP32: faces a..d above bins m0..m0+3; vote: 1 all positive,
// 2 all negative, 0 mixed over the warp.
__device__ __forceinline__ Q kappa_flux(Q c, Q ck, int vote, Edges e, int l, int L, int lane) {
    const int m0 = e.m0, Nk = e.Nk;
    const float k0 = c.a.x, k1 = c.a.y, k2 = c.b.x, k3 = c.b.y;
    const bool dn = l >= 1, up = l < L - 1;
    auto below = [&](float v, float clamp) {
        const float s = __shfl_sync(FULL, v, lane - 1);
        return dn ? s : clamp;
    };
    auto above = [&](float v, float clamp) {
        const float s = __shfl_sync(FULL, v, lane + 1);
        return up ? s : clamp;
    };
    if (vote) {
        float2 Fab, Fcd;
        const bool ha = e.full(m0), hb = e.full(m0 + 1), hc = e.full(m0 + 2), hd = e.full(m0 + 3);
        if (vote == 1) {
            const float km2 = below(k2, k0), km1 = below(k3, k0), kp4 = above(k0, k3), kp5 = above(k1, k3);
            Fab = weno5_2(make_float2(km2, km1), make_float2(km1, k0), make_float2(k0, k1), make_float2(k1, k2),
                          make_float2(k2, k3));
            Fcd = weno5_2(make_float2(k0, k1), make_float2(k1, k2), make_float2(k2, k3), make_float2(k3, kp4),
                          make_float2(kp4, kp5));
            Fab = make_float2(ha ? Fab.x : k0, hb ? Fab.y : k1);
            Fcd = make_float2(hc ? Fcd.x : k2, hd ? Fcd.y : k3);
        } else {
            const float km1 = below(k3, k0), kp4 = above(k0, k3), kp5 = above(k1, k3), kp6 = above(k2, k3);
            Fab = weno5_2(make_float2(k3, kp4), make_float2(k2, k3), make_float2(k1, k2), make_float2(k0, k1),
                          make_float2(km1, k0));
            Fcd = weno5_2(make_float2(kp5, kp6), make_float2(kp4, kp5), make_float2(k3, kp4), make_float2(k2, k3),
                          make_float2(k1, k2));
            Fab = make_float2(ha ? Fab.x : k1, hb ? Fab.y : k2);
            Fcd = make_float2(hc ? Fcd.x : k3, hd ? Fcd.y : kp4);
        }
        const float lo = __shfl_sync(FULL, Fcd.y, lane - 1);
        const float2 La = make_float2(m0 == 0 ? 0.f : lo, Fab.x), Lb = make_float2(Fab.y, Fcd.x);
        return {sub2(mul2(ck.a, zero_top(Fab, m0, Nk)), mul2(ck.a, La)),
                sub2(mul2(ck.b, zero_top(Fcd, m0 + 2, Nk)), mul2(ck.b, Lb))};
    }
    // mixed signs: both faces of every bin in the bin's own orientation
    const float km3 = below(k1, k0), km2 = below(k2, k0), km1 = below(k3, k0);
    const float kp4 = above(k0, k3), kp5 = above(k1, k3), kp6 = above(k2, k3);
    const bool pa = pos1(ck.a.x), pb = pos1(ck.a.y), pc = pos1(ck.b.x), pd = pos1(ck.b.y);
    float2 Fab = weno5_2(make_float2(pa ? km2 : k3, pb ? km1 : kp4), make_float2(pa ? km1 : k2, pb ? k0 : k3),
                         make_float2(pa ? k0 : k1, pb ? k1 : k2), make_float2(pa ? k1 : k0, pb ? k2 : k1),
                         make_float2(pa ? k2 : km1, pb ? k3 : k0));
    float2 Fcd = weno5_2(make_float2(pc ? k0 : kp5, pd ? k1 : kp6), make_float2(pc ? k1 : kp4, pd ? k2 : kp5),
                         make_float2(pc ? k2 : k3, pd ? k3 : kp4), make_float2(pc ? k3 : k2, pd ? kp4 : k3),
                         make_float2(pc ? kp4 : k1, pd ? kp5 : k2));
    float2 La = weno5_2(make_float2(pa ? km3 : k2, pb ? km2 : k3), make_float2(pa ? km2 : k1, pb ? km1 : k2),
                        make_float2(pa ? km1 : k0, pb ? k0 : k1), make_float2(pa ? k0 : km1, pb ? k1 : k0),
                        make_float2(pa ? k1 : km2, pb ? k2 : km1));
    float2 Lb = weno5_2(make_float2(pc ? km1 : kp4, pd ? k0 : kp5), make_float2(pc ? k0 : k3, pd ? k1 : kp4),
                        make_float2(pc ? k1 : k2, pd ? k2 : k3), make_float2(pc ? k2 : k1, pd ? k3 : k2),
                        make_float2(pc ? k3 : k0, pd ? kp4 : k1));
    const bool hl = e.full(m0 - 1), ha = e.full(m0), hb = e.full(m0 + 1), hc = e.full(m0 + 2), hd = e.full(m0 + 3);
    Fab = make_float2(ha ? Fab.x : (pa ? k0 : k1), hb ? Fab.y : (pb ? k1 : k2));
    Fcd = make_float2(hc ? Fcd.x : (pc ? k2 : k3), hd ? Fcd.y : (pd ? k3 : kp4));
    La = make_float2(m0 == 0 ? 0.f : (hl ? La.x : (pa ? km1 : k0)), ha ? La.y : (pb ? k0 : k1));
    Lb = make_float2(hb ? Lb.x : (pc ? k1 : k2), hc ? Lb.y : (pd ? k2 : k3));
    return {sub2(mul2(ck.a, zero_top(Fab, m0, Nk)), mul2(ck.a, La)),
            sub2(mul2(ck.b, zero_top(Fcd, m0 + 2, Nk)), mul2(ck.b, Lb))};
}

// The same for the two FP64 bins of a lane. Faces a and b of one orientation share their differences.
__device__ __forceinline__ D kappa_flux(D c, D ck, int vote, Edges e, int l, int L, int lane) {
    const int m0 = e.m0, Nk = e.Nk;
    const double k0 = c.a, k1 = c.b;
    const double s_m1 = __shfl_sync(FULL, k1, lane - 1), s_p2 = __shfl_sync(FULL, k0, lane + 1);
    const double s_p3 = __shfl_sync(FULL, k1, lane + 1);
    const bool dn = l >= 1, up = l < L - 1;
    const double km1 = dn ? s_m1 : k0, kp2 = up ? s_p2 : k1, kp3 = up ? s_p3 : k1;
    const bool ha = e.full(m0), hb = e.full(m0 + 1);
    double Fa, Fb, lo0, lo1;
    if (vote) {
        if (vote == 1) {
            const double s_m2 = __shfl_sync(FULL, k0, lane - 1), km2 = dn ? s_m2 : k0;
            const double d1 = km1 - km2, d2 = k0 - km1, d3 = k1 - k0, d4 = kp2 - k1, d5 = kp3 - kp2;
            const double D1 = d2 - d1, D2 = d3 - d2, D3 = d4 - d3, D4 = d5 - d4;
            const double A2 = areg(D2), A3 = areg(D3);
            Fa = weno_face(d1, d2, d3, d4, D1, D2, D3, areg(D1), A2, A3, k0);
            Fb = weno_face(d2, d3, d4, d5, D2, D3, D4, A2, A3, areg(D4), k1);
            Fa = ha ? Fa : k0;
            Fb = hb ? Fb : k1;
        } else {
            const double s_p4 = __shfl_sync(FULL, k0, lane + 2), kp4 = l < L - 2 ? s_p4 : kp3;
            const double d1 = kp3 - kp4, d2 = kp2 - kp3, d3 = k1 - kp2, d4 = k0 - k1, d5 = km1 - k0;
            const double D1 = d2 - d1, D2 = d3 - d2, D3 = d4 - d3, D4 = d5 - d4;
            const double A2 = areg(D2), A3 = areg(D3);
            Fb = weno_face(d1, d2, d3, d4, D1, D2, D3, areg(D1), A2, A3, kp2);
            Fa = weno_face(d2, d3, d4, d5, D2, D3, D4, A2, A3, areg(D4), k1);
            Fa = ha ? Fa : k1;
            Fb = hb ? Fb : kp2;
        }
        lo0 = __shfl_sync(FULL, Fb, lane - 1);
        lo1 = Fa;
    } else {   // mixed signs: both faces of every bin in the bin's own orientation
        const double s_m2 = __shfl_sync(FULL, k0, lane - 1), s_m3 = __shfl_sync(FULL, k1, lane - 2);
        const double s_p4 = __shfl_sync(FULL, k0, lane + 2);
        const double km2 = dn ? s_m2 : k0, km3 = l >= 2 ? s_m3 : km2, kp4 = l < L - 2 ? s_p4 : kp3;
        const bool pa = pos1(ck.a), pb = pos1(ck.b), hl = e.full(m0 - 1);
        Fa = ha ? weno5_1(pa ? km2 : kp3, pa ? km1 : kp2, pa ? k0 : k1, pa ? k1 : k0, pa ? kp2 : km1) : (pa ? k0 : k1);
        Fb = hb ? weno5_1(pb ? km1 : kp4, pb ? k0 : kp3, pb ? k1 : kp2, pb ? kp2 : k1, pb ? kp3 : k0) : (pb ? k1 : kp2);
        lo0 = hl ? weno5_1(pa ? km3 : kp2, pa ? km2 : k1, pa ? km1 : k0, pa ? k0 : km1, pa ? k1 : km2) : (pa ? km1 : k0);
        lo1 = ha ? weno5_1(pb ? km2 : kp3, pb ? km1 : kp2, pb ? k0 : k1, pb ? k1 : k0, pb ? kp2 : km1) : (pb ? k0 : k1);
    }
    Fa = m0 == Nk - 1 ? 0. : Fa;
    Fb = m0 + 1 == Nk - 1 ? 0. : Fb;
    lo0 = m0 == 0 ? 0. : lo0;
    return {__dsub_rn(__dmul_rn(ck.a, Fa), __dmul_rn(ck.a, lo0)), __dsub_rn(__dmul_rn(ck.b, Fb), __dmul_rn(ck.b, lo1))};
}

// element q: u_q >= 0 by its sign bit ? x : y
__device__ __forceinline__ Q pick(Q u, Q x, Q y) {
    return {make_float2(pos1(u.a.x) ? x.a.x : y.a.x, pos1(u.a.y) ? x.a.y : y.a.y),
            make_float2(pos1(u.b.x) ? x.b.x : y.b.x, pos1(u.b.y) ? x.b.y : y.b.y)};
}
__device__ __forceinline__ D pick(D u, D x, D y) { return {pos1(u.a) ? x.a : y.a, pos1(u.b) ? x.b : y.b}; }

// Field f of the coefficient records of the lane's bins.
__device__ __forceinline__ Q coef_field(const double* r, int f, int left, Q) {
    return {make_float2((float)r[f], (float)r[8 * min(1, left) + f]),
            make_float2((float)r[8 * min(2, left) + f], (float)r[8 * min(3, left) + f])};
}
__device__ __forceinline__ D coef_field(const double* r, int f, int left, D) {
    return {r[f], r[8 * min(1, left) + f]};
}

// c_kappa and c_phi of direction n (wave_current_refraction.jl:94-98) from the direction's products, in FP32 in
// the fused kernel's order. Trig entries are stored as packed pairs (FP32).
template <class T> struct Vel;
template <> struct Vel<float> {
    Q mk, Uxx, sum, dif, Uxy, Uyx, Uyy;   // -kappa, U_xx, U_yx + U_xy, U_xx - U_yy, ...
    struct Trig { float2 cc, cs, ss, pad; };
    static __device__ __forceinline__ Trig trig(const WalkArgs<float>& p, int n) {
        const float4 t = __ldg(p.trig32 + n);
        return {f2(t.x), f2(t.y), f2(t.z), f2(0.f)};
    }
    __device__ __forceinline__ void load(const double* r, int left) {
        mk = qneg(coef_field(r, 7, left, Q{}));
        Uxx = coef_field(r, 2, left, Q{});
        Uxy = coef_field(r, 3, left, Q{});
        Uyx = coef_field(r, 4, left, Q{});
        Uyy = coef_field(r, 5, left, Q{});
        sum = qadd(Uyx, Uxy);
        dif = qsub(Uxx, Uyy);
    }
    __device__ __forceinline__ void at(const Trig& t, Q& ck, Q& cp) const {
        auto ckf = [&](float2 m, float2 xx, float2 s, float2 yy) {
            return mul2(m, add2(add2(mul2(t.cc, xx), mul2(t.cs, s)), mul2(t.ss, yy)));
        };
        auto cpf = [&](float2 d, float2 yx, float2 xy) {
            return sub2(add2(mul2(t.cs, d), mul2(t.ss, yx)), mul2(t.cc, xy));
        };
        ck = {ckf(mk.a, Uxx.a, sum.a, Uyy.a), ckf(mk.b, Uxx.b, sum.b, Uyy.b)};
        cp = {cpf(dif.a, Uyx.a, Uxy.a), cpf(dif.b, Uyx.b, Uxy.b)};
    }
};
template <> struct Vel<double> {   // a = -kappa (U_xx, U_yx + U_xy, U_yy), b = (U_xx - U_yy, U_yx, U_xy)
    D a1, a2, a3, b1, b2, b3;
    struct Trig { double cc, cs, ss, pad; };
    static __device__ __forceinline__ Trig trig(const WalkArgs<double>& p, int n) {
        const double c = __ldg(p.cosp + n), s = __ldg(p.sinp + n);
        return {c * c, c * s, s * s, 0.};
    }
    __device__ __forceinline__ void load(const double* r, int left) {
        const D mk = qneg(coef_field(r, 7, left, D{}));
        const D xx = coef_field(r, 2, left, D{}), yy = coef_field(r, 5, left, D{});
        b3 = coef_field(r, 3, left, D{});
        b2 = coef_field(r, 4, left, D{});
        a1 = qmul(mk, xx);
        a2 = qmul(mk, qadd(b2, b3));
        a3 = qmul(mk, yy);
        b1 = qsub(xx, yy);
    }
    __device__ __forceinline__ void at(const Trig& t, D& ck, D& cp) const {
        ck = {fma(t.ss, a3.a, fma(t.cs, a2.a, t.cc * a1.a)), fma(t.ss, a3.b, fma(t.cs, a2.b, t.cc * a1.b))};
        cp = {fma(-t.cc, b3.a, fma(t.ss, b2.a, t.cs * b1.a)), fma(-t.cc, b3.b, fma(t.ss, b2.b, t.cs * b1.b))};
    }
};

__device__ __forceinline__ Q add_source(const StageParams& sp, const Cell64& wc, const Bin64* wb, double cth, double sth,
                                        Q c, Q G) {
    G.a.x += (float)source64(sp, wc, wb[0], cth, sth, c.a.x);
    G.a.y += (float)source64(sp, wc, wb[1], cth, sth, c.a.y);
    G.b.x += (float)source64(sp, wc, wb[2], cth, sth, c.b.x);
    G.b.y += (float)source64(sp, wc, wb[3], cth, sth, c.b.y);
    return G;
}
__device__ __forceinline__ D add_source(const StageParams& sp, const Cell64& wc, const Bin64* wb, double cth, double sth,
                                        D c, D G) {
    return {G.a + source64(sp, wc, wb[0], cth, sth, c.a), G.b + source64(sp, wc, wb[1], cth, sth, c.b)};
}

// The lane's place: cell, bins and what they address.
template <typename T>
struct Lane {
    int lane, l, m0, left;
    bool live;
    int64_t cell, home;
    __device__ __forceinline__ explicit Lane(const WalkArgs<T>& p) {
        const int L = p.L, cpw = 32 / L;
        lane = threadIdx.x & 31;
        const int cw = lane / L;
        l = lane - cw * L;
        const int64_t P = (int64_t)p.Nx * (p.j_hi - p.j_lo);
        const int64_t c = ((int64_t)blockIdx.x * (RTHREADS / 32) + (threadIdx.x >> 5)) * cpw + cw;
        live = cw < cpw && c < P;
        cell = min(c, P - 1) + (int64_t)p.Nx * p.j_lo;
        m0 = LaneVec<T>::N * l;
        left = p.Nk - 1 - m0;
        home = cell * p.Nk + m0;
    }
};

// Stores the lane's result. FP64: a result that is not finite though the action is comes from a face out of weno_face's
// range, or from a state that blows up; it goes into S (Nout itself, or free) as a mark, so that N0 stays
// for redo, and *marked is set.
template <bool AL, typename T, class V>
__device__ __forceinline__ void store_result(const WalkArgs<T>& p, const Lane<T>& me, V c, V out, int64_t off, int* marked) {
    if (qfinite(out)) {
        stv<AL>(p.Nout + off, out, me.left);
        return;
    }
    const bool again = std::is_same<T, double>::value && qfinite(c);
    if (again) *marked = 1;
    else atomicOr(p.err, 1u);
    stv<AL>((again ? p.S : p.Nout) + off, out, me.left);
}

// The lane's marked results once more, from the tendency of the wider range: after the walk and out of line (inside it,
// with the walk's registers live, it cost 12% of a refraction and 33% of an intrinsic stage).
template <bool AL, bool REFRACT, bool BUNDLE>
__device__ __noinline__ void redo(const WalkArgs<double>& p, const StageParams& sp, int per_part) {
    const Lane<double> me(p);
    const int left = me.left, n0 = blockIdx.y * per_part, n1 = min(n0 + per_part, p.Np);
    Cell64 wc;
    Bin64 wb[2];
    if constexpr (BUNDLE) {
        wc = make_cell64(sp, me.cell);
        for (int q = 0; q < 2; ++q) wb[q] = make_bin64(sp, me.m0 + min(q, left));
    }
    for (int n = n0; n < n1; ++n) {
        const int64_t off = (int64_t)p.Nx * p.Ny * p.Nk * n + me.home;
        if (qfinite(ldv<AL>(p.S + off, left))) continue;
        const D c = ldv<AL>(p.Nin + off, left);
        D G{bin_tendency_wide<REFRACT>(p, me.cell, me.m0, n), bin_tendency_wide<REFRACT>(p, me.cell, me.m0 + min(1, left), n)};
        if constexpr (BUNDLE) G = add_source(sp, wc, wb, p.cosp[n], p.sinp[n], c, G);
        if (p.rates) G = qfma(ldv<AL>(p.rates + off, left), c, G);
        const D out = stage_update<double>(G, c, p.stage == 1 ? D{0., 0.} : ldv<AL>(p.N0 + off, left), p.stage, p.dt, p.a, p.b);
        if (!qfinite(out)) atomicOr(p.err, 1u);
        stv<AL>(p.Nout + off, out, left);
    }
}

// Shared memory of ring_kernel in 16-byte slots per thread: the window ring twice, then S and N0 of two steps. Behind
// them the direction table of the CTA's range, TABLE_NP entries (32 KiB) at most.
constexpr int WIN = 16, SLOTS = WIN + 4, TABLE_NP = 1024;

template <typename T, bool AL, bool BUNDLE, bool RATES>
__global__ void __launch_bounds__(RTHREADS, BUNDLE ? 2 : 4)
ring_kernel(const __grid_constant__ WalkArgs<T> p, const __grid_constant__ StageParams sp, int per_part) {
    using LV = LaneVec<T>;
    using V = typename LV::V;
    using Trig = typename Vel<T>::Trig;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_marked[RTHREADS];   // per thread: some of its results are to be made again
    s_marked[threadIdx.x] = 0;
    V* slot = reinterpret_cast<V*>(smem) + threadIdx.x;
    Trig* trig = reinterpret_cast<Trig*>(smem + SLOTS * RTHREADS * 16);
    const int Nk = p.Nk, Np = p.Np;
    const int n0 = blockIdx.y * per_part, n1 = min(n0 + per_part, Np);
    for (int n = n0 + threadIdx.x; n < n1; n += RTHREADS) trig[n - n0] = Vel<T>::trig(p, n);
    __syncthreads();
    const int64_t slice = (int64_t)p.Nx * p.Ny * Nk;
    const Lane<T> me(p);
    const int left = me.left;
    const Edges edge{me.m0, Nk};
    const T* own = p.Nin + me.home;
    auto window = [&](int s, const T* src) {   // a direction's slice into ring slot s
        copy_async<AL>(slot + s * RTHREADS, src, left);
        copy_async<AL>(slot + (s + 8) * RTHREADS, src, left);
    };
    auto streams = [&](int par, int64_t off) {  // S and N0 of one step
        copy_async<AL>(slot + (WIN + 2 * par) * RTHREADS, p.S + off, left);
        if (p.stage != 1) copy_async<AL>(slot + (WIN + 2 * par + 1) * RTHREADS, p.N0 + off, left);
    };
    {   // directions n0-3 .. n0+3 into slots 0..6 (refraction needs Np >= 3, so one wrap suffices)
#pragma unroll
        for (int d = 0; d < 7; ++d) {
            const int n = n0 - 3 + d;
            window(d, own + slice * (n < 0 ? n + Np : (n >= Np ? n - Np : n)));
        }
        streams(0, slice * n0 + me.home);
        copy_commit();
    }
    Vel<T> vel;
    vel.load(p.coef + 8 * me.home, left);
    Cell64 wc;
    Bin64 wb[LV::N];
    if constexpr (BUNDLE) {
        wc = make_cell64(sp, me.cell);
#pragma unroll
        for (int q = 0; q < LV::N; ++q) wb[q] = make_bin64(sp, me.m0 + min(q, left));
    }
    V prevF = LV::zero();
    int carried = 0;   // orientation of prevF over the whole warp (1, 2), 0: none
    int nn = (n0 + 4) % Np, b = 0;
    int64_t off = slice * n0 + me.home;
    for (int n = n0; n < n1; ++n) {
        copy_wait<0>();
        if (n + 1 < n1) {   // the next step's window entry and streams
            window((b + 7) & 7, own + slice * nn);
            streams((b + 1) & 1, off + slice);
        }
        copy_commit();
        nn = nn + 1 == Np ? 0 : nn + 1;
        const V* w = slot + b * RTHREADS;
        auto W = [&](int d) { return lds(w + d * RTHREADS); };   // direction n-3+d
        const V* st = slot + (WIN + 2 * (b & 1)) * RTHREADS;
        const V c = W(3);
        V rate = LV::zero();
        if (RATES) rate = ldv<AL>(p.rates + off, left);
        V ck, cp;
        vel.at(trig[n - n0], ck, cp);
        const int vk = __all_sync(FULL, all_pos(ck)) ? 1 : (__all_sync(FULL, all_neg(ck)) ? 2 : 0);
        const V fk = qmuls(kappa_flux(c, ck, vk, edge, me.l, p.L, me.lane), p.dk_inv);
        const int vp = __all_sync(FULL, all_pos(cp)) ? 1 : (__all_sync(FULL, all_neg(cp)) ? 2 : 0);
        V Fpp, Fpm = prevF;
        if (vp == 1) Fpp = qweno(W(1), W(2), c, W(4), W(5));
        else if (vp == 2) Fpp = qweno(W(6), W(5), W(4), c, W(2));
        else Fpp = qweno(pick(cp, W(1), W(6)), pick(cp, W(2), W(5)), pick(cp, c, W(4)), pick(cp, W(4), c), pick(cp, W(5), W(2)));
        if (vp == 0 || vp != carried)
            Fpm = qweno(pick(cp, W(0), W(5)), pick(cp, W(1), W(4)), pick(cp, W(2), c), pick(cp, c, W(2)), pick(cp, W(4), W(1)));
        prevF = Fpp;
        carried = vp;
        const V fp = qmuls(qmul(cp, qsub(Fpp, Fpm)), p.dp_inv);
        V G = qneg(qadd(qadd(lds(st), fk), fp));
        if constexpr (BUNDLE) G = add_source(sp, wc, wb, __ldg(p.cosp + n), __ldg(p.sinp + n), c, G);
        if (RATES) G = qfma(rate, c, G);   // SourceTermSet rates of this stage, state layout
        const V out = stage_update<T>(G, c, p.stage == 1 ? LV::zero() : lds(st + RTHREADS), p.stage, p.dt, p.a, p.b);
        if (me.live) store_result<AL>(p, me, c, out, off, &s_marked[threadIdx.x]);
        off += slice;
        b = (b + 1) & 7;
    }
    if constexpr (std::is_same<T, double>::value)
        if (s_marked[threadIdx.x]) redo<AL, true, BUNDLE>(p, sp, per_part);
}

// Second pass of an intrinsic stage with the FP64 source bundle: G = -S, the sources and the stage update. A
// thread walks a range of the ring with the cell's wind constants and its bins' constants loaded once; S, the
// action and N0 are staged three steps ahead.
constexpr int DEPTH = 4;

template <typename T, bool AL, bool RATES>
__global__ void __launch_bounds__(RTHREADS, 4) bundle_kernel(const __grid_constant__ WalkArgs<T> p,
                                                               const __grid_constant__ StageParams sp, int per_part) {
    using LV = LaneVec<T>;
    using V = typename LV::V;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_marked[RTHREADS];   // per thread: some of its results are to be made again
    s_marked[threadIdx.x] = 0;
    V* slot = reinterpret_cast<V*>(smem) + threadIdx.x;
    const int64_t slice = (int64_t)p.Nx * p.Ny * p.Nk;
    const Lane<T> me(p);
    const int left = me.left, n0 = blockIdx.y * per_part, n1 = min(n0 + per_part, p.Np);
    auto issue = [&](int n) {
        if (n < n1) {
            V* s = slot + (n & (DEPTH - 1)) * 3 * RTHREADS;
            const int64_t off = slice * n + me.home;
            copy_async<AL>(s, p.Nin + off, left);
            copy_async<AL>(s + RTHREADS, p.S + off, left);
            if (p.stage != 1) copy_async<AL>(s + 2 * RTHREADS, p.N0 + off, left);
        }
        copy_commit();
    };
#pragma unroll
    for (int d = 0; d < DEPTH - 1; ++d) issue(n0 + d);
    const Cell64 wc = make_cell64(sp, me.cell);
    Bin64 wb[LV::N];
#pragma unroll
    for (int q = 0; q < LV::N; ++q) wb[q] = make_bin64(sp, me.m0 + min(q, left));
    for (int n = n0; n < n1; ++n) {
        copy_wait<DEPTH - 2>();
        issue(n + DEPTH - 1);
        const int64_t off = slice * n + me.home;
        const V* s = slot + (n & (DEPTH - 1)) * 3 * RTHREADS;
        const V c = lds(s);
        V G = add_source(sp, wc, wb, __ldg(p.cosp + n), __ldg(p.sinp + n), c, qneg(lds(s + RTHREADS)));
        if (RATES) G = qfma(ldv<AL>(p.rates + off, left), c, G);
        const V out = stage_update<T>(G, c, p.stage == 1 ? LV::zero() : lds(s + 2 * RTHREADS), p.stage, p.dt, p.a, p.b);
        if (me.live) store_result<AL>(p, me, c, out, off, &s_marked[threadIdx.x]);
    }
    if constexpr (std::is_same<T, double>::value)
        if (s_marked[threadIdx.x]) redo<AL, false, true>(p, sp, per_part);
}

template <typename T, bool AL>
cudaError_t launch_al(const WalkArgs<T>& a, const StageParams& p, bool refract, bool bundle, cudaStream_t s) {
    if (a.L < 1) return cudaErrorInvalidValue;   // no lane geometry (walk_supported)
    const int64_t P = (int64_t)a.Nx * (a.j_hi - a.j_lo), per = (RTHREADS / 32) * (32 / a.L);
    const unsigned blocks = (unsigned)((P + per - 1) / per);
    // ranges of the ring: one unless that leaves the GPU without eight CTAs per SM, then as many as that
    // takes, of at least three directions each (a range pays a 7-deep window and one more face); never more
    // directions in a range than its table holds
    const int64_t parts = std::max<int64_t>({1, std::min<int64_t>((8 * 148 + blocks - 1) / blocks, a.Np / 3),
                                             (a.Np + TABLE_NP - 1) / TABLE_NP});
    const int per_part = (int)((a.Np + parts - 1) / parts);
    const dim3 grid(blocks, (unsigned)((a.Np + per_part - 1) / per_part));
    const bool rates = a.rates != nullptr;
    auto go = [&](auto k, size_t smem) {
        if (smem > 48 * 1024) {   // the most any model takes: the attribute is the kernel's, shared by all threads
            constexpr int most = SLOTS * RTHREADS * 16 + TABLE_NP * (int)sizeof(typename Vel<T>::Trig);
            cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
            if (e != cudaSuccess) return e;
        }
        k<<<grid, RTHREADS, smem, s>>>(a, p, per_part);
        return cudaGetLastError();
    };
    const size_t ring = SLOTS * RTHREADS * 16 + per_part * sizeof(typename Vel<T>::Trig);
    if (refract && bundle) return rates ? go(ring_kernel<T, AL, true, true>, ring) : go(ring_kernel<T, AL, true, false>, ring);
    if (refract) return rates ? go(ring_kernel<T, AL, false, true>, ring) : go(ring_kernel<T, AL, false, false>, ring);
    const size_t staged = DEPTH * 3 * RTHREADS * 16;
    if (bundle) return rates ? go(bundle_kernel<T, AL, true>, staged) : go(bundle_kernel<T, AL, false>, staged);
    return cudaErrorInvalidValue;   // intrinsic transport without the bundle is one pass
}

}  // namespace

template <typename T>
cudaError_t launch_ring(const WalkArgs<T>& a, const StageParams& p, bool refract, bool bundle, cudaStream_t s) {
    if (a.Nk % LaneVec<T>::N == 0) return launch_al<T, true>(a, p, refract, bundle, s);
    return launch_al<T, false>(a, p, refract, bundle, s);
}
template cudaError_t launch_ring<float>(const WalkArgs<float>&, const StageParams&, bool, bool, cudaStream_t);
template cudaError_t launch_ring<double>(const WalkArgs<double>&, const StageParams&, bool, bool, cudaStream_t);

}  // namespace rpl
