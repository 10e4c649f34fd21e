// rpl_xyw.cuh -- the x/y pass of a stage as a y-walk, FP32 and FP64: the x and y fluxes
// u (N(+1/2) - N(-1/2)) / spacing of every cell-bin (wave_current_refraction.jl:104-123), written as
// S = fx + fy in the state layout for the second pass (rpl_ring.cu, ks_kernel and kp_kernel of
// rpl_tile32.cu); for intrinsic transport without the bundle or learned sources the same kernel applies
// the stage update itself (one pass).
//
// Layout of the work: a CTA owns one direction bin n, CX consecutive cells in x (the first of them only
// supplies a face: CX-1 cells are written) and a segment of `seg` rows, with L lanes per cell and one
// 16-byte vector of adjacent kappa bins per lane (four FP32 or two FP64 bins). L = ceil(Nk / bins per
// lane), so every Nk takes this path; where a column is not a whole number of vectors its accesses go
// element by element (ldv/stv). The threads walk the rows j of the segment:
//  * every face is reconstructed once. The x face between cells s and s+1 is computed by the lane of
//    cell s and handed to cell s+1 through shared memory one row later; the y face j+1/2 of a column
//    is the upper face of row j and the lower face of row j+1 in the same thread;
//  * FP32: the y and x stencils come from a ring of staged rows in shared memory. FP64: the y stencil lives
//    in registers, where the first and second differences and the regularised squares slide by one row per
//    step (one new difference each instead of four, three and three); only row j passes through shared
//    memory, for the x stencil (two row buffers, one barrier per row);
//  * upwinding: the reference upwinds each cell's two faces by the sign of the cell-centre velocity.
//    Where a CTA's x (or y) velocities share one sign, each face needs one reconstruction and the
//    body has no per-element selects. The velocity of bin (m, n) is u = c g(m,n) + U (c the per-cell c_g
//    magnitude when the depth varies, else 1 with c_g in the table g), so it has the sign of g(m,n)
//    wherever |g(m,n)| > |U| / c. vel_kernel stores, per region of cells and kappa bin, the maximum of
//    |U| / c enlarged by 1e-5 (FP32); a CTA whose every bin passes |g| (1 - 1e-5) > that maximum, with
//    one sign, runs a body without selects along that axis; elsewhere both candidates are reconstructed where
//    needed and selected per element. The margins cover the FP32 roundings of the product, the division and the
//    test. Both bodies give the same face values bit for bit (a stencil read backwards changes the sign
//    of its odd differences only, exactly), in FP32 those of the fused tile kernel.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "rpl_flux.cuh"
#include "rpl_vec.cuh"
#include "rpl_walk.h"

namespace rpl {

namespace xyw {

using namespace w32;

constexpr int XTHREADS = 256;                    // most threads per CTA
constexpr int MAXL = 32;                         // most lanes per cell
constexpr int ROWV64 = XTHREADS + 5 * MAXL;      // FP64: vectors per staged row, the CTA's cells and five halo cells
enum { POS = 0, NEG = 1, MIX = 2 };
// x/y pass without and with currents; whole intrinsic stage without and with the SourceTermSet rates
enum { PASS = 0, PASS_CURRENTS = 1, STAGE = 2, STAGE_RATES = 3 };

// FP32: the y stencil from a ring of staged rows in shared memory (16 rows of ROWV vectors; a row is written
// twice, slots s and s+8, so the seven rows around j sit at constant offsets from one slot; row j+3 is
// written in step j into the slot of row j-5, which no thread reads after step j-2). The FP32 body is bound by the reciprocals (MUFU) and by how many warps hide them: holding the
// stencil's differences in registers as the FP64 body does saves 18 of 132 packed operations per vector and
// row but spills at 128 registers (two CTAs per SM) and was slower, 1.29 against 0.99 ms per stage at
// 448 x 448 x 32 x 36 (1.17 at 168 registers, 12 warps per SM).
// One phase of `bar` per row: a warp arrives when its x faces of the row are stored and its reads of the previous
// row's are done, and waits at the next row's start, so that the row's y face hides the slowest warp.
__device__ __forceinline__ void row_arrive(unsigned bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Every warp of the CTA arrives once per row, so the wait ends; it is bounded all the same (error word bit 3).
__device__ __forceinline__ void row_wait(unsigned bar, int parity, unsigned* err) {
#pragma unroll 1
    for (int t = 0; t < (1 << 20); ++t) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, P1;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return;
    }
    atomicOr(err, 8u);
}

template <bool AL, int ROWV, int XM, int YM, int MODE>
__device__ __forceinline__ void xyw_body_ring(const WalkArgs<float>& p, Q* ring, Q* fsm, Q* priv, int* sg, unsigned bar,
                                              int n, int tx, int js, int je) {
    using LV = LaneVec<float>;
    constexpr bool XMIX = XM == MIX, FUSED = MODE >= STAGE, RATES = MODE == STAGE_RATES, curr = MODE == PASS_CURRENTS;
    // whole vectors, no currents: rows and c_g by cp.async (882 against 962 us per stage with the SourceTermSet
    // rates at 384 x 384 x 32 x 36, 716 against 739 without at 601 x 417 x 24 x 24; with currents 1040 against 996
    // at 448 x 448, element by element 542 against 418)
    constexpr bool ASYNC = AL && !curr;
    // Rows divided by row_arrive / row_wait: at a barrier a warp stood 0.9 of its 7.4 cycles per instruction.
    // Against the barrier, cases of 384 x 384 to 1024 x 1024 x 32 x 36: two steps with SourceTermSet rates 8.42 -> 8.06 ms,
    // tides at 448 x 448 7.48 -> 7.28, self-coupled 11.53 -> 11.2, 1024 x 1024 64.1 -> 63.1; 64 x 64 x 4 x 16, one
    // step, 112 -> 114 us (latency). Vectors copied element by element keep the barrier: 7.68 against 7.92 ms
    // at 389 x 251 x 25 x 24.
    constexpr bool SPLIT = AL;
    const int Nx = p.Nx, Ny = p.Ny, Nk = p.Nk, L = p.L, CX = p.CX;
    const int64_t slice = (int64_t)Nx * Ny * Nk;
    const int tid = threadIdx.x, l = tid % L;
    const bool act = tid / L < CX;                             // threads past the last cell repeat it
    const int slot = min(tid / L, CX - 1);
    const int cnt = je - js;
    const int ibase = tx * (CX - 1) - 1;                       // x of slot 0
    const int my_i = ((ibase + slot) % Nx + Nx) % Nx;
    const bool own = act && slot >= 1 && ibase + slot < Nx;
    const int m0 = LV::N * l, left = Nk - 1 - m0;
    // halo columns: 2 on the left, 3 on the right, loaded by the first 5*L threads
    const bool hal = tid < 5 * L;
    const int hs = tid / L < 2 ? tid / L - 2 : CX + tid / L - 2;
    const int hi_x = hal ? ((ibase + hs) % Nx + Nx) % Nx : 0;
    const int rs = Nx * Nk;                                    // row stride within a direction slice
    const float* base = p.Nin + slice * n;
    float* Sn = (FUSED ? p.Nout : p.S) + slice * n;
    const float* N0n = p.N0 + slice * n;
    const int colm = my_i * Nk + m0, hcol = hi_x * Nk + m0;
    const float2* gt = p.cg32 + m0 + (int64_t)Nk * n;
    const float2 g0 = __ldg(gt), g1 = __ldg(gt + min(1, left)), g2 = __ldg(gt + min(2, left)),
                 g3 = __ldg(gt + min(3, left));
    const Q gx = LV::make(g0.x, g1.x, g2.x, g3.x), gy = LV::make(g0.y, g1.y, g2.y, g3.y);
    const bool cgp = p.cg_per_cell != 0;
    auto modr = [&](int r) { return (r % Ny + Ny) % Ny; };
    auto ld = [&](int r, int col) { return ldv<AL>(base + r * rs + col, left); };
    const int own_off = (slot + 2) * L + l, hal_off = (hs + 2) * L + l;
    auto put = [&](int s, int off, Q q) {
        sts(ring + s * ROWV + off, q);
        sts(ring + (s + 8) * ROWV + off, q);
    };
    // prologue: rows js-3 .. js+2 of the own column, rows js .. js+2 of the halo columns (ring slots 0..5)
    for (int d = -3; d <= 2; ++d) {
        const Q v = ld(modr(js + d), colm);
        if (act) put(d + 3, own_off, v);
    }
    if (hal)
        for (int d = 0; d <= 2; ++d) put(d + 3, hal_off, ld(modr(js + d), hcol));
    // row j+3 comes one row ahead: by cp.async straight into the ring and c_g into a slot of the thread (ASYNC),
    // or through registers
    Q nw = qz(), hv = qz();
    Q vx = qz(), vy = qz(), vc = {f2(1.f), f2(1.f)};
    Q* mine = priv + tid;
    auto rload = [&](int s, int r) {
        if constexpr (ASYNC) {
            const float* src = base + r * rs + colm;
            if (act) {
                copy_async<AL>(ring + s * ROWV + own_off, src, left);
                copy_async<AL>(ring + (s + 8) * ROWV + own_off, src, left);
            }
            if (hal) {
                const float* hsrc = base + r * rs + hcol;
                copy_async<AL>(ring + s * ROWV + hal_off, hsrc, left);
                copy_async<AL>(ring + (s + 8) * ROWV + hal_off, hsrc, left);
            }
        } else {
            nw = ld(r, colm);
            if (hal) hv = ld(r, hcol);
        }
    };
    rload(6, modr(js + 3));
    auto vload = [&](int r) {
        const int e = r * rs + colm;
        if constexpr (ASYNC) {
            if (cgp) copy_async<AL>(mine, p.cg + e, left);
            copy_commit();
            return;
        }
        if (curr) {
            vx = ldgv<AL>(p.ux + e, left);
            vy = ldgv<AL>(p.uy + e, left);
        }
        if (cgp) vc = ldgv<AL>(p.cg + e, left);
    };
    // velocities in the fused kernel's order: (c_g * direction table) + U (intrinsic: no U)
    auto velo = [&](Q& ux, Q& uy) {
        ux = gx;
        uy = gy;
        if constexpr (ASYNC) copy_wait<0>();
        if constexpr (ASYNC)
            if (cgp) vc = lds(mine);
        if (cgp) {
            ux = qmul(vc, ux);
            uy = qmul(vc, uy);
        }
        if (curr) {
            ux = qadd(ux, vx);
            uy = qadd(uy, vy);
        }
    };
    // fused stage: the inputs of the row being finished, loaded one row ahead (after that row's faces)
    Q pn0 = qz(), plr = qz();
    auto pend = [&](int j) {
        const int off = j * rs + colm;
        if (p.stage != 1) pn0 = ldv<AL>(N0n + off, left);
        if (RATES) plr = ldv<AL>(p.rates + slice * n + off, left);
    };
    vload(modr(js));
    Q ux0, uy0;
    velo(ux0, uy0);
    Q uy1 = qz();
    vload(modr(js + 1));
    if constexpr (XMIX)
        if (act) {
            sg[slot * L + l] = own ? codeq(ux0) : 0;           // the first row's codes
            if (slot == 0) {
                sg[CX * L + l] = 0;
                sg[(2 * CX + 1) * L + l] = 0;
            }
        }
    __syncthreads();
    const Q* q = ring + own_off;
    Q pLy = qz(), pRy = qz();   // the two candidates of the lower y face of the current row
    {
        auto R = [&](int d) { return lds(q + d * ROWV); };     // row js-3+d
        if constexpr (YM == POS) pLy = qweno(R(0), R(1), R(2), R(3), R(4));
        else if constexpr (YM == NEG) pRy = qweno(R(5), R(4), R(3), R(2), R(1));
        else {
            const int need = own ? codeq(uy0) : 0;
            if (__any_sync(FULL, need & 1)) pLy = qweno(R(0), R(1), R(2), R(3), R(4));
            if (__any_sync(FULL, need & 2)) pRy = qweno(R(5), R(4), R(3), R(2), R(1));
        }
    }
    int rl = modr(js + 4), rv = modr(js + 2);
    int sw = 6, sq = 0;                                         // ring slots of rows j+3 and j-3
    const float dxi = p.dx_inv, dyi = p.dy_inv;
    Q Fx_prev = qz(), fy_prev = qz(), ux_prev = qz();
    int outoff = js * rs + colm;
    auto step = [&](int k, auto bufc) {
        constexpr int buf = decltype(bufc)::value;
        const bool row = k < cnt;
        Q ux1 = qz();
        if (row) {
            if constexpr (!ASYNC) {
                if (act) put(sw, own_off, nw);
                if (hal) put(sw, hal_off, hv);
            }
            velo(ux1, uy1);   // also waits for row j+3
            if constexpr (!ASYNC) {
                rload(0, rl);
                vload(rv);
            }
        }
        if constexpr (!SPLIT) __syncthreads();
        else row_wait(bar, buf, p.err);                         // the x faces of row j-1 are all stored
        if constexpr (ASYNC) {
            if (row) {   // row j+4 into the slot of row j-4, whose readers have arrived since
                rload((sw + 1) & 7, rl);
                vload(rv);
            }
        }
        // the previous row: its lower x face from the left neighbour's candidates, then S
        if (k > 0 && slot >= 1) {
            Q Flo;
            if constexpr (XMIX) {
                const Q* f = fsm + (((1 - buf) * CX + slot - 1) * L + l) * 2;
                Flo = selq(ux_prev, lds(f), lds(f + 1));
            } else {
                Flo = lds(fsm + ((1 - buf) * CX + slot - 1) * L + l);
            }
            const Q fx = qmuls(qmul(ux_prev, qsub(Fx_prev, Flo)), dxi);
            if constexpr (!FUSED) {
                if (own) stv<AL>(Sn + outoff - rs, qadd(fx, fy_prev), left);
            } else {
                const Q cv = lds(q + (sq + 2) * ROWV);          // the finished row's action
                Q G = qneg(qadd(fx, fy_prev));
                if (RATES) G = qfma(plr, cv, G);              // SourceTermSet rates of this stage
                const Q o = stage_update<float>(G, cv, pn0, p.stage, p.dt, p.a, p.b);
                if (own) {
                    if (!qfinite(o)) atomicOr(p.err, 1u);
                    stv<AL>(Sn + outoff - rs, o, left);
                }
            }
        }
        if (!row) {   // the CTA does not end with the last row's copies, which nothing reads, in flight
            if constexpr (ASYNC) copy_wait<0>();
            return false;
        }
        if constexpr (XMIX)
            if (act) sg[((1 - buf) * (CX + 1) + slot) * L + l] = own ? codeq(ux1) : 0;   // for the next row
        if constexpr (FUSED) pend(js + k);
        const Q* qq = q + sq * ROWV;
        auto R = [&](int d) { return lds(qq + d * ROWV); };     // own column, row j-3+d
        const Q c = R(3);
        {
            const Q* xr = qq + 3 * ROWV;                         // row j
            auto X = [&](int d) { return lds(xr + d * L); };     // cell slot+d
            if constexpr (XM == POS) {
                Fx_prev = qweno(X(-2), X(-1), c, X(1), X(2));
                if (act) sts(fsm + (buf * CX + slot) * L + l, Fx_prev);
            } else if constexpr (XM == NEG) {
                Fx_prev = qweno(X(3), X(2), X(1), c, X(-1));
                if (act) sts(fsm + (buf * CX + slot) * L + l, Fx_prev);
            } else {
                const int need = (own ? codeq(ux0) : 0) | sg[(buf * (CX + 1) + slot + 1) * L + l];
                Q Lx = qz(), Rx = qz();
                if (__any_sync(FULL, need & 1)) Lx = qweno(X(-2), X(-1), c, X(1), X(2));
                if (__any_sync(FULL, need & 2)) Rx = qweno(X(3), X(2), X(1), c, X(-1));
                if (act) {
                    sts(fsm + ((buf * CX + slot) * L + l) * 2, Lx);
                    sts(fsm + ((buf * CX + slot) * L + l) * 2 + 1, Rx);
                }
                Fx_prev = selq(ux0, Lx, Rx);
            }
            ux_prev = ux0;
        }
        if constexpr (SPLIT) row_arrive(bar);
        {
            Q Fhi, Flo;
            if constexpr (YM == POS) {
                Fhi = qweno(R(1), R(2), c, R(4), R(5));
                Flo = pLy;
                pLy = Fhi;
            } else if constexpr (YM == NEG) {
                Fhi = qweno(R(6), R(5), R(4), c, R(2));
                Flo = pRy;
                pRy = Fhi;
            } else {
                const int need = own ? (codeq(uy0) | (k + 1 < cnt ? codeq(uy1) : 0)) : 0;
                Q Ly = qz(), Ry = qz();
                if (__any_sync(FULL, need & 1)) Ly = qweno(R(1), R(2), c, R(4), R(5));
                if (__any_sync(FULL, need & 2)) Ry = qweno(R(6), R(5), R(4), c, R(2));
                Fhi = selq(uy0, Ly, Ry);
                Flo = selq(uy0, pLy, pRy);
                pLy = Ly;
                pRy = Ry;
            }
            fy_prev = qmuls(qmul(uy0, qsub(Fhi, Flo)), dyi);
        }
        ux0 = ux1;
        uy0 = uy1;
        rl = rl + 1 == Ny ? 0 : rl + 1;
        rv = rv + 1 == Ny ? 0 : rv + 1;
        sw = sw + 1 == 8 ? 0 : sw + 1;
        sq = sq + 1 == 8 ? 0 : sq + 1;
        outoff += rs;
        return true;
    };
    if constexpr (SPLIT) row_arrive(bar);                      // the phase the first row waits for
    for (int k = 0;; k += 2) {
        if (!step(k, std::integral_constant<int, 0>{})) break;
        if (!step(k + 1, std::integral_constant<int, 1>{})) break;
    }
}

// FP64: the y stencil in registers, shifted by one row per step. The next row, its velocities and the halo cells
// of the next row come by cp.async into shared memory (`priv`: five slots of the thread), issued after a
// row's barrier and waited for at its end: in registers they spilled, and L1 returns a warp's loads in
// order, so a spilled value then waited for the row's loads from DRAM (1.30 against 1.07 ms per stage at
// 320 x 320 x 32 x 36). Four copies of the step with the stencil in rings indexed at compile time need no
// moves and take 1.03 ms there, but a small grid pays for fetching the longer code: 17.4 against 14.9 us at
// 64 x 64 x 4 x 16. Bound: the FP64 pipe (55% busy with currents, 57%
// without), issue (62%) and the barrier per row.
template <bool AL, int XM, int YM, int MODE>
__device__ __forceinline__ void xyw_body(const WalkArgs<double>& p, D* rowb, D* fsm, D* priv, int* sg, int* marked, int n,
                                         int tx, int js, int je) {
    using T = double;
    using LV = LaneVec<T>;
    using V = typename LV::V;
    constexpr int ROWV = ROWV64;
    constexpr bool XMIX = XM == MIX, YMIX = YM == MIX, FUSED = MODE >= STAGE, RATES = MODE == STAGE_RATES, curr = MODE == PASS_CURRENTS;
    const int Nx = p.Nx, Ny = p.Ny, Nk = p.Nk, L = p.L, CX = p.CX;
    const int64_t slice = (int64_t)Nx * Ny * Nk;
    const int tid = threadIdx.x, l = tid % L;
    const bool act = tid / L < CX;                             // threads past the last cell repeat it
    const int slot = min(tid / L, CX - 1);
    const int cnt = je - js;
    const int ibase = tx * (CX - 1) - 1;                       // x of slot 0
    const int my_i = ((ibase + slot) % Nx + Nx) % Nx;
    const bool own = act && slot >= 1 && ibase + slot < Nx;
    const int m0 = LV::N * l, left = Nk - 1 - m0;
    // halo columns: 2 on the left, 3 on the right, loaded by the first 5*L threads
    const bool hal = tid < 5 * L;
    const int hs = tid / L < 2 ? tid / L - 2 : CX + tid / L - 2;
    const int hi_x = hal ? ((ibase + hs) % Nx + Nx) % Nx : 0;
    const int rs = Nx * Nk;                                    // row stride within a direction slice
    const T* base = p.Nin + slice * n;
    T* Sn = (FUSED ? p.Nout : p.S) + slice * n;
    const T* N0n = p.N0 + slice * n;
    const int colm = my_i * Nk + m0, hcol = hi_x * Nk + m0;
    const V gx = ldgv<false>(p.cgx + m0 + (int64_t)Nk * n, left), gy = ldgv<false>(p.cgy + m0 + (int64_t)Nk * n, left);
    const bool cgp = p.cg_per_cell != 0;
    auto modr = [&](int r) { return (r % Ny + Ny) % Ny; };
    auto ld = [&](int r, int col) { return ldv<AL>(base + r * rs + col, left); };
    V* own_at = rowb + (slot + 2) * L + l;
    V* hal_at = rowb + (hs + 2) * L + l;
    D* mine = priv + threadIdx.x;                              // slots 0, 1: rows; 2, 3, 4: U_x, U_y, c_g
    auto vload = [&](int r) {
        const int e = r * rs + colm;
        if (curr) {
            copy_async<AL>(mine + 2 * XTHREADS, p.ux + e, left);
            copy_async<AL>(mine + 3 * XTHREADS, p.uy + e, left);
        }
        if (cgp) copy_async<AL>(mine + 4 * XTHREADS, p.cg + e, left);
    };
    auto rload = [&](int slot_, int r) { copy_async<AL>(mine + slot_ * XTHREADS, base + r * rs + colm, left); };
    // velocities in the reference's order: (c_g * direction table) + U (intrinsic: no U)
    auto velo = [&](V& ux, V& uy) {
        ux = gx;
        uy = gy;
        if (cgp) {
            const V vc = lds(mine + 4 * XTHREADS);
            ux = qmul(vc, ux);
            uy = qmul(vc, uy);
        }
        if (curr) {
            ux = qadd(ux, lds(mine + 2 * XTHREADS));
            uy = qadd(uy, lds(mine + 3 * XTHREADS));
        }
    };
    // fused stage: the inputs of the row being finished, loaded one row ahead (after that row's faces)
    V pn0 = LV::zero(), plr = LV::zero();
    auto pend = [&](int j) {
        const int off = j * rs + colm;
        if (p.stage != 1) pn0 = ldv<AL>(N0n + off, left);
        if (RATES) plr = ldv<AL>(p.rates + slice * n + off, left);
    };
    V ux0, uy0;
    vload(modr(js));
    copy_commit();
    copy_wait<0>();
    velo(ux0, uy0);

    // the y stencil. Uniform bodies: row (or difference) q in slot (q - j) & 3: rows sw, oriented first
    // differences dw (POS: s[q+1] - s[q]; NEG: s[q] - s[q+1]), second differences ew and their regularised
    // squares aw (POS: e[q] = d[q] - d[q-1]; NEG: e[q] = d[q] - d[q+1]). General body: rows j-2 .. j+3 in w.
    V sw[4], dw[4], ew[4], aw[4], w[6];
    V pLy = LV::zero(), pRy = LV::zero();   // the candidates of the lower y face of the current row
    if (XMIX && slot == 0 && act) {
        sg[CX * L + l] = 0;
        sg[(2 * CX + 1) * L + l] = 0;
    }
    if constexpr (YMIX) {
#pragma unroll
        for (int d = -2; d <= 3; ++d) w[d + 2] = ld(modr(js + d), colm);
        const V below = ld(modr(js - 3), colm);
        const int need = own ? codeq(uy0) : 0;
        if (__any_sync(FULL, need & 1)) pLy = qweno_each(below, w[0], w[1], w[2], w[3]);
        if (__any_sync(FULL, need & 2)) pRy = qweno_each(w[4], w[3], w[2], w[1], w[0]);
        rload(0, modr(js + 4));
    } else if constexpr (YM == POS) {
        const V r0 = ld(modr(js - 3), colm), r1 = ld(modr(js - 2), colm), r2 = ld(modr(js - 1), colm);
        sw[0] = ld(js, colm);
        sw[1] = ld(modr(js + 1), colm);
        rload(0, modr(js + 2));
        const V d1 = qsub(r1, r0);
        dw[2] = qsub(r2, r1);
        dw[3] = qsub(sw[0], r2);
        dw[0] = qsub(sw[1], sw[0]);
        const V e2 = qsub(dw[2], d1), a2 = qareg(e2);
        ew[3] = qsub(dw[3], dw[2]);
        ew[0] = qsub(dw[0], dw[3]);
        aw[3] = qareg(ew[3]);
        aw[0] = qareg(ew[0]);
        sw[3] = r2;
        pLy = qface(d1, dw[2], dw[3], dw[0], e2, ew[3], ew[0], a2, aw[3], aw[0], r2);
    } else {
        const V r1 = ld(modr(js - 2), colm);
        sw[3] = ld(modr(js - 1), colm);
        sw[0] = ld(js, colm);
        sw[1] = ld(modr(js + 1), colm);
        sw[2] = ld(modr(js + 2), colm);
        rload(0, modr(js + 3));
        const V d2 = qsub(r1, sw[3]);
        dw[3] = qsub(sw[3], sw[0]);
        dw[0] = qsub(sw[0], sw[1]);
        dw[1] = qsub(sw[1], sw[2]);
        const V e2 = qsub(d2, dw[3]), a2 = qareg(e2);
        ew[3] = qsub(dw[3], dw[0]);
        ew[0] = qsub(dw[0], dw[1]);
        aw[3] = qareg(ew[3]);
        aw[0] = qareg(ew[0]);
        pLy = qface(dw[1], dw[0], dw[3], d2, ew[0], ew[3], e2, aw[0], aw[3], a2, sw[0]);
    }
    if (hal) copy_async<AL>(hal_at, base + js * rs + hcol, left);
    // general body: the velocity of row j+1 is known during row j
    if constexpr (YMIX) vload(modr(js + 1));
    copy_commit();
    copy_wait<0>();
    // rows the next loads touch
    constexpr int AHEAD = YMIX ? 5 : (YM == POS ? 3 : 4);
    int rl = modr(js + AHEAD), rv = modr(js + (YMIX ? 2 : 1)), rh = modr(js + 1);
    const T dxi = p.dx_inv, dyi = p.dy_inv;
    V Fx_prev = LV::zero(), fy_prev = LV::zero(), ux_prev = LV::zero();
    int outoff = js * rs + colm;
    auto step = [&](int k) {
        const int buf = k & 1;
        const bool row = k < cnt;
        V c, ux1 = LV::zero(), uy1 = LV::zero();
        if constexpr (YMIX) c = w[2];
        else c = sw[0];
        if (row) {
            if (act) sts(own_at + buf * ROWV, c);
            if constexpr (XMIX)
                if (act) sg[(buf * (CX + 1) + slot) * L + l] = own ? codeq(ux0) : 0;
            if constexpr (YMIX) velo(ux1, uy1);
        }
        __syncthreads();
        if (row) {   // row j is complete in rowb; the other buffer's last readers have passed this barrier
            rload(1 - buf, rl);
            vload(rv);
            if (hal) copy_async<AL>(hal_at + (1 - buf) * ROWV, base + rh * rs + hcol, left);
            copy_commit();
        }
        // the previous row: its lower x face from the left neighbour's candidates, then S
        if (k > 0 && slot >= 1) {
            V Flo;
            if constexpr (XMIX) {
                const V* f = fsm + (((1 - buf) * CX + slot - 1) * L + l) * 2;
                Flo = selq(ux_prev, lds(f), lds(f + 1));
            } else {
                Flo = lds(fsm + ((1 - buf) * CX + slot - 1) * L + l);
            }
            const V fx = qmuls(qmul(ux_prev, qsub(Fx_prev, Flo)), dxi);
            if constexpr (!FUSED) {
                if (own) stv<AL>(Sn + outoff - rs, qadd(fx, fy_prev), left);
            } else {
                V cv;                                          // the finished row's action
                if constexpr (YMIX) cv = w[1];
                else cv = sw[3];
                V G = qneg(qadd(fx, fy_prev));
                if (RATES) G = qfma(plr, cv, G);             // SourceTermSet rates of this stage
                const V o = stage_update<T>(G, cv, pn0, p.stage, p.dt, p.a, p.b);
                if (own) {   // a result that is not finite is marked in S, as store_result (rpl_ring.cu) does
                    if (qfinite(o)) {
                        stv<AL>(Sn + outoff - rs, o, left);
                    } else {
                        const bool again = qfinite(cv);
                        if (again) marked[threadIdx.x] = 1;
                        else atomicOr(p.err, 1u);
                        stv<AL>((again ? p.S + slice * n : Sn) + outoff - rs, o, left);
                    }
                }
            }
        }
        if (!row) return false;
        if constexpr (FUSED) pend(js + k);
        {
            const V* xr = own_at + buf * ROWV;
            auto X = [&](int d) { return lds(xr + d * L); };   // cell slot+d of row j
            if constexpr (XM == POS) {
                Fx_prev = qweno(X(-2), X(-1), c, X(1), X(2));
                if (act) sts(fsm + (buf * CX + slot) * L + l, Fx_prev);
            } else if constexpr (XM == NEG) {
                Fx_prev = qweno(X(3), X(2), X(1), c, X(-1));
                if (act) sts(fsm + (buf * CX + slot) * L + l, Fx_prev);
            } else {
                const int need = (own ? codeq(ux0) : 0) | sg[(buf * (CX + 1) + slot + 1) * L + l];
                V Lx = LV::zero(), Rx = LV::zero();
                if (__any_sync(FULL, need & 1)) Lx = qweno_each(X(-2), X(-1), c, X(1), X(2));
                if (__any_sync(FULL, need & 2)) Rx = qweno_each(X(3), X(2), X(1), c, X(-1));
                if (act) {
                    sts(fsm + ((buf * CX + slot) * L + l) * 2, Lx);
                    sts(fsm + ((buf * CX + slot) * L + l) * 2 + 1, Rx);
                }
                Fx_prev = selq(ux0, Lx, Rx);
            }
            ux_prev = ux0;
        }
        {
            V Fhi, Flo;
            if constexpr (YMIX) {
                const int need = own ? (codeq(uy0) | (k + 1 < cnt ? codeq(uy1) : 0)) : 0;
                V Ly = LV::zero(), Ry = LV::zero();
                if (__any_sync(FULL, need & 1)) Ly = qweno_each(w[0], w[1], w[2], w[3], w[4]);
                if (__any_sync(FULL, need & 2)) Ry = qweno_each(w[5], w[4], w[3], w[2], w[1]);
                Fhi = selq(uy0, Ly, Ry);
                Flo = selq(uy0, pLy, pRy);
                pLy = Ly;
                pRy = Ry;
            } else if constexpr (YM == POS) {
                sw[2] = lds(mine + buf * XTHREADS);            // row j+2
                dw[1] = qsub(sw[2], sw[1]);
                ew[1] = qsub(dw[1], dw[0]);
                aw[1] = qareg(ew[1]);
                Fhi = qface(dw[2], dw[3], dw[0], dw[1], ew[3], ew[0], ew[1], aw[3], aw[0], aw[1], c);
                Flo = pLy;
                pLy = Fhi;
            } else {
                sw[3] = lds(mine + buf * XTHREADS);            // row j+3
                dw[2] = qsub(sw[2], sw[3]);
                ew[1] = qsub(dw[1], dw[2]);
                aw[1] = qareg(ew[1]);
                Fhi = qface(dw[2], dw[1], dw[0], dw[3], ew[1], ew[0], ew[3], aw[1], aw[0], aw[3], sw[1]);
                Flo = pLy;
                pLy = Fhi;
            }
            fy_prev = qmuls(qmul(uy0, qsub(Fhi, Flo)), dyi);
        }
        if constexpr (YMIX) {
#pragma unroll
            for (int q = 0; q < 5; ++q) w[q] = w[q + 1];
            w[5] = lds(mine + buf * XTHREADS);
            ux0 = ux1;
            uy0 = uy1;
            copy_wait<0>();
        } else {
            auto turn = [](V* r) {   // row j+1 is the next step's row j
                const V t = r[0];
                r[0] = r[1];
                r[1] = r[2];
                r[2] = r[3];
                r[3] = t;
            };
            turn(sw);
            turn(dw);
            turn(ew);
            turn(aw);
            copy_wait<0>();
            velo(ux0, uy0);
        }
        rl = rl + 1 == Ny ? 0 : rl + 1;
        rv = rv + 1 == Ny ? 0 : rv + 1;
        rh = rh + 1 == Ny ? 0 : rh + 1;
        outoff += rs;
        return true;
    };
    for (int k = 0; step(k); ++k) {}
}

// The results of the thread's column that the whole-stage body marked, once more from the tendency of the wider range
// (redo in rpl_ring.cu).
template <bool AL>
__device__ __noinline__ void redo_column(const WalkArgs<double>& p, int n, int tx, int js, int je) {
    const int l = threadIdx.x % p.L, slot = threadIdx.x / p.L, i = tx * (p.CX - 1) - 1 + slot;   // own cells only
    const int m0 = 2 * l, left = p.Nk - 1 - m0;
    for (int j = js; j < je; ++j) {
        const int64_t cell = (int64_t)j * p.Nx + i, off = ((int64_t)p.Nx * p.Ny * n + cell) * p.Nk + m0;
        if (qfinite(ldv<AL>(p.S + off, left))) continue;
        D G = {bin_tendency_wide<false>(p, cell, m0, n), bin_tendency_wide<false>(p, cell, m0 + min(1, left), n)};
        const D c = ldv<AL>(p.Nin + off, left);
        if (p.rates) G = qfma(ldv<AL>(p.rates + off, left), c, G);
        const D o = stage_update<double>(G, c, p.stage == 1 ? D{0., 0.} : ldv<AL>(p.N0 + off, left), p.stage, p.dt, p.a, p.b);
        if (!qfinite(o)) atomicOr(p.err, 1u);
        stv<AL>(p.Nout + off, o, left);
    }
}

template <typename T, bool AL, int LB, int XM, int YM, int MODE>
__device__ __forceinline__ void run_body(const WalkArgs<T>& p, unsigned char* smem, int* sg, int* marked, unsigned bar, int n,
                                         int tx, int js, int je) {
    if constexpr (std::is_same<T, float>::value) {
        constexpr int ROWV = XTHREADS + 5 * LB;
        Q* ring = reinterpret_cast<Q*>(smem);
        xyw_body_ring<AL, ROWV, XM, YM, MODE>(p, ring, ring + 16 * ROWV, ring + 16 * ROWV + 4 * XTHREADS, sg, bar, n, tx, js,
                                              je);
    } else {
        D* rows = reinterpret_cast<D*>(smem);
        xyw_body<AL, XM, YM, MODE>(p, rows, rows + 2 * ROWV64, rows + 2 * ROWV64 + 4 * XTHREADS, sg, marked, n, tx, js, je);
    }
}

// Shared memory: the staged rows, then the x faces of two rows (two candidates each in the general body), FP64
// then the threads' private slots.
template <typename T, int LB> constexpr size_t xyw_smem() {
    return ((std::is_same<T, float>::value ? 16 * (XTHREADS + 5 * LB) + (LB <= 8 ? 1 : 0) * XTHREADS : 2 * ROWV64 + 5 * XTHREADS) +
            4 * XTHREADS) * 16;
}

// One CTA per (direction, x tile, row segment), direction fastest so the CTAs of one region run together.
// LB: most lanes per cell the staged rows have room for.
template <typename T, bool AL, int LB, int MODE>
__global__ void __launch_bounds__(XTHREADS, 2)
xyw_kernel(const __grid_constant__ WalkArgs<T> p, int seg0) {
    constexpr int N = LaneVec<T>::N;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int sg[2 * (XTHREADS + MAXL)];
    // FP64 whole stage, per thread: some of its results are to be made again
    constexpr bool MARKS = std::is_same<T, double>::value && MODE >= STAGE;
    __shared__ int marked[MARKS ? XTHREADS : 1];
    if (MARKS) marked[threadIdx.x] = 0;
    __shared__ __align__(8) unsigned long long row_bar;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&row_bar);
    if (std::is_same<T, float>::value && threadIdx.x == 0)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(blockDim.x / 32) : "memory");
    int b = blockIdx.x;
    const int n = b % p.Np;
    b /= p.Np;
    const int tx = b % p.tiles_x, seg = seg0 + b / p.tiles_x;
    const int js = max(p.j_lo, seg * p.seg), je = min(p.j_hi, (seg + 1) * p.seg);
    // the uniform test of the thread's bins against the region's ratios
    const int Nk = p.Nk, m0 = N * (threadIdx.x % p.L), left = Nk - 1 - m0;
    const int64_t region = (int64_t)seg * p.tiles_x + tx;
    const unsigned* rx = p.rmax + (2 * region) * Nk + m0;
    const unsigned* ry = rx + Nk;
    const float2* g = p.cg32 + m0 + (int64_t)Nk * n;
    bool xp = true, xn = true, yp = true, yn = true;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        const int o = min(q, left);
        const float2 gq = __ldg(g + o);
        constexpr float SH = 1.0f - 1e-5f;
        const bool cx = fabsf(gq.x) * SH > __uint_as_float(__ldg(rx + o));
        const bool cy = fabsf(gq.y) * SH > __uint_as_float(__ldg(ry + o));
        xp = xp && cx && gq.x > 0.f;
        xn = xn && cx && gq.x < 0.f;
        yp = yp && cy && gq.y > 0.f;
        yn = yn && cy && gq.y < 0.f;
    }
    const int allxp = __syncthreads_and(xp), allxn = __syncthreads_and(xn);
    const int allyp = __syncthreads_and(yp), allyn = __syncthreads_and(yn);
    const int xm = allxp ? POS : (allxn ? NEG : MIX), ym = allyp ? POS : (allyn ? NEG : MIX);
    // one body per pair of signs, mixed ones included: 5 to 17% of the directions run along an axis, where one
    // component's sign depends on the current. Against the four uniform bodies and one general body: 407 against
    // 431 us per stage at 389 x 251 x 25 x 24 FP32, 1041 against 1068 at 320 x 320 x 32 x 36 FP64.
#define RPL_BODY(X, Y) \
    if (xm == X && ym == Y) run_body<T, AL, LB, X, Y, MODE>(p, smem, sg, marked, bar, n, tx, js, je)
    RPL_BODY(POS, POS);
    else RPL_BODY(POS, NEG);
    else RPL_BODY(NEG, POS);
    else RPL_BODY(NEG, NEG);
    else RPL_BODY(POS, MIX);
    else RPL_BODY(NEG, MIX);
    else RPL_BODY(MIX, POS);
    else RPL_BODY(MIX, NEG);
    else RPL_BODY(MIX, MIX);
#undef RPL_BODY
    if constexpr (MARKS)
        if (marked[threadIdx.x]) redo_column<AL>(p, n, tx, js, je);
}

template <typename T, bool AL, int LB, int MODE>
cudaError_t launch_xyw_lb(const WalkArgs<T>& a, const WalkGeom& g, cudaStream_t s) {
    constexpr size_t smem = xyw_smem<T, LB>();
    const int seg0 = a.j_lo / g.seg, seg1 = (a.j_hi - 1) / g.seg;
    const unsigned blocks = (unsigned)((int64_t)a.Np * g.tiles_x * (seg1 - seg0 + 1));
    auto k = xyw_kernel<T, AL, LB, MODE>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    k<<<blocks, g.threads, smem, s>>>(a, seg0);
    return cudaGetLastError();
}

// The instances, spread over translation units (rpl_xyw_f32.cu: whole lane vectors up to Nk = 32;
// rpl_xyw_f32u.cu: any Nk up to 64; rpl_xyw_f64.cu).
#define RPL_XYW_INSTANCES(EXT, T, AL, LB)                                                                   \
    EXT template cudaError_t launch_xyw_lb<T, AL, LB, PASS>(const WalkArgs<T>&, const WalkGeom&, cudaStream_t);          \
    EXT template cudaError_t launch_xyw_lb<T, AL, LB, PASS_CURRENTS>(const WalkArgs<T>&, const WalkGeom&, cudaStream_t); \
    EXT template cudaError_t launch_xyw_lb<T, AL, LB, STAGE>(const WalkArgs<T>&, const WalkGeom&, cudaStream_t);         \
    EXT template cudaError_t launch_xyw_lb<T, AL, LB, STAGE_RATES>(const WalkArgs<T>&, const WalkGeom&, cudaStream_t);

}  // namespace xyw
}  // namespace rpl
