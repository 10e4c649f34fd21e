// rpl_walk.h -- arguments and launchers of the two-pass stage kernels: the x/y pass as a y-walk
// (rpl_xyw.cu) and the kappa/phi/source pass as a walk of the phi ring (rpl_ring.cu), FP32 and FP64.
#pragma once

#include "rpl_internal.h"

namespace rpl {

template <typename T>
struct WalkArgs {
    const T* Nin;
    const T* N0;
    T* Nout;
    T* S;                      // x+y flux sums between the passes (state layout); may be Nout itself
    const T* ux;               // planes of U_x, U_y and the c_g magnitude per (i,j,m), device order;
    const T* uy;               // ux, uy null for intrinsic transport
    const T* cg;
    const T* rates;            // SourceTermSet rates per cell-bin (state layout) or null
    const double* coef;
    const float4* trig32;
    const float2* cg32;
    const double* cgx;
    const double* cgy;
    const double* cosp;
    const double* sinp;
    const unsigned* rmax;
    unsigned* err;
    int Nx, Ny, Nk, Np, stage, cg_per_cell, j_lo, j_hi;
    int L, CX, tiles_x, seg;   // lanes per cell, cells per CTA row (one supplies a face only), tiles, rows per segment
    T dx_inv, dy_inv, dk_inv, dp_inv, dt, a, b;
};

// Geometry of the y-walk for a model: lanes per cell, cells per CTA (the first supplies a face only), x
// tiles, rows per segment and threads per CTA.
WalkGeom walk_geometry(const rpl_desc& d);
bool walk_supported(const rpl_desc& d);

template <typename T>
WalkArgs<T> make_walk_args(const Handle& h, const StageParams& p, const void* Nin, const void* N0, void* Nout);

// The x/y pass: S = fx + fy of rows [j_lo, j_hi).
template <typename T> cudaError_t launch_xy_pass(const WalkArgs<T>& a, const WalkGeom& g, cudaStream_t s);
// The whole stage of intrinsic transport (no currents, no bundle or learned sources) in one pass.
template <typename T> cudaError_t launch_xy_stage(const WalkArgs<T>& a, const WalkGeom& g, cudaStream_t s);
// The second pass: kappa and phi fluxes (refraction), SourceTermSet rates or the FP64 source bundle, update.
template <typename T>
cudaError_t launch_ring(const WalkArgs<T>& a, const StageParams& p, bool refract, bool bundle, cudaStream_t s);

}  // namespace rpl
