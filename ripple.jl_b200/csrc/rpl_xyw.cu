// rpl_xyw.cu -- set-up and dispatch of the y-walk x/y pass (rpl_xyw.cuh): the CTA geometry, the velocity planes
// and upwind ratios, the kernels' arguments.
#include "rpl_xyw.cuh"

#include <algorithm>

namespace rpl {

namespace xyw {
RPL_XYW_INSTANCES(extern, float, true, 8)
RPL_XYW_INSTANCES(extern, float, false, 8)
RPL_XYW_INSTANCES(extern, float, false, 16)
RPL_XYW_INSTANCES(extern, double, true, 32)
RPL_XYW_INSTANCES(extern, double, false, 32)
}  // namespace xyw

namespace {

using namespace xyw;

// Velocity planes (U_x, U_y, c_g magnitude per (i,j,m), device order, type T) from the coefficient records,
// and per region (x tile of per_tile cells, seg rows) and bin m the maxima of |U_x| / c and |U_y| / c
// (c the per-cell c_g magnitude, or 1 when c_g is folded into the direction table), enlarged by 1e-5,
// at rmax[(2 region + axis) Nk + m] as bit patterns (non-negative floats order like them). One thread per
// (bin, column, VROWS rows of a segment).
constexpr int VROWS = 4;

template <typename T>
__global__ void vel_kernel(int Nx, int Ny, int Nk, int per_tile, int tiles_x, int seg_rows, const double* __restrict__ coef,
                           int cg_per_cell, T* ux_p, T* uy_p, T* cg_p, unsigned* rmax) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int chunks = (Ny + VROWS - 1) / VROWS;   // seg_rows is a multiple of VROWS
    if (t >= (int64_t)Nk * Nx * chunks) return;
    const int m = (int)(t % Nk), i = (int)((t / Nk) % Nx), ch = (int)(t / ((int64_t)Nk * Nx));
    float rx = 0.f, ry = 0.f;
    const float inf = __int_as_float(0x7f800000);
    const int jend = min(Ny, (ch + 1) * VROWS);
    for (int j = ch * VROWS; j < jend; ++j) {
        const int64_t e = ((int64_t)j * Nx + i) * Nk + m;
        const double* r = coef + 8 * e;
        const double2 u = *reinterpret_cast<const double2*>(r);
        const float ux = (float)u.x, uy = (float)u.y, cm = (float)r[6];
        if (ux_p) {
            ux_p[e] = (T)u.x;
            uy_p[e] = (T)u.y;
        }
        cg_p[e] = (T)r[6];
        const float c = cg_per_cell ? cm : 1.0f;
        rx = fmaxf(rx, c > 0.f ? fabsf(ux) / c * (1.0f + 1e-5f) : inf);
        ry = fmaxf(ry, c > 0.f ? fabsf(uy) / c * (1.0f + 1e-5f) : inf);
    }
    const int64_t region = (int64_t)(ch * VROWS / seg_rows) * tiles_x + i / per_tile;
    atomicMax(rmax + (2 * region) * Nk + m, __float_as_uint(rx));
    atomicMax(rmax + (2 * region + 1) * Nk + m, __float_as_uint(ry));
}

template <int MODE>
cudaError_t launch_xyw(const WalkArgs<float>& a, const WalkGeom& g, cudaStream_t s) {
    if (g.L > 8) return launch_xyw_lb<float, false, 16, MODE>(a, g, s);
    return a.Nk % 4 == 0 ? launch_xyw_lb<float, true, 8, MODE>(a, g, s) : launch_xyw_lb<float, false, 8, MODE>(a, g, s);
}
template <int MODE>
cudaError_t launch_xyw(const WalkArgs<double>& a, const WalkGeom& g, cudaStream_t s) {
    return a.Nk % 2 == 0 ? launch_xyw_lb<double, true, 32, MODE>(a, g, s) : launch_xyw_lb<double, false, 32, MODE>(a, g, s);
}

}  // namespace

bool walk_supported(const rpl_desc& d) {
    // at most 32 lanes per cell; offsets within one direction slice are 32-bit
    return (d.transport == RPL_TRANSPORT_REFRACTION || d.transport == RPL_TRANSPORT_INTRINSIC) && d.Nk <= 64 &&
           d.Nx * d.Ny * d.Nk < (int64_t)1 << 31 && d.Nx >= 3 && d.Ny >= 3 &&
           (d.transport != RPL_TRANSPORT_REFRACTION || d.Np >= 3);
}

// Cells per CTA: as many as 256 threads hold, spread evenly over the tiles a row needs (a row of 64 cells
// takes one tile of 65 slots, not one of 128 with half of them idle). Rows per segment: a segment pays a
// prologue of six row loads and one face per column, so long segments are cheaper, but a small grid then
// leaves SMs without a CTA: the largest of 128, 64, 32, 16, 8, 4 rows that gives two CTAs per SM.
WalkGeom walk_geometry(const rpl_desc& d) {
    WalkGeom g;
    const int N = d.precision == RPL_FP64 ? 2 : 4;
    g.L = (int)((d.Nk + N - 1) / N);
    const int64_t most = XTHREADS / g.L - 1;
    g.tiles_x = (int)((d.Nx + most - 1) / most);
    g.CX = (int)((d.Nx + g.tiles_x - 1) / g.tiles_x) + 1;
    g.threads = ((std::max(g.CX, 5) * g.L + 31) / 32) * 32;   // at least the five halo columns' threads
    g.seg = 128;
    while (g.seg > 4 && d.Np * g.tiles_x * ((d.Ny + g.seg - 1) / g.seg) < 2 * 148) g.seg /= 2;
    return g;
}

cudaError_t launch_vel(const Handle& h, cudaStream_t s) {
    if (!h.d_vel) return cudaSuccess;
    pin_planes(h, s);
    const rpl_desc& d = h.desc;
    const int64_t c3 = d.Nx * d.Ny * d.Nk;
    const int per_tile = h.walk.CX - 1;
    cudaError_t e = cudaMemsetAsync(h.d_rmax, 0, 2 * h.vel_regions * d.Nk * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    const int64_t threads = d.Nk * d.Nx * ((d.Ny + VROWS - 1) / VROWS);
    const unsigned blocks = (unsigned)((threads + 255) / 256);
    // refraction: U_x, U_y and c_g planes; intrinsic transport (no currents): the c_g plane only
    const bool refract = d.transport == RPL_TRANSPORT_REFRACTION;
    auto go = [&](auto* v) {
        auto* ux = refract ? v : nullptr;
        auto* uy = refract ? v + c3 : nullptr;
        auto* cg = refract ? v + 2 * c3 : v;
        vel_kernel<<<blocks, 256, 0, s>>>((int)d.Nx, (int)d.Ny, (int)d.Nk, per_tile, h.walk.tiles_x, h.walk.seg, h.d_coef,
                                          h.d_cgmag != nullptr, ux, uy, cg, h.d_rmax);
    };
    if (h.precision == RPL_FP64) go((double*)h.d_vel);
    else go((float*)h.d_vel);
    return cudaGetLastError();
}

template <typename T>
WalkArgs<T> make_walk_args(const Handle& h, const StageParams& p, const void* Nin, const void* N0, void* Nout) {
    WalkArgs<T> a{};
    const rpl_desc& d = h.desc;
    a.Nin = (const T*)Nin;
    a.N0 = (const T*)N0;
    a.Nout = (T*)Nout;
    a.S = (T*)stage_scratch(h, Nout);
    const int64_t c3 = d.Nx * d.Ny * d.Nk;
    const T* v = (const T*)h.d_vel;
    if (v && d.transport == RPL_TRANSPORT_REFRACTION) {
        a.ux = v;
        a.uy = v + c3;
        a.cg = v + 2 * c3;
    } else {
        a.cg = v;
    }
    a.rates = (const T*)p.lin_rates;
    a.coef = p.coef;
    a.trig32 = p.trig32;
    a.cg32 = p.cg32;
    a.cgx = p.cg_x;
    a.cgy = p.cg_y;
    a.cosp = p.cosp;
    a.sinp = p.sinp;
    a.rmax = h.d_rmax;
    a.err = p.err;
    a.Nx = (int)d.Nx;
    a.Ny = (int)d.Ny;
    a.Nk = (int)d.Nk;
    a.Np = (int)d.Np;
    a.stage = p.stage;
    a.cg_per_cell = p.cg_per_cell;
    a.j_lo = (int)p.j_lo;
    a.j_hi = (int)p.j_hi;
    a.L = h.walk.L;
    a.CX = h.walk.CX;
    a.tiles_x = h.walk.tiles_x;
    a.seg = h.walk.seg;
    a.dx_inv = (T)p.dx_inv;
    a.dy_inv = (T)p.dy_inv;
    a.dk_inv = (T)p.dk_inv;
    a.dp_inv = (T)p.dp_inv;
    a.dt = (T)p.dt;
    a.a = (T)p.a;
    a.b = (T)p.b;
    return a;
}
template WalkArgs<float> make_walk_args<float>(const Handle&, const StageParams&, const void*, const void*, void*);
template WalkArgs<double> make_walk_args<double>(const Handle&, const StageParams&, const void*, const void*, void*);

template <typename T>
cudaError_t launch_xy_pass(const WalkArgs<T>& a, const WalkGeom& g, cudaStream_t s) {
    return a.ux ? launch_xyw<PASS_CURRENTS>(a, g, s) : launch_xyw<PASS>(a, g, s);
}
template <typename T>
cudaError_t launch_xy_stage(const WalkArgs<T>& a, const WalkGeom& g, cudaStream_t s) {
    return a.rates ? launch_xyw<STAGE_RATES>(a, g, s) : launch_xyw<STAGE>(a, g, s);
}
template cudaError_t launch_xy_pass<float>(const WalkArgs<float>&, const WalkGeom&, cudaStream_t);
template cudaError_t launch_xy_pass<double>(const WalkArgs<double>&, const WalkGeom&, cudaStream_t);
template cudaError_t launch_xy_stage<float>(const WalkArgs<float>&, const WalkGeom&, cudaStream_t);
template cudaError_t launch_xy_stage<double>(const WalkArgs<double>&, const WalkGeom&, cudaStream_t);

}  // namespace rpl
