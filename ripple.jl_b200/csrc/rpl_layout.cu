// rpl_layout.cu -- conversions between the caller's layout and the device layout of the state,
// and the per-(i,j,kappa) coefficient records the stage kernels read.
//
// Caller layout (RPL_LAYOUT_XFAST, the reference's flat_data interior): (i,j,m,n) at
//   c + P*(m + Nk*n),   c = i + Nx*j, P = Nx*Ny.
// Device layout of the state: kappa fastest, one contiguous spectral column slice per (i,j,n):
//   (n*P + c)*Nk + m.
// For each direction bin n this is the transpose of an Nk x P matrix, done in tiles through shared memory
// so both sides are read and written in full lines.
#include <cuda_runtime.h>

#include "rpl_internal.h"

namespace rpl {

namespace {

// Tiles of CT cells x 32 kappa bins through shared memory. Each thread holds all of its tile's loads (eight) in
// flight before the first is stored: the pass is bound by memory latency (32 x 32 tiles with four loads in
// flight took 648 us for 448 x 448 x 32 x 36 FP32, 2.9 TB/s; one read and one write of the state are 287 us).
// VEC: sixteen bytes (four cells) per access on the caller's side, where its rows are 16-byte aligned.
constexpr int CT = 64, MT = 32, LTHREADS = 256, PAD = 1;

template <typename S> struct Four { S v[4]; };

// src: rows m0 .. m0+mc-1 of slices n0 .. n0+nc-1 in caller layout, starting at (n0, m0)
// dst: device layout, whole array. err: bit 2 is set where a converted value is not finite.
template <typename S, typename D, bool VEC>
__global__ void __launch_bounds__(LTHREADS) to_device_kernel(const S* __restrict__ src, D* __restrict__ dst, int64_t P, int64_t Nk,
                                 int64_t n0, int64_t m0, int64_t mc, int64_t src_slice_stride, unsigned int* err) {
    __shared__ D tile[MT][CT + PAD];
    const int64_t c0 = (int64_t)blockIdx.x * CT, mb = (int64_t)blockIdx.y * MT;
    const int64_t n = n0 + blockIdx.z;
    const S* s = src + (int64_t)blockIdx.z * src_slice_stride;
    const int nm = (int)min((int64_t)MT, mc - mb), nc = (int)min((int64_t)CT, P - c0);
    bool bad = false;
    if (VEC) {
        constexpr int PER = MT * CT / 4 / LTHREADS;
        Four<S> v[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int q = threadIdx.x + k * LTHREADS, r = q / (CT / 4), x = (q % (CT / 4)) * 4;
            if (r < nm && x < nc) {   // P is a multiple of 4: four cells or none
                const S* at = s + (mb + r) * P + c0 + x;
                if constexpr (sizeof(S) == 4) {
                    const float4 f = __ldcs(reinterpret_cast<const float4*>(at));
                    v[k] = {(S)f.x, (S)f.y, (S)f.z, (S)f.w};
                } else {
                    const double2 f = __ldcs(reinterpret_cast<const double2*>(at)), g = __ldcs(reinterpret_cast<const double2*>(at) + 1);
                    v[k] = {(S)f.x, (S)f.y, (S)g.x, (S)g.y};
                }
            }
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int q = threadIdx.x + k * LTHREADS, r = q / (CT / 4), x = (q % (CT / 4)) * 4;
            if (r < nm && x < nc) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const D d = (D)v[k].v[j];
                    bad |= !isfinite(d);
                    tile[r][x + j] = d;
                }
            }
        }
    } else {
        constexpr int PER = MT * CT / LTHREADS;
        S v[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int q = threadIdx.x + k * LTHREADS, r = q / CT, x = q % CT;
            if (r < nm && x < nc) v[k] = __ldcs(s + (mb + r) * P + c0 + x);
        }
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int q = threadIdx.x + k * LTHREADS, r = q / CT, x = q % CT;
            if (r < nm && x < nc) {
                const D d = (D)v[k];
                bad |= !isfinite(d);
                tile[r][x] = d;
            }
        }
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(err, 2u);
    D* out = dst + (n * P + c0) * Nk + m0 + mb;
#pragma unroll
    for (int k = 0; k < MT * CT / LTHREADS; ++k) {
        const int q = threadIdx.x + k * LTHREADS, x = q / MT, r = q % MT;
        if (r < nm && x < nc) out[x * Nk + r] = tile[r][x];
    }
}

template <typename S, typename D, bool VEC>
__global__ void __launch_bounds__(LTHREADS) from_device_kernel(const S* __restrict__ src, D* __restrict__ dst, int64_t P, int64_t Nk,
                                   int64_t n0, int64_t m0, int64_t mc, int64_t dst_slice_stride) {
    __shared__ D tile[MT][CT + PAD];
    const int64_t c0 = (int64_t)blockIdx.x * CT, mb = (int64_t)blockIdx.y * MT;
    const int64_t n = n0 + blockIdx.z;
    D* d = dst + (int64_t)blockIdx.z * dst_slice_stride;
    const int nm = (int)min((int64_t)MT, mc - mb), nc = (int)min((int64_t)CT, P - c0);
    const S* in = src + (n * P + c0) * Nk + m0 + mb;
    S v[MT * CT / LTHREADS];
#pragma unroll
    for (int k = 0; k < MT * CT / LTHREADS; ++k) {
        const int q = threadIdx.x + k * LTHREADS, x = q / MT, r = q % MT;
        if (r < nm && x < nc) v[k] = __ldcs(in + x * Nk + r);
    }
#pragma unroll
    for (int k = 0; k < MT * CT / LTHREADS; ++k) {
        const int q = threadIdx.x + k * LTHREADS, x = q / MT, r = q % MT;
        if (r < nm && x < nc) tile[r][x] = (D)v[k];
    }
    __syncthreads();
    if (VEC) {
#pragma unroll
        for (int k = 0; k < MT * CT / 4 / LTHREADS; ++k) {
            const int q = threadIdx.x + k * LTHREADS, r = q / (CT / 4), x = (q % (CT / 4)) * 4;
            if (r < nm && x < nc) {
                D* at = d + (mb + r) * P + c0 + x;
                const D* t = &tile[r][x];
                if constexpr (sizeof(D) == 4) {
                    __stcs(reinterpret_cast<float4*>(at), make_float4(t[0], t[1], t[2], t[3]));
                } else {
                    __stcs(reinterpret_cast<double2*>(at), make_double2(t[0], t[1]));
                    __stcs(reinterpret_cast<double2*>(at) + 1, make_double2(t[2], t[3]));
                }
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < MT * CT / LTHREADS; ++k) {
            const int q = threadIdx.x + k * LTHREADS, r = q / CT, x = q % CT;
            if (r < nm && x < nc) d[(mb + r) * P + c0 + x] = tile[r][x];
        }
    }
}

// Coefficient record per (i,j,m), device order (j*Nx + i)*Nk + m, 8 doubles:
// Ux, Uy, Ux_x, Ux_y, Uy_x, Uy_y, c_g magnitude (depth field; else 0), kappa.
__global__ void coef_kernel(int64_t Nx, int64_t Ny, int64_t Nk, const double* __restrict__ coupling,
                            const double* __restrict__ cgmag, const double* __restrict__ kappa,
                            double* __restrict__ coef) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t P = Nx * Ny, c3 = P * Nk;
    if (t >= c3) return;
    const int64_t m = t % Nk, c = t / Nk;     // device order
    const int64_t x = c + P * m;              // caller order of the coupling arrays
    double* r = coef + 8 * t;
    if (coupling) {
        r[0] = coupling[x];
        r[1] = coupling[c3 + x];
        r[2] = coupling[4 * c3 + x];
        r[3] = coupling[5 * c3 + x];
        r[4] = coupling[6 * c3 + x];
        r[5] = coupling[7 * c3 + x];
    } else {
        r[0] = r[1] = r[2] = r[3] = r[4] = r[5] = 0.0;
    }
    r[6] = cgmag ? cgmag[x] : 0.0;
    r[7] = kappa[m];
}

constexpr int COEF_THREADS = 256;

// Coefficient records (Ux, Uy, Ux_x, Ux_y, Uy_x, Uy_y; fields 6 and 7 are kept) from the device-order
// velocity, with the periodic centred gradients of wave_current_refraction.jl:7-19. A block's 256
// records are assembled in shared memory and written back whole with 16-byte stores, so every DRAM
// sector is written in full.
__global__ void __launch_bounds__(COEF_THREADS)
coef_from_U_kernel(int64_t Nx, int64_t Ny, int Nk, const double* __restrict__ U, double dx_inv, double dy_inv,
                   double* __restrict__ coef) {
    __shared__ double2 rec[COEF_THREADS * 4];
    const int64_t P = Nx * Ny, c3 = P * Nk;
    const int64_t t0 = (int64_t)blockIdx.x * COEF_THREADS, t = t0 + threadIdx.x;
    if (t < c3) {
        const int64_t c = t / Nk, m = t - c * Nk;
        const int64_t j = c / Nx, i = c - j * Nx;
        const int64_t ip = i == Nx - 1 ? 0 : i + 1, im = i == 0 ? Nx - 1 : i - 1;
        const int64_t jp = j == Ny - 1 ? 0 : j + 1, jm = j == 0 ? Ny - 1 : j - 1;
        const int64_t xp = (j * Nx + ip) * Nk + m, xm = (j * Nx + im) * Nk + m;
        const int64_t yp = (jp * Nx + i) * Nk + m, ym = (jm * Nx + i) * Nk + m;
        const double* Uy = U + c3;
        double2* r = rec + threadIdx.x * 4;
        r[0] = make_double2(U[t], Uy[t]);
        r[1] = make_double2((U[xp] - U[xm]) * (dx_inv / 2.0), (U[yp] - U[ym]) * (dy_inv / 2.0));
        r[2] = make_double2((Uy[xp] - Uy[xm]) * (dx_inv / 2.0), (Uy[yp] - Uy[ym]) * (dy_inv / 2.0));
        r[3] = *reinterpret_cast<const double2*>(coef + 8 * t + 6);
    }
    __syncthreads();
    const int n = (int)(min((int64_t)COEF_THREADS, c3 - t0) * 4);
    double2* out = reinterpret_cast<double2*>(coef + 8 * t0);
    for (int k = threadIdx.x; k < n; k += COEF_THREADS) out[k] = rec[k];
}

// Device-order velocity -> the caller-order coupling arrays Ux, Uy, dUx/dkappa, dUy/dkappa (x fastest).
__global__ void export_U_kernel(int64_t P, int Nk, const double* __restrict__ U, double* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t c3 = P * Nk;
    if (t >= c3) return;
    const int64_t c = t / Nk, m = t - c * Nk;
    const int64_t x = c + P * m;
#pragma unroll
    for (int a = 0; a < 4; ++a) out[a * c3 + x] = U[a * c3 + t];
}

// Whether the caller's rows of P cells start on 16-byte boundaries.
bool aligned_rows(const void* p, int64_t P) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && P % 4 == 0; }

template <typename S, typename D>
cudaError_t to_dev(const void* src, void* dst, const Handle& h, int64_t n0, int64_t nc, int64_t m0, int64_t mc,
                   cudaStream_t s) {
    const int64_t P = h.cells, Nk = h.desc.Nk;
    const dim3 grid((unsigned)((P + CT - 1) / CT), (unsigned)((mc + MT - 1) / MT), (unsigned)nc);
    auto k = aligned_rows(src, P) ? to_device_kernel<S, D, true> : to_device_kernel<S, D, false>;
    k<<<grid, LTHREADS, 0, s>>>((const S*)src, (D*)dst, P, Nk, n0, m0, mc, Nk * P, h.d_err);
    return cudaGetLastError();
}

template <typename S, typename D>
cudaError_t from_dev(const void* src, void* dst, const Handle& h, int64_t n0, int64_t nc, int64_t m0, int64_t mc,
                     cudaStream_t s) {
    const int64_t P = h.cells, Nk = h.desc.Nk;
    const dim3 grid((unsigned)((P + CT - 1) / CT), (unsigned)((mc + MT - 1) / MT), (unsigned)nc);
    auto k = aligned_rows(dst, P) ? from_device_kernel<S, D, true> : from_device_kernel<S, D, false>;
    k<<<grid, LTHREADS, 0, s>>>((const S*)src, (D*)dst, P, Nk, n0, m0, mc, Nk * P);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_to_device_layout(const Handle& h, const void* src, int src_dtype, void* dst, int dst_dtype,
                                    int64_t n0, int64_t nc, int64_t m0, int64_t mc, cudaStream_t s) {
    if (src_dtype == RPL_F64 && dst_dtype == RPL_F64) return to_dev<double, double>(src, dst, h, n0, nc, m0, mc, s);
    if (src_dtype == RPL_F64 && dst_dtype == RPL_F32) return to_dev<double, float>(src, dst, h, n0, nc, m0, mc, s);
    if (src_dtype == RPL_F32 && dst_dtype == RPL_F64) return to_dev<float, double>(src, dst, h, n0, nc, m0, mc, s);
    return to_dev<float, float>(src, dst, h, n0, nc, m0, mc, s);
}

cudaError_t launch_from_device_layout(const Handle& h, const void* src, int src_dtype, void* dst, int dst_dtype,
                                      int64_t n0, int64_t nc, int64_t m0, int64_t mc, cudaStream_t s) {
    if (src_dtype == RPL_F64 && dst_dtype == RPL_F64) return from_dev<double, double>(src, dst, h, n0, nc, m0, mc, s);
    if (src_dtype == RPL_F64 && dst_dtype == RPL_F32) return from_dev<double, float>(src, dst, h, n0, nc, m0, mc, s);
    if (src_dtype == RPL_F32 && dst_dtype == RPL_F64) return from_dev<float, double>(src, dst, h, n0, nc, m0, mc, s);
    return from_dev<float, float>(src, dst, h, n0, nc, m0, mc, s);
}

cudaError_t launch_coef(const Handle& h, cudaStream_t s) {
    const rpl_desc& d = h.desc;
    const int64_t c3 = d.Nx * d.Ny * d.Nk;
    coef_kernel<<<(unsigned)((c3 + 255) / 256), 256, 0, s>>>(d.Nx, d.Ny, d.Nk, h.currents_set ? h.d_coupling : nullptr,
                                                             h.d_cgmag, h.d_kappa, h.d_coef);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? launch_vel(h, s) : e;
}

cudaError_t launch_coef_from_U(const Handle& h, cudaStream_t s) {
    const rpl_desc& d = h.desc;
    const int64_t c3 = d.Nx * d.Ny * d.Nk;
    coef_from_U_kernel<<<(unsigned)((c3 + COEF_THREADS - 1) / COEF_THREADS), COEF_THREADS, 0, s>>>(
        d.Nx, d.Ny, (int)d.Nk, h.d_U, 1.0 / d.dx, 1.0 / d.dy, h.d_coef);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? launch_vel(h, s) : e;
}

cudaError_t launch_export_U(const Handle& h, cudaStream_t s) {
    const int64_t c3 = h.cells * h.desc.Nk;
    export_U_kernel<<<(unsigned)((c3 + 255) / 256), 256, 0, s>>>(h.cells, (int)h.desc.Nk, h.d_U, h.d_coupling);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_gradients(h, s);
}

}  // namespace rpl
