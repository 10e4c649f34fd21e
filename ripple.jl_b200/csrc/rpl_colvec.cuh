// rpl_colvec.cuh -- the per-column reductions over the spectrum (diagnostics, SourceTermSet integrals,
// pseudomomentum moments): a lane holds one 16-byte vector of adjacent kappa bins of a column (four FP32 or two
// FP64 bins), L = ceil(Nk / bins per lane) lanes make a column and a warp takes floor(32 / L) consecutive
// columns, so one load per lane covers a direction of all of them and a bin table entry read from shared memory
// serves the warp's columns at once. Several directions' loads are issued together. The tables must not come
// through L1: it returns a warp's loads in order, so a table entry read behind the streaming loads waits for
// DRAM with them. More than 32 lanes' worth of bins are walked in chunks.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "rpl_vec.cuh"

namespace rpl {

template <typename T>
struct ColVec {
    static constexpr int N = w32::LaneVec<T>::N;
    int lane, l, L, cpw;
    bool used;
    __device__ __forceinline__ explicit ColVec(int Nk) {
        lane = threadIdx.x & 31;
        L = min((Nk + N - 1) / N, 32);
        cpw = 32 / L;
        used = lane / L < cpw;
        l = lane % L;
    }
    __device__ __forceinline__ int col() const { return min(lane / L, cpw - 1); }
};

// Values of a lane vector as T[N]; elements past the column's last repeat it (their table entries are zero).
template <bool AL> __device__ __forceinline__ void ld_bins(const float* p, int left, float (&v)[4]) {
    if constexpr (AL) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = __ldg(p + min(q, left));
    }
}
template <bool AL> __device__ __forceinline__ void ld_bins(const double* p, int left, double (&v)[2]) {
    if constexpr (AL) {
        const double2 f = __ldg(reinterpret_cast<const double2*>(p));
        v[0] = f.x; v[1] = f.y;
    } else {
        v[0] = __ldg(p);
        v[1] = __ldg(p + min(1, left));
    }
}

// Bins per direction of a staged table: whole lane vectors (and whole chunks of 32 lanes), zero past Nk.
template <typename T> __host__ __device__ inline int table_stride(int Nk) {
    const int N = w32::LaneVec<T>::N, L = (Nk + N - 1) / N;
    return (L <= 32 ? L : (L + 31) / 32 * 32) * N;
}
template <typename A> __device__ __forceinline__ void stage_table(A* dst, const A* src, int Nk, int Np, int stride) {
    for (int e = threadIdx.x; e < stride * Np; e += blockDim.x) {
        const int n = e / stride, m = e - n * stride;
        dst[e] = m < Nk ? src[m + Nk * n] : A(0);
    }
}

// Most bytes of tables a CTA stages; a model with more takes the kernels' global-memory tables. Every launch allows its
// kernel this much dynamic shared memory, whatever the model needs of it: the attribute belongs to the kernel, not to
// the launch, and handles launch from several threads.
constexpr size_t kTableBytes = 200 * 1024;

}  // namespace rpl
