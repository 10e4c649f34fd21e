"""rcpd (csrc/rpl_vec.cuh), the FP64 reciprocal under every WENO5 face of the two-pass stage, against CUDA's division.

Bound: the truncated term e^3 is below 2^-58 and e itself is rounded below 2^-72, so the value before its last rounding is
within 0.02 units in the last place of 1/x; that rounding and the quotient's own add half a unit each.
"""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "rpl_vec.cuh"
__global__ void compare(int exponent, unsigned long long seed, unsigned long long* worst) {
    unsigned long long s = seed + 0x9e3779b97f4a7c15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
    unsigned long long most = 0;
    for (int k = 0; k < 64; ++k) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        unsigned long long m = s >> 12;
        if (k == 0) m = 0;
        if (k == 1) m = (1ull << 52) - 1;
        const double x = __longlong_as_double(((long long)(exponent + 1023) << 52) | (long long)m);
        const long long a = __double_as_longlong(rpl::w32::rcpd(x)), b = __double_as_longlong(1.0 / x);
        most = max(most, (unsigned long long)(a > b ? a - b : b - a));
    }
    atomicMax(worst, most);
}
extern "C" int run(int exponent, unsigned long long seed, unsigned long long* out) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return 1;
    compare<<<32, 128>>>(exponent, seed, d);
    const cudaError_t e = cudaMemcpy(out, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 1;
}
"""


def test_reciprocal_within_one_unit_in_the_last_place(tmp_path):
    import build
    src, lib = tmp_path / "rcp.cu", tmp_path / "rcp.so"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, *build.FLAGS, "-I", build.CSRC, "-shared", "-o", str(lib), str(src)],
                   check=True, cwd=os.path.dirname(build.CSRC))
    run, worst = ctypes.CDLL(str(lib)).run, ctypes.c_ulonglong()
    run.argtypes = [ctypes.c_int, ctypes.c_ulonglong, ctypes.POINTER(ctypes.c_ulonglong)]
    for exponent in range(-160, 851):   # the denominators' range: (4 eps)^4 ~ 2^-147 to 2^850
        assert run(exponent, 7919 * (exponent + 200), ctypes.byref(worst)) == 0
        assert worst.value <= 1, exponent
