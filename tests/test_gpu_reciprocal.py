"""rcp_series (csrc/lj_impl.cuh), the reciprocal of the FP64 pair kernels,
compiled into a kernel of its own and compared with CUDA's correctly rounded
1.0 / x."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "lj_impl.cuh"
using namespace mrmd_impl;
__global__ void k(const double* x, int n, double* series, double* exact, double* residual)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x[i]));
    series[i] = rcp_series(x[i]);
    exact[i] = 1.0 / x[i];
    residual[i] = __fma_rn(-x[i], y, 1.0);
}
extern "C" int reciprocals(const double* x, int n, double* out)
{
    double* d = nullptr;
    const size_t bytes = sizeof(double) * n;
    if (cudaMalloc(&d, 4 * bytes) != cudaSuccess) return 1;
    cudaMemcpy(d, x, bytes, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d, n, d + n, d + 2 * n, d + 3 * n);
    const cudaError_t e = cudaMemcpy(out, d + n, 3 * bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e != cudaSuccess;
}
"""


def test_rcp_series_is_within_an_ulp(tmp_path):
    """The seed takes and gives 20 fraction bits: truncating the operand costs
    below 2^-20, rounding the result at most 2^-20, so |e| < 2^-19 and the
    series' rest e^3 < 2^-57, an eighth of an ulp at most; with the last
    rounding the result is the correctly rounded one or its neighbour."""
    from mrmd_gb300 import build as B

    src, lib = tmp_path / "rcp.cu", tmp_path / "rcp.so"
    src.write_text(SOURCE)
    subprocess.run([B.nvcc()] + B.NVCC_FLAGS + ["-shared", str(src), "-o", str(lib)], check=True)
    f = ctypes.CDLL(str(lib)).reciprocals
    rng = np.random.default_rng(1)
    # mantissas at the operand's 20-bit steps and around them, and random ones
    m = np.concatenate([1.0 + rng.integers(0, 1 << 52, 1 << 20) * 2.0 ** -52,
                        1.0 + np.arange(1 << 20) * 2.0 ** -20, 1.0 + np.arange(1, 1 << 20) * 2.0 ** -20 - 2.0 ** -52,
                        [1.0 + 2.0 ** -20 - 2.0 ** -52, 2.0 - 2.0 ** -52, 1.0, 1.0 + 2.0 ** -52]])
    x = np.concatenate([m, np.ldexp(m[-300000:], rng.integers(-340, 1000, 300000)),
                        np.ldexp([1.0, 2.0 - 2.0 ** -52], [-340, 999])])
    out = np.empty((3, len(x)))
    p = lambda v: v.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    assert f(p(x), len(x), p(out)) == 0
    series, exact, e = out
    assert np.abs(e).max() < 2.0 ** -19
    ulps = np.abs(series.view(np.int64) - exact.view(np.int64))
    print("largest residual 2^%.2f, %.2f%% of the results a neighbour" % (np.log2(np.abs(e).max()), 100 * np.mean(ulps > 0)))
    assert ulps.max() <= 1
