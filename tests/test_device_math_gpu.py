"""The device arithmetic of dg_common.cuh against correctly rounded FP64.

rcp_r, sqrt_r and sqrt_rsqrt_r take a hardware seed (error e <= 2^-20) to
e^3 <= 2^-60 with one third-order step; what remains is the rounding of the
step itself: half an ulp of the last FMA, plus for the root a quarter and for
the reciprocal root a half ulp that the rounding of x y puts into h.  All
stay within 2 ulp.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "climatemachine.jl_gb300", "csrc")

SOURCE = r"""
#include "dg_common.cuh"
using namespace cmdg;
__global__ void k(const double* x, double* r, double* s, double* l, double* rl, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = rcp_r(x[i]);
    s[i] = sqrt_r(x[i]);
    sqrt_rsqrt_r(x[i], l[i], rl[i]);
}
extern "C" int run(const double* x, double* out, int n) {
    double* d = nullptr;
    const size_t b = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d, 5 * b) != cudaSuccess) return 1;
    cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n, d + 4 * (size_t)n, n);
    const cudaError_t e = cudaMemcpy(out, d + n, 4 * b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def device_math(tmp_path_factory):
    d = tmp_path_factory.mktemp("device_math")
    src, lib = d / "t.cu", d / "t.so"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", CSRC, "-Xcompiler", "-fPIC", "-shared", "-o", str(lib), str(src)],
                   check=True, capture_output=True)
    return ctypes.CDLL(str(lib))


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi", [(0.5, 2.0), (1e-3, 1e3), (1e-290, 1e290)])
def test_reciprocal_and_roots_within_two_ulp(device_math, lo, hi):
    n = 1 << 18
    x = np.exp(np.random.default_rng(7).uniform(np.log(lo), np.log(hi), n))
    out = np.empty((4, n))
    assert device_math.run(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data), n) == 0
    for got, want in zip(out, (1 / x, np.sqrt(x), np.sqrt(x), 1 / np.sqrt(x))):
        assert np.max(np.abs(got - want) / np.spacing(want)) <= 2


@pytest.mark.gpu
def test_root_of_zero_is_zero(device_math):
    x, out = np.zeros(32), np.empty((4, 32))
    assert device_math.run(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data), 32) == 0
    assert np.all(out[1] == 0)
