"""The FP64 device arithmetic of dg_common.cuh beside IEEE division and square
root.

Error: the seeds carry e <= 2^-19 (reciprocal) and 2^-19.4 (reciprocal root);
one third-order step leaves e^3 <= 2^-57, two simplified Newton steps
3/2 e^3 <= 2^-57.6, i.e. at most 2^-4 of an ulp beside the last rounding's
half: 0.57 ulp (1 ulp for a root whose residual underflows).  Zeros,
infinities, NaN and negative radicands: the IEEE results, bit for bit;
subnormals count as zeros."""
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
__global__ void k(const double* x, double* r, double* s, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = rcp_r(x[i]);
    s[i] = sqrt_r(x[i]);
}
extern "C" int run(const double* x, double* out, int n) {
    double* d = nullptr;
    const size_t b = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d, 3 * b) != cudaSuccess) return 1;
    cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, n);
    const cudaError_t e = cudaMemcpy(out, d + n, 2 * b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("device_math_edges")
    src, lib = d / "t.cu", d / "t.so"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", CSRC, "-Xcompiler", "-fPIC", "-shared", "-o", str(lib), str(src)],
                   check=True, capture_output=True)
    dll = ctypes.CDLL(str(lib))

    def call(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out = np.empty((2, x.size))
        assert dll.run(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(out.ctypes.data), x.size) == 0
        return out

    return call


def _bits(a):
    return np.where(np.isnan(a), np.uint64(0x7FF8000000000000), np.ascontiguousarray(a).view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi", [(1.0, 4.0), (1e-3, 1e13), (1e-270, 1e300)])
def test_error_in_ulp(run, lo, hi):
    x = np.exp(np.random.default_rng(11).uniform(np.log(lo), np.log(hi), 1 << 18))
    rcp, root = run(x)
    xl = x.astype(np.longdouble)
    assert np.finfo(np.longdouble).eps < 1e-18
    for got, want in ((rcp, 1 / xl), (root, np.sqrt(xl))):
        err = np.abs(got.astype(np.longdouble) - want) / np.spacing(want.astype(np.float64))
        assert float(err.max()) <= 0.57


@pytest.mark.gpu
def test_edges(run):
    tiny, big = np.finfo(float).tiny, np.finfo(float).max
    x = np.array([0.0, np.inf, np.nan, 5e-324, 5.6e-309, np.nextafter(tiny, 0), tiny, 2.0 ** -1000, 2.0 ** -927,
                  2.0 ** -200, 2.0 ** 1021, np.nextafter(2.0 ** 1022, 0), np.nextafter(2.0 ** 1022, np.inf), big])
    x = np.concatenate((x, -x))
    rcp, root = run(x)
    flushed = np.where(np.abs(x) < tiny, np.copysign(0.0, x), x)
    with np.errstate(all="ignore"):
        r, s = 1 / flushed, np.sqrt(flushed)
        s = np.where(s == 0, 0.0, s)
        # a reciprocal below the normal range: itself, or zero where the seed flushed
        below = (np.abs(r) < tiny) & (r != 0)
        r = np.where(below & (rcp == 0), np.copysign(0.0, r), r)
        for got, want in ((rcp, r), (root, s)):
            exact = ~np.isfinite(want) | (want == 0)
            assert np.array_equal(_bits(got)[exact], _bits(want)[exact])
            assert np.all(np.abs(got - want)[~exact] <= np.spacing(np.abs(want[~exact])))
