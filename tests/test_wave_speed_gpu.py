"""The larger of two wave speeds: max_nonneg of dg_common.cuh, a comparison of
bits in FP64, and the Rusanov penalty that takes it.  As fmax it leaves a NaN
for the other value: a node whose sound speed does not exist (negative internal
energy) takes the other side's."""
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
__global__ void k(const double* x, const double* y, double* m, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) m[i] = max_nonneg(x[i], y[i]);
}
extern "C" int run(const double* x, const double* y, double* out, int n) {
    double* d = nullptr;
    const size_t b = sizeof(double) * (size_t)n;
    if (cudaMalloc(&d, 3 * b) != cudaSuccess) return 1;
    cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, n);
    const cudaError_t e = cudaMemcpy(out, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
"""


def _bits(a):
    return np.where(np.isnan(a), np.uint64(0x7FF8000000000000), np.ascontiguousarray(a).view(np.uint64))


@pytest.mark.gpu
def test_larger_of_two_leaves_a_nan(tmp_path):
    src, lib = tmp_path / "t.cu", tmp_path / "t.so"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", CSRC, "-Xcompiler", "-fPIC", "-shared", "-o", str(lib), str(src)],
                   check=True, capture_output=True)
    v = [0.0, 5e-324, 1.0, 340.0, np.finfo(float).max, np.inf, np.nan, -np.nan]
    a, b = (np.ascontiguousarray(g.ravel()) for g in np.meshgrid(v, v))
    out = np.empty_like(a)
    ptr = [ctypes.c_void_p(x.ctypes.data) for x in (a, b, out)]
    assert ctypes.CDLL(str(lib)).run(*ptr, a.size) == 0
    assert np.array_equal(_bits(out), _bits(np.fmax(a, b)))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["brick", "shell", "arrays", "les"])
def test_node_without_a_sound_speed(kind):
    """An FP64 state with one node of negative internal energy: the tendency stays
    finite with a clean status word."""
    torch = pytest.importorskip("torch")
    from cmdg import workloads

    if kind == "brick":
        dg = workloads.bubble_model(ne=(3, 3, 3), N=3)
        Q = workloads.rising_bubble(dg.grid.coordinates())
    elif kind == "shell":
        dg = workloads.gcm_shell_model(nhorz=2, nvert=2, N=3)
        Q = workloads.gcm_initial_state(dg.grid.coordinates())
    elif kind == "arrays":
        dg, _perm, xyz = workloads.bubble_arrays_model(ne=(3, 3, 3), N=3)
        Q = workloads.rising_bubble(xyz)
    else:
        L = (300.0, 300.0, 300.0)
        dg = workloads.les_model(ne=(3, 3, 3), N=3, L=L)
        Q = workloads.les_initial_state(dg.grid.coordinates(), L, nmodes=2)
    node = (1 * 4 + 1) * 4  # on the xi1 face of an element, at no edge of it
    Q[1, 4, node] -= 4e5 * Q[1, 0, node]  # cv T = 2.15e5 J/kg at 300 K
    T = torch.zeros(Q.shape, dtype=torch.float64, device="cuda")
    dg(T, dg.init_ode_state(Q), None, 0.0)
    torch.cuda.synchronize()
    if kind != "les":  # theta_v of a negative pressure is NaN in the closure itself
        assert torch.isfinite(T).all() and dg.status_word() == 0
    else:
        assert torch.isfinite(T[:, 0]).all()
