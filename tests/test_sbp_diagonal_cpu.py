"""The identity behind the kernels' zero derivative diagonals (KParams::DhatC,
DC): on Legendre-Gauss-Lobatto points the diagonal of the weak-form
derivative Dhat[i][n] = D[n][i] w_n / w_i and of the strong-form D is zero at
interior nodes and -+1/(2 w_0) at the ends, and there it cancels the interior
half of a central face term with lift 1/w_0.  Bound: a few roundings of the
largest entry, N (N + 1) / 4."""
import numpy as np
import pytest

pytest.importorskip("torch")


def _matrices(N):
    from cmdg.workloads import lgl

    x, w = lgl(N)
    n = N + 1
    bary = np.array([1 / np.prod([x[j] - x[i] for i in range(n) if i != j]) for j in range(n)])
    D = np.zeros((n, n))
    for j in range(n):
        for k in range(n):
            D[j, k] = (bary[k] / bary[j]) / (x[j] - x[k]) if j != k else sum(1 / (x[k] - x[m]) for m in range(n) if m != k)
    return D, D.T * w[None, :] / w[:, None], w


@pytest.mark.parametrize("N", [2, 3, 4, 5])
def test_zero_diagonal_with_far_half_equals_full_form(N):
    D, Dhat, w = _matrices(N)
    tol = 64 * np.finfo(float).eps * N * (N + 1)
    ends = np.zeros(N + 1)
    ends[0], ends[N] = -0.5 / w[0], 0.5 / w[0]
    assert np.abs(np.diag(D) - ends).max() <= tol
    assert np.abs(np.diag(Dhat) - ends).max() <= tol
    rng = np.random.default_rng(N)
    F, G = rng.normal(size=(2, N + 1))
    far = rng.normal(size=2)  # values across the two faces

    def off(A):
        return A - np.diag(np.diag(A))

    # weak form: Dhat F - lift F*.n with F* = (F- + F+) / 2
    full = Dhat @ F
    full[0] += 0.5 / w[0] * (F[0] + far[0])
    full[N] -= 0.5 / w[0] * (F[N] + far[1])
    half = off(Dhat) @ F
    half[0] += 0.5 / w[0] * far[0]
    half[N] -= 0.5 / w[0] * far[1]
    assert np.abs(full - half).max() <= tol * 4
    # strong form: D G + lift n (G* - G-), G* = (G- + G+) / 2 inside, G+ on walls
    for c in (0.5, 1.0):
        full = D @ G
        full[0] -= c / w[0] * (far[0] - G[0])
        full[N] += c / w[0] * (far[1] - G[N])
        half = off(D) @ G
        half[0] -= (c * far[0] - (c - 0.5) * G[0]) / w[0]
        half[N] += (c * far[1] - (c - 0.5) * G[N]) / w[0]
        assert np.abs(full - half).max() <= tol * 4
