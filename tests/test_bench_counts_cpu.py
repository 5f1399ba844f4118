"""The counts behind bench.py's lines: the entries of the column LU that a
substitution reads, against a factorization of a matrix with the vertical
operator's coupling, and the launches of an ensemble's stage."""
import numpy as np
import pytest

import bench


@pytest.mark.parametrize("N", [2, 3, 4, 5])
def test_factor_entries_are_the_nonzeros_of_an_interior_level(N):
    nb, nz = 5 * (N + 1), 5
    n = nb * nz
    rng = np.random.default_rng(N)
    A = np.zeros((n, n))
    for v in range(nz):
        b = slice(v * nb, (v + 1) * nb)
        A[b, b] = rng.normal(size=(nb, nb)) + 4 * nb * np.eye(nb)
        if v + 1 < nz:  # the facing layers: the top 5 unknowns of v, the bottom 5 of v + 1
            top, bottom = slice((v + 1) * nb - 5, (v + 1) * nb), slice((v + 1) * nb, (v + 1) * nb + 5)
            A[bottom, top], A[top, bottom] = rng.normal(size=(2, 5, 5))
    LU = A.copy()
    for k in range(n):
        LU[k + 1:, k] /= LU[k, k]
        LU[k + 1:, k + 1:] -= np.outer(LU[k + 1:, k], LU[k, k + 1:])
    nonzero = LU != 0
    # columns of an interior level: below the diagonal, and on and above it
    cols = range(2 * nb, 3 * nb)
    assert sum(int(nonzero[:, c].sum()) for c in cols) == bench.hevi_factor_entries(N)


def test_ensemble_launches():
    assert bench.ensemble_launches([(4, 64000)] * 3) == 3
    assert bench.ensemble_launches([(4, 63999)]) == 1
    per_set = (24 << 20) // (100 * 50000)  # 5 members of 50,000 nodes
    assert bench.ensemble_launches([(3, 50000)] * per_set) == 1
    assert bench.ensemble_launches([(3, 50000)] * (per_set + 1)) == 2
    assert bench.ensemble_launches([(3, 1000), (4, 1000), (3, 2000), (5, 70000)]) == 3
