"""The modified Cholesky above the sizes whose rows stay in shared memory: rows left
in S (n above ~1,700), and the panel in global memory too (n above 9,300)."""
import numpy as np
import pytest

import oracle
import psba_gb300 as P

pytestmark = pytest.mark.gpu


def _matrix(n, rank, shift, seed):
    G = np.random.default_rng(seed).normal(size=(n, rank)) / np.sqrt(rank)
    A = G @ G.T
    A[np.diag_indices(n)] += shift
    return np.tril(A)


@pytest.mark.parametrize("shift", [0.5, -0.05])
def test_rows_left_in_the_matrix(shift):
    # the tolerance of the smaller sizes' test, against the oracle
    n = 1800
    A = _matrix(n, 24, shift, 1)
    Lo, Eo = oracle.cholmod(A)
    Lg, Eg = P.cholmod(A)
    scale = np.abs(Lo).max()
    tol = 50 * n * 2.0 ** -53 * max(1.0, scale ** 2 / np.abs(A).max())
    assert np.abs(np.tril(Lg) - np.tril(Lo)).max() <= tol * scale
    assert np.abs(Eg - Eo).max() <= tol * max(1.0, np.abs(Eo).max(), scale ** 2)
    assert not np.triu(Lg, 1).any()


def test_panel_in_global_memory():
    # positive definite: no entry is above beta and no pivot is changed, so L is the
    # Cholesky factor, whose rows are off by (n + 1) u sqrt(A_ii) sqrt(cond) at most
    n = 9303
    A = _matrix(n, 24, 4.0, 2)
    L = np.linalg.cholesky(A + np.tril(A, -1).T)
    Lg, Eg = P.cholmod(A)
    tol = n * 2.0 ** -53 * np.sqrt(np.abs(A).max()) * 11.0  # cond(A) is 107
    worst = max(np.abs(np.tril(Lg[r:r + 500] - L[r:r + 500], r)).max() for r in range(0, n, 500))
    assert worst <= tol
    assert np.abs(Eg).max() <= n * 2.0 ** -53 * np.abs(A).max()
    assert not np.triu(Lg[:600, :600], 1).any() and not Lg[0, 1:].any()
