"""The dense solve at the edges of its 16 x 16 tiles.

Sizes around one, two and three tiles, where the panel has no sub-diagonal
tile, one, or the first tasks of the other CTAs (and the largest):
* the residual: a Cholesky solve's backward error is within (n + 1) eps of
  sqrt(a_ii a_jj) per entry, and the products with the tiles' explicit inverses
  multiply it by the tile factor's condition, sqrt(1e2) at most here; the
  bound is 4 times that;
* powers of two on rows and columns (up to 2^+-400 each, and 2^+-480 on all)
  change no bit of the scaled result: the factor scales each tile's diagonal to
  one by powers of two;
* a negative, NaN or infinite pivot is refused at every position.
"""
import numpy as np
import pytest

import psba_gb300 as P

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 160]


@pytest.fixture(scope="module", autouse=True)
def built():
    P.build()


def system(n, seed):
    rng = np.random.default_rng(seed)
    Q, _ = np.linalg.qr(rng.normal(size=(n, n)))
    A = (Q * np.geomspace(1.0, 1e2, n)) @ Q.T
    return np.tril(A) + np.tril(A, -1).T, rng.normal(size=n)


@pytest.mark.parametrize("n", SIZES)
def test_residual(n):
    A, b = system(n, n)
    st, x = P.dense_solve(np.tril(A), b)
    assert st == 0
    d = np.sqrt(np.diag(A))
    bound = 4 * 10 * (n + 1) * np.finfo(float).eps * d * (d @ np.abs(x))
    assert np.all(np.abs(A @ x - b) <= bound)


@pytest.mark.parametrize("n", [2528, 2561, 4096])  # the back solve's shared memory below and above 40 KB, the largest
def test_residual_large(n):
    rng = np.random.default_rng(n)
    B = rng.normal(size=(n, 64))
    A, b = B @ B.T / 64 + 3 * np.eye(n), rng.normal(size=n)  # condition below 100
    st, x = P.dense_solve(np.tril(A), b)
    assert st == 0
    d = np.sqrt(np.diag(A))
    bound = 4 * 10 * (n + 1) * np.finfo(float).eps * d * (d @ np.abs(x))
    assert np.all(np.abs(A @ x - b) <= bound)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("spread, shift", [(400, 0), (0, 480), (0, -480), (7, 3)])
def test_powers_of_two_change_nothing(n, spread, shift):
    A, b = system(n, n)
    e = np.random.default_rng(n + 1).integers(-spread, spread + 1, n) + shift
    st0, x0 = P.dense_solve(np.tril(A), b)
    st1, x1 = P.dense_solve(np.tril(np.ldexp(A, e[:, None] + e)), np.ldexp(b, e))
    assert st0 == st1 == 0
    assert np.array_equal(np.ldexp(x1, e), x0)


@pytest.mark.parametrize("bad", [-1.0, 0.0, np.nan, np.inf])
def test_bad_pivots_are_refused_at_every_position(bad):
    A, b = system(40, 40)
    for j in range(40):
        B = A.copy()
        B[j, j] = bad
        assert P.dense_solve(np.tril(B), b)[0] == 1, j
