"""The modified Cholesky at the sizes where its launch changes shape (one CTA,
fewer rows than threads, more rows than one pass of a CTA's threads, several
rows a CTA), with every path of a block step: plain, redone for a pivot,
redone for an entry above beta.  Against the oracle, which rounds the same
operations in another order: the factor's backward error grows with n."""
import numpy as np
import pytest

import oracle
import psba_gb300 as P

pytestmark = pytest.mark.gpu


def _matrix(n, seed, indefinite):
    rng = np.random.default_rng(seed)
    Q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    w = np.linspace(0.5, 4.0, n)
    if indefinite:
        w[: max(1, n // 10)] = -1.0
    return (Q * w) @ Q.T


@pytest.mark.parametrize("indefinite", [False, True])
@pytest.mark.parametrize("n", [3, 6, 24, 27, 255, 258, 261, 771])
def test_cholmod_sizes(n, indefinite):
    A = np.tril(_matrix(n, n, indefinite))
    Lo, Eo = oracle.cholmod(A)
    Lg, Eg = P.cholmod(A)
    scale = np.abs(Lo).max()
    # an indefinite matrix's redone columns amplify earlier roundings by up to |L|^2 / |A|
    tol = 50 * n * 2.0 ** -53 * max(1.0, scale ** 2 / np.abs(A).max())
    assert np.abs(np.tril(Lg) - np.tril(Lo)).max() <= tol * scale
    assert np.abs(Eg - Eo).max() <= tol * max(1.0, np.abs(Eo).max(), scale ** 2)
    assert not np.triu(Lg, 1).any()
