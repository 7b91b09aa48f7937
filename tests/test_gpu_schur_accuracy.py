"""The FP64 form's fixed-point sums (psba_schurfx.cu) against 80-bit sums of the
same factors, entry by entry, in units of what an FP64 sum is held to: 2^-53 of
the sum of the products' magnitudes.  Scenes whose factors lie many binary
orders apart within a block: an FP64 sum keeps each factor's 53 bits there, and
so must these.

Tolerance, from the method (u = 2^-53, m = the sum of magnitudes): Y's three
products are formed in FP64 (4 u m); a chunk's sum is rounded once and added
once, as are the units' sums and the last term (2 u m per chunk and four more);
a factor is cut 2^-73 of its block's unit below, and the block's largest value is
at least half a unit, on either side, with weights within a factor of 2 each (the
FP32 sum of the small terms is nearer): 2^-69 of the largest product, per
product; 2^-68 is allowed.
"""
import numpy as np
import pytest

import psba_gb300 as P
from psba_gb300 import scenes

pytestmark = pytest.mark.gpu
X = np.longdouble
u, cut = X(2.0) ** -53, X(2.0) ** -68


def _scene(cnp, n_pts, depths, sigma, seed):
    sc = scenes.arc_scene(seed=seed, n_cams=5, n_pts=n_pts, arc_deg=8.0, min_views=3)
    if cnp > 6:
        sc = scenes.with_intrinsics(sc, cnp, seed=3)
    if depths:
        sc.pts *= np.exp(np.random.default_rng(seed).uniform(np.log(depths[0]), np.log(depths[1]), size=(sc.n_pts, 1)))
    return scenes.with_covariance(sc, seed=1, sigma=sigma) if sigma else sc


SCENES = [(40, None, None, 1), (300, (0.2, 400.0), None, 7), (300, (0.2, 400.0), (1e-3, 1e2), 7),
          (120, (0.5, 50.0), (1e-6, 1e6), 8)]


@pytest.mark.parametrize("cnp", [6, 11, 16])
@pytest.mark.parametrize("n_pts,depths,sigma,seed", SCENES)
def test_reduced_system(cnp, n_pts, depths, sigma, seed):
    sc, mu = _scene(cnp, n_pts, depths, sigma, seed), 1e-3
    nc, N = sc.n_cams, sc.n_cams * cnp
    with P.Solver(sc) as s:
        U, _, W, g = s.eval_normal(1.0)
        Vinv, _, S, ea = s.eval_reduced(mu)
    W, Vi, gb = W.astype(X), Vinv.astype(X), g[N:].reshape(-1, 3).astype(X)
    opt, oc = np.asarray(sc.obs_pt), np.asarray(sc.obs_cam)
    Y = np.einsum("ork,okj->orj", W, Vi[opt])
    Ya = np.einsum("ork,okj->orj", np.abs(W), np.abs(Vi[opt]))
    d = np.sqrt(np.einsum("krr->kr", U)).astype(X)
    my, mw = (np.abs(Y).max(2) / d[oc]).max(1), (np.abs(W).max(2) / d[oc]).max(1)
    by_cam = [dict(zip(opt[oc == k].tolist(), np.nonzero(oc == k)[0].tolist())) for k in range(nc)]
    for k in range(nc):
        for l in range(k + 1):
            common = [i for i in by_cam[k] if i in by_cam[l]]
            a = np.array([by_cam[k][i] for i in common], dtype=int)
            b = np.array([by_cam[l][i] for i in common], dtype=int)
            n = len(a)
            if n == 0:
                continue
            ref = -np.einsum("trj,tcj->rc", Y[a], W[b])
            mag = np.einsum("trj,tcj->rc", Ya[a], np.abs(W[b]))
            bound = (8 + 2 * np.ceil(n / 32)) * u * mag + 3 * n * cut * np.outer(d[k], d[l]) * (my[a] * mw[b]).max()
            if k == l:
                ref = ref + U[k] + mu * np.eye(cnp)
                bound = bound + 2 * u * (np.abs(U[k]) + mu)
            err = np.abs(S[cnp * k:cnp * k + cnp, cnp * l:cnp * l + cnp] - ref)
            if k == l:
                err = np.tril(err)
            assert (err <= bound).all(), (k, l, n, float((err / bound).max()))
        a = np.nonzero(oc == k)[0]
        n = len(a)
        if n == 0:
            continue
        ga = g[cnp * k:cnp * k + cnp]
        gp = gb[opt[a]]
        ref = ga - np.einsum("trj,tj->r", Y[a], gp)
        bound = ((8 + 2 * np.ceil(n / 32)) * u * np.einsum("trj,tj->r", Ya[a], np.abs(gp)) + 2 * u * np.abs(ga) +
                 3 * n * cut * d[k] * (my[a] * np.abs(gp).max(1)).max())
        err = np.abs(ea[cnp * k:cnp * k + cnp] - ref)
        assert (err <= bound).all(), ("ea", k, float((err / bound).max()))


@pytest.mark.parametrize("cnp", [6, 11, 16])
@pytest.mark.parametrize("n_pts,depths,sigma,seed", SCENES)
def test_camera_blocks(cnp, n_pts, depths, sigma, seed):
    sc = _scene(cnp, n_pts, depths, sigma, seed)
    with P.Solver(sc) as s:
        A, _ = s.eval_jacobian()
        U = s.eval_normal(1.0)[0]
    A, oc = A.astype(X), np.asarray(sc.obs_cam)
    for k in range(sc.n_cams):
        a = np.nonzero(oc == k)[0]
        n = len(a)
        top = np.abs(A[a]).max((0, 1))
        # (the 6-parameter cameras' are FP64 sums of up to 8 observations a thread and 128 threads)
        steps = 8 + 2 * np.ceil(n / 32) + (26 if cnp == 6 else 0)
        bound = steps * u * np.einsum("tir,tic->rc", np.abs(A[a]), np.abs(A[a])) + 2 * n * cut * np.outer(top, top)
        err = np.triu(np.abs(U[k] - np.einsum("tir,tic->rc", A[a], A[a])))
        assert (err <= bound).all(), (k, n, float((err / bound).max()))
