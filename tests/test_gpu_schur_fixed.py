"""The FP64 Schur complement's products run in block fixed point
(psba_schurfx.cu): S and ea of psba_eval_reduced against extended-precision
sums of the same W and V^-1, at the sizes where the kernels' chunks of 32
entries end, with spread-out magnitudes and with a NaN.

Tolerance, from the method: Y is formed in FP64 (3 roundings of its terms);
a limb row is cut 2^-56 below its observation's largest value (after the row
weights), a W row once more to the largest product of its 32 entries, and the
low limbs' product is left out: less than 2^-53 of the largest product of the
block per product; the chunks' sums are added in FP64.
"""
import numpy as np
import pytest

import psba_gb300 as P
from psba_gb300 import scenes

pytestmark = pytest.mark.gpu
X = np.longdouble


def _reduced(sc, mu):
    with P.Solver(sc) as s:
        U, _, W, g = s.eval_normal(1.0)
        Vinv, Y, S, ea = s.eval_reduced(mu)
    return U, W, g, Vinv, Y, S, ea


def _check(sc, mu=1e2, skip=()):
    nc, cnp, N = sc.n_cams, sc.cnp, sc.n_cams * sc.cnp
    U, W, g, Vinv, Y, S, ea = _reduced(sc, mu)
    W, Vi = W.astype(X), Vinv.astype(X)
    gb = g[N:].reshape(-1, 3).astype(X)
    opt, oc = np.asarray(sc.obs_pt), np.asarray(sc.obs_cam)
    Yx = np.einsum("ork,okj->orj", W, Vi[opt])
    Ya = np.einsum("ork,okj->orj", np.abs(W), np.abs(Vi[opt]))
    # weights: within a factor 2 of sqrt(U_rr)
    s = np.sqrt(np.maximum(np.einsum("krr->kr", U), 1e-300))
    my = (np.abs(Yx).max(2) / s[oc]).max(1)
    mw = (np.abs(W).max(2) / s[oc]).max(1)
    by_cam = [dict(zip(opt[oc == k].tolist(), np.nonzero(oc == k)[0].tolist())) for k in range(nc)]
    eps = X(2.0) ** -53
    for k in range(nc):
        for l in range(k + 1):
            common = [i for i in by_cam[k] if i in by_cam[l]]
            if (k, l) in skip:
                continue
            a = np.array([by_cam[k][i] for i in common], dtype=int)
            b = np.array([by_cam[l][i] for i in common], dtype=int)
            ref = -np.einsum("trj,tcj->rc", Yx[a], W[b]) if len(a) else np.zeros((cnp, cnp), X)
            bound = np.zeros((cnp, cnp), X)
            if len(a):
                bound = 4 * eps * np.einsum("trj,tcj->rc", Ya[a], np.abs(W[b]))  # Y's roundings
                # 3 n products, the factor 8 for weights and exponents within a factor 2 each
                bound += 3 * len(a) * 8 * eps * np.outer(s[k], s[l]) * (my[a] * mw[b]).max()
            if k == l:
                ref = ref + U[k] + mu * np.eye(cnp)
                bound = bound + 4 * eps * (np.abs(U[k]) + mu)
            bound = bound + 2 * eps * (np.ceil(len(a) / 32) + 2) * np.abs(ref)  # FP64 sums of the chunks and units
            got = S[cnp * k:cnp * k + cnp, cnp * l:cnp * l + cnp]
            d = np.abs(got - ref)
            if k == l:
                d, bound = np.tril(d), bound
            assert (d <= bound).all(), (k, l, len(a), float((d / np.maximum(bound, X(1e-300))).max()))
        a = np.nonzero(oc == k)[0]
        if (k, k) in skip:
            continue
        ref = g[cnp * k:cnp * k + cnp] - np.einsum("trj,tj->r", Yx[a], gb[opt[a]])
        bound = 4 * eps * np.einsum("trj,tj->r", Ya[a], np.abs(gb[opt[a]]))
        if len(a):
            bound = bound + 3 * len(a) * 8 * eps * s[k] * (my[a] * np.abs(gb[opt[a]]).max(1)).max()
        bound = bound + 2 * eps * (np.ceil(len(a) / 32) + 2) * (np.abs(ref) + np.abs(g[cnp * k:cnp * k + cnp]))
        d = np.abs(ea[cnp * k:cnp * k + cnp] - ref)
        assert (d <= bound).all(), ("ea", k, float((d / bound).max()))


@pytest.mark.parametrize("cnp", [6, 11, 16])
@pytest.mark.parametrize("n_pts", [1, 31, 32, 33, 65, 130])
def test_blocks_at_chunk_edges(cnp, n_pts):
    sc = scenes.arc_scene(seed=n_pts, n_cams=4, n_pts=n_pts, arc_deg=10.0, min_views=3)
    _check(sc if cnp == 6 else scenes.with_intrinsics(sc, cnp, seed=1))


@pytest.mark.parametrize("cnp", [6, 11, 16])
def test_blocks_with_units_of_several_chunks(cnp):
    # a camera pair of ~1,500 common points: units of more than one chunk, several units a pair
    sc = scenes.arc_scene(seed=3, n_cams=3, n_pts=1500, arc_deg=5.0, min_views=3)
    _check(sc if cnp == 6 else scenes.with_intrinsics(sc, cnp, seed=2), mu=1.0)


@pytest.mark.parametrize("cnp", [6, 16])
def test_spread_magnitudes(cnp):
    # points from 0.02 to 2,000 units deep: W rows over ten decades, and cost-scale differences by covariance
    sc = scenes.arc_scene(seed=7, n_cams=5, n_pts=120, arc_deg=8.0, min_views=3)
    if cnp > 6:
        sc = scenes.with_intrinsics(sc, cnp, seed=3)
    sc.pts *= np.exp(np.random.default_rng(0).uniform(np.log(0.2), np.log(400.0), size=(sc.n_pts, 1)))
    _check(scenes.with_covariance(sc, seed=1, sigma=(1e-3, 1e2)), mu=1e-3)


@pytest.mark.parametrize("cnp", [6, 11])
def test_nan_stays_where_it_is(cnp):
    # one point's coordinates are NaN: the blocks of the cameras that see it are NaN, the others are not
    sc = scenes.arc_scene(seed=11, n_cams=6, n_pts=90, arc_deg=30.0, k_range=(3, 4))
    if cnp > 6:
        sc = scenes.with_intrinsics(sc, cnp, seed=4)
    sc.pts[17] = np.nan
    see = set(np.asarray(sc.obs_cam)[np.asarray(sc.obs_pt) == 17].tolist())
    assert len(see) < sc.n_cams
    S = _reduced(sc, 1.0)[5]
    skip = {(k, l) for k in see for l in see}
    for k, l in skip:
        if l < k:
            assert np.isnan(S[cnp * k:cnp * k + cnp, cnp * l:cnp * l + cnp]).all()
    for k in range(sc.n_cams):
        for l in range(k):
            if not (k in see and l in see):
                assert np.isfinite(S[cnp * k:cnp * k + cnp, cnp * l:cnp * l + cnp]).all()
