"""The batched engine's in-CTA dense solve at every panel width (16, 8 and 4 columns
in shared memory, 16 in global memory): one iteration against the single-problem
solver's, on arcs of as many cameras as each begins or ends with, one of them
without observations.

Tolerance: both are FP64 solves of the same damped system, whose step is off by
cond(S) 2^-53 in either; the first damping factor (1e-3 of the largest diagonal
entry) keeps cond(S) below 1e6 here, so steps agree to 1e-9 of the largest; the
cost falls by about half in the step, so it agrees to 1e-8.  The mixed form
holds its products to 24 bits: 1e-3 of the step and 1e-4 of the cost.
"""
import numpy as np
import pytest

import psba_gb300 as P
from psba_gb300 import scenes
from psba_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _scene(n_cams):
    sc = scenes.arc_scene(seed=n_cams, n_cams=n_cams, n_pts=6 * n_cams, arc_deg=160.0, k_range=(3, 5))
    keep = np.asarray(sc.obs_cam) != n_cams // 2
    sc.meas, sc.obs_pt, sc.obs_cam = sc.meas[keep], sc.obs_pt[keep], sc.obs_cam[keep]
    return sc


@pytest.mark.parametrize("n_cams,precision,tol,tol_cost", [
    (64, P.PREC_FP64, 1e-9, 1e-8), (65, P.PREC_FP64, 1e-9, 1e-8), (129, P.PREC_FP64, 1e-9, 1e-8),
    (256, P.PREC_FP64, 1e-9, 1e-8), (257, P.PREC_FP64, 1e-9, 1e-8), (513, P.PREC_FP64, 1e-9, 1e-8),
    (65, P.PREC_MIXED, 1e-3, 1e-4), (257, P.PREC_MIXED, 1e-3, 1e-4)])
def test_one_iteration_is_the_single_solvers(n_cams, precision, tol, tol_cost):
    sc = _scene(n_cams)
    kw = dict(allow_switch=0, max_iter=1)
    with P.Solver(sc) as s:
        r = s.levmar(**kw)
    with Batch([sc, scenes.arc_scene(seed=1, n_cams=5, n_pts=40)]) as b:
        res, _ = b.levmar(precision=precision, **kw)
        cams, pts = b.get_params(0)
    assert res["iterations"][0] == r.iterations and res["n_trials"][0] == r.n_trials
    assert abs(res["final_cost"][0] - r.final_cost) <= tol_cost * r.final_cost
    for got, ref, at in ((cams, r.cams, sc.cams), (pts, r.pts, sc.pts)):
        step = np.abs(np.asarray(ref) - np.asarray(at)).max()
        assert step > 0
        assert np.abs(np.asarray(got).reshape(np.shape(ref)) - ref).max() <= tol * step
