"""The FP64 camera blocks at the sizes where their kernel changes.

Up to 33 units (cameras of up to 1,024 observations) go to nine CTAs each, up
to 152 to three, more to one.  U_j = sum A^T A and ga_j = sum A^T e are checked
against sums of the device's own Jacobian in extended precision; a sum of n
products is within (n + 2) eps of the sum of their magnitudes.
"""
import numpy as np
import pytest

import psba_gb300 as P
from psba_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    P.build()


@pytest.mark.parametrize("n_cams, n_pts", [(7, 40), (7, 1500), (33, 60), (34, 60), (152, 60), (153, 60)])
def test_camera_blocks(n_cams, n_pts):
    sc = scenes.arc_scene(3, n_cams=n_cams, n_pts=n_pts)
    with P.Solver(sc) as s:
        A = s.eval_jacobian()[0].reshape(-1, 2, 6).astype(np.longdouble)
        U, _, _, g = s.eval_normal(1.0)
        e = s.eval_residual()[0].reshape(-1, 2).astype(np.longdouble)
    cam = np.asarray(sc.obs_cam)
    eps = np.finfo(float).eps
    for j in range(n_cams):
        a, r = A[cam == j], e[cam == j]
        n = 2 * len(a) + 2
        assert np.all(np.abs(U[j] - np.einsum("oki,okj->ij", a, a)) <= n * eps * np.einsum("oki,okj->ij", abs(a), abs(a)))
        gj = g[6 * j:6 * j + 6]
        assert np.all(np.abs(gj - np.einsum("oki,ok->i", a, r)) <= n * eps * np.einsum("oki,ok->i", abs(a), abs(r)))
