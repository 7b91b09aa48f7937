"""The work that users of this framework have it do, as cases that can be timed.

Every case is a pass through a public entry point: an LM solve of a problem
that is resident on the device (``Solver``), the same from host arrays and
back (create, solve, destroy), a batch of independent problems (``Batch``), a
burst of requests to a server (``Server``), the trust-region driver's modified
Cholesky (``cholmod``) and the allocation-free cost (``psba_cost_noalloc``).
Sizes are those of the benchmark's workloads and of the tests, and odd ones
between them.

Solves are cut at a few LM iterations.  LM amplifies the last bits of its sums
from step to step (with 2% outliers the 88-camera problem is chaotic past
about 20 iterations), so outputs of longer runs could not be compared.  The
trust-region driver is stood for by its own dense kernel and by the stages
that it shares with LM: its first Gauss-Newton step factors a matrix that is
singular up to rounding (the gauge), and one ulp in the points moves its
lambda by up to 80%.
"""
import ctypes
import math

import numpy as np
import torch

import psba_gb300 as P
from psba_gb300 import batch as batch_mod
from psba_gb300 import scenes
from psba_gb300 import serve as serve_mod

MIXED = {"fp64": P.PREC_FP64, "mixed": P.PREC_MIXED}


def listed():
    return [
        # the CPU-runnable problem: launches, waits and the small stages count
        {"name": "lm_arc7x500_fp64", "kind": "lm", "scene": "arc", "cams": 7, "pts": 500, "vmin": 3, "vmax": 7,
         "cnp": 6, "cov": False, "precision": "fp64", "iters": 10},
        # a problem of the middle of the serving range, in the mixed form
        {"name": "lm_arc24x3001_mixed", "kind": "lm", "scene": "arc", "cams": 24, "pts": 3001, "vmin": 4, "vmax": 6,
         "cnp": 6, "cov": False, "precision": "mixed", "iters": 8},
        # one problem from host arrays to host arrays, weighted measurements: handle and lists count
        {"name": "oneshot_arc41x7001_cov_fp64", "kind": "oneshot", "scene": "arc", "cams": 41, "pts": 7001, "vmin": 3,
         "vmax": 8, "cnp": 6, "cov": True, "precision": "fp64", "iters": 6},
        # the headline: 88 cameras x 64,298 points, power-law views, in both forms
        {"name": "lm_circle88x64298_fp64", "kind": "lm", "scene": "circle", "cams": 88, "pts": 64298, "vmin": 2,
         "vmax": 40, "cnp": 6, "cov": False, "precision": "fp64", "iters": 8},
        {"name": "lm_circle88x64298_mixed", "kind": "lm", "scene": "circle", "cams": 88, "pts": 64298, "vmin": 2,
         "vmax": 40, "cnp": 6, "cov": False, "precision": "mixed", "iters": 8},
        # variable intrinsics: the benchmark's size in FP64, and with distortion a smaller one in the mixed form
        {"name": "lm_circle52x64053_cnp11_fp64", "kind": "lm", "scene": "circle", "cams": 52, "pts": 64053, "vmin": 2,
         "vmax": 40, "cnp": 11, "cov": False, "precision": "fp64", "iters": 6},
        {"name": "lm_circle21x11315_cnp16_mixed", "kind": "lm", "scene": "circle", "cams": 21, "pts": 11315, "vmin": 2,
         "vmax": 20, "cnp": 16, "cov": False, "precision": "mixed", "iters": 6},
        # batches of independent problems: 5-30 cameras, 200-3,000 points, 3-8 views
        {"name": "batch64_fp64", "kind": "batch", "problems": 64, "vmin": 3, "vmax": 8, "precision": "fp64",
         "iters": 6},
        {"name": "batch304_mixed", "kind": "batch", "problems": 304, "vmin": 3, "vmax": 8, "precision": "mixed",
         "iters": 8},
        # a burst of requests, half with 6 and half with 11 parameters per camera
        {"name": "serve_burst12", "kind": "serve", "requests": 12, "vmin": 4, "vmax": 6, "precision": "mixed",
         "iters": 6},
        # the trust-region driver's modified Cholesky at 88 cameras
        {"name": "cholmod528", "kind": "cholmod", "n": 528},
        # the cost alone, on device arrays of the caller
        {"name": "cost_circle88x64298", "kind": "cost", "scene": "circle", "cams": 88, "pts": 64298, "vmin": 2,
         "vmax": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lm", "lm", "lm", "lm", "lm", "oneshot", "batch", "batch", "serve", "cholmod", "cost"])
    if kind in ("lm", "oneshot"):
        scene = rng.choice(["arc", "circle"])
        cnp = rng.choice([6, 6, 6, 11, 16])
        cams = _log_int(rng, 5, {6: 88, 11: 52, 16: 30}[cnp]) if scene == "arc" else _log_int(
            rng, 12, {6: 88, 11: 52, 16: 30}[cnp])
        top = 64298 if kind == "lm" and cnp != 16 else 16000
        vmin, vmax = (3, rng.randint(4, min(9, cams))) if scene == "arc" else (2, min(40, cams - 1))
        return {"kind": kind, "scene": scene, "cams": cams, "pts": _log_int(rng, 300, top), "vmin": vmin,
                "vmax": vmax, "cnp": cnp, "cov": rng.random() < 0.25, "precision": rng.choice(["fp64", "fp64", "mixed"]),
                "iters": rng.randint(4, 8)}
    if kind == "batch":
        return {"kind": "batch", "problems": _log_int(rng, 8, 200), "vmin": 3, "vmax": rng.randint(4, 8),
                "precision": rng.choice(["fp64", "mixed"]), "iters": rng.randint(4, 6)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(2, 12), "vmin": 4, "vmax": 6,
                "precision": rng.choice(["fp64", "mixed"]), "iters": rng.randint(3, 6)}
    if kind == "cholmod":
        return {"kind": "cholmod", "n": 3 * _log_int(rng, 14, 176)}
    cams = _log_int(rng, 7, 138)
    return {"kind": "cost", "scene": "circle" if cams >= 12 else "arc", "cams": cams, "pts": _log_int(rng, 500, 64298),
            "vmin": 2 if cams >= 12 else 3, "vmax": min(40, cams - 1)}


# ---------------------------------------------------------------------------
# inputs

def _scene(case, seed):
    """One problem: host arrays as a caller of the solver has them."""
    cams, pts = case["cams"], case["pts"]
    if case["scene"] == "arc":
        sc = scenes.arc_scene(seed=seed, n_cams=cams, n_pts=pts, arc_deg=min(max(30.0, 2.0 * cams), 160.0),
                              k_range=(case["vmin"], case["vmax"]))
    else:
        sc = scenes.circle_scene(seed=seed, n_cams=cams, n_pts=pts, kmin=case["vmin"], kmax=case["vmax"])
    if case.get("cnp", 6) > 6:
        sc = scenes.with_intrinsics(sc, case["cnp"], seed=seed + 1000)
    if case.get("cov"):
        sc = scenes.with_covariance(sc, seed=seed + 2000)
    return sc


def _problems(case, seed):
    """The problems of a batch or of a burst of requests.  The sizes are a
    fixed spread of the workload's ranges, the same for every seed; the
    scenes are not."""
    out = []
    if case["kind"] == "batch":
        sizes = np.random.default_rng(case["problems"])
        for q in range(case["problems"]):
            cams, pts = int(sizes.integers(5, 31)), int(sizes.integers(200, 3001))
            out.append(scenes.arc_scene(seed=100000 * seed + q, n_cams=cams, n_pts=pts, arc_deg=max(30.0, 4.0 * cams),
                                        k_range=(case["vmin"], case["vmax"])))
        return out
    n = case["requests"]
    for q, (cams, pts) in enumerate(_burst(n)):
        sc = scenes.arc_scene(seed=1000 * seed + q, n_cams=cams, n_pts=pts,
                              arc_deg=float(min(max(30.0, 2.0 * cams), 160.0)), k_range=(case["vmin"], case["vmax"]))
        out.append(scenes.with_intrinsics(sc, 11, seed=1000 * seed + 500 + q) if q % 2 else sc)
    return out


def _burst(n):
    """Cameras and points of n requests: 5-138 and 500-20,000, log-spread."""
    return [(int(round(5 * (138 / 5) ** (((7 * q + 3) % n + 0.5) / n))), int(round(500 * 40 ** ((q + 0.5) / n))))
            for q in range(n)]


def _schur_like(n, seed):
    """A symmetric matrix as the trust-region fallback meets one: a Gram
    matrix of camera rows with mixed scales (rotations far above
    translations) whose last 7 columns depend on the others, as the gauge's
    do, less a little on their diagonal.  The pivots that fail are the last
    ones and stay well away from rounding, unlike the gauge's."""
    rng = np.random.default_rng(seed)
    scale = np.where(np.arange(n) % 6 < 3, 40.0, 1.0)
    J = rng.normal(size=(3 * n, n))
    J[:, n - 7:] = J[:, :n - 7] @ rng.normal(size=(n - 7, 7)) / math.sqrt(n)
    A = (J * scale).T @ (J * scale) / n
    A[np.arange(n - 7, n), np.arange(n - 7, n)] -= 0.01 * scale[n - 7:] ** 2
    return np.tril(A)


class _Server(serve_mod.Server):
    """A server that ends with the program's last use of it."""

    def __del__(self):
        self.close()


def _opts(case):
    return P.default_opts(allow_switch=0, max_iter=case["iters"], precision=MIXED[case["precision"]])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cholmod":
        return {"kind": kind, "S": _schur_like(case["n"], seed)}
    if kind == "lm":
        return {"kind": kind, "solver": P.Solver(_scene(case, seed)), "opts": _opts(case)}
    if kind == "oneshot":
        return {"kind": kind, "scene": _scene(case, seed), "opts": _opts(case)}
    if kind == "batch":
        return {"kind": kind, "batch": batch_mod.Batch(_problems(case, seed)), "opts": _opts(case)}
    if kind == "serve":
        return {"kind": kind, "requests": _problems(case, seed),
                "server": _Server(precision=MIXED[case["precision"]], max_iter=case["iters"],
                                  hbm_budget_bytes=4e9)}
    sc = _scene(case, seed)
    dev = {f: torch.from_numpy(np.ascontiguousarray(getattr(sc, f))).cuda()
           for f in ("K", "q0", "cams", "pts", "meas", "obs_pt", "obs_cam")}
    fn = P.lib().psba_cost_noalloc
    fn.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p] * 9
    return {"kind": kind, "sizes": (sc.n_cams, sc.n_pts, sc.n_obs), "dev": dev, "fn": fn,
            "cost": torch.empty(1, dtype=torch.float64, device="cuda")}


# ---------------------------------------------------------------------------
# one pass

def run(state):
    kind = state["kind"]
    if kind == "lm":
        s = state["solver"]
        s.reset_params()
        r = s.levmar(state["opts"])
        return {"cams": r.cams, "pts": r.pts, "cost": np.float64(r.final_cost)}
    if kind == "oneshot":
        with P.Solver(state["scene"]) as s:
            r = s.levmar(state["opts"])
        return {"cams": r.cams, "pts": r.pts, "cost": np.float64(r.final_cost)}
    if kind == "batch":
        b = state["batch"]
        b.reset()
        res, _ = b.levmar(state["opts"])
        got = [b.get_params(q) for q in range(b.n)]
        return {"cams": np.concatenate([c.ravel() for c, _ in got]), "pts": np.concatenate([p for _, p in got]),
                "cost": res["final_cost"]}
    if kind == "serve":
        s = state["server"]
        tickets = [s.submit(sc) for sc in state["requests"]]
        got = [s.wait(t) for t in tickets]
        return {"cams": np.concatenate([g.cams.ravel() for g in got]), "pts": np.concatenate([g.pts for g in got]),
                "cost": np.array([g.final_cost for g in got])}
    if kind == "cholmod":
        L, E = P.cholmod(state["S"])
        return {"L": np.tril(L), "E": E}
    d = state["dev"]
    rc = state["fn"](*state["sizes"], *(d[f].data_ptr() for f in ("K", "q0", "cams", "pts", "meas", "obs_pt",
                                                                  "obs_cam")),
                     state["cost"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc != P.PSBA_OK:
        raise RuntimeError("psba_cost_noalloc: %d" % rc)
    return state["cost"]


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _views(case):
    """Mean views per point and mean camera pairs per point."""
    lo, hi = case["vmin"], case["vmax"]
    k = np.arange(lo, hi + 1)
    w = k ** -1.835 if case.get("scene") == "circle" else np.ones(len(k))
    w = w / w.sum()
    return float((w * k).sum()), float((w * k * (k - 1) / 2).sum())


def _lm_work(case, cams, pts, cnp, iters):
    v, pairs = _views(case)
    obs, n = v * pts, cnp * cams
    per_obs = 100 + 6 * cnp + cnp * (cnp + 1) + 18 + 9 * cnp + 3 * cnp * (cnp + 1) / 2 + 3 * cnp + 30
    fma = per_obs * obs + 3 * cnp * cnp * pairs * pts + 60 * pts + n ** 3 / 6 + n * n
    # measurements and indices, cameras and points in and out
    nbytes = 24 * obs + 8 * (2 * n + 9 * cams + 6 * pts) + (24 * obs if case.get("cov") else 0)
    return nbytes, 2.0 * fma * iters


def work(case):
    kind = case["kind"]
    if kind in ("lm", "oneshot"):
        b, f = _lm_work(case, case["cams"], case["pts"], case["cnp"], case["iters"])
    elif kind == "batch":
        b, f = _lm_work(case, 17.5, 1600, 6, case["iters"])
        b, f = b * case["problems"], f * case["problems"]
    elif kind == "serve":
        b = f = 0.0
        for q, (cams, pts) in enumerate(_burst(case["requests"])):
            bq, fq = _lm_work(case, cams, pts, 11 if q % 2 else 6, case["iters"])
            b, f = b + bq, f + fq
    elif kind == "cholmod":
        n = case["n"]
        b, f = 8.0 * (n * (n + 1) + n), n ** 3 / 3
    else:
        v, _ = _views(case)
        obs = v * case["pts"]
        b, f = 24 * obs + 24 * case["pts"] + 120 * case["cams"], 2 * 25 * obs
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch and numpy

def _project(cam, q0, K, X):
    """Cameras (n, cnp), their initial rotations (n, 4) and fixed intrinsics
    (n, 5) on points (n, 3): image points (n, 2)."""
    v0, v1, v2 = cam[:, 0], cam[:, 1], cam[:, 2]
    s0, a1, a2, a3 = q0.unbind(1)
    sl = torch.sqrt(1 - v0 * v0 - v1 * v1 - v2 * v2)
    s = sl * s0 - (a1 * v0 + a2 * v1 + a3 * v2)
    a = s0 * v0 + sl * a1 + a3 * v1 - a2 * v2
    b = s0 * v1 + sl * a2 + a1 * v2 - a3 * v0
    c = s0 * v2 + sl * a3 + a2 * v0 - a1 * v1
    d = s * s - (a * a + b * b + c * c)
    X0, X1, X2 = X.unbind(1)
    xc = (d + 2 * a * a) * X0 + 2 * (a * b - s * c) * X1 + 2 * (a * c + s * b) * X2 + cam[:, 3]
    yc = 2 * (a * b + s * c) * X0 + (d + 2 * b * b) * X1 + 2 * (b * c - s * a) * X2 + cam[:, 4]
    zc = 2 * (a * c - s * b) * X0 + 2 * (b * c + s * a) * X1 + (d + 2 * c * c) * X2 + cam[:, 5]
    x, y = xc / zc, yc / zc
    fx, cx, cy, ar, sk = (cam[:, 6:11] if cam.shape[1] > 6 else K).unbind(1)
    if cam.shape[1] == 16:
        k1, k2, p1, p2, k3 = cam[:, 11:16].unbind(1)
        r2 = x * x + y * y
        rad = 1 + r2 * (k1 + r2 * (k2 + r2 * k3))
        x, y = (rad * x + 2 * p1 * x * y + p2 * (r2 + 2 * x * x), rad * y + p1 * (r2 + 2 * y * y) + 2 * p2 * x * y)
    return torch.stack([fx * x + sk * y + cx, fx * ar * y + cy], 1)


class _Exact:
    """levmar() on one problem in 64 bits: dense Schur complement, LU solve."""

    def __init__(self, sc, cnp):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
        self.cnp = cnp
        self.cams, self.pts, self.q0, self.K, self.meas = (t(x) for x in (sc.cams, sc.pts, sc.q0, sc.K, sc.meas))
        self.i, self.j = t(sc.obs_pt.astype(np.int64)), t(sc.obs_cam.astype(np.int64))
        cov = getattr(sc, "cov", None)
        # e' cov^-1 e through the upper factor L of cov^-1 (L' L = cov^-1)
        self.L = None if cov is None else torch.linalg.cholesky(torch.linalg.inv(t(cov))).transpose(1, 2)

    def _white(self, m):
        return m if self.L is None else self.L @ m

    def residual(self, cams, pts):
        e = self.meas - _project(cams[self.j], self.q0[self.j], self.K[self.j], pts[self.i])
        return self._white(e.unsqueeze(2))

    def jacobian(self):
        cols = []
        cam, X = self.cams[self.j], self.pts[self.i]
        for c in range(self.cnp + 3):
            tc, tx = torch.zeros_like(cam), torch.zeros_like(X)
            (tc if c < self.cnp else tx)[:, c if c < self.cnp else c - self.cnp] = 1.0
            f = lambda a, b: _project(a, self.q0[self.j], self.K[self.j], b)  # noqa: E731
            cols.append(torch.func.jvp(f, (cam, X), (tc, tx))[1])
        J = self._white(torch.stack(cols, 2))
        return J[:, :, :self.cnp], J[:, :, self.cnp:]

    def solve(self, iters, tau=1e-3):
        nc, npt, cnp = self.cams.shape[0], self.pts.shape[0], self.cnp
        n, mu, nu = nc * cnp, None, 2
        e = self.residual(self.cams, self.pts)
        cost = float((e * e).sum())
        for _ in range(iters):
            A, B = self.jacobian()
            z = lambda *s: torch.zeros(s, dtype=torch.float64, device=A.device)  # noqa: E731
            U = z(nc, cnp, cnp).index_add_(0, self.j, A.transpose(1, 2) @ A)
            V = z(npt, 3, 3).index_add_(0, self.i, B.transpose(1, 2) @ B)
            ga = z(nc, cnp, 1).index_add_(0, self.j, A.transpose(1, 2) @ e).reshape(-1)
            gb = z(npt, 3, 1).index_add_(0, self.i, B.transpose(1, 2) @ e)
            W = z(nc, npt, cnp, 3)
            W[self.j, self.i] = A.transpose(1, 2) @ B
            W = W.permute(0, 2, 1, 3).reshape(n, npt, 3)
            if mu is None:
                mu = tau * max(float(torch.diagonal(U, dim1=1, dim2=2).max()),
                               float(torch.diagonal(V, dim1=1, dim2=2).max()))
            while True:
                Vi = torch.linalg.inv(V + mu * torch.eye(3, dtype=V.dtype, device=V.device))
                Y = torch.einsum("npk,pkl->npl", W, Vi)
                S = torch.block_diag(*U) - Y.reshape(n, -1) @ W.reshape(n, -1).T
                S += mu * torch.eye(n, dtype=S.dtype, device=S.device)
                da = torch.linalg.solve(0.5 * (S + S.T), ga - Y.reshape(n, -1) @ gb.reshape(-1))
                db = (Vi @ (gb - torch.einsum("npk,n->pk", W, da).unsqueeze(2))).squeeze(2)
                e1 = self.residual(self.cams + da.reshape(nc, cnp), self.pts + db)
                new = float((e1 * e1).sum())
                den = float((da * (mu * da + ga)).sum() + (db * (mu * db + gb.squeeze(2))).sum())
                rho = (cost - new) / den
                if rho > 0:
                    mu *= max(1 / 3, 1 - (2 * rho - 1) ** 3)
                    nu = 2
                    self.cams, self.pts, cost, e = self.cams + da.reshape(nc, cnp), self.pts + db, new, e1
                    break
                mu *= nu
                nu *= 2
        return self.cams.cpu().numpy(), self.pts.cpu().numpy(), np.float64(cost)


def _cholmod64(S):
    """The modified Cholesky by columns of 3, right-looking, in numpy."""
    n = S.shape[0]
    A = np.tril(S) + np.tril(S, -1).T
    off = np.abs(A - np.diag(np.diag(A))).max()
    gam = np.abs(np.diag(A)).max()
    delta = 1e-15 * max(off + gam, 1.0)
    beta = math.sqrt(max(gam, 1e-15, off / math.sqrt(n * n - 1.0)))
    T, L, a0 = A.copy(), np.zeros((n, n)), np.diag(A).copy()
    for j in range(0, n, 3):
        try:
            D = np.linalg.cholesky(T[j:j + 3, j:j + 3])
            R = np.linalg.solve(D, T[j + 3:, j:j + 3].T).T
            ok = not (R > beta).any()
        except np.linalg.LinAlgError:
            ok = False
        if ok:
            L[j:j + 3, j:j + 3], L[j + 3:, j:j + 3] = D, R
            T[j + 3:, j + 3:] -= R @ R.T
            continue
        for x in range(j, j + 3):
            d = math.sqrt(max(abs(T[x, x]), delta))
            c = T[x + 1:, x].copy()
            if (c / d > beta).any():
                d = np.abs(c).max() / beta
            L[x, x], L[x + 1:, x] = d, c / d
            T[x + 1:, x + 1:] -= np.outer(L[x + 1:, x], L[x + 1:, x])
    return L, (L * L).sum(1) - a0


def exact(case, seed):
    kind = case["kind"]
    if kind == "cholmod":
        L, E = _cholmod64(_schur_like(case["n"], seed))
        return {"L": L, "E": E}
    if kind == "cost":
        sc = _scene(case, seed)
        e = _Exact(sc, 6).residual(torch.from_numpy(sc.cams).to("cuda"), torch.from_numpy(sc.pts).to("cuda"))
        return (e * e).sum().reshape(1)
    if kind in ("lm", "oneshot"):
        cams, pts, cost = _Exact(_scene(case, seed), case["cnp"]).solve(case["iters"])
        return {"cams": cams, "pts": pts, "cost": cost}
    if kind == "batch" and case["problems"] * case["iters"] > 1500:
        return None  # over 20 seconds
    got = [_Exact(sc, sc.cnp).solve(case["iters"]) for sc in _problems(case, seed)]
    return {"cams": np.concatenate([c.ravel() for c, _, _ in got]), "pts": np.concatenate([p for _, p, _ in got]),
            "cost": np.array([c for _, _, c in got])}
