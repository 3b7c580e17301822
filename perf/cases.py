"""The framework's timed workloads: whole calls of the friction-solve path as a program that steps a rigid-body
simulation (or differentiates one) makes them, from a handful of contacts to the 200 000-contact problem.

Problems come from the package's seeded generators: random body pairs (small scenes, batches, the gradient
workload) or bodies on a jittered grid (large scenes). Solves start from r = 0 unless stated and run with the
reference's defaults but for the iteration budget, which bounds a pass. Host arrays go in and come out, as they do
for a program that uses the classes of bogus_gpu; the handle (W, its device copies, workspaces) is kept between
passes, except in the `step` cases, where every pass assembles its problem anew.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "so-bogus_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bogus_gpu  # noqa: E402
from bogus_gpu import generator  # noqa: E402

COMPLIANCE = generator.ADJOINT_COMPLIANCE


def listed():
    return [
        # one articulated figure or a small pile, solved every frame: launches and latency are all there is
        {"name": "apgd_33", "kind": "pg", "n": 33, "bodies": 11, "variant": "apgd", "coulomb": False, "iters": 300},
        # the 500-contact scene with exact Coulomb friction: the Cadoux fixed point over SPG, the facade's default
        {"name": "cadoux_spg_500", "kind": "cadoux", "n": 500, "bodies": 200, "outer": 5, "iters": 100},
        # an interactive granular scene
        {"name": "apgd_20000", "kind": "pg", "n": 20000, "bodies": 5000, "variant": "apgd", "coulomb": False,
         "iters": 150},
        # the offline scene: 50 000 bodies, W larger than the L2 cache
        {"name": "apgd_200000", "kind": "pg", "n": 200000, "bodies": 50000, "variant": "apgd", "coulomb": False,
         "iters": 100},
        # the FP32-refined solve with FP32 correction products, on a scene of intermediate size
        {"name": "refined_50000", "kind": "refined", "n": 50000, "bodies": 12500, "iters": 200, "refine": 100,
         "refresh": 25},
        # Gauss-Seidel in the contacts' own order, the reference's default solver, on a small scene
        {"name": "gs_501", "kind": "gs", "n": 501, "bodies": 200, "coloring": False, "iters": 100},
        # colored Gauss-Seidel on a large scene
        {"name": "gs_colored_50000", "kind": "gs", "n": 50000, "bodies": 12500, "coloring": True, "iters": 25},
        # many independent scenes (a learning environment): problems of 16 to 1024 contacts in one call
        {"name": "batch_256", "kind": "batch", "problems": 256, "largest": 1024, "iters": 100},
        # the backward pass of a differentiable simulation: gradients with respect to b and mu at the solution
        {"name": "adjoint_4x2500", "kind": "adjoint", "problems": 4, "n": 2500, "iters": 150},
        # the primal solvers, which never form W
        {"name": "admm_30000", "kind": "admm", "n": 30000, "bodies": 7500, "iters": 100},
        {"name": "dama_9999", "kind": "dama", "n": 9999, "bodies": 2500, "iters": 100},
        # one whole time step: W and b assembled from the bodies' Jacobians, the solve, the resulting velocities
        {"name": "step_15001", "kind": "step", "n": 15001, "bodies": 3750, "iters": 50},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pg", "pg", "cadoux", "refined", "gs", "gs", "batch", "adjoint", "admm", "dama", "step"])
    if kind == "pg":
        n = _log_int(rng, 16, 200000)
        return {"kind": kind, "n": n, "bodies": max(3, n // rng.choice([3, 4])), "variant": rng.choice(["apgd", "apgd", "spg"]),
                "coulomb": rng.random() < 0.3, "iters": 300 if n < 2000 else 150 if n < 30000 else 80}
    if kind == "cadoux":
        n = _log_int(rng, 100, 5000)
        return {"kind": kind, "n": n, "bodies": max(3, n // 3), "outer": rng.randint(2, 5), "iters": 100}
    if kind == "refined":
        n = _log_int(rng, 2000, 100000)
        return {"kind": kind, "n": n, "bodies": n // 4, "iters": 150, "refine": 80, "refresh": rng.choice([0, 25, 50])}
    if kind == "gs":
        if rng.random() < 0.5:
            n = _log_int(rng, 64, 2000)
            return {"kind": kind, "n": n, "bodies": max(3, n // 3), "coloring": False, "iters": 50}
        n = _log_int(rng, 2000, 70000)
        return {"kind": kind, "n": n, "bodies": n // 4, "coloring": True, "iters": 20}
    if kind == "batch":
        return {"kind": kind, "problems": _log_int(rng, 24, 400), "largest": _log_int(rng, 64, 1024), "iters": 100}
    if kind == "adjoint":
        return {"kind": kind, "problems": rng.randint(1, 4), "n": _log_int(rng, 150, 2500), "iters": 150}
    if kind == "step":
        n = _log_int(rng, 500, 30000)
        return {"kind": kind, "n": n, "bodies": n // 4, "iters": 50}
    n = _log_int(rng, 200, 60000)
    return {"kind": kind, "n": n, "bodies": max(3, n // 4), "iters": 80}


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _data(case, seed):
    """The generated bodies and contacts of a case, and the contact ranges of its problems."""
    if case["kind"] == "batch":
        return _batch(case["problems"], case["largest"], seed)
    if case["kind"] == "adjoint":
        return generator.adjoint_batch(case["problems"], case["n"], seed=seed)
    n, nb = case["n"], case["bodies"]
    # scenes below a thousand contacts are random pairs; larger ones live on the grid
    d = generator.random_pairs(nb, n, seed=seed) if n < 1000 else generator.grid(nb, n, seed=seed)
    return d, np.array([0, n], np.int32)


def _batch(problems, largest, seed):
    """generator.batch with the problems' sizes (log-uniform from 16 contacts) fixed by the case, not by the seed."""
    rng = np.random.default_rng(problems * 100003 + largest)
    sizes = np.exp(rng.uniform(math.log(16), math.log(largest + 1), problems)).astype(int)
    parts = [generator.random_pairs(max(2, n // 3), int(n), seed=seed * 100003 + p) for p, n in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum([d.nbodies for d in parts])])
    cat = lambda f: np.concatenate([f(d, o) for d, o in zip(parts, off)])  # noqa: E731
    d = generator.PrimalData(
        cat(lambda d, o: d.minv), cat(lambda d, o: d.objA + o).astype(np.int32),
        cat(lambda d, o: np.where(d.objB >= 0, d.objB + o, -1)).astype(np.int32), cat(lambda d, o: d.HA),
        cat(lambda d, o: d.HB), cat(lambda d, o: d.b), cat(lambda d, o: d.mu), seed, "batch")
    return d, np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)


def _dual(data):
    D = bogus_gpu.DualFrictionProblem(0)
    D.computeFrom(bogus_gpu.PrimalFrictionProblem.from_generated(data))
    return D


def _pg(case):
    pg = bogus_gpu.ProjectedGradient()
    pg.setMaxIters(case["iters"])
    if case["kind"] == "cadoux" or case.get("variant") == "spg":
        pg.setDefaultVariant(bogus_gpu.SPG)
    if case["kind"] == "refined":
        pg.setMixedPrecision(True, case["refine"])
        pg.setFp32CorrectionProducts(case["refresh"])
    return pg


def prepare(case, seed):
    kind = case["kind"]
    data, cptr = _data(case, seed)
    st = {"case": case, "data": data, "r0": np.zeros(3 * data.n)}
    if kind in ("admm", "dama", "step"):
        P = bogus_gpu.PrimalFrictionProblem.from_generated(data)
        if kind == "dama":
            P.computeMInv(np.linalg.inv(data.minv))
        st["P"] = P
        st["v0"] = np.zeros(6 * data.nbodies)
        if kind == "step":
            st["solver"] = _pg(case)
        else:
            st["solver"] = bogus_gpu.ADMM() if kind == "admm" else bogus_gpu.DualAMA()
            st["solver"].setMaxIters(case["iters"])
        return st
    D = st["D"] = _dual(data)
    if kind == "gs":
        gs = bogus_gpu.GaussSeidel()
        gs.setMaxIters(case["iters"])
        gs.coloring().update(case["coloring"])
        st["solver"] = gs
        return st
    if kind == "batch":
        D.setBatch(cptr)
        st["solver"] = _pg(case)
        return st
    if kind == "adjoint":
        D.add_compliance(COMPLIANCE)
        D.setBatch(cptr)
        pg = bogus_gpu.ProjectedGradient()
        pg.setMaxIters(400)
        pg.setTol(1e-10)
        r = np.zeros(3 * data.n)
        D.solveBatchWith(pg, r)
        st["r"] = r
        st["g"] = np.random.default_rng(seed + 1).standard_normal(3 * data.n)
        return st
    st["solver"] = _pg(case)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "adjoint":
        D = st["D"]
        db, dmu = D.adjoint(st["r"], st["g"], tol=1e-10, max_iters=case["iters"])
        return {"db": db, "dmu": dmu, "iterations": D.last_adjoint_iterations}
    r = st["r0"].copy()
    if kind in ("admm", "dama"):
        P, v = st["P"], st["v0"].copy()
        res = P.solveWith(st["solver"], 0.0, v, r) if kind == "admm" else P.solveWith(st["solver"], v, r)
        return {"r": r, "v": v, "residual": res, "iterations": P.last_iterations}
    if kind == "batch":
        res, its = st["D"].solveBatchWith(st["solver"], r)
        return {"r": r, "residual": res, "iterations": its.astype(np.int64)}
    if kind == "step":
        D = bogus_gpu.DualFrictionProblem(0)
        D.computeFrom(st["P"])
        res = D.solveWith(st["solver"], r)
        return {"r": r, "u": D.multiply(r) + st["P"].w, "residual": res, "iterations": D.last_iterations}
    D = st["D"]
    if kind == "cadoux":
        res = D.solveCadoux(st["solver"], r, case["outer"])
    elif kind == "pg":
        res = D.solveWith(st["solver"], r, staticProblem=not case["coulomb"])
    else:
        res = D.solveWith(st["solver"], r)
    return {"r": r, "residual": res, "iterations": D.last_iterations}


def work(case):
    """Bytes: W (or H and M^-1) and the vectors once. Flops: the budgeted iterations' products and per-contact law."""
    kind = case["kind"]
    if kind == "batch":
        # contacts log-uniform in [16, largest], a third as many bodies: about 11 blocks in a row
        n = case["problems"] * (case["largest"] - 16) / math.log(case["largest"] / 16)
        per_row = 11.0
    elif kind == "adjoint":
        n, per_row = case["problems"] * case["n"], 11.5
    else:
        n = case["n"]
        per_row = 3.6 * n / case["bodies"]
    blocks = n * per_row
    if kind in ("admm", "dama"):
        bodies = case["bodies"]
        nbytes = n * (1.9 * (144 + 4) + 8 * 10) + bodies * 8 * (36 + 12)
        return {"bytes": nbytes, "flops": case["iters"] * (n * (1.9 * 72 + 150) + bodies * 72)}
    nbytes = 76 * blocks + 8 * 11 * n
    if kind == "gs":
        return {"bytes": nbytes, "flops": case["iters"] * (18 * blocks + 1000 * n)}
    if kind == "adjoint":
        return {"bytes": nbytes, "flops": case["iters"] * (18 * blocks + 120 * n)}
    iters = case["iters"] * (case["outer"] if kind == "cadoux" else 1) + case.get("refine", 0)
    passes = 1.0 if kind == "cadoux" or case.get("variant") == "spg" else 2.3
    flops = iters * (passes * 18 * blocks + 200 * n)
    if kind == "step":
        nbytes = n * (2 * 144 + 8 * 11) + case["bodies"] * 288
        flops += blocks * 18 * 12
    return {"bytes": nbytes, "flops": flops}


# ---- the same results in plain 64-bit torch -------------------------------------------------------------------------

class _Plain:
    """H, M^-1, scalings and segment sums of generated data, for problems [ptr[p], ptr[p + 1]) side by side."""

    def __init__(self, data, ptr, compliance=0.0):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float64))  # noqa: E731
        self.n, self.nb = data.n, data.nbodies
        self.HA, self.HB = t(data.HA), t(data.HB)
        self.iA = torch.from_numpy(data.objA.astype(np.int64))
        self.iB = torch.from_numpy(np.where(data.objB >= 0, data.objB, 0).astype(np.int64))  # H is zero on the ground
        self.minv, self.b, self.mu = t(data.minv), t(data.b), t(data.mu)
        self.c = compliance
        self.seg = torch.from_numpy(np.repeat(np.arange(len(ptr) - 1), np.diff(ptr)))
        self.size = torch.from_numpy(np.diff(ptr).astype(np.float64))
        tr = 0.0
        for H, i in ((self.HA, self.iA), (self.HB, self.iB)):
            tr = tr + torch.einsum("nrk,nkl,nrl->n", H, self.minv[i], H)
        self.scaling = torch.clamp(tr / 3.0 + compliance, min=1.0)

    def Ht(self, r):
        v = torch.zeros(self.nb, 6, dtype=torch.float64)
        v.index_add_(0, self.iA, torch.einsum("nrk,nr->nk", self.HA, r))
        v.index_add_(0, self.iB, torch.einsum("nrk,nr->nk", self.HB, r))
        return v

    def Hv(self, v):
        return torch.einsum("nrk,nk->nr", self.HA, v[self.iA]) + torch.einsum("nrk,nk->nr", self.HB, v[self.iB])

    def W(self, r):
        return self.Hv(torch.einsum("bkl,bl->bk", self.minv, self.Ht(r))) + self.c * r

    def dot(self, a, b):
        return torch.zeros(len(self.size), dtype=torch.float64).index_add_(0, self.seg, (a * b).sum(1))


def _project(mu, x):
    t = torch.linalg.vector_norm(x[:, 1:], dim=1)
    p = (x[:, 0] + mu * t) / (1 + mu * mu)
    q = torch.cat([p[:, None], x[:, 1:] * (mu * p / torch.where(t > 0, t, torch.ones_like(t)))[:, None]], 1)
    q = torch.where((mu * t <= -x[:, 0])[:, None], torch.zeros_like(q), q)
    return torch.where((t <= mu * x[:, 0])[:, None], x, q)


def _law(mu, x, y, coulomb):
    """Fischer-Burmeister function of the cone's complementarity."""
    s = mu * torch.linalg.vector_norm(y[:, 1:], dim=1) if coulomb else torch.zeros_like(mu)
    xh = torch.cat([(mu * x[:, 0])[:, None], x[:, 1:]], 1)
    yh = torch.cat([(y[:, 0] + s)[:, None], mu[:, None] * y[:, 1:]], 1)
    z0 = (xh * xh).sum(1) + (yh * yh).sum(1)
    zt = xh[:, :1] * xh[:, 1:] + yh[:, :1] * yh[:, 1:]
    nt = torch.linalg.vector_norm(zt, dim=1)
    u = torch.where((nt < 2.3e-16)[:, None], torch.tensor([[1.0, 0.0]], dtype=torch.float64),
                    zt / torch.where(nt > 0, nt, torch.ones_like(nt))[:, None])
    r1, r2 = torch.sqrt(torch.clamp(z0 - 2 * nt, min=0.0)), torch.sqrt(z0 + 2 * nt)
    z = 0.5 * torch.cat([(r1 + r2)[:, None], (r2 - r1)[:, None] * u], 1)
    return xh + yh - z


def _nesterov(theta):
    t2 = theta * theta
    new = 0.5 * (torch.sqrt(t2 * t2 + 4 * t2) - t2)
    return new, (theta - t2) / (t2 + new)


def _descend(A, b, x, variant, coulomb, iters, tol):
    """APGD or SPG (Core/BlockSolvers/ProjectedGradient.impl.hpp) on every problem at once; (best x, its residual)."""
    mu, seg, spg = A.mu, A.seg, variant == "spg"
    one = torch.ones(len(A.size), dtype=torch.float64)
    at = lambda s: s[seg][:, None]  # noqa: E731
    x = _project(mu, x)
    Mx = A.W(x)
    d = A.W(x - 1)
    den = A.dot(d, d)
    alpha = torch.where(den > 1e-16, torch.clamp(A.dot(x - 1, x - 1) / den, max=1.0), one)
    prev, theta, best, least = x, one.clone(), x.clone(), torch.full_like(one, math.inf)
    live = torch.ones_like(one, dtype=torch.bool)
    for _ in range(iters):
        y = Mx + b
        f = _law(mu, x * A.scaling[:, None], y, coulomb)
        res = A.dot(f, f) / (1 + A.size)
        better = live & (res < least)
        least = torch.where(better, res, least)
        best = torch.where(at(better), x, best)
        live = live & ~(res < tol)
        if not bool(live.any()):
            break
        s = torch.zeros_like(y)
        if coulomb:
            s[:, 0] = mu * torch.linalg.vector_norm(y[:, 1:], dim=1)
        y = y + s
        if spg:
            xs = _project(mu, x - at(alpha) * y)
            mom = A.dot(xs - prev, y) < 0
            new, beta = _nesterov(theta)
            theta = torch.where(mom, new, one)
            w = xs + at(torch.where(mom, beta, 0 * beta)) * (xs - prev) - x
            z = A.W(x + w) - Mx
            x, Mx, prev = x + w, Mx + z, xs
            alpha = torch.clamp(A.dot(w, z) / A.dot(z, z), 1e-6, 1e6)
            continue
        J = A.dot(x, 0.5 * Mx + b + s)
        alpha = alpha * 1.25
        trying = live.clone()
        xs, Mxs = x, Mx
        for ls in range(8):
            t = _project(mu, x - at(alpha) * y)
            xs = torch.where(at(trying), t, xs)
            Mxs = A.W(xs)
            dx = xs - x
            ok = A.dot(xs, 0.5 * Mxs + b + s) < J + A.dot(y, dx) + 0.5 / alpha * A.dot(dx, dx)
            trying = trying & ~ok
            alpha = torch.where(trying, 0.5 * alpha, alpha)
            if not bool(trying.any()):
                break
        mom = A.dot(xs - prev, y) < 0
        new, beta = _nesterov(theta)
        theta = torch.where(mom, new, one)
        x = xs + at(torch.where(mom, beta, 0 * beta)) * (xs - prev)
        prev, Mx = xs, A.W(x)
    return best, least


def _primal_admm(A, iters, tol):
    """Accelerated primal ADMM with lambda = 0 (Core/BlockSolvers/ADMM.impl.hpp), step size 1e-2, from v = r = 0."""
    g, im, w = 1e-2, 1.0 / A.mu, A.b
    r = torch.zeros_like(w)
    ut = w.clone()
    z, yp = _project(im, ut - r / g), -r / g
    theta, last, res = torch.ones(1, dtype=torch.float64), -1.0, -1.0
    v = torch.zeros(A.nb, 6, dtype=torch.float64)
    for _ in range(iters):
        v = torch.einsum("bkl,bl->bk", A.minv, A.Ht(r))
        ut = w + A.Hv(v)
        f = _law(im, ut, r, False)
        res = float((f * f).sum()) / (1 + A.n) + float(((ut - z) ** 2).sum()) / (1 + 3 * A.n)
        if res < tol:
            break
        zn = _project(im, ut - r / g)
        if res < last:
            theta, beta = _nesterov(theta)
            y = (ut - zn) - r / g
            r, yp = -g * (y + beta * (y - yp)), y
        else:
            theta = torch.ones_like(theta)
            r = r + g * (zn - ut)
            yp = -r / g
        z, last = zn, res
    return r, v, res


def _gradients(A, r, g, ptr):
    """dL/db and dL/dmu by the implicit function theorem, one dense system for each problem."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    db, dmu = torch.zeros(A.n, 3, dtype=torch.float64), torch.zeros(A.n, dtype=torch.float64)
    al = 1.0 / A.scaling
    x = r - al[:, None] * (A.W(r) + A.b)
    t = torch.linalg.vector_norm(x[:, 1:], dim=1)
    mu, xn = A.mu, x[:, 0]
    u = x[:, 1:] / torch.where(t > 0, t, torch.ones_like(t))[:, None]
    c = 1 / (1 + mu * mu)
    pn = c * (xn + mu * t)
    e = torch.cat([torch.ones(A.n, 1, dtype=torch.float64), mu[:, None] * u], 1)
    o = torch.stack([torch.zeros_like(t), -u[:, 1], u[:, 0]], 1)
    rho = mu * pn / torch.where(t > 0, t, torch.ones_like(t))
    J = c[:, None, None] * e[:, :, None] * e[:, None, :] + rho[:, None, None] * o[:, :, None] * o[:, None, :]
    dpn = t * c - 2 * mu * (xn + mu * t) * c * c
    K = torch.cat([dpn[:, None], (pn + mu * dpn)[:, None] * u], 1)
    polar, inside = mu * t <= -xn, t <= mu * xn
    J = torch.where(polar[:, None, None], torch.zeros_like(J), J)
    J = torch.where((inside & ~polar)[:, None, None], torch.eye(3, dtype=torch.float64).expand_as(J), J)
    K = torch.where((polar | inside)[:, None], torch.zeros_like(K), K)
    for p in range(len(ptr) - 1):
        a, z = int(ptr[p]), int(ptr[p + 1])
        n = z - a
        first = int(min(A.iA[a:z].min(), A.iB[a:z][A.HB[a:z].abs().sum((1, 2)) > 0].min()))
        nb = int(max(A.iA[a:z].max(), A.iB[a:z].max())) + 1 - first
        H = torch.zeros(n, 3, nb, 6, dtype=torch.float64)
        i = torch.arange(n)
        H[i, :, A.iA[a:z] - first] += A.HA[a:z]
        touches = A.HB[a:z].abs().sum((1, 2)) > 0
        H[i[touches], :, (A.iB[a:z] - first)[touches]] += A.HB[a:z][touches]
        H = H.reshape(3 * n, 6 * nb).to(dev)
        root = torch.block_diag(*torch.linalg.cholesky(A.minv[first:first + nb])).to(dev)
        HL = H @ root
        W = HL @ HL.T + A.c * torch.eye(3 * n, dtype=torch.float64, device=dev)
        Jd, ad = J[a:z].to(dev), al[a:z].to(dev)
        WAJ = torch.einsum("rnk,nkl->rnl", W.reshape(3 * n, n, 3) * ad[None, :, None], Jd).reshape(3 * n, 3 * n)
        S = torch.eye(3 * n, dtype=torch.float64, device=dev) - torch.block_diag(*Jd) + WAJ
        lam = torch.linalg.solve(S, g[a:z].reshape(-1).to(dev)).reshape(n, 3)
        db[a:z] = -(ad[:, None] * torch.einsum("nkl,nl->nk", Jd, lam)).cpu()
        dmu[a:z] = (K[a:z].to(dev) * lam).sum(1).cpu()
    return db, dmu


def exact(case, seed):
    """None for Gauss-Seidel (its sweep is sequential: minutes in plain Python), DualAMA and the FP32-refined solve
    (its first part's iterates are 32-bit ones)."""
    kind = case["kind"]
    if kind in ("gs", "dama", "refined"):
        return None
    data, ptr = _data(case, seed)
    A = _Plain(data, ptr, COMPLIANCE if kind == "adjoint" else 0.0)
    x0 = torch.zeros(data.n, 3, dtype=torch.float64)
    if kind == "adjoint":
        st = prepare(case, seed)  # the solution at which the gradients are taken is an input
        db, dmu = _gradients(A, torch.from_numpy(st["r"]).reshape(-1, 3), torch.from_numpy(st["g"]).reshape(-1, 3), ptr)
        return {"db": db.reshape(-1), "dmu": dmu, "iterations": None}
    if kind == "admm":
        r, v, res = _primal_admm(A, case["iters"], 1e-6)
        return {"r": r.reshape(-1), "v": v.reshape(-1), "residual": res, "iterations": None}
    if kind == "cadoux":
        x, res = x0, None
        for it in range(case["outer"] + 1):
            y = A.W(x) + A.b
            f = _law(A.mu, x * A.scaling[:, None], y, True)
            res = float((f * f).sum()) / (1 + A.n)
            if it == case["outer"] or (it > 0 and res < 1e-6):
                break
            b = A.b.clone()
            b[:, 0] += A.mu * torch.linalg.vector_norm(y[:, 1:], dim=1)
            x, _ = _descend(A, b, x, "spg", False, case["iters"], 0.1 * max(1e-6, min(res, 1.0)))
        return {"r": x.reshape(-1), "residual": res, "iterations": None}
    x, res = _descend(A, A.b, x0, case.get("variant", "apgd"), bool(case.get("coulomb")), case["iters"], 1e-6)
    out = {"r": x.reshape(-1), "residual": res if kind == "batch" else float(res[0]), "iterations": None}
    if kind == "step":
        out["u"] = (A.W(x) + A.b).reshape(-1)
    return out
