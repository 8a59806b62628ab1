"""Workloads of the q-LSKUM solver, through its public Python interface.

Every case is a call that a program of this library makes in real use:

  solve   a steady solve's iterations on one cloud: set the state, iterate
          (Solver.q_lskum, or Solver.fpi_solver call by call), read the state
  batch   the same over several clouds at once (batch.run_batch), or in
          lockstep groups (batch.run_grouped)
  first   time to the first result of a cloud given as raw points: neighbour
          search, set-up on the device, the first iteration
  serve   a burst of requests to the request server

Clouds are the seeded shell clouds of mfcfd.cloud (spheres and ellipsoids);
the flow starts impulsively, as Solver.initial_conditions does.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(_ROOT, "3d-mfcfd_b200"), _ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from mfcfd import _lib, batch, cloud, serve  # noqa: E402
from mfcfd.solver import Solver  # noqa: E402

PRECISION = {"fp64": _lib.PRECISION_FP64, "mixed": _lib.PRECISION_MIXED, "mixed_dc": _lib.PRECISION_MIXED_DC}
# operations of one point in one iteration, counted by running the solver
# with counting arithmetic (1.1M sphere); least bytes: coordinates, frame,
# neighbours, state and increments read, state and increments written
FLOPS_PER_POINT = 95180
BYTES_PER_POINT = 24 + 72 + 4 * 28 + 80 + 80


def listed():
    return [
        # one fpi_solver call on a small test cloud: launches and latency
        {"name": "step_600", "kind": "solve", "shells": 6, "per": 100, "r1": 1.5, "aspect_y": 1.0, "aspect_z": 1.0,
         "precision": "fp64", "iters": 1, "by_call": True},
        # a coarse cloud of odd size, iterated by single calls (a host that logs every residual)
        {"name": "solve_9k_fp64", "kind": "solve", "shells": 26, "per": 361, "r1": 10.0, "aspect_y": 1.0,
         "aspect_z": 1.0, "precision": "fp64", "iters": 3, "by_call": True},
        # an ellipsoid in the defect-correction form that converged solves use
        {"name": "solve_21k_mixed_dc", "kind": "solve", "shells": 33, "per": 643, "r1": 10.0, "aspect_y": 1.4,
         "aspect_z": 1.2, "precision": "mixed_dc", "iters": 20, "by_call": False},
        # the 62,400-point sphere, the reference's kind of cloud, in FP64 and in mixed precision
        {"name": "solve_62k_fp64", "kind": "solve", "shells": 48, "per": 1300, "r1": 10.0, "aspect_y": 1.0,
         "aspect_z": 1.0, "precision": "fp64", "iters": 10, "by_call": False},
        {"name": "solve_62k_mixed", "kind": "solve", "shells": 48, "per": 1300, "r1": 10.0, "aspect_y": 1.0,
         "aspect_z": 1.0, "precision": "mixed", "iters": 10, "by_call": False},
        # a mid-size cloud of odd size
        {"name": "solve_260k_fp64", "kind": "solve", "shells": 61, "per": 4273, "r1": 10.0, "aspect_y": 1.0,
         "aspect_z": 1.0, "precision": "fp64", "iters": 4, "by_call": False},
        # the 1,104,000-point sphere, the benchmark's cloud, in FP64 and in the defect-correction form
        {"name": "solve_1m_fp64", "kind": "solve", "shells": 96, "per": 11500, "r1": 10.0, "aspect_y": 1.0,
         "aspect_z": 1.0, "precision": "fp64", "iters": 4, "by_call": False},
        {"name": "solve_1m_mixed_dc", "kind": "solve", "shells": 96, "per": 11500, "r1": 10.0, "aspect_y": 1.0,
         "aspect_z": 1.0, "precision": "mixed_dc", "iters": 4, "by_call": False},
        # a sweep of design points: clouds of uneven size iterated side by side
        {"name": "batch_12_mixed", "kind": "batch", "clouds": 12, "n_min": 10000, "n_max": 40000,
         "precision": "mixed", "iters": 20, "grouped": False},
        # the same as lockstep groups, in the form of converged batches
        {"name": "group_12_mixed_dc", "kind": "batch", "clouds": 12, "n_min": 10000, "n_max": 40000,
         "precision": "mixed_dc", "iters": 20, "grouped": True},
        # a new cloud of odd size from raw points to its first iteration
        {"name": "first_250k", "kind": "first", "shells": 60, "per": 4177, "r1": 10.0, "precision": "fp64"},
        # a burst of requests to the server, each iterated for a few chunks
        {"name": "serve_8", "kind": "serve", "clouds": 8, "n_min": 7000, "n_max": 20000, "precision": "mixed",
         "iters": 40},
    ]


def _shape(n):
    """Shells and points per shell of a cloud of about n points."""
    shells = max(6, int(round(1.21 * n ** (1.0 / 3.0))))
    return shells, max(100, int(round(n / shells)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "batch", "first"])
    precision = rng.choice(["fp64", "mixed", "mixed_dc"])
    if kind == "solve":
        n = math.exp(rng.uniform(math.log(600), math.log(900000)))
        shells, per = _shape(n)
        small = n < 2000
        return {"kind": kind, "shells": shells, "per": per, "r1": 1.5 if small else 10.0,
                "aspect_y": 1.0 if small else round(rng.uniform(1.0, 1.5), 3),
                "aspect_z": 1.0 if small else round(rng.uniform(1.0, 1.5), 3), "precision": precision,
                "iters": rng.randint(1, 3) if n > 200000 else rng.randint(2, 12), "by_call": n < 30000 and rng.random() < 0.5}
    if kind == "batch":
        n_min = rng.randint(5000, 15000)
        return {"kind": kind, "clouds": rng.randint(3, 14), "n_min": n_min, "n_max": rng.randint(2 * n_min, 50000),
                "precision": precision, "iters": 2 * rng.randint(3, 8), "grouped": rng.random() < 0.5}
    shells, per = _shape(math.exp(rng.uniform(math.log(5000), math.log(400000))))
    return {"kind": "first", "shells": shells, "per": per, "r1": 10.0, "precision": precision}


def _flow(rng):
    return float(rng.uniform(0.3, 0.6)), float(rng.uniform(-3.0, 3.0))


def _clouds(case, seed):
    """[(cloud, Mach, angle of attack)] of a case, from the seed alone."""
    rng = np.random.Generator(np.random.PCG64(90001 + 7 * seed))
    if case["kind"] in ("solve", "first"):
        aspect = (1.0, case.get("aspect_y", 1.0), case.get("aspect_z", 1.0))
        c = cloud.shell_cloud(case["shells"], case["per"], r1=case["r1"], jitter=0.02, seed=1000 + seed, aspect=aspect,
                              knn_device=0)
        return [(c,) + _flow(rng)]
    out = []
    for j in range(case["clouds"]):
        f = (j + 0.5) / case["clouds"]      # log-spaced sizes
        shells, per = _shape(case["n_min"] * (case["n_max"] / case["n_min"]) ** f)
        out.append((cloud.shell_cloud(shells, per, jitter=0.02, seed=100 * (1000 + seed) + j, knn_device=0),) + _flow(rng))
    return out


def prepare(case, seed):
    flows = _clouds(case, seed)
    state = {"case": case}
    prec = PRECISION[case["precision"]]
    if case["kind"] == "solve":
        c, m, a = flows[0]
        s = Solver(c, m, a, device=0, precision=prec, gpu_setup=1)
        prim = cloud.initial_state(c, m, a)
        # pinned host buffers, as a program that exchanges its state keeps
        pin = [torch.from_numpy(v).pin_memory() for v in (prim, np.zeros_like(prim), np.zeros_like(prim), np.zeros_like(prim))]
        state.update(solver=s, pinned=pin, buf=[p.numpy() for p in pin])
    elif case["kind"] == "batch":
        ss = [Solver(c, m, a, device=0, precision=prec, gpu_setup=1) for c, m, a in flows]
        # fewer warps per cloud than alone, so that more clouds share the device
        for s in ss:
            s.set_chain_warps(max(4, s.info()["max_level_width"]))
        state.update(solvers=ss, prims=[cloud.initial_state(c, m, a) for c, m, a in flows])
    elif case["kind"] == "first":
        state.update(flow=flows[0])
    else:
        state.update(server=serve.Server(device=0, setup_threads=4, chunk=10), flows=flows,
                     prims=[cloud.initial_state(c, m, a) for c, m, a in flows])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        s, (prim, zero, prim_out, delu_out) = state["solver"], state["buf"]
        s.set_state(prim, zero, 0.0)
        if case["by_call"]:
            hist = np.array([s.fpi_solver(t) for t in range(1, case["iters"] + 1)])
        else:
            hist = s.q_lskum(case["iters"])
        s.get_state(out=(prim_out, delu_out))
        return {"history": hist, "prim": prim_out, "delu": delu_out}
    if case["kind"] == "batch":
        ss = state["solvers"]
        for s, prim in zip(ss, state["prims"]):
            s.initial_conditions(prim)
            s.history.clear()
        hist = (batch.run_grouped if case["grouped"] else batch.run_batch)(ss, case["iters"])
        states = [s.get_state() for s in ss]
        return {"history": hist, "prim": [p for p, _, _ in states], "delu": [d for _, d, _ in states]}
    if case["kind"] == "first":
        c, m, a = state["flow"]
        nbhs, conn, min_dist = cloud.knn(c.x, c.y, c.z, 26, device=0)
        c.nbhs, c.conn, c.min_dist = nbhs, conn, min_dist
        s = Solver(c, m, a, device=0, precision=PRECISION[case["precision"]], gpu_setup=1)
        s.initial_conditions()
        res = s.fpi_solver(1)
        prim, delu, _ = s.get_state()
        alias, _ = s.alias()
        s.close()
        return {"nbhs": nbhs, "conn": conn, "min_dist": min_dist, "alias": alias, "history": np.array([res]),
                "prim": prim, "delu": delu}
    srv = state["server"]
    ids = [srv.submit(c, m, a, max_iters=case["iters"], residue_target=-20.0, prim=prim,
                      precision=PRECISION[case["precision"]])
           for (c, m, a), prim in zip(state["flows"], state["prims"])]
    res = [srv.wait(i) for i in ids]
    return {"history": np.array([[r["res_new"], r["residue"]] for r in res]),
            "prim": [r["prim"] for r in res]}


def work(case):
    if case["kind"] in ("solve", "first"):
        points = case["shells"] * case["per"]
    else:
        a, b = case["n_min"], case["n_max"]
        points = case["clouds"] * (b - a) / math.log(b / a)      # mean of a log-uniform size
    iters = case.get("iters", 1)
    return {"bytes": points * iters * BYTES_PER_POINT, "flops": points * iters * FLOPS_PER_POINT}


# ------------------------------------------------------------ 64-bit values

def _flux(kind, prim, fr):
    """Split (kind 0-5: x+ x- y+ y- z+ z-) and octant fluxes (6-9 wall, 10-13
    outer: x+ x- y+ y-) of primitive states in frames (t1, t2, n)."""
    rho, vel, pr = prim[..., 0], prim[..., 1:4], prim[..., 4]
    u = [(f * vel).sum(-1) for f in fr]
    usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    beta = 0.5 * rho / pr

    def terms(a):
        S = u[a] * np.sqrt(beta)
        B = 0.5 * np.exp(-S * S) / np.sqrt(math.pi * beta)
        e = torch.erf(torch.from_numpy(np.ascontiguousarray(S))).numpy()
        return 0.5 * (1 + e), 0.5 * (1 - e), B

    a = kind // 2 if kind < 6 else ((kind - 6) % 4) // 2
    pos = kind % 2 == 0
    Ap, An, B = terms(a)
    A, sg = (Ap, 1.0) if pos else (An, -1.0)
    t1 = u[a] * A + sg * B
    G = [rho * t1] + [rho * u[c] * t1 for c in range(3)]
    G[1 + a] = G[1 + a] + pr * A
    t = 2.5 * pr + 0.5 * rho * usq
    G.append((t + pr) * u[a] * A + sg * (t + 0.5 * pr) * B)
    if kind >= 6:
        zp, zn, B3 = terms(2)
        A3, s3 = (zn, -1.0) if kind < 10 else (zp, 1.0)
        last = G[4] * A3 + s3 * 0.5 * rho * u[2] * B3 * t1
        G = [G[0] * A3, G[1] * A3, G[2] * A3, rho * t1 * (u[2] * A3 + s3 * B3), last]
    return np.stack(G, -1)


def _kind(cls, d):
    if cls == 0:
        return d
    if cls == 1:
        return 6 + d if d < 4 else (5 if d == 5 else None)
    return 10 + d if d < 4 else (4 if d == 4 else None)


def _to_prim(U, fr):
    v = (fr[0] * U[..., 1:2] + fr[1] * U[..., 2:3] + fr[2] * U[..., 3:4]) / U[..., 0:1]
    p = 0.4 * (U[..., 4] - 0.5 * U[..., 0] * (v * v).sum(-1))
    return np.concatenate([U[..., 0:1], v, p[..., None]], -1)


class _Reference:
    """The iteration in plain numpy for a sphere or ellipsoid shell cloud
    (interior points in the global axes, unit least-squares weights)."""

    def __init__(self, c, mach, aoa):
        n = self.n = c.n
        self.inf = np.array(cloud.freestream(mach, aoa))
        self.cls = c.status.astype(int)
        self.xyz = np.stack([c.x, c.y, c.z], 1)
        self.fr = (c.tan1, c.tan2, c.nor)
        self.conn = c.conn.astype(np.int64) - 1
        self.has = np.arange(27)[None, :] < c.nbhs[:, None]
        self.conn[~self.has] = 0
        self.eps2 = ((2.0 * c.min_dist) ** 3) ** 2
        d = self.xyz[self.conn] - self.xyz[:, None]
        self.dx = np.where(self.has[..., None], d, 0.0)
        loc = [(d * f[:, None]).sum(-1) for f in self.fr]
        inner = (self.cls == 0)[:, None]
        # the six lists, stored 22 entries to a point with longer lists
        # running on into the next point's, points by class then index
        cap = 22
        order = np.concatenate([np.flatnonzero(self.cls == k) for k in (0, 1, 2)])
        self.idx = np.zeros((6, n, 27), np.int64)
        self.on = np.zeros((6, n, 27), bool)
        for k in range(6):
            v = loc[k // 2]
            take = (v <= 0) if k % 2 == 0 else np.where(inner, v > 0, v >= 0)
            if k == 4:
                take = np.where((self.cls == 2)[:, None], True, np.where((self.cls == 1)[:, None], False, take))
            if k == 5:
                take = np.where((self.cls == 1)[:, None], True, np.where((self.cls == 2)[:, None], False, take))
            take = take & self.has
            cnt = take.sum(1)
            flat = np.zeros(cap * n + 64, np.int64)
            rank = take.cumsum(1) - 1
            rows, cols = np.nonzero(take[order])
            pts = order[rows]
            flat[pts * cap + rank[pts, cols]] = self.conn[pts, cols]
            at = np.arange(n)[:, None] * cap + np.arange(27)[None]
            self.on[k] = np.arange(27)[None] < cnt[:, None]
            self.idx[k] = np.where(self.on[k], flat[np.minimum(at, flat.size - 1)], 0)
            if k == 5:
                wall = self.cls == 1
                self.idx[k][wall] = np.where(self.has[wall], self.conn[wall], 0)
        self.w = np.zeros((6, n, 27, 3))
        for k in range(6):
            d = self.xyz[self.idx[k]] - self.xyz[:, None]
            for a in range(3):
                self.w[k, :, :, a] = np.where(self.on[k], (d * self.fr[a][:, None]).sum(-1), 0.0)
        # row a = k // 2 of each list's inverse moment matrix
        M = np.einsum("knja,knjb->knab", self.w, self.w)
        self.row = np.zeros((6, n, 3))
        for k in range(6):
            good = self.on[k].sum(1) > 2
            self.row[k][good] = np.linalg.inv(M[k][good])[:, k // 2]
        # sweep order: breadth-first from the first point, whose own entry its first neighbour takes
        alias = [0] * (n + 1)
        pwa = [0] * (n + 2)
        nb = (c.conn * self.has).tolist()
        num = c.nbhs.tolist()
        alias[1] = pwa[1] = 1
        count = 0
        for i in range(1, n + 1):
            p = pwa[i]
            if p:
                for k in nb[p - 1][:num[p - 1]]:
                    if not alias[k]:
                        count += 1
                        alias[k] = count
                        pwa[count] = k
        self.alias = np.array(alias[1:])
        seq = [p - 1 for p in pwa[1:n + 1] if p and self.cls[p - 1] < 2]
        self.swept = np.zeros(n, bool)
        self.swept[seq] = True
        self.dirs = []
        for forward in (True, False):
            use = self.on & ((self.alias[self.idx] < self.alias[None, :, None]) if forward
                             else (self.alias[self.idx] > self.alias[None, :, None]))
            level = np.full(n, -1)
            dep = [np.unique(self.idx[:, p][use[:, p]]) for p in range(n)]
            for p in (seq if forward else seq[::-1]):
                lv = level[dep[p]]
                level[p] = (lv.max() if lv.size else -1) + 1
            self.dirs.append((use, [np.flatnonzero(level == v) for v in range(level.max() + 1)]))

    def _solve(self, k, p, t, use):
        """Derivative of list k at points p from the terms t (len(p), 27, 5)."""
        s = np.einsum("pja,pjc->pac", self.w[k, p] * use[..., None], t)
        return np.einsum("pa,pac->pc", self.row[k, p], s)

    def _recon(self, j, d, q, dq, qmax, qmin):
        qj = q[j]
        temp = (d[..., None, :] * dq[j]).sum(-1)
        neg = (qj - 0.5 * temp) - qj
        pos = np.where(neg > 0, qmax[j], qmin[j]) - qj
        e = self.eps2[j][..., None]
        num = (pos * pos + e) * neg + 2 * neg * neg * pos
        den = (pos * pos + 2 * neg * neg + neg * pos + e) * neg
        small = np.abs(neg) <= float(np.float32(10e-6))
        phi = np.where(small, 1.0, np.minimum(num / np.where(small, 1.0, den), 1.0))
        qt = qj - 0.5 * phi * temp
        b = -0.5 * qt[..., 4]
        v = qt[..., 1:4] * (0.5 / b)[..., None]
        rho = np.exp(qt[..., 0] + b * (v * v).sum(-1) - 2.5 * np.log(b))
        return np.concatenate([rho[..., None], v, (rho * 0.5 / b)[..., None]], -1)

    def step(self, prim, delu):
        n, fr = self.n, self.fr
        rot = np.stack([(f * prim[:, 1:4]).sum(-1) for f in fr], 1)
        U = np.concatenate([prim[:, :1], prim[:, :1] * rot,
                            (2.5 * prim[:, 4] + 0.5 * prim[:, 0] * (prim[:, 1:4] ** 2).sum(1))[:, None]], 1)
        beta = 0.5 * prim[:, 0] / prim[:, 4]
        q = np.empty((n, 5))
        q[:, 0] = np.log(prim[:, 0]) + 2.5 * np.log(beta) - beta * (prim[:, 1:4] ** 2).sum(1)
        q[:, 1:4] = 2 * beta[:, None] * prim[:, 1:4]
        q[:, 4] = -2 * beta
        qn = np.where(self.has[..., None], q[self.conn], q[:, None])
        qmax, qmin = qn.max(1), qn.min(1)
        M = np.einsum("nja,njb->nab", self.dx, self.dx)
        dq = np.einsum("nab,nbc->nca", np.linalg.inv(M), np.einsum("nja,njc->nac", self.dx, qn - q[:, None]))
        pk = prim[self.conn]
        dt = 5.0 * np.sqrt((self.dx ** 2).sum(-1)) / (np.sqrt((pk[..., 1:4] ** 2).sum(-1)) + 3 * np.sqrt(pk[..., 4] / pk[..., 0]))
        dt = np.minimum(np.where(self.has, dt, 1.0).min(1), 1.0)
        # flux residual and D_inv
        res, diag = np.zeros((n, 5)), np.zeros(n)
        snd = np.sqrt(1.4 * prim[:, 4] / prim[:, 0])
        for cls in range(3):
            p = np.flatnonzero(self.cls == cls)
            f = [v[p][:, None] for v in fr]
            for k in range(6):
                kind = _kind(cls, k)
                if kind is None:
                    continue
                j, on = self.idx[k, p], self.on[k, p]
                d = np.where(on[..., None], self.xyz[j] - self.xyz[p][:, None], 0.0)
                t = _flux(kind, self._recon(j, d, q, dq, qmax, qmin), f) - \
                    _flux(kind, self._recon(np.broadcast_to(p[:, None], j.shape), d, q, dq, qmax, qmin), f)
                res[p] += self._solve(k, p, t, on)
                g = np.einsum("pa,pa->p", self.row[k, p], self.w[k, p].sum(1))
                v = prim[p, 1 + k // 2]
                lam = np.maximum(v + snd[p], 0.0) if k % 2 == 0 else -np.maximum(snd[p] - v, 0.0)
                diag[p] += lam * g
            if cls == 1:
                res[p] *= 2.0
                diag[p] *= 2.0
        dinv = 1.0 / (1.0 / dt - diag)
        # sweeps: interior points read the neighbours' flux increments in the global axes
        eye = [np.eye(3)[a] for a in range(3)]
        flux6 = lambda P: np.stack([_flux(k, P, eye) for k in range(6)], 0)     # noqa: E731
        g_old = flux6(prim)
        d = delu.copy()
        for forward in (True, False):
            use, levels = self.dirs[0 if forward else 1]
            base = d.copy()
            inc = np.zeros((6, n, 5))
            fixed = np.flatnonzero(~self.swept)
            inc[:, fixed] = flux6(_to_prim(U[fixed] + d[fixed], [v[fixed] for v in fr])) - g_old[:, fixed]
            for pts in levels:
                for cls in (0, 1):
                    p = pts[self.cls[pts] == cls]
                    if not p.size:
                        continue
                    lu = np.zeros((p.size, 5))
                    f = [v[p][:, None] for v in fr]
                    for k in range(6):
                        kind = _kind(cls, k)
                        if kind is None:
                            continue
                        j, on = self.idx[k, p], use[k, p]
                        if cls == 0:
                            t = inc[k, j]
                        else:
                            t = _flux(kind, _to_prim(U[j] + d[j], [v[j] for v in fr]), f) - _flux(kind, prim[j], f)
                        lu += self._solve(k, p, t, on)
                    lu *= 2.0 if cls == 1 else 1.0
                    d[p] = -dinv[p, None] * (res[p] + lu) if forward else base[p] - dinv[p, None] * lu
                inc[:, pts] = flux6(_to_prim(U[pts] + d[pts], [v[pts] for v in fr])) - g_old[:, pts]
        # state update: outer points take the far field's half-range state
        out = self.cls == 2
        Un = U + d
        terms = []
        for P, sg in ((np.broadcast_to(self.inf, (int(out.sum()), 5)), -1.0), (prim[out], 1.0)):
            ur = np.stack([(f[out] * P[:, 1:4]).sum(-1) for f in fr], 1)
            b = 0.5 * P[:, 0] / P[:, 4]
            S = ur[:, 2] * np.sqrt(b)
            B = np.exp(-S * S) / (2 * np.sqrt(math.pi * b))
            A = 0.5 * (1 + sg * torch.erf(torch.from_numpy(S)).numpy())
            e = 2.5 * P[:, 4] + 0.5 * P[:, 0] * (ur ** 2).sum(1)
            rho = P[:, 0]
            terms.append(np.stack([rho * A, rho * ur[:, 0] * A, rho * ur[:, 1] * A, rho * (ur[:, 2] * A + sg * B),
                                   e * A + sg * 0.5 * rho * ur[:, 2] * B], 1))
        Un[out] = terms[0] + terms[1] + d[out]
        res_new = math.sqrt(float(((Un - U)[~out, 0] ** 2).sum())) / n
        return _to_prim(Un, fr), d, res_new

    def iterate(self, prim, iters):
        d = np.zeros_like(prim)
        hist, res_old = [], 0.0
        for t in range(1, iters + 1):
            prim, d, r = self.step(prim, d)
            if t <= 2:
                res_old, residue = r, 0.0
            else:
                residue = math.log10(r / res_old)
            hist.append((r, residue))
        return np.array(hist), prim, d


def _nearest(x, y, z):
    """Distance to the nearest neighbour of every point, by search over all."""
    p = torch.from_numpy(np.stack([x, y, z], 1)).cuda()
    best = torch.empty(len(x), dtype=torch.float64)
    for a in range(0, len(x), 256):
        d = (p[a:a + 256, None, :] - p[None]).square().sum(-1)
        d[torch.arange(d.shape[0]), torch.arange(a, a + d.shape[0])] = math.inf
        best[a:a + 256] = d.min(1).values.cpu()
    return best.sqrt().numpy()


def exact(case, seed):
    flows = _clouds(case, seed)
    points, iters = sum(c.n for c, _, _ in flows), case.get("iters", 1)
    # seconds: two sweeps of about 7 sqrt(n) levels at 2.4 ms, the rest 0.1 ms a point
    cost = sum(iters * (2 * 2.4e-3 * 7.0 * c.n ** 0.5 + 1e-4 * c.n) for c, _, _ in flows)
    if case["kind"] != "first" and cost > 18.0:
        return None
    out = {"history": [], "prim": [], "delu": []}
    if case["kind"] == "first":
        c, m, a = flows[0]
        out = {"nbhs": None, "conn": None, "min_dist": _nearest(c.x, c.y, c.z) if points < 300000 else None,
               "alias": None}
        small = cost < 18.0
        h, p, d = _Reference(c, m, a).iterate(cloud.initial_state(c, m, a), 1) if small else (None, None, None)
        out.update(history=h, prim=p, delu=d)
        return out
    for c, m, a in flows:
        h, p, d = _Reference(c, m, a).iterate(cloud.initial_state(c, m, a), iters)
        out["history"].append(h)
        out["prim"].append(p)
        out["delu"].append(d)
    if case["kind"] == "solve":
        return {k: v[0] for k, v in out.items()}
    return {"history": np.array(out["history"]), "prim": out["prim"], "delu": out["delu"]}
