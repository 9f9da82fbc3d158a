"""The workloads that the framework's speed is measured on, through its public entry points.

Each case is one call that a Graph-SLAM program makes over and over:
  city     a Gauss-Newton round of an SE(2) pose graph (odometry and loop closures of a
           city-grid walk), host poses in and out (PoseGraph.round_io)
  log      the same round of a reference-format landmark log (ObsEdge / MotionEdge factors)
  batch    a round of many independent graphs on one handle (PoseGraphBatch)
  adjoint  the implicit-function gradient of an SE(2) graph (PoseGraph.adjoint)
  dense    the dense Gauss-Jordan solve of a small graph's system (gslam_gj_solve)
Solver settings are the library's defaults (tolerance 1e-6, at most 500 PCG iterations per
round: the reference's) unless the case says otherwise.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

G = importlib.import_module("g-slam_on_gpu_and_fpga_b200")

MAX_ITER, TOL = 500, 1e-6
ANCHOR = 1e6
MAX_POSES, MAX_BATCH_POSES = 100_000, 300_000


def listed():
    return [
        # a short log on the reference's factors, library defaults: the smallest call, all
        # latency
        {"name": "log-100", "kind": "log", "n": 100, "lam": 0.1, "precision": 0, "round_graph": False},
        # an ordinary log: landmark cliques make rows of many blocks
        {"name": "log-2k", "kind": "log", "n": 2001, "lam": 0.1, "precision": 0, "round_graph": False},
        # the size of Victoria Park as an SE(2) graph with far closures
        {"name": "city-7k", "kind": "city", "n": 7120, "k": 6, "radius": 3.0, "far": 0.02, "lam": 1.0,
         "precision": 0, "round_graph": True},
        # a district map
        {"name": "city-20k", "kind": "city", "n": 20_000, "k": 3, "radius": 2.0, "far": 0.0, "lam": 0.1,
         "precision": 0, "round_graph": True},
        # large maps: the reference's recurrence, the one-reduction FP64 solver and the
        # mixed-precision one
        {"name": "city-50k", "kind": "city", "n": 50_000, "k": 3, "radius": 2.0, "far": 0.0, "lam": 0.1,
         "precision": 0, "round_graph": True},
        {"name": "city-100k", "kind": "city", "n": 100_000, "k": 3, "radius": 2.0, "far": 0.0, "lam": 0.1,
         "precision": 0, "round_graph": True},
        {"name": "city-100k-one-reduction", "kind": "city", "n": 100_000, "k": 3, "radius": 2.0, "far": 0.0,
         "lam": 0.1, "precision": 2, "round_graph": True},
        {"name": "city-100k-mixed", "kind": "city", "n": 100_000, "k": 3, "radius": 2.0, "far": 0.0, "lam": 0.1,
         "precision": 1, "round_graph": True},
        # many maps at once (48 sizes, one map at 16 lambdas), in FP64 and mixed precision
        {"name": "batch-64", "kind": "batch", "graphs": 48, "sweep": 16, "n_lo": 500, "n_hi": 20_000, "n_sweep": 5000,
         "precision": 0},
        {"name": "batch-64-mixed", "kind": "batch", "graphs": 48, "sweep": 16, "n_lo": 500, "n_hi": 20_000,
         "n_sweep": 5000, "precision": 1},
        # learning the edge weights: the backward pass after a Gauss-Newton run
        {"name": "adjoint-10k", "kind": "adjoint", "n": 10_000, "lam": 0.5},
        # the dense check of an 800-pose graph
        {"name": "dense-2400", "kind": "dense", "n": 800, "lam": 0.1},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["city"] * 5 + ["log"] * 2 + ["batch"] * 2 + ["adjoint", "dense"])
    lam = rng.choice([0.06, 0.1, 0.5, 1.0])
    if kind == "city":
        far = rng.choice([0.0, 0.0, 0.02])
        return {"kind": kind, "n": _log_uniform(rng, 100, MAX_POSES), "k": rng.choice([2, 3, 6]),
                "radius": rng.choice([2.0, 3.0]), "far": far, "lam": lam, "precision": rng.choice([0, 0, 0, 1, 2]),
                "round_graph": rng.random() < 0.7}
    if kind == "log":
        return {"kind": kind, "n": _log_uniform(rng, 100, 20_000), "lam": lam, "precision": 0,
                "round_graph": rng.random() < 0.5}
    if kind == "batch":
        graphs, sweep = rng.randint(2, 48), rng.choice([0, 0, 4, 16])
        n_hi = _log_uniform(rng, 600, 20_000)
        return {"kind": kind, "graphs": graphs, "sweep": sweep, "n_lo": rng.randint(100, 500), "n_hi": n_hi,
                "n_sweep": rng.randint(500, 5000), "precision": rng.choice([0, 0, 1])}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_uniform(rng, 300, 20_000), "lam": lam}
    return {"kind": kind, "n": rng.randint(60, 800), "lam": lam}


# ---------------------------------------------------------------------------- inputs


def _city(case, seed):
    return G.synth.city_grid(case["n"], seed=seed, k_closures=case.get("k", 3), radius=case.get("radius", 2.0),
                             far_fraction=case.get("far", 0.0))


def _learning_map(case, seed):
    """One map (walk and closures) whose measurements are new with every seed, and poses near
    the optimum, as a finished Gauss-Newton run leaves them."""
    c = G.synth.city_grid(case["n"], seed=1)
    rng = np.random.default_rng(seed)
    sigma = np.array([0.05, 0.05, 0.01])
    meas = c.meas + rng.normal(size=c.meas.shape) * sigma
    poses = c.gt + 0.2 * rng.normal(size=c.gt.shape) * sigma
    return c, meas, poses, rng.normal(size=c.gt.shape)


def _batch_graphs(case, seed):
    """The batch's graphs and lambdas: log-uniform sizes, then one graph at several lambdas."""
    rng = np.random.default_rng(case["graphs"])
    sizes = np.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), case["graphs"])).astype(int)
    while sizes.sum() + case["sweep"] * case["n_sweep"] > MAX_BATCH_POSES:
        sizes = np.maximum(case["n_lo"], sizes * 9 // 10)
    graphs = [G.synth.city_grid(int(n), seed=1000 * (seed % 100_000) + q) for q, n in enumerate(sizes)]
    lams = [0.1] * case["graphs"]
    if case["sweep"]:
        graphs += [G.synth.city_grid(case["n_sweep"], seed=1000 * (seed % 100_000) + 999)] * case["sweep"]
        lams += list(np.geomspace(0.01, 10.0, case["sweep"]))
    return graphs, lams


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a, np.float64))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _pinned_like(a):
    return _pinned(np.zeros_like(a))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dense":
        A, b = _dense_system(case, seed)
        A, b = A.cuda(), b.cuda()
        return {"kind": kind, "A": A, "b": b, "x": torch.empty_like(b)}
    if kind == "adjoint":
        c, meas, poses, grad = _learning_map(case, seed)
        g = G.PoseGraph.from_se2(poses, c.edge_i, c.edge_j, meas, c.log_w, case["lam"])
        return {"kind": kind, "graph": g, "grad": grad}
    if kind == "log":
        log = G.synth.landmark_log(case["n"], seed=seed)
        g = G.PoseGraph.from_log(log, case["lam"], precision=case["precision"], round_graph=int(case["round_graph"]))
        start = log.x
    elif kind == "city":
        c = _city(case, seed)
        g = G.PoseGraph.from_se2(c.init, c.edge_i, c.edge_j, c.meas, c.log_w, case["lam"], precision=case["precision"],
                                 round_graph=int(case["round_graph"]))
        start = c.init
    else:
        graphs, lams = _batch_graphs(case, seed)
        opts = {"inner_tol": 1e-5} if case["precision"] == 1 else {}
        g = G.PoseGraphBatch.from_se2_list(graphs, lams, precision=case["precision"], **opts)
        start = g.init_poses
    return {"kind": kind, "graph": g, "in": _pinned(start), "out": _pinned_like(start)}


def run(state):
    kind = state["kind"]
    if kind == "dense":
        A, b, x = state["A"], state["b"], state["x"]
        n = A.shape[0]
        G.abi.check(G.abi.lib().gslam_gj_solve(n, ctypes.c_void_p(A.data_ptr()), n, ctypes.c_void_p(b.data_ptr()),
                                               ctypes.c_void_p(x.data_ptr()),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), None))
        return x
    if kind == "adjoint":
        d_lam, d_log_w, mu, _ = state["graph"].adjoint(state["grad"])
        return {"d_lam": d_lam, "d_log_w": d_log_w, "mu": mu}
    state["graph"].round_io(state["in"], state["out"])
    return state["out"]


# ---------------------------------------------------------------------------- work


def _counts(case):
    """(poses, edges, 3x3 blocks) of a case, about: a walk has N - 1 odometry edges and some
    closures per pose, a landmark log the cliques of its landmarks."""
    n = case["n"] if "n" in case else 0
    if case["kind"] == "log":
        e = 2 * n
    elif case["kind"] == "batch":
        lo, hi = case["n_lo"], max(case["n_hi"], case["n_lo"] + 1)
        n = int(case["graphs"] * (hi - lo) / math.log(hi / lo)) + case["sweep"] * case["n_sweep"]
        n = min(n, MAX_BATCH_POSES)
        e = int(1.4 * n)
    else:
        e = int((1.55 if case.get("k", 3) < 4 else 1.75) * n)
    return n, e, n + 2 * e


def work(case):
    if case["kind"] == "dense":
        n = 3 * case["n"]
        return {"bytes": 8.0 * (n * n + 2 * n), "flops": 2.0 * n ** 3}
    n, e, nb = _counts(case)
    per_iter = 18 * nb + 18 * n + 2 * 15 * n   # A p, D^-1 r, the vector updates and products
    inputs = 8 * 3 * n + e * (8 + 48)
    outputs = 8 * 3 * n if case["kind"] != "adjoint" else 8 * (3 * n + 3 * e)
    return {"bytes": float(inputs + outputs), "flops": float(MAX_ITER) * per_iter + 250.0 * e}


# ---------------------------------------------------------------------------- exact values


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev()).to(dtype)


def _wrap(a):
    return torch.remainder(a + math.pi, 2 * math.pi) - math.pi


def _sum_at(n, index, values):
    out = torch.zeros((n,) + values.shape[1:], dtype=torch.float64, device=values.device)
    return out.index_add_(0, index, values)


def _se2_edges(poses, ei, ej, meas, w):
    """Jacobians and residuals of the SE(2) between-factors, and the weights: (Ji, Jj, e, w)."""
    xi, xj = poses[ei], poses[ej]
    s, c = torch.sin(xi[:, 2]), torch.cos(xi[:, 2])
    dx, dy = xj[:, 0] - xi[:, 0], xj[:, 1] - xi[:, 1]
    o, z = torch.ones_like(s), torch.zeros_like(s)
    r = torch.stack([c * dx + s * dy - meas[:, 0], c * dy - s * dx - meas[:, 1],
                     _wrap(xj[:, 2] - xi[:, 2] - meas[:, 2])], 1)
    Ji = torch.stack([-c, -s, c * dy - s * dx, s, -c, -c * dx - s * dy, z, z, -o], 1).view(-1, 3, 3)
    Jj = torch.stack([c, s, z, -s, c, z, z, z, o], 1).view(-1, 3, 3)
    return Ji, Jj, r, w


def _normal_blocks(Ji, Jj, r, W):
    """(UL, UR, BL, BR, xi of i, xi of j) of J^T W J dx = -J^T W r."""
    WJi, WJj, Wr = W @ Ji, W @ Jj, (W @ r[:, :, None])[:, :, 0]
    T = lambda m: m.transpose(1, 2)  # noqa: E731
    return (T(Ji) @ WJi, T(Ji) @ WJj, T(Jj) @ WJi, T(Jj) @ WJj,
            -(T(Ji) @ Wr[:, :, None])[:, :, 0], -(T(Jj) @ Wr[:, :, None])[:, :, 0])


def _log_edges(log, lam):
    """The reference's factors of a log at its recorded poses: (ei, ej, the six blocks)."""
    poses, z = _t(log.x), _t(log.z)
    step = _t(log.z_step.astype(np.int64), torch.int64)
    groups = {}
    for k, lm in enumerate(log.z_lm.tolist()):
        groups.setdefault(lm, []).append(k)
    pairs = [(g[a], g[b]) for g in groups.values() for a in range(len(g)) for b in range(a + 1, len(g))]
    pa, pb = (_t(np.array([p[q] for p in pairs], np.int64), torch.int64) for q in (0, 1))

    def seen(p):  # observed point, its covariance and its derivative by the pose
        x, (rng, brg) = poses[step[p]], z[p].unbind(1)
        s, c = torch.sin(x[:, 2] + brg), torch.cos(x[:, 2] + brg)
        R = torch.stack([c, -rng * s, s, rng * c], 1).view(-1, 2, 2)
        Q = torch.stack([(rng * 0.14) ** 2, torch.zeros_like(rng), torch.zeros_like(rng),
                         torch.full_like(rng, 0.05 ** 2)], 1).view(-1, 2, 2)
        o, n = torch.ones_like(s), torch.zeros_like(s)
        J = torch.stack([o, n, -rng * s, n, o, rng * c], 1).view(-1, 2, 3)
        return torch.stack([x[:, 0] + rng * c, x[:, 1] + rng * s], 1), R @ Q @ R.transpose(1, 2), J

    m1, S1, J1 = seen(pa)
    m2, S2, J2 = seen(pb)
    obs = _normal_blocks(-J1, J2, m2 - m1, torch.linalg.inv(S1 + S2))
    # motion factors between consecutive poses, controls of the later one
    u, dt = _t(log.u)[1:], float(log.delta)
    x1, x2 = poses[:-1], poses[1:]
    nu, om = u[:, 0], torch.where(u[:, 1].abs() < 1e-5, torch.full_like(u[:, 1], 1e-5), u[:, 1])
    mn = (0.19, 0.001, 0.13, 0.2)
    M = torch.zeros((len(nu), 2, 2), dtype=torch.float64, device=nu.device)
    M[:, 0, 0] = (mn[0] ** 2 * nu.abs() + mn[1] ** 2 * om.abs()) / dt
    M[:, 1, 1] = (mn[2] ** 2 * nu.abs() + mn[3] ** 2 * om.abs()) / dt
    st, ct = torch.sin(x1[:, 2]), torch.cos(x1[:, 2])
    sw, cw = torch.sin(x1[:, 2] + om * dt), torch.cos(x1[:, 2] + om * dt)
    zero = torch.zeros_like(nu)
    A = torch.stack([(sw - st) / om, nu / om * dt * cw - nu / om ** 2 * (sw - st),
                     (ct - cw) / om, nu / om * dt * sw - nu / om ** 2 * (ct - cw),
                     zero, torch.full_like(nu, dt)], 1).view(-1, 3, 2)
    F = torch.eye(3, dtype=torch.float64, device=nu.device).repeat(len(nu), 1, 1)
    F[:, 0, 2] = nu / om * (cw - ct)
    F[:, 1, 2] = nu / om * (sw - st)
    Sg = A @ M @ A.transpose(1, 2) + 1e-4 * torch.eye(3, dtype=torch.float64, device=nu.device)
    t = float(int(dt))
    moved = torch.stack([nu / om * (torch.sin(x1[:, 2] + om * t) - st), nu / om * (ct - torch.cos(x1[:, 2] + om * t)),
                         om * t], 1)
    I3 = torch.eye(3, dtype=torch.float64, device=nu.device).expand(len(nu), 3, 3)
    mot = _normal_blocks(-F, I3, x2 - (x1 + moved), lam * torch.linalg.inv(Sg))
    n = len(poses)
    seq = torch.arange(n - 1, device=nu.device)
    return (torch.cat([step[pa], seq]), torch.cat([step[pb], seq + 1]),
            tuple(torch.cat([a, b]) for a, b in zip(obs, mot)))


class _System:
    """Omega of a set of edge blocks, its block-Jacobi inverse and PCG, per graph."""

    def __init__(self, n, ei, ej, blocks, anchors, graph=None, n_graphs=1):
        self.n, self.ei, self.ej, self.graph, self.G = n, ei, ej, graph, n_graphs
        UL, self.UR, self.BL, BR, _, _ = blocks
        self.D = _sum_at(n, ei, UL) + _sum_at(n, ej, BR)
        for row, a in anchors:
            self.D[row] += a * torch.eye(3, dtype=torch.float64, device=self.D.device)
        self.Dinv = torch.linalg.inv(self.D)

    def apply(self, p):
        q = (self.D @ p[:, :, None])[:, :, 0]
        q.index_add_(0, self.ei, (self.UR @ p[self.ej][:, :, None])[:, :, 0])
        return q.index_add_(0, self.ej, (self.BL @ p[self.ei][:, :, None])[:, :, 0])

    def dot(self, a, b):
        v = (a * b).sum(1)
        return v.sum()[None] if self.graph is None else _sum_at(self.G, self.graph, v)

    def rows(self, s):
        return s[:, None] if self.graph is None else s[self.graph][:, None]

    def solve(self, b):
        x, r = torch.zeros_like(b), b.clone()
        z = (self.Dinv @ r[:, :, None])[:, :, 0]
        p, rz, tol = z.clone(), self.dot(r, z), TOL * self.dot(b, b).sqrt()
        live = self.dot(r, r).sqrt() >= tol
        for _ in range(MAX_ITER):
            q = self.apply(p)
            pq = self.dot(p, q)
            alpha = torch.where(live & (pq != 0), rz / pq, torch.zeros_like(pq))
            x += self.rows(alpha) * p
            r -= self.rows(alpha) * q
            z = (self.Dinv @ r[:, :, None])[:, :, 0]
            live = live & (self.dot(r, r).sqrt() >= tol)
            rz_new = self.dot(r, z)
            p = z + self.rows(torch.where(live, rz_new / rz, torch.zeros_like(rz))) * p
            rz = rz_new
        return x


def _dense_system(case, seed):
    """Omega and xi of a small graph at its initial guess, as dense matrices."""
    c = _city(case, seed)
    poses = torch.from_numpy(np.ascontiguousarray(c.init))
    ei, ej = torch.from_numpy(c.edge_i.astype(np.int64)), torch.from_numpy(c.edge_j.astype(np.int64))
    Ji, Jj, r, w = _se2_edges(poses, ei, ej, torch.from_numpy(c.meas), torch.from_numpy(np.exp(c.log_w)) * case["lam"])
    UL, UR, BL, BR, bi, bj = _normal_blocks(Ji, Jj, r, torch.diag_embed(w))
    n = case["n"]
    A = torch.zeros((n * n, 3, 3), dtype=torch.float64)
    for a, b, blk in ((ei, ei, UL), (ei, ej, UR), (ej, ei, BL), (ej, ej, BR)):
        A.index_add_(0, a * n + b, blk)
    A = A.view(n, n, 3, 3).permute(0, 2, 1, 3).reshape(3 * n, 3 * n).contiguous()
    A[:3, :3] += ANCHOR * torch.eye(3, dtype=torch.float64)
    b = (_sum_at(n, ei, bi) + _sum_at(n, ej, bj)).reshape(-1)
    return A, b


def exact(case, seed):
    kind = case["kind"]
    if kind == "dense":
        A, b = _dense_system(case, seed)
        x = torch.linalg.solve(A, b)
        for _ in range(3):
            x = x + torch.linalg.solve(A, b - A @ x)
        return x
    if kind == "log":
        log = G.synth.landmark_log(case["n"], seed=seed)
        ei, ej, blocks = _log_edges(log, case["lam"])
        S = _System(case["n"], ei, ej, blocks, [(0, ANCHOR)])
        b = _sum_at(S.n, ei, blocks[4]) + _sum_at(S.n, ej, blocks[5])
        return (_t(log.x) + S.solve(b)).cpu().numpy()
    if kind == "batch":
        graphs, lams = _batch_graphs(case, seed)
        off = np.concatenate([[0], np.cumsum([(g.n_poses + 31) // 32 * 32 for g in graphs])])
        n = int(off[-1])
        poses = np.zeros((n, 3))
        graph = np.zeros(n, np.int64)
        anchors = []
        for q, g in enumerate(graphs):
            poses[off[q]:off[q] + g.n_poses] = g.init
            graph[off[q]:off[q + 1]] = q
            anchors.append((int(off[q]), ANCHOR))
            anchors.append((slice(int(off[q]) + g.n_poses, int(off[q + 1])), 1.0))
        ei = np.concatenate([g.edge_i.astype(np.int64) + off[q] for q, g in enumerate(graphs)])
        ej = np.concatenate([g.edge_j.astype(np.int64) + off[q] for q, g in enumerate(graphs)])
        meas = np.concatenate([g.meas for g in graphs])
        w = np.concatenate([np.exp(g.log_w) * lam for g, lam in zip(graphs, lams)])
        per_graph = {"graph": _t(graph, torch.int64), "n_graphs": len(graphs)}
    else:
        if kind == "city":
            c = _city(case, seed)
            meas, poses = c.meas, c.init
        else:
            c, meas, poses, grad = _learning_map(case, seed)
        n, ei, ej = case["n"], c.edge_i.astype(np.int64), c.edge_j.astype(np.int64)
        w, anchors, per_graph = np.exp(c.log_w) * case["lam"], [(0, ANCHOR)], {}
    poses, ei, ej, meas, w = _t(poses), _t(ei, torch.int64), _t(ej, torch.int64), _t(meas), _t(w)
    Ji, Jj, r, w = _se2_edges(poses, ei, ej, meas, w)
    blocks = list(_normal_blocks(Ji, Jj, r, torch.diag_embed(w)))
    if kind != "adjoint":
        S = _System(n, ei, ej, blocks, anchors, **per_graph)
        b = _sum_at(n, ei, blocks[4]) + _sum_at(n, ej, blocks[5])
        return (poses + S.solve(b)).cpu().numpy()
    # the exact Hessian: the second derivatives of the residuals, which involve theta of pose i
    s, cs = torch.sin(poses[ei, 2]), torch.cos(poses[ei, 2])
    d = poses[ej] - poses[ei]
    a0, a1 = w[:, 0] * r[:, 0], w[:, 1] * r[:, 1]
    h_tt = -a0 * (cs * d[:, 0] + s * d[:, 1]) + a1 * (s * d[:, 0] - cs * d[:, 1])
    h_t = torch.stack([a0 * s + a1 * cs, a1 * s - a0 * cs], 1)
    for blk, row, sign in ((0, 2, 1), (1, 2, -1)):
        blocks[blk][:, row, :2] += sign * h_t
    for blk, col, sign in ((0, 2, 1), (2, 2, -1)):
        blocks[blk][:, :2, col] += sign * h_t
    blocks[0][:, 2, 2] += h_tt
    S = _System(n, ei, ej, blocks, anchors)
    mu = S.solve(_t(grad))
    jm = (Ji @ mu[ei][:, :, None] + Jj @ mu[ej][:, :, None])[:, :, 0]
    d_log_w = -w * r * jm
    return {"d_lam": float(d_log_w.sum() / case["lam"]), "d_log_w": d_log_w.cpu().numpy(), "mu": mu.cpu().numpy()}
