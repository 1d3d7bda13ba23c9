"""Performance cases of the collision-operator library: what a user's program
asks of it, from the smallest hook call to a whole implicit step, each through
the public `collops` interface.

`listed()` are the fixed cases and `draw(rng)` gives further ones of the same
ranges; `prepare(case, seed)` makes what the program holds before the call
(markers, weights, the workspace of its mesh, a network); `run(state)` is one
call; `work(case)` the bytes and flops it cannot do without; `exact(case, seed)`
the result in plain 64-bit numpy/torch, where the call computes one directly
(the iterated solves have no such value).

Marker sets, meshes and solver settings are those of the repository's
configurations: the 16x16 mesh with 2,048 anisotropic Gaussian markers, the
32x32 mesh with 16,384 bimodal ones, the 64x64 mesh with 131,072, and the
default SimParameters (10,000 markers, a graded mesh, dt = 0.001).
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "collisionoperators.jl_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

N_QUAD = 6


def listed():
    return [
        # the projection hook (L2PROJ_FN) at the smallest configuration: a call of
        # a few microseconds of work, once per map and once per diagnostic
        dict(name="project_2k", kind="project", N=2048, n=16, half=6.0, sx=1.0, sy=0.5, peak=0.0),
        # one Landau Picard map of the smallest configuration (FP64, Gonzalez)
        dict(name="map_landau_2k", kind="map", model="landau", precision="fp64", logsq=False,
             N=2048, n=16, half=6.0, sx=1.0, sy=0.5, peak=0.0, dt=0.05),
        # one LB Picard map of the bimodal configuration
        dict(name="map_lb_16k", kind="map", model="lb", precision="fp64", logsq=False, N=16384,
             n=32, half=8.0, sx=math.sqrt(0.5), sy=math.sqrt(0.5), peak=2.0, dt=0.05),
        # the same markers under the Landau operator
        dict(name="map_landau_16k", kind="map", model="landau", precision="fp64", logsq=False,
             N=16384, n=32, half=8.0, sx=math.sqrt(0.5), sy=math.sqrt(0.5), peak=2.0, dt=0.05),
        # F and the metric A (COLLMETRIC_FN) of the default parameters: graded
        # mesh, a marker count that fills no tile evenly
        dict(name="metric_10k", kind="metric", N=10000, n=0, half=6.0, sx=4 / 3, sy=0.5, peak=0.0),
        # the gpu_fp32 collision hook at an odd marker count, unequal weights
        dict(name="collision32_50k", kind="collision32", N=50021, n=48, half=6.0, sx=1.1, sy=0.6,
             peak=0.0, weights="random"),
        # the plain FP64 collision hook (COLLISION_FN) at the largest configuration
        dict(name="collision_131k", kind="collision", N=131072, n=64, half=6.0, sx=1.0, sy=0.5,
             peak=0.0, weights="equal"),
        # the FP64-accurate map of the mixed precision form at the same size
        dict(name="map_ds_131k", kind="map", model="landau", precision="mixed_ds", logsq=True,
             N=131072, n=64, half=6.0, sx=1.0, sy=0.5, peak=0.0, dt=0.02),
        # one implicit step of the default parameters (step_anderson!, FP64)
        dict(name="step_10k", kind="step", N=10000, n=0, half=6.0, sx=4 / 3, sy=0.5, peak=0.0,
             dt=0.001),
        # one whole learned step (predictor, network, mixed defect correction) at a
        # time step of the production presets
        dict(name="step_learned_131k", kind="learned", N=131072, n=64, half=6.0, sx=1.0, sy=0.5,
             peak=0.0, dt=0.001),
        # a batched step of independent ensembles of uneven sizes, half of them LB
        dict(name="batch_8", kind="batch", count=8, N=1500, N_max=9000, n=16, dt=0.005),
        # training of the warm-start network: one Adam step on a minibatch
        dict(name="train_8192", kind="train", N=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A further case: kind, marker count (log-uniform over its range, any
    residue), mesh, distribution and weights drawn independently."""
    kind = rng.choice(["project", "map", "map", "map_lb", "map_ds", "metric", "collision",
                       "collision", "collision32", "step", "batch", "train", "learned"])
    c = dict(kind=kind, N=0, n=rng.randint(12, 64), half=rng.choice([6.0, 8.0]),
             sx=rng.uniform(0.5, 1.3), sy=rng.uniform(0.45, 1.2),
             peak=rng.choice([0.0, 0.0, 2.0]))
    if c["peak"]:
        c["half"] = 8.0
    if kind == "project":
        c["N"] = _log_int(rng, 500, 262144)
    elif kind in ("map", "map_lb", "map_ds"):
        lo, hi = {"map": (600, 65536), "map_lb": (600, 262144), "map_ds": (600, 131072)}[kind]
        c.update(kind="map", model="lb" if kind == "map_lb" else "landau",
                 precision="mixed_ds" if kind == "map_ds" else "fp64",
                 logsq=kind == "map_ds", N=_log_int(rng, lo, hi), dt=rng.choice([0.02, 0.05]))
    elif kind == "metric":
        c["N"] = _log_int(rng, 600, 32768)
    elif kind == "collision":
        c.update(N=_log_int(rng, 600, 131072), weights=rng.choice(["equal", "random"]))
    elif kind == "collision32":
        c.update(N=_log_int(rng, 1100, 131072), weights=rng.choice(["equal", "random"]))
    elif kind == "step":
        c.update(N=_log_int(rng, 2000, 12000), n=0, half=6.0, peak=0.0, sx=rng.uniform(1.0, 4 / 3),
                 sy=rng.uniform(0.5, 0.8), dt=0.001)
    elif kind == "learned":
        c.update(N=_log_int(rng, 20000, 131072), n=rng.randint(32, 64), half=6.0, peak=0.0,
                 sx=rng.uniform(0.9, 1.1), sy=rng.uniform(0.5, 0.7), dt=0.001)
    elif kind == "batch":
        c = dict(kind="batch", count=rng.randint(4, 12), N=rng.randint(600, 2500),
                 N_max=rng.randint(4000, 10000), n=rng.randint(14, 20), dt=0.005)
    elif kind == "train":
        c = dict(kind="train", N=_log_int(rng, 1000, 32768))
    return c


# ------------------------------------------------------------------ inputs

def _breaks(c):
    if c["n"] == 0:      # the graded mesh of the default SimParameters
        return (np.concatenate([[-6.0, -5.0], np.linspace(-4.0, 4.0, 17), [5.0, 6.0]]),
                np.concatenate([[-6.0], np.linspace(-2.5, 2.5, 13), [6.0]]))
    b = np.linspace(-c["half"], c["half"], c["n"] + 1)
    return b, b


def _markers(c, rng):
    N = c["N"]
    v = np.zeros((N, 2), order="F")
    v[:, 0] = c["sx"] * rng.standard_normal(N)
    if c["peak"]:
        v[:, 0] += np.where(np.arange(N) < N // 2, -c["peak"], c["peak"])
    v[:, 1] = c["sy"] * rng.standard_normal(N)
    if c.get("weights") == "random":
        w = rng.uniform(0.2, 1.8, N)
        w /= w.sum()
    else:
        w = np.full(N, 1.0 / N)
    return v, w


def _inputs(c, seed):
    """Everything a call takes, as host arrays from the seed alone."""
    rng = np.random.default_rng(seed)
    kind = c["kind"]
    d = {}
    if kind == "train":
        B = c["N"]
        d["X"] = rng.standard_normal((B, 15)).astype(np.float32)
        a = rng.standard_normal((15, 2)) * 0.4
        d["T"] = (np.tanh(d["X"] @ a) + 0.3 * rng.standard_normal((B, 2))).astype(np.float32)
        p = []
        for i, o in ((15, 64), (64, 64), (64, 64), (64, 2)):
            p += [rng.uniform(-1, 1, i * o) * math.sqrt(6.0 / i), 0.1 * rng.standard_normal(o)]
        d["params"] = np.concatenate(p).astype(np.float32)
        return d
    if kind == "batch":
        d["inst"], d["v"], d["w"] = [], [], []
        for k in range(c["count"]):
            t = k / max(1, c["count"] - 1)
            N = int(round(c["N"] * (c["N_max"] / c["N"]) ** t)) + 13 * (k % 5)
            n = c["n"] + 2 * (k % 4)
            sx, sy = rng.uniform(0.7, 1.1), rng.uniform(0.5, 1.0)
            b = np.linspace(-6.0, 6.0, n + 1)
            d["inst"].append(dict(bp1=b, bp2=b, model="lb" if k % 2 else "landau",
                                  nu=rng.uniform(0.5, 2.0), N=N))
            d["v"].append(np.stack([sx * rng.standard_normal(N), sy * rng.standard_normal(N)]))
            d["w"].append(np.full(N, 1.0 / N))
        return d
    v, w = _markers(c, rng)
    d["v"], d["w"] = v, w
    if kind in ("collision", "collision32", "metric"):
        # the entropy gradient of a near-Gaussian density with sampling noise
        s2 = np.array([c["sx"] ** 2 + c["peak"] ** 2, c["sy"] ** 2])
        G = -v / s2 + 0.2 * np.sin(2.0 * v[:, ::-1]) + 0.05 * rng.standard_normal(v.shape)
        d["G"] = np.asfortranarray(G)
    if kind == "map":
        # v_in: a predictor's guess, O(dt) away
        d["v_in"] = np.asfortranarray(v + c["dt"] * (-0.3 * v + 0.1 * rng.standard_normal(v.shape)))
    if kind in ("map", "step", "learned"):
        m = _Mesh(c)
        d["S0"] = m.entropy(m.project(v, w), c.get("logsq", kind == "learned"))
    return d


def prepare(c, seed):
    import collops
    from collops import learned

    d = _inputs(c, seed)
    kind, N = c["kind"], c["N"]
    s = dict(kind=kind, case=c, api=collops)
    if kind == "train":
        s["mlp"] = learned.MLP(seed=0)
        s["mlp"].set_params(d["params"])
        s["X"], s["T"] = torch.from_numpy(d["X"]).cuda(), torch.from_numpy(d["T"]).cuda()
        return s
    if kind == "batch":
        s["batch"] = collops.Batch(d["inst"])
        s["opts"] = collops.SimParameters(m_anderson=5, damping=0.7, tol=1e-12, abs_floor=0.0,
                                          max_iter=400, use_gonzalez=False).opts()
        s["v"] = torch.from_numpy(np.concatenate([x.reshape(-1) for x in d["v"]])).cuda()
        s["w"] = torch.from_numpy(np.concatenate(d["w"])).cuda()
        s["S0"] = np.zeros(c["count"])      # only the Gonzalez form reads it
        s["v1"] = torch.empty_like(s["v"])
        return s
    bp1, bp2 = _breaks(c)
    if kind == "learned":
        p = collops.SimParameters(bp1=bp1, bp2=bp2, use_logsq=True, precision="mixed_ds", tol=1e-12,
                                  abs_floor=1e-10, stag_window=50, stag_rel_tol=0.01, max_iter=400)
        s["warm"] = learned.WarmStart.load(os.path.join(PKG, "collops", "warmstart_c3.npz"),
                                           relax=0.75)
        s["opts"] = p.opts()
        s["dopt"] = collops.CoDefectOpts(0.02, 100, 5, 0.9, 0, 0, 0, 1e-3, 0, 0, 2)
        s["x"] = torch.from_numpy(np.ascontiguousarray(d["v"].T)).cuda()
        s["w"] = torch.from_numpy(d["w"]).cuda()
        s["v1"] = torch.empty_like(s["x"])
    else:
        p = collops.SimParameters(bp1=bp1, bp2=bp2, collision_model=c.get("model", "landau"),
                                  use_logsq=bool(c.get("logsq", False)),
                                  gpu_fp32=kind == "collision32")
        s.update(d)
    s["S0"] = d.get("S0")
    s["ws"] = collops.build_workspace(p)
    if kind == "project":
        s["f"] = np.zeros(s["ws"].n_dofs)
    else:
        s["out"] = np.zeros((N, 2), order="F")
        s["A"] = np.zeros((N, 3), order="F")
    return s


def run(s):
    api, c, kind = s["api"], s["case"], s["kind"]
    if kind == "project":
        api.l2_project_gpu(s["ws"], s["f"], s["v"], s["w"])
        return s["f"]
    if kind == "collision":
        api.compute_collision_gpu(s["ws"], s["out"], s["v"], s["w"], s["G"])
        return s["out"]
    if kind == "collision32":
        api.compute_collision_gpu32(s["ws"], s["out"], s["v"], s["w"], s["G"])
        return s["out"]
    if kind == "metric":
        api.compute_collision_metric_gpu(s["ws"], s["out"], s["A"], s["v"], s["w"], s["G"])
        return [s["out"], s["A"]]
    if kind == "map":
        api.picard_map(s["ws"], s["out"], s["v_in"], s["v"], s["w"], s["S0"], c["dt"],
                       precision=c["precision"])
        return s["out"]
    if kind == "step":
        # the time loop of the default parameters: explicit predictor, then the
        # implicit solve from it
        api.predictor(s["ws"], s["out"], s["v"], s["w"], c["dt"])
        p = s["ws"].p
        api.step_anderson(s["ws"], s["out"], s["v"], s["w"], s["S0"], c["dt"], m=p.m_anderson,
                          max_iter=p.max_iter, tol=p.tol, abs_floor=p.abs_floor, damping=p.damping)
        return s["out"]
    if kind == "learned":
        rec = s["warm"].step(s["ws"], s["opts"], s["dopt"], s["x"], s["w"], s["S0"], c["dt"],
                             s["v1"])
        return [s["v1"], rec["S_new"]]
    if kind == "batch":
        s["batch"].predictor(s["opts"], s["v1"], s["v"], s["w"], c["dt"])
        s["batch"].step(s["opts"], s["v1"], s["v"], s["w"], s["S0"], c["dt"])
        return s["v1"]
    if kind == "train":
        loss = s["mlp"].train_step(s["X"], s["T"], 2e-3)
        return [loss, s["mlp"].get_params()]
    raise ValueError(kind)


# ------------------------------------------------------------------ work

def work(c):
    kind, N = c["kind"], c["N"]
    if kind == "train":
        P = 15 * 64 + 2 * 64 * 64 + 64 * 2
        return dict(bytes=4 * N * 17 + 4 * 9538 * 6, flops=6 * P * N)
    if kind == "batch":
        b = f = 0
        for k in range(c["count"]):
            n = c["N"] * (c["N_max"] / c["N"]) ** (k / max(1, c["count"] - 1))
            b += 56 * n
            f += 10 * (120 * n + (0 if k % 2 else 23 * n * n))   # about ten maps a step
        return dict(bytes=b, flops=f)
    nd = (c["n"] + 2) ** 2 if c["n"] else 23 * 16
    chain = 120 * N + 4 * nd * (2 * math.sqrt(nd))
    pair = 23.0 * N * N
    if kind == "project":
        return dict(bytes=24 * N + 8 * nd, flops=40 * N + 4 * nd * math.sqrt(nd))
    if kind in ("collision", "collision32"):
        return dict(bytes=56 * N, flops=pair)
    if kind == "metric":
        return dict(bytes=80 * N, flops=35.0 * N * N)
    if kind == "map":
        return dict(bytes=56 * N, flops=chain + (0 if c["model"] == "lb" else pair))
    # whole solves: the predictor and about ten maps
    return dict(bytes=56 * N, flops=10 * (chain + pair))


# ------------------------------------------------------------------ exact values

class _Mesh:
    """The clamped C1 quadratic spline space and its L2 projection in plain
    64-bit numpy: local basis per cell, dense 1D mass matrices, Gauss rule."""

    def __init__(self, c):
        self.bp = _breaks(c)
        x, w = np.polynomial.legendre.leggauss(N_QUAD)
        self.xq, self.wq = 0.5 * (x + 1.0), 0.5 * w
        x3, w3 = np.polynomial.legendre.leggauss(3)
        x3, w3 = 0.5 * (x3 + 1.0), 0.5 * w3
        self.n = [len(b) - 1 for b in self.bp]
        self.nd = [n + 2 for n in self.n]
        self.h, self.cl, self.cr, self.M, self.Bq = [], [], [], [], []
        for b in self.bp:
            h = np.diff(b)
            hl, hr = np.concatenate([[0.0], h[:-1]]), np.concatenate([h[1:], [0.0]])
            self.h.append(h)
            self.cl.append(h / (hl + h))
            self.cr.append(h / (h + hr))
        for d in range(2):
            e = np.arange(self.n[d])
            M = np.zeros((self.nd[d], self.nd[d]))
            for q in range(3):
                p = self.basis(d, e, np.full(len(e), x3[q]))[0]
                for a in range(3):
                    for b in range(3):
                        np.add.at(M, (e + a, e + b), p[a] * p[b] * w3[q] * self.h[d])
            self.M.append(M)
            self.Bq.append(np.stack([self.basis(d, e, np.full(len(e), x))[0] for x in self.xq], -1))

    def basis(self, d, e, x):
        """(3, n) values and reference derivatives of the cell's basis functions."""
        cl, cr = self.cl[d][e], self.cr[d][e]
        om = 1.0 - x
        p0, p2 = cl * om * om, cr * x * x
        q0, q2 = -2.0 * cl * om, 2.0 * cr * x
        return np.stack([p0, 1.0 - p0 - p2, p2]), np.stack([q0, -q0 - q2, q2])

    def locate(self, v):
        inside = np.ones(len(v), bool)
        out = []
        for d in range(2):
            b, x = self.bp[d], v[:, d]
            inside &= (x > b[0]) & (x < b[-1])
            e = np.clip(np.searchsorted(b, x, side="right") - 1, 0, self.n[d] - 1)
            out.append((e, (x - b[e]) / self.h[d][e]))
        return inside, out

    def project(self, v, w):
        """Coefficients (nd1, nd2) of the L2 projection of sum_a w_a delta(v_a)."""
        inside, ((e1, x1), (e2, x2)) = self.locate(v)
        p1, p2 = self.basis(0, e1, x1)[0], self.basis(1, e2, x2)[0]
        rhs = np.zeros(self.nd[0] * self.nd[1])
        ww = np.where(inside, w, 0.0)
        for a in range(3):
            for b in range(3):
                rhs += np.bincount((e1 + a) * self.nd[1] + e2 + b, ww * p1[a] * p2[b],
                                   minlength=rhs.size)
        return self.solve(rhs.reshape(self.nd))

    def solve(self, r):
        return np.linalg.solve(self.M[1], np.linalg.solve(self.M[0], r).T).T

    def _quad(self, f):
        F = np.zeros((self.n[0], N_QUAD, self.n[1], N_QUAD))
        for a in range(3):
            for b in range(3):
                F += np.einsum("ij,ip,jq->ipjq", f[a:a + self.n[0], b:b + self.n[1]],
                               self.Bq[0][a], self.Bq[1][b])
        W = np.einsum("i,p,j,q->ipjq", self.h[0], self.wq, self.h[1], self.wq)
        return F, W

    def entropy(self, f, logsq):
        F, W = self._quad(f)
        ok = np.abs(F) > 1e-30 if logsq else F > 1e-30
        return float(-np.sum(np.where(ok, F * np.log(np.where(ok, np.abs(F), 1.0)), 0.0) * W))

    def r(self, f, logsq):
        F, W = self._quad(f)
        ok = np.abs(F) > 1e-30 if logsq else F > 1e-30
        I = np.where(ok, 1.0 + np.log(np.where(ok, np.abs(F), 1.0)), 0.0) * W
        r = np.zeros(self.nd)
        for a in range(3):
            for b in range(3):
                r[a:a + self.n[0], b:b + self.n[1]] += np.einsum("ipjq,ip,jq->ij", I,
                                                                 self.Bq[0][a], self.Bq[1][b])
        return r

    def evaluate(self, f, v):
        """f, its two derivatives at the markers, and who is inside."""
        inside, ((e1, x1), (e2, x2)) = self.locate(v)
        (p1, q1), (p2, q2) = self.basis(0, e1, x1), self.basis(1, e2, x2)
        val, d1, d2 = (np.zeros(len(v)) for _ in range(3))
        for a in range(3):
            for b in range(3):
                k = f[e1 + a, e2 + b]
                val += k * p1[a] * p2[b]
                d1 += k * q1[a] * p2[b]
                d2 += k * p1[a] * q2[b]
        return val, d1 / self.h[0][e1], d2 / self.h[1][e2], inside


def _pair_sum(v, w, G, inside, metric=False):
    """sum_a w_a U(v_g - v_a)(G_a - G_g), and the metric sum_a w_a U, in 64 bits
    over all ordered pairs of markers inside the domain."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    idx = np.nonzero(inside)[0]
    x, g = (torch.from_numpy(np.ascontiguousarray(a[idx].T)).to(dev) for a in (v, G))
    wt = torch.from_numpy(np.ascontiguousarray(w[idx])).to(dev)
    n = len(idx)
    F, A = torch.zeros(2, n, dtype=torch.float64), torch.zeros(3, n, dtype=torch.float64)
    step = max(1, (1 << 26) // max(n, 1))
    for i in range(0, n, step):
        s = slice(i, min(n, i + step))
        d1, d2 = x[0, s, None] - x[0], x[1, s, None] - x[1]
        r2 = d1 * d1 + d2 * d2
        r2 = torch.where(r2 < 1e-24, math.inf, r2)
        k = wt / (r2 * torch.sqrt(r2))
        c = (g[0] - g[0, s, None]) * d2 - (g[1] - g[1, s, None]) * d1
        F[0, s], F[1, s] = (k * c * d2).sum(1).cpu(), -(k * c * d1).sum(1).cpu()
        if metric:
            A[0, s], A[1, s] = (k * d2 * d2).sum(1).cpu(), -(k * d1 * d2).sum(1).cpu()
            A[2, s] = (k * d1 * d1).sum(1).cpu()
    out, am = np.zeros_like(v, order="F"), np.zeros((len(v), 3), order="F")
    out[idx], am[idx] = F.numpy().T, A.numpy().T
    return (out, am) if metric else out


def _exact_map(c, d):
    m = _Mesh(c)
    v0, v_in, w, dt = d["v"], d["v_in"], d["w"], c["dt"]
    vm, dv = 0.5 * (v0 + v_in), v_in - v0
    f = m.project(vm, w)
    dS = m.entropy(m.project(v_in, w), c["logsq"]) - d["S0"]
    if c["model"] == "lb":
        val, d1, d2, inside = m.evaluate(f, vm)
        inv = 1.0 / np.maximum(np.abs(val), 1e-30)
        g = np.clip(np.stack([d1 * inv, d2 * inv], 1), -100.0, 100.0) * inside[:, None]
        lam = (dS + np.sum(w[:, None] * dv * g)) / np.sum(dv * dv)
        g = g - lam * dv / w[:, None]
        M = np.array([[w.sum(), 0.0, w @ vm[:, 0]], [0.0, w.sum(), w @ vm[:, 1]],
                      [w @ vm[:, 0], w @ vm[:, 1], np.sum(w * (vm ** 2).sum(1))]])
        rhs = -np.array([w @ g[:, 0], w @ g[:, 1], np.sum(w * (vm * g).sum(1))])
        a = np.linalg.solve(M, rhs)
        return v0 - dt * (g + a[:2] + a[2] * vm)      # nu = 1
    L = m.solve(m.r(f, c["logsq"]))
    _, g1, g2, inside = m.evaluate(L, vm)
    G = np.stack([g1, g2], 1) * inside[:, None]
    lam = (dS + np.sum(w[:, None] * dv * G)) / np.sum(dv * dv)
    return v0 + dt * _pair_sum(vm, w, G - lam * dv / w[:, None], inside)


def _exact_train(d):
    """One Adam step of the network with BF16-rounded weights in the products."""
    p = torch.from_numpy(d["params"])
    X, T = torch.from_numpy(d["X"]).double(), torch.from_numpy(d["T"]).double()
    at, leaves, h = 0, [], X
    for k, (i, o) in enumerate(((15, 64), (64, 64), (64, 64), (64, 2))):
        W = p[at:at + i * o].bfloat16().double().reshape(o, i).requires_grad_()
        b = p[at + i * o:at + i * o + o].double().requires_grad_()
        at += i * o + o
        leaves += [W, b]
        h = h @ W.T + b
        if k < 3:
            h = torch.nn.functional.gelu(h)
    loss = ((h - T) ** 2).mean()
    loss.backward()
    g = torch.cat([x.grad.reshape(-1) for x in leaves])
    return [float(loss), (p.double() - 2e-3 * g / (g.abs() + 1e-8)).numpy()]


def exact(c, seed):
    kind = c["kind"]
    if kind in ("step", "learned", "batch"):
        return None
    d = _inputs(c, seed)
    if kind == "train":
        return _exact_train(d)
    if kind == "project":
        return np.ascontiguousarray(_Mesh(c).project(d["v"], d["w"]).T).reshape(-1)
    if kind == "map":
        return np.asfortranarray(_exact_map(c, d))
    inside = _Mesh(c).locate(d["v"])[0]
    if kind == "metric":
        F, A = _pair_sum(d["v"], d["w"], d["G"], inside, metric=True)
        return [F, A]
    return _pair_sum(d["v"], d["w"], d["G"], inside)
