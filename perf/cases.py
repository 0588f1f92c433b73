"""Timed cases: what programs built on this package have it do.

Every case is one call sequence of a user's program through the public entry
points: the LSRK45 time loop of an affine problem with its state copied in
and out (the reference's WaveSetData3d / Wave_RK / WaveGetData3d pattern),
single stages on a tiny mesh, batched shots with sources and receivers, the
forward + adjoint gradient, the curvilinear loop, and the three kernel-level
launches of a stage on device arrays.

A case is a dict: ``kind`` ("steps" | "stages" | "shots" | "adjoint" |
"curved" | "kernels"), polynomial degree ``N``, mesh size ``n`` (n^3 x 6
tetrahedra, Kuhn box or ball), cubature ``rule`` ("table": the reference's
rule, from the committed fixtures; "default": the package's own), ``steps``,
and for the affine kinds ``variant``, ``precision`` and ``bc``; ``shots`` and
``receivers`` where they apply.

Meshes, operators and node coordinates are built once per size (a user's
program has them on disk); the medium, the initial state, sources, receivers
and observed traces are made from the seed.
"""
import dataclasses
import functools
import math
import os

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from bbwadg_b200 import RK4A, RK4B, RK4C, WaveSolver, _lib, make_problem
from bbwadg_b200.curved import CurvedSolver, make_curved_problem
from bbwadg_b200.problem import gaussian_source, receiver_weights, source_entries

F0, AMPLITUDE = 4.0, 1e4  # Ricker peak frequency and amplitude of the shots


def listed():
    return [
        # single stages driven by the caller on a tiny mesh: launches and host calls
        dict(name="stages_n3_box4", kind="stages", N=3, n=4, rule="table", variant="nodal",
             precision="fp32", bc="pressure_release", steps=2),
        # the plain small run: N=3, 8^3 x 6, rigid walls, 100 steps
        dict(name="nodal_n3_box8", kind="steps", N=3, n=8, rule="table", variant="nodal",
             precision="fp32", bc="rigid", steps=100),
        # low order on an odd mesh with the package's own rule
        dict(name="nodal_n2_box25", kind="steps", N=2, n=25, rule="default", variant="nodal",
             precision="fp32", bc="pressure_release", steps=20),
        # the benchmark workload in its default (FP32) form ...
        dict(name="nodal_n5_box32", kind="steps", N=5, n=32, rule="table", variant="nodal",
             precision="fp32", bc="pressure_release", steps=20),
        # ... and in the split-FP16 form
        dict(name="f16x3_n5_box32", kind="steps", N=5, n=32, rule="table", variant="nodal",
             precision="f16x3", bc="pressure_release", steps=20),
        # the Bernstein-Bezier form at the middle size of the h-refinement
        dict(name="bb_n5_box24", kind="steps", N=5, n=24, rule="table", variant="bb",
             precision="fp32", bc="pressure_release", steps=20),
        # high order: the precision study's N=7, FP32
        dict(name="nodal_n7_box16", kind="steps", N=7, n=16, rule="table", variant="nodal",
             precision="fp32", bc="pressure_release", steps=10),
        # batched shots: N=4, Ricker sources, receivers recorded every step
        dict(name="shots8_n4_box16", kind="shots", N=4, n=16, rule="table", variant="nodal",
             precision="fp32", bc="pressure_release", steps=20, shots=8, receivers=64),
        # gradient of a receiver misfit: forward with tape, then the adjoint
        dict(name="adjoint8_n4_box16", kind="adjoint", N=4, n=16, rule="table", variant="nodal",
             precision="fp32", bc="pressure_release", steps=20, shots=8, receivers=64),
        # curvilinear path at the bench size, and a higher order on a small odd ball
        dict(name="curved_n3_ball24", kind="curved", N=3, n=24, rule="table", steps=20),
        dict(name="curved_n5_ball10", kind="curved", N=5, n=10, rule="table", steps=10),
        # a caller that launches the reference's three kernels itself
        dict(name="kernels_n5_box16", kind="kernels", N=5, n=16, rule="table", variant="nodal",
             precision="fp32", bc="pressure_release", steps=2),
    ]


def _np(N):
    return (N + 1) * (N + 2) * (N + 3) // 6


def _nfp(N):
    return (N + 1) * (N + 2) // 2


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "stages", "shots", "adjoint", "curved",
                       "kernels"])
    bc = rng.choice(["pressure_release", "pressure_release", "rigid"])
    if kind == "curved":
        N = rng.choice([2, 3, 3, 4, 5])
        n = 2 * _log_int(rng, 2, {2: 12, 3: 12, 4: 8, 5: 6}[N])
        return dict(kind=kind, N=N, n=n, rule="table" if N >= 3 else "default",
                    steps=rng.randint(5, 20))
    if kind == "stages":
        return dict(kind=kind, N=rng.randint(2, 6), n=rng.randint(1, 6), rule="default",
                    variant=rng.choice(["nodal", "nodal", "bb"]), precision="fp32", bc=bc,
                    steps=rng.randint(1, 4))
    if kind == "kernels":
        N = rng.randint(2, 6)
        return dict(kind=kind, N=N, n=_log_int(rng, 4, {2: 24, 3: 22, 4: 20, 5: 16, 6: 12}[N]),
                    rule="table" if N >= 3 else "default", variant="nodal", precision="fp32",
                    bc=bc, steps=rng.randint(1, 3))
    if kind in ("shots", "adjoint"):
        N = rng.choice([2, 3, 4, 4, 5])
        return dict(kind=kind, N=N, n=_log_int(rng, 6, {2: 18, 3: 16, 4: 14, 5: 10}[N]),
                    rule="table" if N >= 3 else "default",
                    variant=rng.choice(["nodal", "nodal", "bb"]),
                    precision=rng.choice(["fp32", "fp32", "f16x3"]), bc=bc,
                    steps=rng.randint(4, 16), shots=rng.randint(2, 8),
                    receivers=rng.randint(8, 64))
    precision = rng.choice(["fp32", "fp32", "fp32", "f16x3", "bf16x3"])
    N = rng.choice([2, 3, 4, 5, 5, 6, 7]) if precision == "fp32" else rng.randint(2, 5)
    return dict(kind=kind, N=N,
                n=_log_int(rng, 5, {2: 40, 3: 36, 4: 32, 5: 28, 6: 18, 7: 13}[N]),
                rule="table" if N >= 5 else "default" if N == 2 else rng.choice(["table", "default"]),
                variant=rng.choice(["nodal", "nodal", "bb"]), precision=precision, bc=bc,
                steps=rng.randint(6, 20))


# ------------------------------------------------------------------ inputs
def _rule(N, name):
    if name != "table":
        return None, None
    g = np.load(os.path.join("tests", "golden", "ops_N%d.npz" % N))
    m = int(g["Nfq"][0])
    return (g["rq"], g["sq"], g["tq"], g["wq"]), (g["rfq"][:m], g["sfq"][:m], g["wfqFace"])


@functools.lru_cache(maxsize=3)
def _affine(N, n, rule, variant):
    """Mesh and operators; dt for c^2 <= 2; the smooth part of the medium."""
    cub, tri = _rule(N, rule)
    p = make_problem(N, n, variant=variant, c2="sine", ic=lambda x, y, z, t: 0.0 * x,
                     cubature=cub, tri_cubature=tri)
    fmax = float(p.mesh["fgeo"].reshape(p.K, 4, 4)[:, :, 0].max())
    p.dt = float(np.float32(0.25 / ((N + 1) ** 2 * fmax * math.sqrt(2.0))))
    return p


@functools.lru_cache(maxsize=3)
def _ball(N, n, rule):
    cub, tri = _rule(N, rule)
    return make_curved_problem(N, n, cubature=cub, tri_cubature=tri)


def _medium(p, seed):
    """Smooth field plus a jump per element, c^2 in (0.5, 2)."""
    jump = 0.5 * np.random.default_rng(seed).random((p.K, 1), np.float32)
    return np.ascontiguousarray(p.c2q.reshape(p.K, -1) + jump, np.float32)


def _initial(p, seed):
    """Nodal state: a Gaussian pulse off centre over smooth modes, in pinned memory."""
    rng = np.random.default_rng(seed + 1)
    x, y, z = (torch.from_numpy(p.mesh[c]).cuda() for c in ("x", "y", "z"))
    cx, cy, cz = rng.uniform(-0.3, 0.3, 3)
    a = rng.uniform(0.05, 0.3, 4)
    k = rng.integers(1, 4, (4, 3)) * math.pi
    Q = torch.empty(p.K, 4, p.Np, dtype=torch.float32, device="cuda")
    for f in range(4):
        v = a[f] * torch.cos(k[f][0] * x) * torch.sin(k[f][1] * y + 0.5) * torch.cos(k[f][2] * z)
        if f == 0:
            v = v + torch.exp(-50.0 * ((x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2))
        Q[:, f] = v
    if getattr(p, "variant", "nodal") == "bb":
        inv = torch.from_numpy(p.ops["invVB64"].reshape(p.Np, p.Np).T.copy()).cuda()
        Q = (Q.double() @ inv.T).float()
    return _pinned(Q)


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy().ravel()


@functools.lru_cache(maxsize=3)
def _cubature_xyz(p_key):
    return _affine(*p_key).cubature_xyz()


def _sources(case, p, seed):
    rng = np.random.default_rng(seed + 2)
    xyz = _cubature_xyz((case["N"], case["n"], case["rule"], case["variant"]))
    ent = [source_entries(gaussian_source(p, c, a=20.0, xyz=xyz), shot=i)
           for i, c in enumerate(rng.uniform(-0.8, 0.8, (case["shots"], 3)))]
    return [np.concatenate(e) for e in zip(*ent)]


def _receivers(case, p, seed):
    rng = np.random.default_rng(seed + 3)
    return receiver_weights(p, rng.uniform(-0.8, 0.8, (case["receivers"], 3)))


def _observed(case, seed):
    rng = np.random.default_rng(seed + 4)
    return rng.standard_normal((case["shots"], case["receivers"], case["steps"])).astype(np.float32)


def _problem(case, seed):
    base = _affine(case["N"], case["n"], case["rule"], case["variant"])
    return dataclasses.replace(base, c2q=_medium(base, seed))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "curved":
        base = _ball(case["N"], case["n"], case["rule"])
        p = dataclasses.replace(base, c2q=_medium(base, seed))
        return dict(case=case, p=p, s=CurvedSolver(p), Q0=_initial(p, seed))
    p = _problem(case, seed)
    if kind == "kernels":
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        o, g = p.ops_dict(), p.geo_dict()
        d = {k: dev(o[k]) for k in ("Dr", "Ds", "Dt", "LIFT", "Vq", "Pq", "Fmask")}
        d.update({k: dev(g[k]) for k in ("vgeo", "fgeo", "vmapP", "Jq", "c2q")})
        d["Q0"] = dev(_initial(p, seed))
        d.update({k: torch.zeros_like(d["Q0"]) for k in ("Q", "res", "rhs")})
        return dict(case=case, p=p, d=d, ptr={k: t.data_ptr() for k, t in d.items()})
    s = WaveSolver(p, bc=case["bc"], precision=case["precision"])
    st = dict(case=case, p=p, s=s)
    if kind in ("shots", "adjoint"):
        s.set_shots(case["shots"])
        s.set_sources(*_sources(case, p, seed), f0=F0, amplitude=AMPLITUDE, stage_times=True)
        s.set_receivers(*_receivers(case, p, seed), case["steps"])
        st["Q0"] = _pinned(torch.zeros(s.state_size))
        st["observed"] = _observed(case, seed)
    else:
        st["Q0"] = _initial(p, seed)
    st["out"] = _pinned(torch.zeros(s.state_size))
    return st


# ------------------------------------------------------------------ one pass
def run(state):
    case, p = state["case"], state["p"]
    kind = case["kind"]
    if kind == "kernels":
        return _run_kernels(case, p, state["d"], state["ptr"])
    s = state["s"]
    s.set_data(state["Q0"])
    if kind == "curved":
        s.steps(p.dt, case["steps"])
        return s.get_data()
    if kind == "stages":
        for _ in range(case["steps"]):
            for a, b in zip(RK4A, RK4B):
                s.rk_step(a, b, p.dt)
        return s.get_data(out=state["out"])
    if kind == "steps":
        s.steps(p.dt, case["steps"])
        return s.get_data(out=state["out"])
    s.set_time(0.0)
    if kind == "shots":
        s.steps(p.dt, case["steps"])
        return s.get_traces(), s.get_data(out=state["out"])
    s.set_residual(state["Q0"])
    tape = s.forward(p.dt, case["steps"])
    traces = s.get_traces()
    grad = s.backward(tape, traces - state["observed"])
    tape.free()
    return traces, grad


def _run_kernels(case, p, d, a):
    bc = 1 if case["bc"] == "rigid" else 0
    d["Q"].copy_(d["Q0"])
    d["res"].zero_()
    N, K = p.N, p.K
    for _ in range(case["steps"]):
        for fa, fb in zip(RK4A, RK4B):
            _lib.call("bbw_rk_volume", N, K, a["vgeo"], a["Dr"], a["Ds"], a["Dt"], a["Q"],
                      a["rhs"], None)
            _lib.call("bbw_rk_surface", N, K, bc, a["fgeo"], a["Fmask"], a["vmapP"], a["LIFT"],
                      a["Q"], a["rhs"], None)
            _lib.call("bbw_rk_update_wadg", N, K, p.Nq, a["Vq"], a["Pq"], a["Jq"], a["c2q"],
                      float(fa), float(fb), p.dt, a["rhs"], a["res"], a["Q"], None)
    return d["Q"], d["res"]


# ------------------------------------------------------------------ the work
_TABLE_NQ = {3: (31, 15), 4: (57, 19), 5: (95, 28), 6: (146, 40), 7: (214, 54)}


def work(case):
    """Bytes: per stage and element, state and residual read and written
    (64 Np), the medium (4 Nq), geometry and connectivity; the state in and
    out once.  Operations: the contractions in the form the path uses."""
    N, K, S = case["N"], 6 * case["n"] ** 3, case.get("shots", 1)
    Np, Nfp = _np(N), _nfp(N)
    Nq, Nfq = _TABLE_NQ[N] if case["rule"] == "table" else ((N + 1) ** 3, (N + 1) ** 2)
    stages = 5 * case["steps"]
    state = 16 * Np * K * S
    wadg = 2 * Nq * Np
    if case["kind"] == "curved":
        # share of curved elements of the ball: those that touch the sphere
        kc = 1.0 - max(0.0, 1.0 - 2.0 / case["n"]) ** 3
        planar = 64 * Np + 4 * Nq + 132
        curved = 64 * Np + 48 * Nq + 64 * Nfq + 16 * Nfp
        fp = 6 * Np * Np + 4 * Np * Nfp + wadg
        fc = 12 * Nq * Np + 28 * Nfq * Nfp + 16 * Nfq * Np + 8 * Nq * Np
        return dict(bytes=K * stages * ((1 - kc) * planar + kc * curved) + 2 * state,
                    flops=2.0 * K * stages * ((1 - kc) * fp + kc * fc))
    if case.get("variant") == "bb":
        fma = 24 * Np + 7 * 4 * Nfp + 4 * 4 * Np + 16 * Np + wadg
    else:
        fma = 6 * Np * Np + 4 * Np * Nfp + wadg
    nbytes = S * K * stages * 64 * Np + K * stages * (4 * Nq + 132) + 2 * state
    flops = 2.0 * S * K * stages * fma
    if case["kind"] == "kernels":
        nbytes = K * stages * (64 * Np + 8 * Nq + 100 + 16 * Nfp)
    if case["kind"] == "adjoint":  # the reverse sweep does the transposed work once more
        nbytes, flops = 2 * nbytes + S * K * stages * 8 * Nq + 8 * K * Nq, 2 * flops
    return dict(bytes=float(nbytes), flops=flops)


# ------------------------------------------------------------------ in 64 bits
def _mat(a, rows, cols):
    """Column-major operator as an FP64 matrix on the GPU."""
    return torch.from_numpy(np.asarray(a, np.float64).reshape(cols, rows).T.copy()).cuda()


def _f64(a, *shape):
    return torch.from_numpy(np.asarray(a, np.float64).reshape(shape)).cuda()


def _bb_dense(N, o):
    """Dense Dr, Ds, Dt and LIFT of the sparse Bernstein-Bezier operators."""
    Np, Nfp = _np(N), _nfp(N)
    D = np.zeros((3, Np, Np))
    vals = np.asarray(o["Dvals4"], np.float64).reshape(Np, 4)
    for j in range(4):
        ids = np.asarray(o["D_ids%d" % (j + 1)]).reshape(Np, 4)
        for n in range(Np):
            for d in range(3):
                D[d, n, ids[n, d + 1]] += 0.5 * vals[n, j]
                D[d, n, ids[n, 0]] -= 0.5 * vals[n, j]
    L0 = np.zeros((Nfp, Nfp))
    li, lv = np.asarray(o["L0_ids"]).reshape(-1, Nfp), np.asarray(o["L0_vals"], np.float64).reshape(-1, Nfp)
    for l in range(len(li)):
        np.add.at(L0, (np.arange(Nfp), li[l]), lv[l])
    E = np.zeros((Np, 4 * Nfp))
    ei, ev = np.asarray(o["EEL_ids"]).reshape(-1, Np), np.asarray(o["EEL_vals"], np.float64).reshape(-1, Np)
    for j in range(len(ei)):
        np.add.at(E, (np.arange(Np), ei[j]), ev[j])
    return D, E @ np.kron(np.eye(4), L0)


class _Affine64:
    def __init__(self, p, bc):
        N, K = p.N, p.K
        self.K, self.Np, self.Nfp, self.bc = K, _np(N), _nfp(N), bc
        Np, NF = self.Np, 4 * self.Nfp
        o, g = p.ops_dict(), p.geo_dict()
        if p.variant == "bb":
            D, L = _bb_dense(N, o)
            self.D, self.L = [torch.from_numpy(d).cuda() for d in D], torch.from_numpy(L).cuda()
        else:
            self.D = [_mat(o[k], Np, Np) for k in ("Dr", "Ds", "Dt")]
            self.L = _mat(o["LIFT"], Np, NF)
        self.Vq, self.Pq = _mat(o["Vq"], p.Nq, Np), _mat(o["Pq"], Np, p.Nq)
        self.G = _f64(g["vgeo"], K, 9)
        fg = _f64(g["fgeo"], K, 4, 4)
        self.Fs, self.n = fg[:, :, 0, None], fg[:, :, 1:4].transpose(1, 2)[..., None]
        self.Fm = torch.from_numpy(np.asarray(o["Fmask"], np.int64)).cuda()
        vm = torch.from_numpy(np.asarray(g["vmapP"], np.int64).reshape(K, NF)).cuda()
        self.k2, self.n2 = vm // (4 * Np), vm % (4 * Np)
        self.wall = (self.k2 == torch.arange(K, device="cuda")[:, None]) & (self.n2 == self.Fm)

    def rhs(self, Q, c2q):
        """[K][4][Np] -> projected rhs and nothing else."""
        K, Np, Nfp, G = self.K, self.Np, self.Nfp, self.G
        p, u, v, w = Q[:, 0], Q[:, 1], Q[:, 2], Q[:, 3]
        g = [G[:, i, None] for i in range(9)]
        div = sum((u * g[3 * d] + v * g[3 * d + 1] + w * g[3 * d + 2]) @ self.D[d].T
                  for d in range(3))
        dp = [p @ self.D[d].T for d in range(3)]
        M = Q[:, :, self.Fm]
        flat = Q.reshape(-1)
        at = self.k2 * (4 * Np) + self.n2
        jump = torch.stack([flat[at + c * Np] - M[:, c] for c in range(4)], 1)
        if self.bc == 0:
            jump = torch.where(self.wall[:, None], torch.cat([-2 * M[:, :1], 0 * M[:, 1:]], 1), jump)
        else:
            jump = torch.where(self.wall[:, None], torch.cat([0 * M[:, :1], -2 * M[:, 1:]], 1), jump)
        jump = jump.reshape(K, 4, 4, Nfp)
        un = (jump[:, 1:] * self.n).sum(1)
        flux = 0.5 * (jump[:, 0] - un) * self.Fs  # [K][4 faces][Nfp]
        lift = lambda f: f.reshape(K, 4 * Nfp) @ self.L.T  # noqa: E731
        rp = -div + lift(flux)
        rp = ((rp @ self.Vq.T) * c2q) @ self.Pq.T
        ru = [-(g[c] * dp[0] + g[3 + c] * dp[1] + g[6 + c] * dp[2]) -
              lift(flux * self.n[:, c]) for c in range(3)]
        return torch.stack([rp] + ru, 1)


def _lsrk(rhs, Q, steps, dt, after_step=None):
    """The time loop with the coefficients as the FP32 path casts them."""
    dt = float(np.float32(dt))
    res = torch.zeros_like(Q)
    for step in range(steps):
        for i, (a, b) in enumerate(zip(RK4A, RK4B)):
            res = float(np.float32(a)) * res + dt * rhs(Q, step, i)
            Q = Q + float(np.float32(b)) * res
        if after_step:
            after_step(Q)
    return Q, res


def _ricker(step, i, dt):
    t = step * float(np.float32(dt)) + float(np.float32(RK4C[i])) * float(np.float32(dt))
    a = math.pi * F0 * (t - 1.0 / F0)
    return AMPLITUDE * (1 - 2 * a * a) * math.exp(-a * a)


def exact(case, seed):
    kind = case["kind"]
    if kind == "curved":
        return _exact_curved(case, seed)
    p = _problem(case, seed)
    A = _Affine64(p, 1 if case["bc"] == "rigid" else 0)
    c2 = _f64(p.c2q, p.K, p.Nq)
    if kind in ("steps", "stages", "kernels"):
        Q = _f64(_initial(p, seed), p.K, 4, p.Np)
        Q, res = _lsrk(lambda q, step, i: A.rhs(q, c2), Q, case["steps"], p.dt)
        if kind == "kernels":
            return Q.reshape(-1).cpu(), res.reshape(-1).cpu()
        return Q.reshape(-1).cpu().numpy()
    shot, elem, vec = _sources(case, p, seed)
    rel, rw = _receivers(case, p, seed)
    rel, rw = torch.from_numpy(rel.astype(np.int64)).cuda(), _f64(rw, len(rel), p.Np)
    grad = torch.zeros_like(c2)
    observed = _f64(_observed(case, seed), case["shots"], case["receivers"], case["steps"])
    traces, finals = [], []
    for sh in range(case["shots"]):
        src = torch.zeros(p.K, p.Np, dtype=torch.float64, device="cuda")
        mine = shot == sh
        src.index_add_(0, torch.from_numpy(elem[mine].astype(np.int64)).cuda(),
                       _f64(vec[mine], int(mine.sum()), p.Np))
        medium = c2.clone().requires_grad_(kind == "adjoint")

        def rhs(Q, step, i, medium=medium, src=src):
            r = A.rhs(Q, medium)
            return torch.cat([r[:, :1] + _ricker(step, i, p.dt) * src[:, None], r[:, 1:]], 1)

        def one_step(Q, res, m, step):
            for i, (a, b) in enumerate(zip(RK4A, RK4B)):
                res = float(np.float32(a)) * res + float(np.float32(p.dt)) * rhs(Q, step, i, m)
                Q = Q + float(np.float32(b)) * res
            return Q, res

        Q = torch.zeros(p.K, 4, p.Np, dtype=torch.float64, device="cuda")
        res, tr = torch.zeros_like(Q), []
        for step in range(case["steps"]):
            if kind == "adjoint":
                Q, res = checkpoint(one_step, Q, res, medium, step, use_reentrant=False)
            else:
                Q, res = one_step(Q, res, medium, step)
            tr.append((rw * Q[rel, 0]).sum(1))
        tr = torch.stack(tr, 1)
        if kind == "adjoint":
            (0.5 * (tr - observed[sh]) ** 2).sum().backward()
            grad += medium.grad
        else:
            finals.append(Q.reshape(-1).cpu())
        traces.append(tr.detach())
    traces = torch.stack(traces).cpu().numpy()
    if kind == "adjoint":
        return traces, grad.cpu().numpy()
    return traces, torch.cat(finals).numpy()


def _exact_curved(case, seed):
    base = _ball(case["N"], case["n"], case["rule"])
    p = dataclasses.replace(base, c2q=_medium(base, seed))
    a, K, Np, Nfp, Nq, Nfq = p.desc_arrays(), p.K, p.Np, p.Nfp, p.Nq, p.Nfq
    NF = 4 * Nfp
    D = [_mat(a[k], Np, Np) for k in ("Dr", "Ds", "Dt")]
    L, Vf, Pf = _mat(a["LIFT"], Np, NF), _mat(a["VfqFace"], Nfq, Nfp), _mat(a["Pfq"], Np, 4 * Nfq)
    V, Vr, Vs, Vt = (_mat(a[k], Nq, Np) for k in ("Vq", "Vrq", "Vsq", "Vtq"))
    P, Pr, Ps, Pt = (_mat(a[k], Np, Nq) for k in ("Pq", "Prq", "Psq", "Ptq"))
    kc, kp = (torch.from_numpy(a[k].astype(np.int64)).cuda() for k in ("KlistCurved", "KlistPlanar"))
    vgeo, fgeo, J = _f64(a["vgeo"], K, 9), _f64(a["fgeo"], K, 4, 4), _f64(a["Jplanar"], K)
    g, Jq = _f64(a["vgeoq"], K, 9, Nq)[kc], _f64(a["Jq"], K, Nq)
    fq = _f64(a["fgeoq"], K, 4, 4, Nfq)[kc]
    c2 = _f64(p.c2q, K, Nq)
    Fm = torch.from_numpy(a["Fmask"].astype(np.int64)).cuda()
    vm = torch.from_numpy(a["vmapP"].astype(np.int64).reshape(K, NF)).cuda()

    def traces(Q, at):
        own = at[:, None] * (4 * Np) + Fm
        flat = Q.reshape(-1)
        M = torch.stack([flat[own + c * Np] for c in range(4)], 1)
        Pl = torch.stack([flat[vm[at] + c * Np] for c in range(4)], 1)
        return M, Pl, (own == vm[at])[:, None]

    def rhs(Q, step, i):
        out = torch.empty_like(Q)
        # planar elements, weighted with J
        G, q, Jp = vgeo[kp], Q[kp], J[kp][:, None]
        U = [sum(q[:, 1 + c] * G[:, 3 * d + c, None] for c in range(3)) for d in range(3)]
        dp = [q[:, 0] @ D[d].T for d in range(3)]
        M, Pl, wall = traces(Q, kp)
        jump = torch.where(wall, torch.cat([-2 * M[:, :1], 0 * M[:, 1:]], 1), Pl - M)
        jump = jump.reshape(len(kp), 4, 4, Nfp)
        n = fgeo[kp][:, :, 1:4].transpose(1, 2)[..., None]
        flux = 0.5 * (jump[:, 0] - (jump[:, 1:] * n).sum(1)) * fgeo[kp][:, :, 0, None]
        lift = lambda f: f.reshape(len(kp), NF) @ L.T  # noqa: E731
        out[kp, 0] = Jp * (lift(flux) - sum(U[d] @ D[d].T for d in range(3)))
        for c in range(3):
            out[kp, 1 + c] = -Jp * (lift(flux * n[:, c]) +
                                    sum(G[:, 3 * d + c, None] * dp[d] for d in range(3)))
        # curved elements, skew form
        q, Jc = Q[kc], Jq[kc]
        uq = [q[:, 1 + c] @ V.T for c in range(3)]
        dr = [q[:, 0] @ m.T for m in (Vr, Vs, Vt)]
        grad = [(g[:, 3 * c] * dr[0] + g[:, 3 * c + 1] * dr[1] + g[:, 3 * c + 2] * dr[2]) * Jc
                for c in range(3)]
        con = [sum(uq[c] * g[:, 3 * c + d] for c in range(3)) * Jc for d in range(3)]
        M, Pl, wall = traces(Q, kc)
        E = len(kc)
        q4 = lambda v: v.reshape(E, 4, Nfp) @ Vf.T  # noqa: E731
        dpq = q4(torch.where(wall[:, 0], -2 * M[:, 0], Pl[:, 0] - M[:, 0]))
        nn = [fq[:, :, c] for c in range(3)]
        du = sum(q4(torch.where(wall[:, 0], 0 * M[:, 1 + c], Pl[:, 1 + c] - M[:, 1 + c])) * nn[c]
                 for c in range(3))
        av = sum(q4(0.5 * (Pl[:, 1 + c] + M[:, 1 + c])) * nn[c] for c in range(3))
        sJ = fq[:, :, 3]
        pf, uf = -(av - 0.5 * dpq) * sJ, -0.5 * (dpq - du) * sJ
        lf = lambda f: f.reshape(E, 4 * Nfq) @ Pf.T  # noqa: E731
        out[kc, 0] = con[0] @ Pr.T + con[1] @ Ps.T + con[2] @ Pt.T + lf(pf)
        for c in range(3):
            out[kc, 1 + c] = -(grad[c] @ P.T) + lf(uf * nn[c])
        t = (out @ V.T) / Jq[:, None]
        t[:, 0] *= c2
        return t @ P.T

    Q, _ = _lsrk(rhs, _f64(_initial(p, seed), K, 4, Np), case["steps"], p.dt)
    return Q.reshape(-1).cpu().numpy()
