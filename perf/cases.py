"""The work that a solve on this library is made of, as timed cases.

Every case is one call (or one short sequence of calls) of the public API on
synthetic bodies with lambda = 1 m and leaf boxes of 0.25 lambda: the FP64 and
the FP32 operator, the dense operator, the two whole solves (CGS with ILUT,
and the mixed-precision block solve with the neighbourhood inverse), the
set-up of the neighbourhood inverse, the RCS sum and the network's gradient.

Bodies are geodesic meshes of frequency f (20 f^2 triangles, 30 f^2 RWG
unknowns; f = 2^level is the icosphere of that level) mapped to
  sphere          radius 6 lambda f / 64: edges of about 0.11 lambda, 4-11
                  unknowns per leaf box;
  superellipsoid  exponent 4, semi-axes (4, 2, 2) lambda f / 64: about 60
                  unknowns per leaf box;
  spheroid        semi-axes (3, 0.75, 0.75) lambda f / 64: about 145 unknowns
                  per leaf box.

FP32 results (complex(8) vectors that hold single-precision sums) are returned
in complex64, the precision in which the mixed solve's inner loop takes them.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from lywell_gb300 import MLFMA, RWG, MoM, _capi, ajustar_polariz, direction, learned, meshes

LEAF = 0.25
MU, EPS = 1.2566370614e-6, 8.8541878176e-12
C2 = torch.complex128


def listed():
    return [
        # one product on a small body: ten launches of a few microseconds each
        dict(name="fp64_op_small", op="fp64", body="sphere", f=8, nrhs=1),
        # the operator of the plain FP64 solve at the size of the headline sphere
        dict(name="fp64_op_large", op="fp64", body="sphere", f=64, nrhs=1),
        # the FP64 residual check of a block of angles, after some have converged
        dict(name="fp64_op_block", op="fp64", body="spheroid", f=20, nrhs=24),
        # the dense method-of-moments operator, several excitations at once
        dict(name="dense_op", op="dense", body="sphere", f=15, nrhs=3),
        # the inner operator of a single mixed-precision solve
        dict(name="fp32_op_single", op="fp32", body="sphere", f=64, nrhs=1, engine=-1),
        # the inner operator of a monostatic sweep where leaf boxes are small
        dict(name="fp32_op_sphere_block", op="fp32", body="sphere", f=48, nrhs=16, engine=-1),
        # the same where leaf boxes are full (the engine that the autotuner takes there)
        dict(name="fp32_op_spheroid_block", op="fp32", body="spheroid", f=32, nrhs=64, engine=4),
        # the reference's own method with its default preconditioner: CGS + ILUT to 1e-4
        dict(name="cgs_ilut", op="cgs", body="sphere", f=6, errmax=1e-4, maxit=400),
        # a block of monostatic angles by the mixed-precision solve
        dict(name="mixed_block", op="mixed", body="spheroid", f=24, nrhs=32, engine=4, errmax=1e-6),
        # the preconditioner's set-up where neighbourhoods hold thousands of unknowns
        dict(name="nearinv_setup", op="nearinv", body="spheroid", f=14),
        # a bistatic RCS cut in 1-degree steps, two planes
        dict(name="rcs_cut", op="rcs", body="sphere", f=32, nang=362),
        # loss and gradient of one training batch of the learned preconditioner
        dict(name="mlp_grad", op="mlp_grad", tokens=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["fp64", "fp64", "fp64", "fp32", "fp32", "fp32", "dense", "cgs", "mixed", "nearinv", "rcs",
                     "mlp_grad"])
    if op == "mlp_grad":
        return dict(op=op, tokens=_log_int(rng, 500, 8192))
    case = dict(op=op, body="sphere", scale=round(rng.uniform(0.95, 1.05), 3))
    if op == "fp64":
        if rng.random() < 0.6:
            return dict(case, body=rng.choice(["sphere", "sphere", "superellipsoid"]), f=_log_int(rng, 8, 60), nrhs=1)
        return dict(case, body=rng.choice(["sphere", "spheroid"]), f=_log_int(rng, 12, 20), nrhs=_log_int(rng, 2, 24))
    if op == "fp32":
        body = rng.choice(["sphere", "superellipsoid", "spheroid"])
        nrhs = 1 if rng.random() < 0.25 else _log_int(rng, 2, 64)
        hi = {"sphere": 60, "superellipsoid": 48, "spheroid": 32}[body]
        f = _log_int(rng, 12, min(hi, int(260 / math.sqrt(nrhs))))
        return dict(case, body=body, f=f, nrhs=nrhs, engine=-1 if body == "sphere" or nrhs == 1 else 4)
    if op == "dense":
        return dict(case, f=_log_int(rng, 6, 15), nrhs=rng.randint(1, 6))
    if op == "cgs":
        return dict(case, f=rng.randint(6, 7), errmax=1e-4, maxit=400)
    if op == "mixed":
        return dict(case, body="spheroid", f=rng.randint(14, 24), nrhs=rng.randint(2, 32), engine=4, errmax=1e-6)
    if op == "nearinv":
        body = rng.choice(["sphere", "superellipsoid", "spheroid"])
        return dict(case, body=body, f=rng.randint(10, 14) if body == "spheroid" else rng.randint(12, 20))
    return dict(case, f=_log_int(rng, 8, 32), nang=_log_int(rng, 2, 361))


# -- bodies --------------------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _geodesic(f):
    """Unit sphere of frequency f: (vertices, faces), every vertex stored once."""
    v, faces = meshes.icosphere_indexed(0)
    at = [(i, j) for i in range(f + 1) for j in range(f + 1 - i)]
    place = {ij: n for n, ij in enumerate(at)}
    w = np.array([(f - i - j, i, j) for i, j in at])
    weights = np.zeros((len(faces), len(at), len(v)), dtype=np.int16)
    for n, face in enumerate(faces):
        weights[n][:, face] = w
    keys, node = np.unique(weights.reshape(-1, len(v)), axis=0, return_inverse=True)
    node = node.reshape(len(faces), len(at))
    p = keys @ v / f
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    tri = [(place[i, j], place[i + 1, j], place[i, j + 1]) for i, j in at if i + j < f]
    tri += [(place[i + 1, j], place[i + 1, j + 1], place[i, j + 1]) for i, j in at if i + j < f - 1]
    return p, np.concatenate([node[:, list(t)] for t in tri])


@functools.lru_cache(maxsize=8)
def _triangles(body, f, scale):
    p, faces = _geodesic(f)
    if body == "sphere":
        p = p * (6.0 * scale * f / 64)
    elif body == "spheroid":
        p = p * (np.array([3.0, 0.75, 0.75]) * scale * f / 64)
    else:
        a = np.array([4.0, 2.0, 2.0]) * scale * f / 64
        p = p * (np.sum(np.abs(p / a) ** 4, axis=1) ** -0.25)[:, None]
    return np.ascontiguousarray(p[faces])


@functools.lru_cache(maxsize=8)
def _rwg(body, f, scale):
    return RWG(_triangles(body, f, scale))


def _geometry(case):
    return case["body"], case["f"], case.get("scale", 1.0)


def _operator(case):
    rwg = _rwg(*_geometry(case))
    if case["op"] == "dense":
        return MoM(rwg)
    m = MLFMA(rwg, lam=1.0, ladomax=LEAF)
    if "engine" in case:
        m.set_block_engine(case["engine"])
    return m


def _columns(case, seed, n):
    """Complex Gaussian columns, (nrhs, n) on the GPU: what Krylov vectors look like."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(case.get("nrhs", 1), n, dtype=C2, device="cuda", generator=g)


def _waves(case, seed):
    """Incidence directions at theta = 90 degrees and their VV or HH polarisations, one per column."""
    rng = np.random.default_rng(seed)
    n = case.get("nrhs", 1)
    d = [direction(90.0, p) for p in rng.uniform(0.0, 180.0) + 0.5 * np.arange(n)]
    kind = "HH" if rng.random() < 0.5 else "VV"
    return np.array(d), np.array([ajustar_polariz(x, kind) for x in d])


def _batch(case, seed):
    """Parameters of the network, tokens and targets of one batch (CPU, FP32)."""
    g = torch.Generator().manual_seed(seed)
    shapes = [(16, 128), (1, 128), (128, 128), (1, 128), (128, 2), (1, 2)]
    P = [(torch.rand(s, generator=g) * 2 - 1) * (math.sqrt(6.0 / (s[0] + s[1])) if s[0] > 1 else 0.05) for s in shapes]
    X = torch.randn(case["tokens"], 16, generator=g)
    T = torch.randn(case["tokens"], 2, generator=g)
    return P, X, T


def _cut(case, seed):
    """Currents, their polarisation and the directions of one bistatic cut."""
    rng = np.random.default_rng(seed)
    n = 30 * case["f"] ** 2
    cur = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    th = np.linspace(0.0, np.pi, (case["nang"] + 1) // 2)
    th, ph = np.concatenate([th, th])[:case["nang"]], np.repeat([0.0, np.pi / 2], len(th))[:case["nang"]]
    return cur * 1e-3, np.array([1.0, 0.0, 0.0], dtype=np.complex128), th, ph


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


# -- the passes ----------------------------------------------------------------------------------------------------


def prepare(case, seed):
    op = case["op"]
    if op == "mlp_grad":
        P, X, T = _batch(case, seed)
        net = learned.MLP(seed=0)
        net.set_params(torch.cat([p.reshape(-1) for p in P]).numpy(), np.repeat([0.0, 1.0], 16))
        return dict(op=op, net=net, X=X.cuda(), T=T.cuda())
    m = _operator(case)
    s = dict(case, m=m)
    if op in ("fp64", "fp32", "dense"):
        s["x"] = _columns(case, seed, m.N)
        torch.cuda.current_stream().synchronize()   # the passes run on a stream of their own
    elif op in ("cgs", "mixed"):
        s["b"] = np.asfortranarray(m.excitation(*_waves(case, seed)))
        if op == "mixed":
            assert m.nearinv() == 0
        else:
            assert m.ilutC() == 0
    elif op == "nearinv":
        rng = np.random.default_rng(seed)   # another body: the near values are those of slightly other edges
        _, _, a = m.near_csr()
        a *= (1.0 + 0.01 * rng.standard_normal(a.size)).astype(np.float32)
        m.set_near_values(a)
    elif op == "rcs":
        s["cut"] = _cut(case, seed)
    return s


def run(state):
    op = state["op"]
    if op == "mlp_grad":
        loss, g = state["net"].grad(state["X"], state["T"])
        return dict(loss=np.float32(loss), grad=g)
    m = state["m"]
    if op in ("fp64", "fp32", "dense"):
        x = state["x"]
        with torch.cuda.stream(_stream()):
            y = torch.empty_like(x)
            if op != "fp32":
                m.matvec_device(x.data_ptr(), y.data_ptr(), x.shape[0], _stream().cuda_stream)
                return y
            code = _capi.load().mlf_matvec32_device(m.handle, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()),
                                                    x.shape[0], m.N, ctypes.c_void_p(_stream().cuda_stream))
            assert code == 0
            return y.to(torch.complex64)
    if op == "cgs":
        return m.cgs(state["b"], errmax=state["errmax"], maxit=state["maxit"], precond="ilu0")["x"]
    if op == "mixed":
        out = m.solve(state["b"], errmax=state["errmax"], maxit=2000, precond="nearinv", mixed=True)
        return out["x"].astype(np.complex64)
    if op == "nearinv":
        assert m.nearinv() == 0
        return m.nearinv_values().astype(np.complex64)
    cur, pol, th, ph = state["cut"]
    return m.rcs(cur, pol, th, ph)


# -- what a pass cannot do without ---------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _counts(body, f, scale):
    """Flops, then pattern and near-field bytes, of one FP64 product; near entries; leaf boxes; sum of cubed near rows."""
    with MLFMA(_rwg(body, f, scale), lam=1.0, ladomax=LEAF) as m:
        c = m.algorithmic_counts()
        ia, _, _ = m.near_csr()
        cubes = float(np.sum(np.diff(ia).astype(float) ** 3))
        return c["flops_total"], c["bytes"]["patterns"] / 2 + c["bytes"]["near"], m.nnz, m.levels[m.nlev]["nb"], cubes


def work(case):
    op = case["op"]
    if op == "mlp_grad":
        n = case["tokens"]
        return dict(bytes=4.0 * n * 18 + 8.0 * 18818, flops=3 * 2.0 * n * (16 * 128 + 128 * 128 + 128 * 2))
    N, nrhs = 30 * case["f"] ** 2, case.get("nrhs", 1)
    if op == "dense":
        return dict(bytes=16.0 * N * (N + 2 * nrhs), flops=8.0 * N * N * nrhs)
    if op == "rcs":
        return dict(bytes=16.0 * N + 8.0 * case["nang"], flops=100.0 * N * case["nang"])
    flops, table, nnz, nb, cubes = _counts(*_geometry(case))
    if op == "nearinv":   # the elimination of each box's neighbourhood; its rows read and written once
        return dict(bytes=24.0 * nnz, flops=8.0 / 3.0 * cubes * nb / N)
    if op == "fp64":
        return dict(bytes=table + 32.0 * N * nrhs, flops=flops * nrhs)
    if op == "fp32":
        return dict(bytes=table / 2 + 32.0 * N * nrhs, flops=flops * nrhs)
    if op == "cgs":       # two products and two sweeps an iteration, about 30 iterations
        return dict(bytes=30 * 2 * (table + 12.0 * nnz), flops=30 * 2 * (flops + 8.0 * nnz))
    return dict(bytes=100 * (table / 2 + 8.0 * nnz), flops=100 * nrhs * (flops + 8.0 * nnz))   # about 100 FP32 steps


# -- the same in 64 bits, from the formulas ------------------------------------------------------------------------


class _Body:
    """Triangle and edge data of a body (torch, on the GPU), edges in the order of their first occurrence."""

    def __init__(self, case):
        tris = _triangles(*_geometry(case))
        T = len(tris)
        _, node = np.unique(tris.reshape(-1, 3), axis=0, return_inverse=True)
        node = node.reshape(T, 3)
        pairs = np.array([(0, 1), (0, 2), (1, 2)])
        ends = np.sort(node[:, pairs].reshape(-1, 2), axis=1)
        order = np.lexsort((np.arange(3 * T), ends[:, 1], ends[:, 0])).reshape(-1, 2)   # closed: every edge twice
        order = order[np.argsort(order[:, 0])]
        up = functools.partial(torch.as_tensor, device="cuda")
        third, two = float(np.float32(1) / np.float32(3)), float(np.float32(2) / np.float32(3))
        p = [tris[:, i] for i in range(3)]
        v = [None, *p]
        for a, b in ((0, 1), (1, 2), (2, 0)):
            v += [p[a] + third * (p[b] - p[a]), p[a] + two * (p[b] - p[a])]
        v.append(third * (p[0] + p[1] + p[2]))
        parts = [(1, 4, 9), (4, 5, 10), (5, 2, 6), (6, 10, 7), (7, 8, 3), (7, 8, 10), (8, 9, 10), (9, 4, 10), (5, 6, 10)]
        self.sub = up(np.stack([third * (v[a] + v[b] + v[c]) for a, b, c in parts], axis=1))
        self.bar = up(v[10])
        self.T, self.N = T, len(order)
        self.tri = up(order // 3)                                        # T+, T- of each edge
        self.tip = up(tris[order // 3, (2 - order % 3)])                 # the vertex opposite to it in each
        a = tris.reshape(-1, 3)[order[:, 0] // 3 * 3 + pairs[order[:, 0] % 3, 0]]
        b = tris.reshape(-1, 3)[order[:, 0] // 3 * 3 + pairs[order[:, 0] % 3, 1]]
        self.long = up(np.linalg.norm(b - a, axis=1))
        self.centre = up((a + b) / 2)

    def product(self, x):
        """Z x of the method of moments, x (N, columns): centroid testing, nine source points a triangle."""
        w = 2 * math.pi / math.sqrt(MU * EPS)
        k, q = w * math.sqrt(MU * EPS), x.shape[1]
        xl = x * self.long[:, None]
        flow = torch.zeros(self.T, 9, 3, q, dtype=C2, device="cuda")
        charge = torch.zeros(self.T, q, dtype=C2, device="cuda")
        for s, sign in ((0, 1.0), (1, -1.0)):
            t = self.tri[:, s]
            for i in range(9):
                arm = sign * (self.sub[t, i] - self.tip[:, s])
                flow[:, i].index_add_(0, t, arm[:, :, None] * xl[:, None])
            charge.index_add_(0, t, sign * xl)
        src = torch.cat([flow, charge[:, None, None].expand(-1, 9, 1, q)], 2).reshape(self.T * 9, 4 * q)
        A = torch.empty(self.T, 4 * q, dtype=C2, device="cuda")
        pts = self.sub.reshape(-1, 3)
        step = max(1, int(2e8 // len(pts)))
        for t in range(0, self.T, step):
            r = torch.linalg.norm(self.bar[t:t + step, None] - pts, dim=2)
            A[t:t + step] = torch.polar(1 / r, -k * r) @ src
        A = A.reshape(self.T, 4, q)
        c72 = float(np.float32(1) / np.float32(72))
        y = torch.zeros_like(x)
        for s, sign in ((0, 1.0), (1, -1.0)):
            t = self.tri[:, s]
            arm = sign * (self.bar[t] - self.tip[:, s])
            y += 0.5j * w * (MU / math.pi * c72) * torch.einsum("nd,ndq->nq", arm.to(C2), A[t, :3])
            y += sign / (36j * math.pi * w * EPS) * A[t, 3]
        return y * self.long[:, None]

    def rcs(self, cur, pol, th, ph):
        k = 2 * math.pi
        lo, hi = self.centre.min(0).values, self.centre.max(0).values
        D = float(torch.linalg.norm(hi - lo))
        R = 10 * max(2 * D * D, 50 * D, 20.0)
        th, ph = torch.as_tensor(th, device="cuda"), torch.as_tensor(ph, device="cuda")
        at = (lo + hi) / 2 + R * torch.stack([th.sin() * ph.cos(), th.sin() * ph.sin(), th.cos()], 1)
        cp, cm = self.bar[self.tri[:, 0]], self.bar[self.tri[:, 1]]
        m = (cm - cp) * (torch.as_tensor(cur, device="cuda") * self.long)[:, None]
        out = []
        for o in at:
            r = o - (cp + cm) / 2
            d = torch.linalg.norm(r, dim=1)
            u = r / d[:, None]
            e = torch.polar(1 / d, -k * d)[:, None] * (u * (m * u).sum(1, keepdim=True) - m)
            out.append((e.sum(0).abs() ** 2).sum())
        fac = 2 * math.pi / math.sqrt(MU * EPS) * MU / (4 * math.pi)
        return torch.stack(out) * fac ** 2 * 4 * math.pi * R * R / float(np.sum(np.abs(pol) ** 2))


def exact(case, seed):
    """The operators' values are those of the method of moments, which the multipole expansion approximates."""
    op = case["op"]
    if op == "mlp_grad":
        P, X, T = _batch(case, seed)
        P = [p.bfloat16().double().requires_grad_() for p in P]
        h = torch.relu(torch.relu(X.double() @ P[0] + P[1]) @ P[2] + P[3])
        loss = ((h @ P[4] + P[5] - T.double()) ** 2).mean()
        loss.backward()
        return dict(loss=loss.detach(), grad=torch.cat([p.grad.reshape(-1) for p in P]))
    if op == "rcs":
        return _Body(case).rcs(*_cut(case, seed))
    if op in ("fp64", "fp32", "dense"):
        nrhs = case["nrhs"]
        greens = 9.0 * (20 * case["f"] ** 2) ** 2
        if greens * (1 + 0.2 * nrhs) > 6e10:   # over about 15 seconds
            return None
        b = _Body(case)
        return b.product(_columns(case, seed, b.N).T).T.contiguous()
    return None
