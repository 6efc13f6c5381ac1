"""The work that a user of this framework gives it, as measurable cases.

A case names one call of the public entry points (``BEM_Solver``,
``solve_linear_equation``, ``listener_pressure``, ``solve_modes``) with its
sizes and options.  ``prepare`` makes what a program holds before the call,
``run`` makes the call, ``work`` says what it cannot do without, and ``exact``
computes the same outputs in 64 bits with plain torch.

Kinds of calls:

* ``listen``    pressures at listeners from both boundary densities
  (``BEM_Solver.boundary2potential``);
* ``assemble``  the CBIE pair V and 1/2 M - K (``BEM_Solver.assemble_vk``);
* ``bm``        the Burton-Miller pair, <2,3> rules of ``neumann2dirichlet``
  or <4,6> rules of ``HBIE`` (``BEM_Solver.assemble_bm``);
* ``solve``     ``solve_linear_equation`` on a dense boundary operator;
* ``gradient``  ``listener_pressure`` and its backward pass (shape and
  velocity optimisation: a new mesh in every step);
* ``problem``   ``BEM_Solver.solve_and_evaluate``;
* ``modes``     ``solve_modes``: one wavenumber and one velocity per mode.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from neuralat_b200.bem import BEM_Solver, solve_linear_equation
from neuralat_b200.bem.adjoint import listener_pressure
from neuralat_b200.bem.modal import solve_modes

SPEED_OF_SOUND = 343.0
RADIUS = 0.15  # metres, before the seeded deformation
PI4 = 4.0 * math.pi


def listed():
    return [
        # the smallest call: an object of 642 vertices heard at 256 points, one field (the plain workload's listeners)
        dict(name="listen-s3-256x1", kind="listen", shape="ico", n=8, hz=1000.0, points=256, rhs=1),
        # the transfer dataset's samples: 1000 listeners around a vibrating object beside a static one, ragged meshes
        dict(name="listen-pair-1000x1", kind="listen", shape="pair", n=17, hz=1730.0, points=1000, rhs=1),
        # many listeners and many modal fields at once, 20 480 triangles
        dict(name="listen-s5-4096x64", kind="listen", shape="ico", n=32, hz=4000.0, points=4096, rhs=64),
        # assembly of a coarse object (320 triangles, the batching workload's smallest): launches and latency count
        dict(name="assemble-s2", kind="assemble", shape="ico", n=4, hz=800.0),
        # assembly of the precision workload's mesh: 20 480 triangles
        dict(name="assemble-s5", kind="assemble", shape="ico", n=32, hz=4000.0),
        # the Burton-Miller system of two objects with odd sizes, as the dataset generator assembles it
        dict(name="bm-pair", kind="bm", shape="pair", n=21, hz=1230.0, approx=True),
        # one right-hand side with the defaults of the reference's signature (FP32, relative residual 1e-5)
        dict(name="solve-2487x1", kind="solve", shape="lathe", n=71, hz=2000.0, rhs=1, precision="fp32", rtol=1e-5),
        # eight modal fields on the tensor cores at the precision workload's size
        dict(name="solve-10242x8", kind="solve", shape="ico", n=32, hz=4000.0, rhs=8, precision="fp16x3", rtol=1e-6),
        # one step of shape optimisation: forward and backward, the differentiation workload's sizes
        dict(name="gradient-s4-128", kind="gradient", shape="ico", n=16, hz=1300.0, points=128),
        # the precision workload as a whole: assemble, solve eight fields, evaluate
        dict(name="problem-s5-256x8", kind="problem", shape="ico", n=32, hz=2000.0, points=256, rhs=8),
        # sixteen vibration modes of one object
        dict(name="modes-lathe-16x256", kind="modes", shape="lathe", n=35, hz=3000.0, points=256, modes=16),
        # the large multi-field workload: 81 920 triangles, 64 fields, 4096 listeners
        dict(name="problem-s6-4096x64", kind="problem", shape="ico", n=64, hz=2000.0, points=4096, rhs=64),
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["listen", "listen", "assemble", "assemble", "bm", "solve", "solve", "gradient", "problem", "modes"])
    shape = rng.choice(["ico", "lathe", "pair"])
    most = {"ico": 32, "lathe": 100, "pair": 24}[shape]  # about 20 000 triangles
    # below the first interior resonance of the deformed sphere where the plain CBIE is solved
    low = round(math.exp(rng.uniform(math.log(100.0), math.log(800.0))), 1)
    any_hz = round(math.exp(rng.uniform(math.log(100.0), math.log(5000.0))), 1)
    if kind == "listen":
        return dict(kind=kind, shape=shape, n=log_int(4, most), hz=any_hz, points=log_int(16, 4096), rhs=log_int(1, 64))
    if kind == "assemble":
        return dict(kind=kind, shape=shape, n=log_int(4, most), hz=any_hz)
    if kind == "bm":
        return dict(kind=kind, shape=shape, n=log_int(4, most), hz=any_hz, approx=rng.random() < 0.7)
    if kind == "solve":
        precision = rng.choice(["fp32", "fp16x3", "fp16x3", "bf16x3", "bf16"])
        return dict(kind=kind, shape=shape, n=log_int(4, most), hz=low, rhs=log_int(1, 64), precision=precision, rtol=1e-6)
    if kind == "gradient":
        return dict(kind=kind, shape=shape, n=log_int(4, {"ico": 20, "lathe": 60, "pair": 14}[shape]), hz=low,
                    points=log_int(16, 1024))
    if kind == "problem":
        return dict(kind=kind, shape=shape, n=log_int(4, most), hz=low, points=log_int(16, 1024), rhs=log_int(1, 32))
    return dict(kind=kind, shape=shape, n=log_int(4, {"ico": 16, "lathe": 50, "pair": 12}[shape]), hz=any_hz,
                points=log_int(16, 1024), modes=log_int(2, 24))


# ---- inputs ------------------------------------------------------------------
def _icosphere(n):
    """Unit sphere from the icosahedron with every edge cut into n: 10 n^2 + 2 vertices, 20 n^2 triangles,
    numbered along the faces."""
    t = (1.0 + math.sqrt(5.0)) / 2.0
    v = np.array([[-1, t, 0], [1, t, 0], [-1, -t, 0], [1, -t, 0], [0, -1, t], [0, 1, t], [0, -1, -t], [0, 1, -t],
                  [t, 0, -1], [t, 0, 1], [-t, 0, -1], [-t, 0, 1]])
    f = np.array([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2],
                  [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5], [2, 4, 11],
                  [6, 2, 10], [8, 6, 7], [9, 8, 1]])
    ij = np.array([(i, j) for i in range(n + 1) for j in range(n + 1 - i)])
    at = -np.ones((n + 2, n + 2), np.int64)
    at[ij[:, 0], ij[:, 1]] = np.arange(len(ij))
    up = np.array([(at[i, j], at[i + 1, j], at[i, j + 1]) for i in range(n) for j in range(n - i)])
    down = [(at[i + 1, j], at[i + 1, j + 1], at[i, j + 1]) for i in range(n) for j in range(n - 1 - i)]
    tri = np.concatenate([up, np.array(down, np.int64).reshape(-1, 3)])
    w = np.stack([n - ij[:, 0] - ij[:, 1], ij[:, 0], ij[:, 1]], 1) / n
    points = np.einsum("pc,fcd->fpd", w, v[f]).reshape(-1, 3)
    tris = (tri[None] + len(ij) * np.arange(20)[:, None, None]).reshape(-1, 3)
    _, first, inverse = np.unique(np.round(points * 1e7).astype(np.int64), axis=0, return_index=True,
                                  return_inverse=True)
    order = np.argsort(first)  # by first appearance along the faces
    rank = np.empty_like(order)
    rank[order] = np.arange(len(order))
    points = points[first[order]]
    return points / np.linalg.norm(points, axis=1, keepdims=True), rank[inverse.reshape(-1)][tris]


def _lathe(nlon):
    """Unit sphere as a body of revolution with nlon meridians: any vertex count, slender triangles at the poles."""
    nlat = max(2, nlon // 2)
    a, b = np.meshgrid(np.arange(1, nlat + 1) * math.pi / (nlat + 1), np.arange(nlon) * 2 * math.pi / nlon, indexing="ij")
    ring = np.stack([np.sin(a) * np.cos(b), np.sin(a) * np.sin(b), np.cos(a)], -1).reshape(-1, 3)
    v = np.concatenate([ring, [[0, 0, 1.0], [0, 0, -1.0]]])
    i, j = np.meshgrid(np.arange(nlat - 1), np.arange(nlon), indexing="ij")
    p, q = i * nlon + j, i * nlon + (j + 1) % nlon
    quads = np.stack([np.stack([p, p + nlon, q], -1), np.stack([q, p + nlon, q + nlon], -1)], 2).reshape(-1, 3)
    j = np.arange(nlon)
    last = (nlat - 1) * nlon
    top = np.stack([np.full(nlon, nlat * nlon), j, (j + 1) % nlon], 1)
    bottom = np.stack([np.full(nlon, nlat * nlon + 1), last + (j + 1) % nlon, last + j], 1)
    return v, np.concatenate([top, quads, bottom])


_SHAPES = {}


def _shape(shape, n):
    if (shape, n) not in _SHAPES:
        if len(_SHAPES) > 8:
            _SHAPES.clear()
        if shape == "ico":
            v, t = _icosphere(n)
        elif shape == "lathe":
            v, t = _lathe(n)
        else:  # a vibrating body of revolution beside a static sphere
            (v0, t0), (v1, t1) = _lathe(2 * n + 1), _icosphere(max(2, n - 3))
            v, t = np.concatenate([0.6 * v0 - [0.7, 0, 0], 0.5 * v1 + [0.7, 0, 0]]), np.concatenate([t0, t1 + len(v0)])
        _SHAPES[shape, n] = (np.ascontiguousarray(v), np.ascontiguousarray(t))
    return _SHAPES[shape, n]


def _mesh(case, seed):
    """The case's shape, scaled along its axes, with smooth bumps and turned, from the seed: float32 / int32 tensors."""
    v, t = _shape(case["shape"], case["n"])
    rng = np.random.default_rng([seed, 1])
    for _ in range(4):
        d = rng.standard_normal(3)
        v = v * (1.0 + 0.02 * np.sin(2.0 * v @ d + rng.uniform(0, 6.28)))[:, None]
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    v = (v * rng.uniform(0.8, 1.2, 3) * RADIUS) @ (q * np.sign(np.linalg.det(q)))
    return torch.from_numpy(v.astype(np.float32)).cuda(), torch.from_numpy(t.astype(np.int32)).cuda()


def _fields(v, t, m, seed, passes=5):
    """m complex Gaussian fields over the vertices, smoothed over the edges `passes` times: (N, m) complex64."""
    gen = torch.Generator(device=v.device).manual_seed(seed)
    x = torch.randn((v.shape[0], m), dtype=torch.complex128, device=v.device, generator=gen)
    t = t.long()
    a, b = torch.cat([t[:, 0], t[:, 1], t[:, 2]]), torch.cat([t[:, 1], t[:, 2], t[:, 0]])
    near = torch.zeros(v.shape[0], dtype=torch.float64, device=v.device).index_add_(0, a, torch.ones(len(a), dtype=torch.float64, device=v.device))
    for _ in range(passes):  # on a closed mesh each edge appears once in either direction
        mean = torch.zeros_like(x).index_add_(0, a, x[b]) / near[:, None]
        x = x + 0.5 * (mean - x)
    return x.to(torch.complex64)


def _points(count, seed, radius=0.5):
    p = np.random.default_rng([seed, 2]).standard_normal((count, 3))
    return torch.from_numpy((p / np.linalg.norm(p, axis=1, keepdims=True) * radius).astype(np.float32)).cuda()


def _k(hz):
    return 2.0 * math.pi * hz / SPEED_OF_SOUND


def _operator(case, seed):
    """A dense boundary operator 1/2 M - K and right-hand sides -V g over the vertices of a mesh, K and V by the
    vertices' shares of the area: the matrix that ``solve_linear_equation`` is given, without an assembly."""
    v, t = _mesh(case, seed)
    k, n, x, t = _k(case["hz"]), len(v), v.double(), t.long()
    c = x[t]
    cross = torch.cross(c[:, 1] - c[:, 0], c[:, 2] - c[:, 0], dim=1)
    size = cross.norm(dim=1) / 2
    area = torch.zeros_like(x[:, 0]).index_add_(0, t.reshape(-1), (size / 3).repeat_interleave(3))
    normal = torch.zeros_like(x).index_add_(0, t.reshape(-1), cross.repeat_interleave(3, 0))
    normal = normal / normal.norm(dim=1, keepdim=True)
    g = _fields(v, t, case["rhs"], seed).to(torch.complex128)
    A = torch.empty((n, n), dtype=torch.complex64, device=v.device)
    b = torch.empty((n, case["rhs"]), dtype=torch.complex64, device=v.device)
    for r0 in range(0, n, 1024):
        r = torch.arange(r0, min(n, r0 + 1024), device=v.device)
        d = x[None] - x[r, None]
        dist = d.norm(dim=2)
        dist[r - r0, r] = 1.0
        G = torch.polar(1.0 / (PI4 * dist), k * dist)
        K = (1.0 - 1j * k * dist) * G / dist**2 * (d * normal[None]).sum(2) * (area[r, None] * area[None])
        K[r - r0, r] = 0.0
        A[r] = K.to(A.dtype)
        G[r - r0, r] = torch.rsqrt(PI4 * area[r]).to(G.dtype)  # about a disc's own potential
        b[r] = (-area[r, None] * (G @ (area[:, None] * g))).to(b.dtype)
    for i in range(3):
        for j in range(3):
            A.view(-1).index_add_(0, t[:, i] * n + t[:, j], (size / (12.0 if i == j else 24.0)).to(A.dtype))
    return A, _one(b)


def _one(x):
    return x[:, 0].contiguous() if x.shape[1] == 1 else x


def _inputs(case, seed):
    """What both the call and its 64-bit counterpart start from."""
    kind = case["kind"]
    if kind == "solve":
        A, b = _operator(case, seed)
        return dict(A=A, b=b)
    v, t = _mesh(case, seed)
    s = dict(v=v, t=t, k=_k(case["hz"]))
    if kind in ("listen", "gradient", "problem", "modes"):
        s["points"] = _points(case["points"], seed)
    if kind == "listen":
        s["neumann"] = _one(_fields(v, t, case["rhs"], seed))
        s["dirichlet"] = _one(_fields(v, t, case["rhs"], seed + 7))
    elif kind == "problem":
        s["neumann"] = _one(_fields(v, t, case["rhs"], seed))
    elif kind == "gradient":
        s["neumann"] = _fields(v, t, 1, seed)[:, 0].contiguous()
    elif kind == "modes":
        s["neumann"] = _fields(v, t, case["modes"], seed).t().contiguous()
        s["ks"] = [float(x) for x in np.geomspace(s["k"] / 8, s["k"], case["modes"])]
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["kind"] == "gradient":  # every step has another mesh: the call builds its own solver
        s["v"].requires_grad_(True)
        s["neumann"].requires_grad_(True)
    elif case["kind"] != "solve":
        s["solver"] = BEM_Solver(s["v"], s["t"])
    return s


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "listen":
        return state["solver"].boundary2potential(state["k"], state["neumann"], state["dirichlet"], state["points"])
    if kind == "assemble":
        return state["solver"].assemble_vk(state["k"])
    if kind == "bm":
        return state["solver"].assemble_bm(state["k"], approx=case["approx"])
    if kind == "solve":
        return solve_linear_equation(state["A"], state["b"], tol=case["rtol"] ** 2, precision=case["precision"])
    if kind == "gradient":
        p = listener_pressure(state["v"], state["neumann"], state["t"], state["points"], state["k"])
        loss = (p.real ** 2 + p.imag ** 2).sum()
        return (p.detach(),) + torch.autograd.grad(loss, (state["v"], state["neumann"]))
    if kind == "problem":
        return state["solver"].solve_and_evaluate(state["k"], state["neumann"], state["points"])
    return solve_modes(state["solver"], state["ks"], state["neumann"], state["points"], return_dirichlet=True)


# ---- what a pass cannot do without ---------------------------------------------
PAIR, POINT = 60.0, 30.0  # operations for one pair of quadrature points (both operators, both orders) and one listener's
MATVECS = 20.0            # applications of the operator that a solve needs at the least


def _assembly(nv, nt, points):
    return dict(bytes=2 * 8.0 * nv * nv + 48.0 * nt, flops=0.5 * nt * nt * points * points * PAIR)


def _listening(nv, nt, p, m):
    return dict(bytes=8.0 * m * (2 * nv + p) + 12.0 * p + 48.0 * nt, flops=6.0 * nt * p * POINT + 16.0 * nv * p * m)


def _solving(n, m):
    return dict(bytes=8.0 * n * n + 16.0 * n * m, flops=8.0 * MATVECS * n * n * m)


def _sum(*parts):
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def work(case):
    kind = case["kind"]
    v, t = _shape(case["shape"], case["n"])
    nv, nt = len(v), len(t)
    if kind == "solve":
        return _solving(nv, case["rhs"])
    if kind == "listen":
        return _listening(nv, nt, case["points"], case["rhs"])
    if kind == "assemble":
        return _assembly(nv, nt, 6)
    if kind == "bm":
        return _assembly(nv, nt, 3 if case["approx"] else 6)
    if kind == "problem":
        return _sum(_assembly(nv, nt, 6), _solving(nv, case["rhs"]), _listening(nv, nt, case["points"], case["rhs"]))
    if kind == "gradient":  # forward, the adjoint solve, and the pairs once more for the derivative
        return _sum(_assembly(nv, nt, 6), _solving(nv, 2), _listening(nv, nt, case["points"], 1),
                    dict(bytes=0.0, flops=0.5 * nt * nt * 36 * 2 * PAIR))
    one = _sum(_assembly(nv, nt, 3), _solving(nv, 1), _listening(nv, nt, case["points"], 1))
    return {k: case["modes"] * x for k, x in one.items()}


# ---- the same in 64 bits ---------------------------------------------------------
def _rule(points):
    """Weights (summing to one) and barycentric coordinates of the 3-point degree-2 and 6-point degree-4 rules."""
    if points == 3:
        orbits = [(1.0 / 6.0, 1.0 / 3.0)]
    else:
        r10, s = math.sqrt(10.0), math.sqrt(38.0 - 44.0 * math.sqrt(0.4))
        w = math.sqrt(213125.0 - 53320.0 * r10)
        orbits = [((8.0 - r10 + s) / 18.0, (620.0 + w) / 3720.0), ((8.0 - r10 - s) / 18.0, (620.0 - w) / 3720.0)]
    phi = torch.cat([torch.full((3, 3), a, dtype=torch.float64) + torch.eye(3, dtype=torch.float64) * (1 - 3 * a) for a, _ in orbits])
    return torch.tensor([w for _, w in orbits for _ in range(3)], dtype=torch.float64).cuda(), phi.cuda()


def _line(points):
    if points == 2:
        x = [1 / math.sqrt(3.0), -1 / math.sqrt(3.0)]
        w = [1.0, 1.0]
    else:
        s = 2.0 / 7.0 * math.sqrt(6.0 / 5.0)
        x = [math.sqrt(3 / 7 + s), math.sqrt(3 / 7 - s), -math.sqrt(3 / 7 - s), -math.sqrt(3 / 7 + s)]
        w = [(18 - math.sqrt(30.0)) / 36, (18 + math.sqrt(30.0)) / 36, (18 + math.sqrt(30.0)) / 36, (18 - math.sqrt(30.0)) / 36]
    return [0.5 * (a + 1) for a in x], [0.5 * a for a in w]


def _touching_rule(common, line):
    """Sauter-Schwab points on the two unit triangles (0,0), (1,0), (1,1): shape functions (R, 3) on the test and on
    the trial triangle and weights (R,)."""
    x, w = _line(line)
    pts = []
    for xi, w0 in zip(x, w):
        for e1, w1 in zip(x, w):
            for e2, w2 in zip(x, w):
                for e3, w3 in zip(x, w):
                    g, e12, e123 = w0 * w1 * w2 * w3, e1 * e2, e1 * e2 * e3
                    if common == 3:
                        g *= xi**3 * e1**2 * e2
                        a = [(1, 1 - e1 + e12, 1 - e123, 1 - e1), (1, e1 - e12 + e123, 1 - e12, e1 - e12),
                             (1 - e123, e1 - e123, 1, e1 - e12)]
                        for x1, x2, y1, y2 in a:
                            pts += [(xi * x1, xi * x2, xi * y1, xi * y2, g), (xi * y1, xi * y2, xi * x1, xi * x2, g)]
                    elif common == 2:
                        g *= xi**3 * e1**2
                        a = [(1, e1 * e3, 1 - e12, e1 * (1 - e2), 1), (1, e1, 1 - e123, e12 * (1 - e3), e2),
                             (1 - e12, e1 * (1 - e2), 1, e123, e2), (1 - e123, e12 * (1 - e3), 1, e1, e2),
                             (1 - e123, e1 * (1 - e2 * e3), 1, e12, e2)]
                        pts += [(xi * x1, xi * x2, xi * y1, xi * y2, g * f) for x1, x2, y1, y2, f in a]
                    else:
                        g *= xi**3 * e2
                        pts += [(xi, xi * e1, xi * e2, xi * e2 * e3, g), (xi * e2, xi * e2 * e3, xi, xi * e1, g)]
    p = torch.tensor(pts, dtype=torch.float64).cuda()

    def shapes(a, b):
        return torch.stack([1 - a, a - b, b], 1)

    return shapes(p[:, 0], p[:, 1]), shapes(p[:, 2], p[:, 3]), p[:, 4].contiguous()


def _touching_pairs(t):
    """{common vertices: (test triangles, trial triangles, their corners with the shared ones first)}."""
    t = t.cpu().numpy().astype(np.int64)
    nt = len(t)
    order = np.argsort(t.reshape(-1), kind="stable")
    tri, vert = order // 3, t.reshape(-1)[order]
    start = np.searchsorted(vert, np.arange(t.max() + 2))
    size = np.diff(start)
    i = np.concatenate([np.repeat(tri[start[v]:start[v + 1]], size[v]) for v in range(len(size))])
    j = np.concatenate([np.tile(tri[start[v]:start[v + 1]], size[v]) for v in range(len(size))])
    key, common = np.unique(i * nt + j, return_counts=True)
    i, j = key // nt, key % nt
    found = {}
    for c in (3, 2, 1):
        a, b = i[common == c], j[common == c]
        p = np.tile(np.arange(3), (len(a), 1))
        q = p.copy()
        same = t[a][:, None, :] == t[b][:, :, None]  # [pair, trial corner, test corner]
        if c == 2:  # shared corners in the trial triangle's order, then the third
            jj = np.argsort(~same.any(2), axis=1, kind="stable")
            q = jj
            p = np.take_along_axis(same.argmax(2), jj, 1)
            p[:, 2] = 3 - p[:, 0] - p[:, 1]
        elif c == 1:  # the shared corner changes places with the first
            at = same.reshape(len(a), 9).argmax(1)
            for r, s in ((p, at % 3), (q, at // 3)):
                n = np.arange(len(a))
                r[n, s] = 0
                r[n, 0] = s
        found[c] = tuple(torch.from_numpy(np.ascontiguousarray(w)).cuda() for w in (a, b, p, q))
    return found


def _green(d, k):
    """G = e^{ikr} / (4 pi r) and H = (1 - ikr) G / r^2 for the differences d, r at least 1e-3."""
    r = (d * d).sum(-1).clamp(min=1e-6).sqrt()
    G = torch.polar(1.0 / (PI4 * r), k * r)
    return G, G * torch.complex(1.0 / (r * r), -k / r)


class _Exact:
    """The Galerkin operators of one mesh, block by block, in 64 bits."""

    def __init__(self, v, t):
        self.t = t.long()
        self.x = v.detach().double()
        self.nv, self.nt = len(v), len(t)
        self.touching = _touching_pairs(t)
        self.set(self.x)

    def set(self, x):
        """(Re)computes what follows from the vertices (with their graph, where they require a gradient)."""
        c = x[self.t]
        n = torch.cross(c[:, 1] - c[:, 0], c[:, 2] - c[:, 0], dim=1)
        size = n.norm(dim=1)
        self.corners, self.normal, self.area = c, n / size[:, None], 0.5 * size

    def curls(self):
        """n x grad phi_b: grad phi_b = n x (edge opposite to b) / (2 area), so minus that edge over 2 area."""
        c = self.corners
        edge = torch.stack([c[:, 2] - c[:, 1], c[:, 0] - c[:, 2], c[:, 1] - c[:, 0]], 1)
        return -edge / (2 * self.area)[:, None, None]

    def regular(self, points, step):
        w, phi = _rule(points)
        quad = torch.einsum("qb,tbd->tqd", phi, self.corners)
        for i0 in range(0, self.nt, step):
            i = torch.arange(i0, min(self.nt, i0 + step), device="cuda")
            apart = torch.ones((len(i), self.nt), dtype=torch.float64, device="cuda")
            for a in range(3):
                for b in range(3):
                    apart.masked_fill_(self.t[i, a][:, None] == self.t[None, :, b], 0.0)
            yield i, quad[i], quad, apart, w, phi

    def close(self, line, step):
        for common, (i, j, p, q) in self.touching.items():
            lx, ly, w = _touching_rule(common, line)
            step_ = max(1, step // len(w))
            for c0 in range(0, len(i), step_):
                c = slice(c0, c0 + step_)
                yield i[c], j[c], p[c], q[c], lx, ly, w


def _blocks(E, k, points, line, need_u, add):
    """Calls add(test, trial, rows, columns, S, T, U) with the 3 x 3 blocks of every pair:
    S = int int G phi phi, T = int int H (y - x).n_y phi phi, U = int int H (x - y).n_x phi phi."""
    step = max(1, int(1.2e7 / (E.nt * points * points)))
    for i, x, y, apart, w, phi in E.regular(points, step):
        ni, m = len(i), points
        d = y.reshape(1, -1, 3) - x.reshape(-1, 1, 3)
        G, H = _green(d, k)
        W = (w[:, None] * phi).to(G.dtype)
        scale = E.area[i][:, None] * E.area[None] * apart

        def fold(F):
            F = F.reshape(ni * m * E.nt, m) @ W
            F = F.reshape(ni, m, E.nt * 3).transpose(1, 2) @ W  # (ni, nt * 3, 3)
            return F.reshape(ni, E.nt, 3, 3).transpose(2, 3) * scale[:, :, None, None]

        S = fold(G)
        T = fold(H * (d.reshape(ni * m, E.nt, m, 3) * E.normal[None, :, None]).sum(-1).reshape(ni * m, -1))
        U = fold(-H * (d.reshape(ni, m, -1, 3) * E.normal[i][:, None, None]).sum(-1).reshape(ni * m, -1)) if need_u else None
        add(i[:, None].expand(ni, E.nt), torch.arange(E.nt, device="cuda")[None].expand(ni, E.nt),
            E.t[i][:, None, :, None].expand(ni, E.nt, 3, 3), E.t[None, :, None, :].expand(ni, E.nt, 3, 3), S, T, U)
    for i, j, p, q, lx, ly, w in E.close(line, 6_000_000):
        a = torch.gather(E.corners[i], 1, p[:, :, None].expand(-1, 3, 3))
        b = torch.gather(E.corners[j], 1, q[:, :, None].expand(-1, 3, 3))
        d = torch.einsum("rc,ncd->nrd", ly, b) - torch.einsum("rc,ncd->nrd", lx, a)
        G, H = _green(d, k)
        W = (w[:, None, None] * lx[:, :, None] * ly[:, None, :]).reshape(-1, 9).to(G.dtype)
        scale = (4.0 * E.area[i] * E.area[j])[:, None, None]

        def fold(F):
            return (F @ W).reshape(-1, 3, 3) * scale

        S = fold(G)
        T = fold(H * (d * E.normal[j][:, None]).sum(-1))
        U = fold(-H * (d * E.normal[i][:, None]).sum(-1)) if need_u else None
        add(i, j, torch.gather(E.t[i], 1, p)[:, :, None].expand(-1, 3, 3), torch.gather(E.t[j], 1, q)[:, None, :].expand(-1, 3, 3),
            S, T, U, p, q)


def _matrix(E):
    return torch.zeros(E.nv * E.nv, dtype=torch.complex128, device="cuda")


def _add_mass(E, A, factor):
    m = (torch.ones((3, 3), dtype=torch.float64, device="cuda") + torch.eye(3, dtype=torch.float64, device="cuda")) / 12.0
    rows, cols = E.t[:, :, None].expand(-1, 3, 3), E.t[:, None, :].expand(-1, 3, 3)
    A.index_add_(0, (rows * E.nv + cols).reshape(-1), (factor * (E.area[:, None, None] * m).to(A.dtype)).reshape(-1))


def _exact_vk(E, k):
    V, A = _matrix(E), _matrix(E)

    def add(i, j, rows, cols, S, T, U, p=None, q=None):
        at = (rows * E.nv + cols).reshape(-1)
        V.index_add_(0, at, S.reshape(-1))
        A.index_add_(0, at, T.reshape(-1))

    _blocks(E, k, 6, 4, False, add)
    _add_mass(E, A, 0.5)
    return V.view(E.nv, E.nv), A.view(E.nv, E.nv)


def _exact_bm(E, k, approx):
    L, R = _matrix(E), _matrix(E)
    curl = E.curls()

    def add(i, j, rows, cols, S, T, U, p=None, q=None):
        at = (rows * E.nv + cols).reshape(-1)
        ci, cj = curl[i], curl[j]
        if p is not None:
            ci = torch.gather(ci, 1, p[:, :, None].expand(-1, 3, 3))
            cj = torch.gather(cj, 1, q[:, :, None].expand(-1, 3, 3))
        cc = ci @ cj.transpose(-1, -2)
        nn = (E.normal[i] * E.normal[j]).sum(-1)[..., None, None]
        total = S.sum((-1, -2), keepdim=True)
        L.index_add_(0, at, (-1j * k * nn * S + T + (1j / k) * total * cc).reshape(-1))
        R.index_add_(0, at, (-S + (1j / k) * U).reshape(-1))

    _blocks(E, k, *((3, 2) if approx else (6, 4)), True, add)
    _add_mass(E, L, 0.5)
    _add_mass(E, R, -0.5j / k)
    return L.view(E.nv, E.nv), R.view(E.nv, E.nv)


def _exact_listen(E, k, neumann, dirichlet, points):
    """-S neumann + D dirichlet with the 6-point rule."""
    w, phi = _rule(6)
    y = torch.einsum("qb,tbd->tqd", phi, E.corners).reshape(-1, 3)
    normal = E.normal[:, None].expand(-1, 6, 3).reshape(-1, 3)

    def density(u):
        return (torch.einsum("qb,tbm->tqm", phi.to(u.dtype), u[E.t]) * (E.area[:, None] * w)[:, :, None]).reshape(-1, u.shape[1])

    g, u = density(neumann), density(dirichlet)
    out = []
    for x in points.double().split(max(1, int(2.5e7 / len(y)))):
        d = y[None] - x[:, None]
        G, H = _green(d, k)
        out.append(-(G @ g) - (H * (d * normal[None]).sum(-1)) @ u)
    return torch.cat(out)


def _exact_gradient(s):
    E, k, points = _Exact(s["v"], s["t"]), s["k"], s["points"]
    g = s["neumann"].detach().to(torch.complex128)
    V, A = _exact_vk(E, k)
    u = torch.linalg.solve(A, -(V @ g))
    p = _exact_listen(E, k, g[:, None], u[:, None], points)[:, 0]
    pbar = 2.0 * p
    # D^H pbar by differentiating Re(pbar^H D u) with respect to u
    z = torch.zeros_like(u).requires_grad_(True)
    gz = torch.zeros_like(u)
    listen = (pbar.conj() * _exact_listen(E, k, gz[:, None], z[:, None], points)[:, 0]).real.sum()
    (dh,) = torch.autograd.grad(listen, z)
    lam = torch.linalg.solve(A.conj().t(), dh)
    grad_g = -(V.conj().t() @ lam)
    del V, A
    # with lam and u fixed: dL/dx of Re[pbar^H (-S g + D u) - lam^H (V g + (1/2 M - K) u)]
    x = E.x.clone().requires_grad_(True)
    gv = g.clone().requires_grad_(True)
    E.set(x)
    zero = (pbar.conj() * _exact_listen(E, k, gv[:, None], u[:, None], points)[:, 0]).real.sum()
    part, gs = torch.autograd.grad(zero, (x, gv))
    grad_x, grad_g = part, grad_g + gs
    E.set(x)
    m = (torch.ones((3, 3), dtype=torch.float64, device="cuda") + torch.eye(3, dtype=torch.float64, device="cuda")) / 12.0
    mass = (torch.einsum("ta,ab,tb->t", lam[E.t].conj(), m.to(u.dtype), u[E.t]).real * E.area).sum()
    grad_x = grad_x + torch.autograd.grad(-0.5 * mass, x)[0]
    with torch.no_grad():
        E.set(x)
        parts = [(r[0], r[3]) for r in E.regular(6, max(1, int(2.4e7 / (E.nt * 36))))]
    w, phi = _rule(6)
    lq, gq, uq = (torch.einsum("qb,tb->tq", phi.to(f.dtype), f[E.t]) for f in (lam.conj(), g, u))
    for i, apart in parts:
        E.set(x)
        quad = torch.einsum("qb,tbd->tqd", phi, E.corners)
        d = quad.reshape(1, -1, 3) - quad[i].reshape(-1, 1, 3)
        G, H = _green(d, k)
        dn = (d.reshape(len(i) * 6, E.nt, 6, 3) * E.normal[None, :, None]).sum(-1).reshape(len(i) * 6, -1)
        wj = (E.area[:, None] * w).reshape(-1)
        F = (G * (gq.reshape(-1) * wj) + H * dn * (uq.reshape(-1) * wj)).reshape(len(i), 6, E.nt, 6).sum(3)
        F = (F * apart[:, None, :]).sum(2) * lq[i] * (E.area[i][:, None] * w)
        grad_x = grad_x - torch.autograd.grad(F.real.sum(), x)[0]
    for i, j, pp, qq, lx, ly, ww in E.close(4, 2_000_000):
        E.set(x)
        a = torch.gather(E.corners[i], 1, pp[:, :, None].expand(-1, 3, 3))
        b = torch.gather(E.corners[j], 1, qq[:, :, None].expand(-1, 3, 3))
        ti, tj = torch.gather(E.t[i], 1, pp), torch.gather(E.t[j], 1, qq)
        d = torch.einsum("rc,ncd->nrd", ly, b) - torch.einsum("rc,ncd->nrd", lx, a)
        G, H = _green(d, k)
        cx, cy = lx.to(u.dtype), ly.to(u.dtype)
        F = (G * (g[tj] @ cy.t()) + H * (d * E.normal[j][:, None]).sum(-1) * (u[tj] @ cy.t())) * (lam.conj()[ti] @ cx.t()) * ww
        F = F.sum(1) * (4.0 * E.area[i] * E.area[j])
        grad_x = grad_x - torch.autograd.grad(F.real.sum(), x)[0]
    return p, grad_x.detach(), grad_g.detach()


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A, b = _operator(case, seed)
        x = torch.linalg.solve(A.to(torch.complex128), b.to(torch.complex128).reshape(len(b), -1))
        return x[:, 0] if b.dim() == 1 else x
    v, t = _shape(case["shape"], case["n"])
    if len(t) > 21000 and kind != "listen":  # minutes, or more than the card holds
        return None
    s = _inputs(case, seed)
    if kind == "gradient":
        return _exact_gradient(s)
    E, k = _Exact(s["v"], s["t"]), s["k"]
    wide = {f: s[f].to(torch.complex128) for f in ("neumann", "dirichlet") if f in s}
    if kind == "listen":
        p = _exact_listen(E, k, wide["neumann"].reshape(E.nv, -1), wide["dirichlet"].reshape(E.nv, -1), s["points"])
        return p[:, 0] if s["neumann"].dim() == 1 else p
    if kind == "assemble":
        return _exact_vk(E, k)
    if kind == "bm":
        return _exact_bm(E, k, case["approx"])
    if kind == "problem":
        V, A = _exact_vk(E, k)
        g = wide["neumann"].reshape(E.nv, -1)
        u = torch.linalg.solve(A, -(V @ g))
        p = _exact_listen(E, k, g, u, s["points"])
        return (u[:, 0], p[:, 0]) if s["neumann"].dim() == 1 else (u, p)
    us, ps = [], []
    for km, g in zip(s["ks"], wide["neumann"]):
        L, R = _exact_bm(E, km, True)
        u = torch.linalg.solve(L, R @ g)
        us.append(u)
        ps.append(_exact_listen(E, km, g[:, None], u[:, None], s["points"])[:, 0])
    return torch.stack(ps), torch.stack(us)
