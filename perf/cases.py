"""The work that programs give this framework, as cases that can be timed.

Every case goes through the public Python entry points.  The sizes are those of this repository's
tests, of its benchmark and of its workloads (sphere, torus, batches of ellipsoids and tori, union of
spheres), from the smallest reconstruction that the tests run (depth 5) to the benchmark's own
(2,000,000 points at depth 10).  Clouds are drawn on the GPU from the seed alone.

A program keeps one context and gives it cloud after cloud, so the cases of one configuration share a
context; the cases that need the state of an earlier call (the operator) hold one of their own.
"""
import math

import numpy as np
import torch

import poissonreconstruction_b200 as prb

# The largest clouds that the ranges reach.
MAX_POINTS = 2_000_000


def listed():
    return [
        # one small object of the test suite: latency, launches and synchronisations
        dict(name="mesh_d5", op="mesh", shape="sphere", points=4_000, depth=5, degree=1, pw=4.0, precision="mixed"),
        # a preview with the quadratic basis, its implicit function wanted rather than its mesh
        dict(name="solve_d6_deg2", op="solve", shape="torus", points=6_000, depth=6, degree=2, pw=4.0,
             precision="mixed"),
        # a scan of one object at the low end of the batched workload, points and depth uneven
        dict(name="mesh_d7", op="mesh", shape="ellipsoid", points=20_011, depth=7, degree=1, pw=4.0,
             precision="mixed"),
        # the plain method's sphere at the default depth, without screening as the defaults have it
        dict(name="mesh_d8_default", op="mesh", shape="sphere", points=100_000, depth=8, degree=1, pw=0.0,
             precision="mixed"),
        # the plain method as its workload names it: quadratic B-splines, screening 4, FP64 throughout
        dict(name="mesh_d8_deg2_f64", op="mesh", shape="sphere", points=100_000, depth=8, degree=2, pw=4.0,
             precision="f64"),
        # an ordinary scan, an odd number of points, the crate's basis
        dict(name="mesh_d9", op="mesh", shape="torus", points=317_003, depth=9, degree=1, pw=4.0,
             precision="mixed"),
        # the benchmark's cloud with the crate's basis, points and mesh resident on the device
        dict(name="device_d10", op="device", shape="torus", points=2_000_000, depth=10, degree=1, pw=4.0,
             precision="mixed"),
        # the benchmark's own workload: degree 2, points and mesh resident on the device
        dict(name="device_d10_deg2", op="device", shape="torus", points=2_000_000, depth=10, degree=2, pw=4.0,
             precision="mixed"),
        # a step of the adjoint workload: forward solve, then the gradients of a loss at surface samples
        dict(name="adjoint_d9", op="adjoint", shape="ellipsoid", points=1_000_000, depth=9, degree=1, pw=4.0,
             precision="mixed", queries=200_000),
        # part of the batched workload: uneven clouds of depth 7 to 9 by size in one call
        dict(name="batch_16", op="batch", points=300_000, low=10_000, clouds=16, pw=4.0, precision="mixed"),
        # a large scene on the narrow band around its points
        dict(name="band_d11", op="device", shape="spheres", points=1_500_001, depth=11, coarse=8, degree=2, pw=4.0,
             precision="mixed"),
        # the operator by itself, as a solver of the user's own applies it: a vector on the device
        dict(name="operator_d9", op="operator", shape="torus", points=200_000, depth=9, degree=1, pw=4.0,
             precision="mixed"),
    ]


def _points_for(rng, depth, low=1_500):
    """Points per surface cell of the grid from sparse scans (0.4) to dense ones (6)."""
    n = 4.0 ** depth * math.exp(rng.uniform(math.log(0.4), math.log(6.0)))
    return int(min(MAX_POINTS, max(low, n)))


def draw(rng):
    op = rng.choice(["mesh", "mesh", "mesh", "device", "device", "solve", "adjoint", "batch", "band", "operator"])
    pw = rng.choice([4.0, 4.0, 4.0, 0.0, round(rng.uniform(1.0, 8.0), 3)])
    if op == "batch":
        low = int(math.exp(rng.uniform(math.log(4_000), math.log(30_000))))
        high = int(math.exp(rng.uniform(math.log(35_000), math.log(300_000))))
        return dict(op=op, points=high, low=low, clouds=rng.randint(3, 16), pw=4.0, precision="mixed")
    if op == "band":
        depth = rng.choice([9, 10, 11])
        return dict(op="device", shape="spheres", points=min(1_500_000, _points_for(rng, depth)), depth=depth,
                    coarse=min(8, depth - rng.choice([2, 3])), degree=2, pw=4.0, precision="mixed")
    degree = rng.choice([1, 1, 2])
    precision = rng.choice(["mixed", "mixed", "mixed", "f64"])
    depth = {"mesh": lambda: rng.randint(5, 9), "device": lambda: rng.randint(7, 10),
             "solve": lambda: rng.randint(4, 8), "adjoint": lambda: rng.randint(6, 9),
             "operator": lambda: rng.randint(6, 9)}[op]()
    if depth == 10:
        precision = "mixed"
    case = dict(op=op, shape=rng.choice(["sphere", "torus", "ellipsoid"]), points=_points_for(rng, depth), depth=depth,
                degree=degree, pw=pw, precision=precision)
    if op == "adjoint":
        case["points"] = min(case["points"], 1_000_000)
        case["queries"] = max(1, case["points"] // rng.choice([1, 3, 5, 20]))
        case["queries"] = min(case["queries"], 200_000)
    return case


# ---------------------------------------------------------------------- clouds
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _uniform(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _tilt(g, nrm, angles):
    a = _normal(g, *nrm.shape)
    a = _unit(a - (a * nrm).sum(1, keepdim=True) * nrm)
    return _unit(torch.cos(angles)[:, None] * nrm + torch.sin(angles)[:, None] * a)


def _sphere(g, n):
    u = _unit(_normal(g, n, 3))
    return torch.cat([u, u], 1)  # FP64, exact normals


def _torus(g, n, R=1.0, r=0.35, noise=0.002, sigma=0.05):
    v = _uniform(g, 3 * n + 4096, 0.0, 2 * math.pi)
    v = v[_uniform(g, v.numel()) < (R + r * torch.cos(v)) / (R + r)][:n]
    u = _uniform(g, n, 0.0, 2 * math.pi)
    cu, su, cv, sv = torch.cos(u), torch.sin(u), torch.cos(v), torch.sin(v)
    pos = torch.stack([(R + r * cv) * cu, (R + r * cv) * su, r * sv], 1) + noise * _normal(g, n, 3)
    nrm = _tilt(g, torch.stack([cv * cu, cv * su, sv], 1), sigma * _normal(g, n))
    return torch.cat([pos, nrm], 1).float().double()


def _ellipsoid(g, n, radii, noise=0.001, sigma=0.0):
    ax = torch.tensor(radii, device="cuda", dtype=torch.float64)
    pos = _unit(_normal(g, n, 3)) * ax
    nrm = _unit(pos / ax ** 2)
    if sigma:
        nrm = _tilt(g, nrm, sigma * _uniform(g, n))
    return torch.cat([pos + noise * _normal(g, n, 3), nrm], 1).float().double()


def _spheres(g, n, count=32):
    c, r = torch.rand(count, 3, generator=g, device="cuda", dtype=torch.float64), _uniform(g, count, 0.05, 0.3)
    m = n - n // 100
    k = torch.multinomial(r * r, 6 * m + 4096, replacement=True, generator=g)
    u = _unit(_normal(g, k.numel(), 3))
    pos = c[k] + r[k, None] * u
    keep = torch.ones_like(k, dtype=torch.bool)
    for j in range(count):
        keep &= ((pos - c[j]).square().sum(1) >= r[j] * r[j]) | (k == j)
    surf = torch.cat([pos, u], 1)[keep]
    surf = surf[torch.arange(m, device="cuda") % surf.shape[0]]
    far = torch.cat([torch.rand(n - m, 3, generator=g, device="cuda", dtype=torch.float64),
                     _unit(_normal(g, n - m, 3))], 1)  # 1% outliers
    return torch.cat([surf, far], 0)[torch.randperm(n, generator=g, device="cuda")].float().double()


def _cloud(g, shape, n):
    if shape == "sphere":
        return _sphere(g, n)
    if shape == "torus":
        return _torus(g, n)
    if shape == "ellipsoid":
        return _ellipsoid(g, n, (1.0, 0.7, 0.5), sigma=math.radians(20.0))
    return _spheres(g, n)


def _batch_sizes(case):
    k = case["clouds"]
    return [int(round(case["low"] * (case["points"] / case["low"]) ** (i / (k - 1)))) for i in range(k)]


def _depth_of(n):
    return 7 if n < 40_000 else (8 if n < 160_000 else 9)  # the batched workload's rule


# ---------------------------------------------------------------------- state
_shared = {"key": None, "context": None}


def _context(case):
    """The program's context: one for all clouds of a configuration."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _shared["key"] != key:
        if _shared["context"] is not None:
            _shared["context"].close()
        _shared["context"] = prb.Context(0) if case["op"] != "batch" else None
        _shared["key"] = key
    return _shared["context"]


def _params(case, depth=None):
    return prb.ReconstructParams(depth=depth or case["depth"], point_weight=case["pw"], degree=case.get("degree", 1),
                                 coarse_depth=case.get("coarse", 0),
                                 precision=prb.PR_PRECISION_FP64 if case["precision"] == "f64"
                                 else prb.PR_PRECISION_MIXED)


def prepare(case, seed):
    g = _generator(seed)
    op = case["op"]
    state = dict(op=op, context=_context(case))
    if op == "batch":
        clouds, params = [], []
        for i, n in enumerate(_batch_sizes(case)):
            a, b, c = (float(t) for t in _uniform(g, 3, 0.3, 1.0).cpu())
            pts = (_ellipsoid(g, n, (a, b, c)) if i % 2 else
                   _torus(g, n, R=max(a, b) + 0.01, r=min(a, b), noise=0.001, sigma=0.0))
            clouds.append(pts.cpu().numpy())
            params.append(_params(case, _depth_of(n)))
        return dict(state, clouds=clouds, params=params, meshes=[_MeshBuffers(p.depth) for p in params])
    state["params"] = _params(case)
    pts = _cloud(g, case["shape"], case["points"])
    if op == "device":
        mesh = _MeshBuffers(case["depth"])
        torch.cuda.synchronize()
        return dict(state, points=pts, mesh=mesh)
    state["points"] = pts.cpu().numpy()
    if op == "adjoint":  # samples of the same surface that are not points of the cloud
        q = _cloud(g, case["shape"], case["queries"])[:, :3]
        return dict(state, queries=q.cpu().numpy())
    if op == "operator":
        stream = torch.cuda.Stream()
        context = prb.Context(0, stream=stream.cuda_stream)
        context.solve(state["points"], state["params"])
        dtype = torch.float64 if case["precision"] == "f64" else torch.float32
        x = torch.randn(8 ** case["depth"], generator=g, device="cuda", dtype=dtype)
        torch.cuda.synchronize()
        return dict(state, context=context, stream=stream, x=x, y=torch.empty_like(x))
    return dict(state, mesh=_MeshBuffers(case["depth"])) if op == "mesh" else state


class _DeviceArray:
    """A library-owned device array, for torch.as_tensor."""

    def __init__(self, ptr, rows, typestr):
        self.__cuda_array_interface__ = dict(shape=(rows, 3), typestr=typestr, data=(ptr, False), version=2)


class _MeshBuffers:
    """Where the program keeps a cloud's mesh, whose size differs from cloud to cloud, beyond the next
    call: a viewer's vertex and triangle buffers on the GPU, with room for any mesh of the depth, zero
    past its end."""

    def __init__(self, depth):
        self.vertices = torch.zeros(12 * 4 ** depth + 4096, 3, dtype=torch.float64, device="cuda")
        self.triangles = torch.zeros(24 * 4 ** depth + 8192, 3, dtype=torch.int64, device="cuda")
        self.used = [0, 0]

    def take(self, vertices, triangles, stats):
        for k, (to, new) in enumerate(((self.vertices, vertices), (self.triangles, triangles))):
            n = new.shape[0]
            to[:n].copy_(new)
            if n < self.used[k]:
                to[n:self.used[k]].zero_()
            self.used[k] = n
        return dict(vertices=self.vertices, triangles=self.triangles, n_vertices=vertices.shape[0],
                    n_triangles=triangles.shape[0], iso=stats.iso_value)

    def take_host(self, mesh, stats):
        return self.take(torch.from_numpy(mesh.vertices), torch.from_numpy(mesh.triangles.view(np.int64)), stats)


def run(state):
    op, context = state["op"], state["context"]
    if op == "mesh":
        return state["mesh"].take_host(*context.reconstruct(state["points"], state["params"]))
    if op == "device":
        points = state["points"]
        stats = context.reconstruct_device(points.data_ptr(), points.shape[0], state["params"])
        dv, nv, dt, nt = context.mesh_device()
        return state["mesh"].take(torch.as_tensor(_DeviceArray(dv, nv, "<f8"), device="cuda"),
                                  torch.as_tensor(_DeviceArray(dt, nt, "<i8"), device="cuda"), stats)
    if op == "solve":
        context.solve(state["points"], state["params"])
        return dict(coefficients=context.coefficients())
    if op == "adjoint":
        context.solve(state["points"], state["params"])
        chi, dpos, dnrm, stats = context.loss_backward(state["queries"])
        return dict(chi=chi, dpositions=dpos, dnormals=dnrm, loss=stats.loss)
    if op == "batch":
        out = prb.reconstruct_batch(state["clouds"], state["params"])
        kept = [b.take_host(*r) for b, r in zip(state["meshes"], out)]
        return [[k["vertices"], k["triangles"], k["iso"]] for k in kept]
    context.apply_operator_device(state["x"].data_ptr(), state["y"].data_ptr(), state["params"].precision)
    return dict(y=state["y"])


# ---------------------------------------------------------------------- work
def _grid_work(n, degree, width):
    """The system's solution cannot do without its right-hand side read and its coefficients written,
    nor with less than one application of the operator (21 or 125 points)."""
    return 2 * width * n, 2 * (21 if degree == 1 else 125) * n


def work(case):
    op = case["op"]
    if op == "batch":
        each = [work(dict(op="mesh", points=n, depth=_depth_of(n), degree=1)) for n in _batch_sizes(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    res = 2 ** case["depth"]
    points = 48 * case["points"]
    if op == "operator":
        width = 8 if case["precision"] == "f64" else 4
        b, f = _grid_work(res ** 3, case["degree"], width)
        # besides the vectors, each point's nodes and weights
        return dict(bytes=b + (8 if case["degree"] == 1 else 27) * (4 + width) * case["points"] * (case["pw"] > 0),
                    flops=f)
    nodes = res ** 3
    if case.get("coarse"):  # 8^3 bricks about the surface (2.6 bricks for each 8 x 8 square of it), and the coarse grid
        nodes = int(2.6 * 512 * (res / 8) ** 2 * 4) + 8 ** case["coarse"]
    b, f = _grid_work(nodes, case["degree"], 8)
    b += points
    if op in ("mesh", "device"):
        b += 8 * nodes + 230 * res * res  # coefficients read, vertices and triangles written
    if op == "adjoint":  # a second solve; chi and both gradients written
        b, f = 2 * b + points + 32 * case["queries"], 2 * f
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------- the values in 64 bits
def _morton(depth, device):
    """Natural index (x fastest) of every Morton index (x in bit 0)."""
    m = torch.arange(8 ** depth, device=device)
    c = [torch.zeros_like(m) for _ in range(3)]
    for bit in range(depth):
        for a in range(3):
            c[a] |= ((m >> (3 * bit + a)) & 1) << bit
    return c[0] + (c[1] << depth) + (c[2] << (2 * depth))


def _filter(x, band, axis):
    """Banded Toeplitz matrix along one axis of a (z, y, x) grid, rows cut at its faces."""
    out, half, n = torch.zeros_like(x), len(band) // 2, x.shape[axis]
    for d in range(-half, half + 1):
        w = band[d + half]
        if w:
            k = n - abs(d)
            out.narrow(axis, max(0, -d), k).add_(x.narrow(axis, max(0, d), k), alpha=w)
    return out


_M = {1: [1 / 6, 2 / 3, 1 / 6], 2: [1 / 120, 13 / 60, 11 / 20, 13 / 60, 1 / 120]}
_S = {1: [-1.0, 2.0, -1.0], 2: [-1 / 6, -1 / 3, 1.0, -1 / 3, -1 / 6]}
_G = {1: [0.5, 0.0, -0.5], 2: [1 / 24, 5 / 12, 0.0, -5 / 12, -1 / 24]}


class _System:
    """A x = b of a cloud in FP64 with plain torch, natural order."""

    def __init__(self, case, points):
        self.degree, depth, pw = case["degree"], case["depth"], case["pw"]
        self.res = 1 << depth
        self.h = 1.0 / self.res
        pos, nrm = points[:, :3], points[:, 3:]
        lo, hi = pos.min(0).values, pos.max(0).values
        u = (pos - 0.5 * (lo + hi)) * (1.1 / (hi - lo).max()) + 0.5
        self.wh3 = pw * self.h ** 3 / 1.5
        self.wg = self.wh3 * 0.005
        self.key, self.phi = self.pairs(u, torch.trunc if self.degree == 1 else torch.floor)
        key, w = self.pairs(u, torch.floor)
        n = self.res ** 3
        field = torch.zeros(3, n + 1, device=u.device, dtype=torch.float64)
        total = torch.zeros(n + 1, device=u.device, dtype=torch.float64).index_add_(0, key.reshape(-1), w.reshape(-1))
        unit = _unit(nrm)
        for a in range(3):
            field[a].index_add_(0, key.reshape(-1), (w * unit[:, a:a + 1]).reshape(-1))
        field = torch.where(total > 0, -field / torch.where(total > 0, total, 1.0), field)[:, :n]
        grid = field.view(3, self.res, self.res, self.res)
        b = torch.zeros_like(grid[0])
        for a in range(3):
            t = grid[a]
            for axis in range(3):
                t = _filter(t, (_G if axis == a else _M)[self.degree], 2 - axis)
            b += self.h ** 2 * t
        self.b = b.reshape(-1) + 0.5 * self.wh3 * self.gather(torch.ones_like(self.phi[:, 0]))

    def pairs(self, u, cell):
        s = u * self.res
        c = cell(s)
        t = s - c
        if self.degree == 1:
            w, first = torch.stack([1 - t, t], 2), 0
        else:
            w, first = torch.stack([0.5 * (1 - t) ** 2, 0.5 * (-2 * t * t + 2 * t + 1), 0.5 * t * t], 2), -1
        k = w.shape[2]
        node = c.long()[:, :, None] + first + torch.arange(k, device=u.device)
        ok = (node >= 0) & (node < self.res)
        x, y, z = node[:, 0], node[:, 1], node[:, 2]
        index = (x[:, None, None, :] + self.res * (y[:, None, :, None] + self.res * z[:, :, None, None]))
        ok = ok[:, 0][:, None, None, :] & ok[:, 1][:, None, :, None] & ok[:, 2][:, :, None, None]
        weight = w[:, 0][:, None, None, :] * w[:, 1][:, None, :, None] * w[:, 2][:, :, None, None]
        index = torch.where(ok, index, self.res ** 3).reshape(len(u), -1)
        return index, torch.where(ok, weight, 0.0).reshape(len(u), -1)

    def gather(self, v):
        """sum_p v_p phi(p)"""
        out = torch.zeros(self.res ** 3 + 1, device=v.device, dtype=torch.float64)
        return out.index_add_(0, self.key.reshape(-1), (self.phi * v[:, None]).reshape(-1))[:-1]

    def apply(self, x):
        M, S = _M[self.degree], _S[self.degree]
        g = x.view(self.res, self.res, self.res)
        mx, sx = _filter(g, M, 2), _filter(g, S, 2)
        mm, ms = _filter(mx, M, 1), _filter(mx, S, 1) + _filter(sx, M, 1)
        y = self.h * (_filter(mm, S, 0) + _filter(ms, M, 0))
        y = y.reshape(-1) + self.wg * x
        if self.wh3:
            y += self.wh3 * self.gather((self.phi * torch.cat([x, x.new_zeros(1)])[self.key]).sum(1))
        return y

    def solve(self, tol=1e-14):
        x, r = torch.zeros_like(self.b), self.b.clone()
        d, rr = r.clone(), r.dot(r)
        stop = tol * tol * rr
        for it in range(20 * self.res):
            q = self.apply(d)
            alpha = rr / d.dot(q)
            x += alpha * d
            r -= alpha * q
            new = r.dot(r)
            if it % 16 == 0 and bool(new <= stop):
                break
            d = r + (new / rr) * d
            rr = new
        return x


def exact(case, seed):
    """Coefficients and operator products; meshes and gradients follow from whole solves at sizes where
    plain torch takes too long, or have no plain form."""
    op = case["op"]
    if op not in ("solve", "operator") or (op == "solve" and case["depth"] > 7):
        return None
    g = _generator(seed)
    system = _System(case, _cloud(g, case["shape"], case["points"]))
    natural = _morton(case["depth"], "cuda")
    if op == "solve":
        return dict(coefficients=system.solve()[natural].cpu().numpy())
    dtype = torch.float64 if case["precision"] == "f64" else torch.float32
    x = torch.randn(8 ** case["depth"], generator=g, device="cuda", dtype=dtype).double()
    grid = torch.empty_like(x)
    grid[natural] = x
    return dict(y=system.apply(grid)[natural])
