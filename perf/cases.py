"""Workloads of the layer-potential operators, for timing and for comparing outputs.

A case is a plain dict; ``prepare`` makes what a program holds before the
call (meshes, densities on the GPU or the host, batches), ``run`` is one pass
through the package's public calls, ``exact`` the same outputs in 64 bits
from plain PyTorch. Kinds:

* ``fused``: SL and DL of one mesh on device pointers (the matvec of an
  iterative solver that lives on the GPU; both operators in one pass);
* ``host``: one operator on host vectors (easybem's own calling convention,
  the matvec of a SciPy solver);
* ``setup``: a new mesh, one DL and one SL apply, and the mesh dropped (easybem's
  driver sequence init_gpu, apply, apply, close_gpu on each refinement);
* ``batch``: SL and DL of many uneven ellipsoids in one pass;
* ``solve``: GMRES with refinement, several meshes with four data sets each;
* ``rhs``: Dirichlet right-hand sides 1/2 M g + K g for several data sets;
* ``hyper`` and ``linear``: the hypersingular operator and the P1 single layer
  on device pointers through the host call;
* ``potential``: the representation formula at points off the surface.

Mixed-precision calls return vectors that are good to about single precision,
and so are solutions known to a residual of 1e-8: their results are handed on
in float32, as a program that post-processes them in single precision does.
FP64 calls return float64.
"""
import functools
import math

import numpy as np
import torch

import easybem_b200 as eb
from easybem_b200 import meshes

# ---------------------------------------------------------------------------
# the cases


def _case(name, kind, shape, size, prec, **more):
    return {"name": name, "kind": kind, "shape": shape, "size": size, "prec": prec, "order": 4, **more}


def listed():
    return [
        # the smallest matvec a driver makes: 1,280 triangles, host vectors, FP64
        _case("host_sl_fp64_1280", "host", "sphere", 3, "fp64", op="sl"),
        # a small mesh on device pointers, where launches and idle SMs count
        _case("fused_mixed_5120", "fused", "sphere", 4, "mixed"),
        # an ordinary mesh whose size divides neither tiles nor cells
        _case("fused_mixed_torus_13530", "fused", "torus", 165, "mixed"),
        # the headline matvec: 81,920 triangles, mixed
        _case("fused_mixed_81920", "fused", "sphere", 6, "mixed"),
        # the default precision at the same scale, another surface
        _case("fused_fp64_torus_81608", "fused", "torus", 404, "fp64"),
        # the largest mesh of the benchmark configurations
        _case("fused_mixed_327680", "fused", "sphere", 7, "mixed"),
        # many uneven meshes in one pass (320 to 20,480 triangles each)
        _case("batch_mixed_24", "batch", "ellipsoids", 24, "mixed"),
        # whole solves to a residual of 1e-8, four data sets per mesh
        _case("solve_mixed_4x4", "solve", "ellipsoids", 4, "mixed"),
        # right-hand sides of a served request: five data sets, one torus
        _case("rhs_fp64_torus_17860x5", "rhs", "torus", 190, "fp64", cols=5),
        # Neumann problems: the hypersingular operator
        _case("hyper_mixed_20480", "hyper", "sphere", 5, "mixed"),
        # post-processing: the solution at points inside the surface
        _case("potential_mixed_50000", "potential", "sphere", 5, "mixed", points=50000),
        # a moving or refined surface: new mesh, DL, SL, dropped
        _case("setup_fp64_torus_5000", "setup", "torus", 100, "fp64"),
    ]


def draw(rng):
    """One more case: the kinds above over their whole ranges (512 to 327,680
    triangles for mixed matvecs, up to 81,920 in FP64), odd sizes among them."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fused", "fused", "fused", "host", "setup", "batch", "solve", "rhs", "hyper", "linear",
                       "potential"])
    prec = rng.choice(["mixed", "fp64"])
    c = {"kind": kind, "shape": "torus", "prec": prec, "order": 4}
    if kind == "fused":
        c["size"] = log_int(32, 790 if prec == "mixed" else 400)
    elif kind == "host":
        c["size"] = log_int(32, 400 if prec == "mixed" else 250)
        c["op"] = rng.choice(["sl", "dl"])
        c["order"] = rng.choice([4, 4, 4, 7, 9])
        if c["order"] > 4:
            c["size"] = min(c["size"], 128)
    elif kind == "setup":
        c["size"] = log_int(32, 250)
        c["order"] = rng.choice([4, 4, 9])
        if c["order"] > 4:
            c["size"] = min(c["size"], 96)
    elif kind == "batch":
        c["shape"] = "ellipsoids"
        c["size"] = log_int(3, 40)
    elif kind == "solve":
        c["shape"] = "ellipsoids"
        c["size"] = rng.randint(1, 6)
        c["prec"] = "mixed"
    elif kind == "rhs":
        c["size"] = log_int(32, 250)
        c["cols"] = rng.randint(1, 8)
    elif kind in ("hyper", "linear"):
        c["size"] = log_int(32, 256)
    else:
        c["size"] = log_int(48, 256)
        c["points"] = log_int(1000, 100000)
    return c


# ---------------------------------------------------------------------------
# inputs


@functools.lru_cache(maxsize=None)
def _icosphere(level):
    return meshes.icosphere(level)


def _surface(case, rng):
    """A smooth closed surface: a sphere whose radius varies by a few percent
    (a seeded combination of polynomials up to degree 4), or a torus."""
    if case["shape"] == "sphere":
        v, f = _icosphere(case["size"])
        x, y, z = v.T
        terms = (x, y, z, x * y, y * z, z * x, x * x - y * y, 3 * z * z - 1, x * y * z, x * (x * x - 3 * y * y),
                 x * y * (x * x - y * y), z * z * (x * x - y * y))
        r = 1.0 + 0.03 * sum(rng.normal() * t for t in terms)
        return v * np.maximum(r, 0.6)[:, None], f
    return meshes.torus(case["size"], float(rng.uniform(0.2, 0.4)))


def _ellipsoids(case, rng):
    """Ellipsoids of uneven size (icospheres of level 2 to 5 in turn), rotated and offset."""
    out = []
    for k in range(case["size"]):
        v, f = _icosphere((4, 2, 5, 3)[k % 4])
        out.append(((v * rng.uniform(0.5, 2.0, size=3)) @ meshes.random_rotation(rng).T + rng.uniform(-5, 5, size=3), f))
    return out


def _sources(rng, nodes, n):
    """n point sources outside the surface, as the data g = 1/|x - p| of a Dirichlet problem."""
    c = nodes.mean(axis=0)
    rad = np.linalg.norm(nodes - c, axis=1).max()
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    p = c + d * (rad * rng.uniform(2.0, 4.0, size=(n, 1)))
    return np.stack([1.0 / np.linalg.norm(nodes - q, axis=1) for q in p])


def _load(nodes, elems, g):
    """b_i = integral of g over triangle i, for P1 data g [n, nnodes]."""
    p = nodes[elems - 1]
    area = 0.5 * np.linalg.norm(np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), axis=1)
    return g[:, elems - 1].mean(axis=2) * area


def _inputs(case, seed):
    """Everything made from the seed, on the host."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("batch", "solve"):
        surf = _ellipsoids(case, rng)
        if kind == "batch":
            return {"surf": surf, "t": [rng.normal(size=len(f)) for _, f in surf],
                    "u": [rng.normal(size=len(v)) for v, _ in surf]}
        return {"surf": surf, "b": [_load(v, f, _sources(rng, v, 4)) for v, f in surf]}
    v, f = _surface(case, rng)
    d = {"surf": [(v, f)]}
    if kind == "rhs":
        d["g"] = _sources(rng, v, case["cols"])
    else:
        d["t"] = rng.normal(size=len(v) if kind == "linear" else len(f))
        d["u"] = rng.normal(size=len(v))
    if kind == "potential":
        # points inside: between the centre (sphere) or the tube's axis (torus) and the surface
        k = rng.integers(0, len(v), size=case["points"])
        axis = np.zeros_like(v[k])
        if case["shape"] == "torus":
            axis[:, :2] = v[k, :2] / np.linalg.norm(v[k, :2], axis=1, keepdims=True)
        d["points"] = axis + (v[k] - axis) * rng.uniform(0.05, 0.9, size=(len(k), 1))
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "setup":
        s.update(nodes=d["surf"][0][0], elems=d["surf"][0][1], t=d["t"], u=d["u"])
        return s
    s["meshes"] = [eb.Mesh(v, f, case["order"]) for v, f in d["surf"]]
    if kind == "fused":
        ne = s["meshes"][0].nelems
        s["t"], s["u"] = (torch.from_numpy(d[k]).cuda() for k in ("t", "u"))
        s["vq"] = torch.empty(2, ne, dtype=torch.float64, device="cuda")
    elif kind == "batch":
        s["batch"] = eb.Batch(s["meshes"], precision=case["prec"], sl_dl=True)
        s["t"], s["u"] = ([torch.from_numpy(x).cuda() for x in d[k]] for k in ("t", "u"))
        s["v"], s["q"] = ([torch.empty_like(x) for x in s["t"]] for _ in range(2))
        s["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()  # the inputs are there before the other stream reads them
    else:
        s.update({k: d[k] for k in ("t", "u", "g", "b", "points") if k in d})
    return s


# ---------------------------------------------------------------------------
# one pass


def run(s):
    case = s["case"]
    kind, prec = case["kind"], case["prec"]
    if kind == "setup":
        with eb.Mesh(s["nodes"], s["elems"], case["order"]) as m:
            q = m.apply_dl(s["u"], prec)
            v = m.apply_sl(s["t"], prec)
        out = [v, q]
        return out if prec == "fp64" else [x.astype(np.float32) for x in out]
    m = s["meshes"][0]
    if kind == "fused":
        v, q = s["vq"]
        m.apply_device(s["t"].data_ptr(), s["u"].data_ptr(), v.data_ptr(), q.data_ptr(), prec)
        return s["vq"] if prec == "fp64" else s["vq"].float()
    if kind == "batch":
        with torch.cuda.stream(s["stream"]):
            ptr = [[x.data_ptr() for x in s[k]] for k in ("t", "u", "v", "q")]
            s["batch"].apply_sl_dl_device(*ptr, stream=s["stream"].cuda_stream)
            out = [torch.cat(s["v"]), torch.cat(s["q"])]
            return out if prec == "fp64" else [x.float() for x in out]
    if kind == "solve":
        got = eb.solve(list(zip(s["meshes"], s["b"])), inner_precision=prec)
        return [x.astype(np.float32) for x, _ in got]
    if kind == "rhs":
        out = m.dirichlet_rhs(s["g"], prec)
    elif kind == "hyper":
        out = m.apply_hypersingular(s["u"], prec)
    elif kind == "linear":
        out = m.apply_sl_p1(s["t"], prec)
    elif kind == "potential":
        out = m.evaluate(s["points"], s["t"], s["u"], prec)
    else:
        out = m.apply_sl(s["t"], prec) if case["op"] == "sl" else m.apply_dl(s["u"], prec)
    return out if prec == "fp64" else out.astype(np.float32)


def _sizes(case):
    """(triangles, vertices) of each mesh."""
    if case["shape"] == "sphere":
        return [(20 * 4 ** case["size"], 10 * 4 ** case["size"] + 2)]
    if case["shape"] == "torus":
        n = case["size"] * max(3, case["size"] // 4)
        return [(2 * n, n)]
    return [(20 * 4 ** L, 10 * 4 ** L + 2) for L in ((4, 2, 5, 3)[k % 4] for k in range(case["size"]))]


def work(case):
    """What any evaluation needs: the geometry (vertices, triangles) and the
    densities read once, the results written once, every near-field integral
    (13 pairs a triangle) used once, every quadrature point formed and
    weighted once for each operator. The pair sum itself is not counted: its
    cost depends on how it is evaluated."""
    kind = case["kind"]
    points = {4: 7, 7: 16, 9: 25}[case["order"]]
    passes = {"rhs": case.get("cols", 1), "hyper": 3, "solve": 4 * 10, "fused": 2, "batch": 2, "setup": 2,
              "potential": 2}.get(kind, 1)
    nbytes = flops = 0
    for ne, nv in _sizes(case):
        nbytes += 24 * nv + 12 * ne + passes * (16 * ne + 12 * 13 * ne)
        flops += passes * ne * (2 * 13 + 10 * points)
    if kind == "potential":
        nbytes += 32 * case["points"]
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits: the Galerkin sums over all quadrature-point pairs of
# triangles without a common vertex, and the Sauter-Schwab integrals of the
# others (index 4: the 7-point rule of degree 5, 5 Gauss-Legendre points)

_R15 = math.sqrt(15.0)
_A, _B = (6.0 - _R15) / 21.0, (6.0 + _R15) / 21.0
_RULE = np.array([[1 / 3, 1 / 3, 9 / 80]] +
                 [[x, y, (155.0 - _R15) / 2400.0] for x, y in ((_A, _A), (_A, 1 - 2 * _A), (1 - 2 * _A, _A))] +
                 [[x, y, (155.0 + _R15) / 2400.0] for x, y in ((_B, _B), (_B, 1 - 2 * _B), (1 - 2 * _B, _B))])
_CHUNK = 1 << 28  # values of one temporary


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return [(float(a), float(b)) for a, b in zip(0.5 * (x + 1.0), 0.5 * w)]


def _dot(a, b):
    return (a * b).sum(-1)


def _cross(a, b):
    return torch.linalg.cross(a, b)


class _Surface:
    def __init__(self, nodes, elems):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.f = torch.from_numpy(np.asarray(elems, dtype=np.int64) - 1).to(dev)
        self.x = torch.from_numpy(nodes).to(dev)
        P = self.P = self.x[self.f]
        e1, e2 = P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]
        n = _cross(e1, e2)
        self.J = n.norm(dim=1)
        self.n = n / self.J[:, None]
        rule = torch.from_numpy(_RULE).to(dev)
        self.w = rule[:, 2]
        self.hat = torch.stack([1 - rule[:, 0] - rule[:, 1], rule[:, 0], rule[:, 1]], 1)  # [Q, 3]
        self.y = P[:, None, 0] + rule[None, :, 0, None] * e1[:, None] + rule[None, :, 1, None] * e2[:, None]
        self.wJ = self.w[None] * self.J[:, None]
        self.ne, self.Q, self.dev = len(self.f), len(rule), dev

    def tensor(self, a):
        return torch.from_numpy(np.asarray(a)).to(self.dev)

    def inverse(self, X):
        """1/|x - y| of points X against all quadrature points."""
        Y = self.y.reshape(-1, 3)
        r2 = (X[:, 0:1] - Y[:, 0]).square_()
        for d in (1, 2):
            t = X[:, d:d + 1] - Y[:, d]
            r2.addcmul_(t, t)
        return r2

    def chunks(self, rows, per_row):
        step = max(1, _CHUNK // (per_row * self.ne * self.Q))
        return [(a, min(rows, a + step)) for a in range(0, rows, step)]

    def dl_sum(self, inv3, X, S):
        """sum over sources of d_j(x) s_b / r^3 for strengths S [ne, Q]."""
        G = (inv3.view(len(X), self.ne, self.Q) * S).sum(-1)
        D = torch.zeros_like(G)
        for d in range(3):
            D.addcmul_(X[:, d:d + 1] - self.P[:, 0, d], self.n[:, d].expand_as(D))
        return (G * D).sum(-1)

    def operators(self, T=None, U=None, matrix=False):
        """V T for T [ne, k], K U for U [nv, k], and the matrix of V."""
        V = torch.zeros_like(T) if T is not None else None
        K = torch.zeros(self.ne, U.shape[1], dtype=torch.float64, device=self.dev) if U is not None else None
        A = torch.zeros(self.ne, self.ne, dtype=torch.float64, device=self.dev) if matrix else None
        S = [self.wJ * (U[self.f][:, None, :, c] * self.hat).sum(-1) for c in range(U.shape[1])] if U is not None else []
        near = []
        for a, b in self.chunks(self.ne, self.Q):
            fa = self.f[a:b]
            share = torch.zeros(b - a, self.ne, dtype=torch.bool, device=self.dev)
            for k in range(3):
                for l in range(3):
                    share |= fa[:, k:k + 1] == self.f[:, l]
            pairs = share.nonzero()
            pairs[:, 0] += a
            near.append(pairs)
            X = self.y[a:b].reshape(-1, 3)
            inv = self.inverse(X)
            inv.view(b - a, self.Q, self.ne, self.Q).masked_fill_(share[:, None, :, None], math.inf)
            inv.rsqrt_()
            w = self.wJ[a:b] / (4 * math.pi)
            if T is not None:
                c = (self.wJ[..., None] * T[:, None]).reshape(-1, T.shape[1])
                V[a:b] = ((inv @ c).view(b - a, self.Q, -1) * w[..., None]).sum(1)
            if matrix:
                A[a:b] = ((inv.view(-1, self.ne, self.Q) * self.wJ).sum(-1).view(b - a, self.Q, -1) * w[..., None]).sum(1)
            if U is not None:
                inv = inv * inv * inv
                for c, s in enumerate(S):
                    K[a:b, c] = (self.dl_sum(inv, X, s).view(b - a, self.Q) * w).sum(1)
            del inv
        i, j = torch.cat(near).T
        sl, dl, cols = self.singular(i, j)
        if T is not None:
            V.index_add_(0, i, sl[:, None] * T[j])
        if matrix:
            A[i, j] += sl
        if U is not None:
            K.index_add_(0, i, (dl[..., None] * U[cols]).sum(1))
        return V, K, A

    def singular(self, i, j):
        """SL value, DL weights and their vertices for pairs with common vertices."""
        fi, fj = self.f[i], self.f[j]
        eq = fj[:, :, None] == fi[:, None, :]  # [pair, k of j, l of i]
        count = eq.sum((1, 2))
        count[i == j] = 0
        sl = torch.zeros(len(i), dtype=torch.float64, device=self.dev)
        dl = torch.zeros(len(i), 3, dtype=torch.float64, device=self.dev)
        cols = fj.clone()
        q = _gauss(5)
        q2 = _gauss(2)

        def moment(s):
            return sum(w * x * (1.0 - x * s) for x, w in q2)

        m2, m1 = sum(w * x * x for x, w in q2), moment(1.0)

        def corner(P, k):
            return P.gather(1, (k % 3)[:, None, None].expand(-1, 1, 3))[:, 0]

        def r1(a):
            return _dot(a, a).rsqrt()

        def flux(a, n):
            return _dot(a, n) * _dot(a, a).rsqrt() ** 3

        sel = (i == j).nonzero()[:, 0]
        P = self.P[i[sel]]
        u, v = P[:, 1] - P[:, 0], P[:, 2] - P[:, 1]
        s = sum(w * (r1(e * u + v) + r1(e * v + u) + r1(e * (u + v) - v)) for e, w in q)
        sl[sel] = _dot(_cross(u, v), _cross(u, v)) * s / (12 * math.pi)

        sel = ((count == 1) & (i != j)).nonzero()[:, 0]
        if len(sel):
            e = eq[sel]
            d, c = e.any(2).long().argmax(1), e.any(1).long().argmax(1)
            Pi, Pj = self.P[i[sel]], self.P[j[sel]]
            p0, p1, p2 = (corner(Pi, c + k) for k in range(3))
            t0, t1, t2 = (corner(Pj, d + k) for k in range(3))
            u, v, w, z = p1 - p0, p2 - p1, t1 - t0, t2 - t1
            nt = _cross(w, z)
            jt = nt.norm(dim=1)
            n, jac = nt / jt[:, None], _cross(u, v).norm(dim=1) * jt
            s = torch.zeros_like(jt)
            k = [torch.zeros_like(jt) for _ in range(3)]
            for e1, w1 in q:
                a, b = u + e1 * v, w + e1 * z
                for e2, w2 in q:
                    for e3, w3 in q:
                        ww = w1 * w2 * w3 * e2
                        va, vb = a - e2 * (w + e3 * z), e2 * (u + e3 * v) - b
                        s += ww * (r1(va) + r1(vb))
                        h, g = ww * flux(va, n), ww * flux(vb, n)
                        k[0] += moment(e2) * h + m1 * g
                        k[1] += m2 * (e2 * (1 - e3) * h + (1 - e1) * g)
                        k[2] += m2 * (e2 * e3 * h + e1 * g)
            sl[sel] = jac * s / (12 * math.pi)
            dl[sel] = torch.stack(k, 1) * (jac / (4 * math.pi))[:, None]
            cols[sel] = fj[sel].gather(1, (d[:, None] + torch.arange(3, device=self.dev)) % 3)

        sel = ((count == 2) & (i != j)).nonzero()[:, 0]
        if len(sel):
            e = eq[sel]
            free = e.any(2).long().argmin(1)  # the vertex of j that is not shared
            c0, c1 = (free + 1) % 3, (free + 2) % 3
            ri = e.any(1).long().argmin(1)
            Pi, Pj = self.P[i[sel]], self.P[j[sel]]
            q0, q1, qr, pr = corner(Pj, c0), corner(Pj, c1), corner(Pj, free), corner(Pi, ri)
            u, v, w = q1 - q0, pr - q1, qr - q1
            nt = _cross(u, w)
            jt = nt.norm(dim=1)
            n, jac = nt / jt[:, None], _cross(u, v).norm(dim=1) * jt
            s = torch.zeros_like(jt)
            k = [torch.zeros_like(jt) for _ in range(3)]
            for e2, w2 in q:
                for e3, w3 in q:
                    a = 0.5 * e2
                    ab = a * e3
                    vs = (e2 * (e3 * (u + w) - w) + v, v - e2 * (u + v + e3 * w), e2 * (v - e3 * (u + v)) - w,
                          v - e2 * (w + e3 * (u + v)), e2 * (u + w) + e3 * v - w)
                    fac = ((moment(1 - ab), 1 - a, a * (1 - e3)), (m1, 1 - ab, ab), (m1, 0.5, 0.5),
                           (m1, 1 - a, a), (moment(1 - a), 0.5, 0.5 * (1 - e2)))
                    for x, (f0, f1, f2), t in zip(vs, fac, (e2, e2, e2, e2, 1.0)):
                        ww = w2 * w3 * t
                        s += ww * r1(x)
                        h = ww * flux(x, n)
                        k[0] += f0 * h
                        k[1] += m2 * f1 * h
                        k[2] += m2 * f2 * h
            sl[sel] = jac * s / (24 * math.pi)
            dl[sel] = torch.stack(k, 1) * (jac / (4 * math.pi))[:, None]
            cols[sel] = torch.stack([fj[sel].gather(1, c[:, None])[:, 0] for c in (c0, c1, free)], 1)
        return sl, dl, cols

    def potential(self, X, t, u):
        out = torch.zeros(len(X), dtype=torch.float64, device=self.dev)
        c = (self.wJ * t[:, None]).reshape(-1)
        S = self.wJ * (u[self.f][:, None] * self.hat).sum(-1)
        for a, b in self.chunks(len(X), 1):
            inv = self.inverse(X[a:b]).rsqrt_()
            out[a:b] = (inv @ c - self.dl_sum(inv * inv * inv, X[a:b], S)) / (4 * math.pi)
        return out

    def curls(self):
        """Surface curls of the three hat functions, [ne, 3 (component), 3 (vertex)]."""
        e1, e2 = self.P[:, 1] - self.P[:, 0], self.P[:, 2] - self.P[:, 0]
        a11, a22, a12 = _dot(e1, e1), _dot(e2, e2), _dot(e1, e2)
        det = (a11 * a22 - a12 * a12)[:, None]
        b1, b2 = _cross(self.n, e1), _cross(self.n, e2)
        y1 = (b1 * a22[:, None] - b2 * a12[:, None]) / det
        y2 = (b2 * a11[:, None] - b1 * a12[:, None]) / det
        return torch.stack([-y1 - y2, y1, y2], 2)


def exact(case, seed):
    kind = case["kind"]
    if case["order"] != 4 or kind == "linear" or max(ne for ne, _ in _sizes(case)) > 90000:
        return None
    d = _inputs(case, seed)
    surf = [_Surface(v, f) for v, f in d["surf"]]
    m = surf[0]
    if kind == "batch":
        vq = [s.operators(s.tensor(t)[:, None], s.tensor(u)[:, None]) for s, t, u in zip(surf, d["t"], d["u"])]
        return [torch.cat([x[k][:, 0] for x in vq]) for k in (0, 1)]
    if kind == "solve":
        return [torch.linalg.solve(s.operators(matrix=True)[2], s.tensor(b).T).T.contiguous().cpu().numpy()
                for s, b in zip(surf, d["b"])]
    if kind == "rhs":
        g = m.tensor(d["g"]).T
        b = m.operators(U=g)[1] + (m.J / 12.0)[:, None] * g[m.f].sum(1)
        return b.T.contiguous().cpu().numpy()
    u = m.tensor(d["u"])
    if kind == "potential":
        return m.potential(m.tensor(d["points"]), m.tensor(d["t"]), u).cpu().numpy()
    if kind == "hyper":
        C = m.curls()
        W = m.operators((C * u[m.f][:, None]).sum(2))[0]
        q = torch.zeros_like(u)
        return q.index_add_(0, m.f.reshape(-1), (C * W[:, :, None]).sum(1).reshape(-1)).cpu().numpy()
    t = m.tensor(d["t"])
    op = case.get("op", "both")
    v, q, _ = m.operators(t[:, None] if op != "dl" else None, u[:, None] if op != "sl" else None)
    if kind == "host":
        return (v if op == "sl" else q)[:, 0].cpu().numpy()
    if kind == "fused":
        return torch.stack([v[:, 0], q[:, 0]])
    return [v[:, 0].cpu().numpy(), q[:, 0].cpu().numpy()]
