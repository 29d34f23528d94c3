"""Timing cases of the matrix fill: what a user of the package has it do, over the sizes it is used at.

A case is a dict of plain values.  `prepare` makes the spaces, operator and configuration a program holds
before it calls the package, `run` is the one call that fills the matrix (`assemble_gpu` or
`assemble_batch`), `work` counts the bytes and operations the fill cannot do without, and `exact` is the
same matrix in 64 bits from plain torch, written from the rules' definitions.

Keys of a case: mesh ("sphere", "box", "plate", "fold", "curve", "ellipsoids") with its sizes, op, k (wave
number), precision ("fp64" or "mixed"), out ("host" or "device"), far_test / far_trial (points of the
far-pair rules, triangle meshes), row0 / nrows (a row window; nrows = 0 is the whole matrix).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import beastgpu_gb300 as bg

DEV = "cuda:0"
F8 = torch.float64

TRI_OPS = {
    "hh_sl": (bg.Helmholtz3D.singlelayer, bg.lagrangec0d1),
    "hh_dl": (bg.Helmholtz3D.doublelayer, bg.lagrangec0d1),
    "hh_dlt": (bg.Helmholtz3D.doublelayer_transposed, bg.lagrangec0d1),
    "hh_hs": (bg.Helmholtz3D.hypersingular, bg.lagrangec0d1),
    "efie": (bg.Maxwell3D.singlelayer, bg.raviartthomas),
    "mfie": (bg.Maxwell3D.doublelayer, bg.raviartthomas),
}
CURVE_OPS = {
    "sl": bg.Helmholtz2D.singlelayer,
    "dl": bg.Helmholtz2D.doublelayer,
    "dlt": bg.Helmholtz2D.doublelayer_transposed,
    "hs": bg.Helmholtz2D.hypersingular,
}


def _case(name, mesh, op, k, precision, out, far_test=3, far_trial=4, row0=0, nrows=0, **sizes):
    c = {"mesh": mesh, "op": op, "k": float(k), "precision": precision, "out": out, "far_test": far_test,
         "far_trial": far_trial, "row0": row0, "nrows": nrows, **sizes}
    return {"name": name, **c} if name else c


def listed():
    pi = math.pi
    return [
        # the reference's correctness case, one step finer: a matrix of a hundred unknowns, all latency
        _case("box_4_hh_sl_fp64_host", "box", "hh_sl", 1.0, "fp64", "host", nx=4, ny=4, nz=4),
        # a small antenna or unit-test scatterer through the drop-in call: 480 RWG, FP64, numpy result
        _case("sphere_2_efie_fp64_host", "sphere", "efie", 2 * pi, "fp64", "host", level=2),
        # the plain FP64 drop-in on a scatterer of ordinary size, matrix left on the device for a solver
        _case("sphere_4_efie_fp64_device", "sphere", "efie", 4 * pi, "fp64", "device", level=4),
        # the reference's benchmark family (Helmholtz single layer on a cuboid) in its own precision
        _case("box_24_hh_sl_fp64_device", "box", "hh_sl", 1.0, "fp64", "device", nx=24, ny=24, nz=24),
        # the benchmark workload: 30,720 RWG, mixed precision, matrix in device memory
        _case("sphere_5_efie_mixed_device", "sphere", "efie", 8 * pi, "mixed", "device", level=5),
        # the reference's benchmark family in mixed precision, an odd box
        _case("box_41_hh_sl_mixed_device", "box", "hh_sl", 1.0, "mixed", "device", nx=41, ny=37, nz=43),
        # near-singular work: two jittered plates almost touching at a fold
        _case("fold_64_mfie_mixed_device", "fold", "mfie", 4 * pi, "mixed", "device", n=64),
        # what the default call hands a CPU solver: a new numpy matrix
        _case("sphere_4_efie_mixed_host", "sphere", "efie", 4 * pi, "mixed", "host", level=4),
        # the other Helmholtz operators of a combined-field formulation: hypersingular
        _case("sphere_4_hh_hs_mixed_device", "sphere", "hh_hs", 4 * pi, "mixed", "device", level=4),
        # a user who asks for more accurate far pairs (6 x 7 points)
        _case("sphere_4_efie_6x7_mixed_device", "sphere", "efie", 4 * pi, "mixed", "device", 6, 7, level=4),
        # many small scatterers of uneven size in one call
        _case("ellipsoids_24_efie_mixed_device", "ellipsoids", "efie", 5.0, "mixed", "device", count=24, top=3),
        # the 2-D path: hypersingular on a curve
        _case("curve_8192_hs_mixed_device", "curve", "hs", 100 * pi, "mixed", "device", n=8192),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    precision = rng.choice(["fp64", "mixed", "mixed"])
    out = rng.choice(["host", "device", "device"])
    kind = rng.choice(["sphere", "box", "box", "plate", "fold", "curve", "ellipsoids"])
    if kind == "curve":
        n = logint(48, 2500 if precision == "fp64" else 9000)
        return _case("", "curve", rng.choice(sorted(CURVE_OPS)), rng.uniform(0.5, 0.04 * n), precision, out, n=n)
    if kind == "ellipsoids":
        return _case("", kind, rng.choice(["efie", "mfie"]), rng.uniform(2.0, 8.0), precision, "device",
                     count=rng.randint(3, 20), top=2 if precision == "fp64" else 3)
    # a plate: no double layer, which vanishes on a plane
    op = rng.choice(["hh_sl", "hh_hs", "efie"] if kind == "plate" else sorted(TRI_OPS))
    far = rng.choice([(3, 4), (3, 4), (3, 4), (4, 6), (6, 7)])
    small = precision == "fp64" or far != (3, 4)
    if kind == "sphere":
        sizes = {"level": rng.randint(1, 3 if small else 4)}
        nfun = {"efie": 30, "mfie": 30}.get(op, 10) * 4 ** sizes["level"] + (0 if op in ("efie", "mfie") else 2)
    elif kind == "box":
        top = 16 if small else 36
        sizes = {"nx": logint(2, top), "ny": logint(2, top), "nz": logint(2, top)}
        cells = 2 * (sizes["nx"] * sizes["ny"] + sizes["ny"] * sizes["nz"] + sizes["nz"] * sizes["nx"])
        nfun = 3 * cells if op in ("efie", "mfie") else cells + 2
    else:
        sizes = {"n": logint(3, (30 if small else 72) if kind == "fold" else (44 if small else 100))}
        n = sizes["n"]
        nfun = (3 * n * n - 2 * n if op in ("efie", "mfie") else (n - 1) ** 2) * (2 if kind == "fold" else 1)
    row0, nrows = 0, 0
    if rng.random() < 0.25:  # one rank's rows of a matrix that is split over several processes
        nrows = rng.randint(max(1, nfun // 8), max(1, nfun // 2))
        row0 = rng.randint(0, nfun - nrows)
    return _case("", kind, op, rng.uniform(0.5, 20.0), precision, out, far[0], far[1], row0, nrows, **sizes)


# ---- inputs --------------------------------------------------------------------------------------


def _mesh(case, rng):
    """The case's surface: its vertices depend on the seed, its connectivity does not."""
    kind = case["mesh"]
    if kind == "sphere":
        return bg.ellipsoid(case["level"], rng.uniform(0.85, 1.15, 3))
    if kind == "box":
        n = np.array([case["nx"], case["ny"], case["nz"]])
        m = bg.meshcuboid(*(float(x) for x in n), 1.0)
        return bg.Mesh(m.vertices / n.max() * rng.uniform(0.95, 1.05, 3), m.triangles)
    if kind == "plate":
        return bg.plate(case["n"], 0.3, int(rng.integers(1 << 30)))
    # the second plate 0.01 beside the first, turned up by 30 degrees about its edge
    m = bg.two_plates(case["n"], 0.3, int(rng.integers(1 << 30)), 0.01)
    v = m.vertices.copy()
    up = v[:, 0] > 1.005
    x = v[up, 0] - 1.01
    v[up, 0], v[up, 2] = 1.01 + x * math.cos(math.pi / 6), x * math.sin(math.pi / 6)
    return bg.Mesh(v, m.triangles)


def _inputs(case, seed):
    """(problems, quadrature): the operator and space of each matrix of the case."""
    rng = np.random.default_rng(seed)
    if case["mesh"] == "curve":
        m = bg.ellipse(case["n"], 1.0, 0.5, jitter=0.2, seed=int(rng.integers(1 << 30)))
        return [(CURVE_OPS[case["op"]](wavenumber=case["k"]), bg.curve_lagrangec0d1(m))], bg.QuadStrat2D()
    make_op, make_space = TRI_OPS[case["op"]]
    qs = bg.QuadStrat(far_test=case["far_test"], far_trial=case["far_trial"])
    if case["mesh"] == "ellipsoids":
        levels = [1 + i % case["top"] for i in range(case["count"])]
        probs = []
        for lev in levels:
            m = bg.ellipsoid(lev, rng.uniform(0.7, 1.4, 3))
            probs.append((make_op(wavenumber=case["k"] * rng.uniform(0.5, 1.5)), make_space(m)))
        return probs, qs
    k = case["k"] * rng.uniform(0.95, 1.05)
    return [(make_op(wavenumber=k), make_space(_mesh(case, rng)))], qs


def prepare(case, seed):
    problems, qs = _inputs(case, seed)
    return {"case": case, "problems": problems, "qs": qs, "config": bg.GPUConfiguration(precision=case["precision"])}


def run(state):
    case, cfg, qs = state["case"], state["config"], state["qs"]
    if case["mesh"] == "ellipsoids":
        return bg.assemble_batch([(op, X, X) for op, X in state["problems"]], cfg, quadstrat=qs, out=case["out"])
    (op, X), = state["problems"]
    rows = (case["row0"], case["nrows"]) if case["nrows"] else None
    return bg.assemble_gpu(op, X, X, cfg, quadstrat=qs, out=case["out"], rows=rows)


def _cells(case):
    """(cells, functions) of each matrix of the case, without making the mesh."""
    kind, rt = case["mesh"], case["op"] in ("efie", "mfie")
    if kind == "curve":
        return [(case["n"], case["n"])]
    if kind in ("sphere", "ellipsoids"):
        levels = [case["level"]] if kind == "sphere" else [1 + i % case["top"] for i in range(case["count"])]
        return [(20 * 4 ** v, 30 * 4 ** v if rt else 10 * 4 ** v + 2) for v in levels]
    if kind == "box":
        q = 2 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nz"] * case["nx"])
        return [(2 * q, 3 * q if rt else q + 2)]
    n, c = case["n"], 2 if kind == "fold" else 1
    return [(c * 2 * n * n, c * (3 * n * n - 2 * n if rt else (n - 1) ** 2))]


def work(case):
    """Each point pair of the far rule: 15 operations and 3 transcendental functions for the kernel and the
    accumulation into the local matrix (45 Helmholtz, 108 EFIE, 180 MFIE; 2-D: 40 in all); each vertex and
    table read once, each matrix entry written once."""
    entry = 16 if case["precision"] == "fp64" else 8
    nbytes = flops = 0.0
    for cells, nfun in _cells(case):
        rows = case["nrows"] or nfun
        if case["mesh"] == "curve":
            flops += cells * cells * 16 * 40
            nbytes += cells * (16 + 8 + 8 + 16) + entry * rows * nfun
            continue
        acc = {"efie": 108, "mfie": 180}.get(case["op"], 45)
        flops += cells * cells * (rows / nfun) * case["far_test"] * case["far_trial"] * (18 + acc)
        nbytes += cells * (12 + 12 + 12 + 24) + entry * rows * nfun
    return {"bytes": nbytes, "flops": flops}


# ---- the same matrices in 64 bits ----------------------------------------------------------------

_RULES = {  # symmetric triangle rules (Dunavant): orbits (barycentric a, b, c; weight), points in u, v order
    3: [((2 / 3, 1 / 6, 1 / 6), 1 / 3)],
    4: [((1 / 3, 1 / 3, 1 / 3), -0.5625), ((0.6, 0.2, 0.2), 25 / 48)],
    6: [((0.10810301816807023, 0.4459484909159649, 0.4459484909159649), 0.22338158967801147),
        ((0.8168475729804585, 0.09157621350977074, 0.09157621350977074), 0.10995174365532187)],
    7: [((1 / 3, 1 / 3, 1 / 3), 0.225),
        ((0.05971587178976982, 0.4701420641051151, 0.4701420641051151), 0.1323941527885062),
        ((0.7974269853530873, 0.10128650732345634, 0.10128650732345634), 0.12593918054482714)],
    12: [((0.5014265096581791, 0.24928674517091043, 0.24928674517091043), 0.11678627572637937),
         ((0.8738219710169955, 0.06308901449150223, 0.06308901449150223), 0.05084490637020682),
         ((0.053145049844816945, 0.3103524510337844, 0.6365024991213987), 0.08285107561837357)],
    13: [((1 / 3, 1 / 3, 1 / 3), -0.14957004446768174),
         ((0.47930806784192037, 0.2603459660790398, 0.2603459660790398), 0.1756152574332078),
         ((0.8697397941955683, 0.06513010290221581, 0.06513010290221581), 0.05334723560883849),
         ((0.04869031542531641, 0.31286549600487384, 0.6384441885698098), 0.07711376089025714)],
}


def _rule(n):
    """Barycentric points [n, 3] and weights [n] (sum 1)."""
    pts, wts = [], []
    for b, w in _RULES[n]:
        seen = sorted({(b[i], b[j], b[3 - i - j]) for i in range(3) for j in range(3) if i != j})
        pts += seen
        wts += [w] * len(seen)
    lam = torch.tensor(pts, dtype=F8, device=DEV)
    lam[:, 2] = 1 - lam[:, 0] - lam[:, 1]
    return lam, torch.tensor(wts, dtype=F8, device=DEV)


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return (x + 1) / 2, w / 2


class _Tri:
    """Per-triangle tables: vertices [n, 3, 3], area, unit normal, surface curls of the hats [n, 3, 3]."""

    def __init__(self, v):
        self.v = v
        nn = torch.linalg.cross(v[:, 0] - v[:, 2], v[:, 1] - v[:, 2])
        two_a = nn.norm(dim=1)
        self.area = two_a / 2
        self.n = nn / two_a[:, None]
        self.curl = (v[:, [1, 2, 0]] - v[:, [2, 0, 1]]) / two_a[:, None, None]

    def at(self, i, perm=None):
        t = object.__new__(_Tri)
        t.v, t.area, t.n, t.curl = self.v[i], self.area[i], self.n[i], self.curl[i]
        if perm is not None:  # vertices (and the hats' curls) taken in another order; the normal stays
            e = perm[:, :, None].expand(-1, -1, 3)
            t.v, t.curl = t.v.gather(1, e), t.curl.gather(1, e)
        return t


def _green(r2, k):
    R = r2.sqrt()
    a = 1 / (4 * math.pi * R)
    return R, a * torch.cos(k * R), -a * torch.sin(k * R)


def _contract(kind, op, A, B, la, lb, K, H):
    """Local matrices [.., i, j] (real, imaginary) of pairs from kernel values K = (re, im) [pair, point]
    at matching points la / lb [point, 3] with the weights in them; H holds G'/R the same way."""
    x, y = torch.einsum("na,pac->pnc", la, A.v), torch.einsum("na,pac->pnc", lb, B.v)
    if kind in ("efie", "mfie"):
        f = (x[:, :, None] - A.v[:, None]) / (2 * A.area)[:, None, None, None]
        g = (y[:, :, None] - B.v[:, None]) / (2 * B.area)[:, None, None, None]
    out = []
    for q in range(2):
        if kind == "hh_sl":
            L = torch.einsum("pn,na,nb->pab", K[q], la, lb)
        elif kind == "hh_dl":
            L = torch.einsum("pn,na,nb->pab", -H[q] * ((x - y) * B.n[:, None]).sum(-1), la, lb)
        elif kind == "hh_dlt":
            L = torch.einsum("pn,na,nb->pab", H[q] * ((x - y) * A.n[:, None]).sum(-1), la, lb)
        elif kind == "hh_hs":
            L = (torch.einsum("pn,na,nb->pab", K[q], la, lb) * (A.n * B.n).sum(-1)[:, None, None],
                 torch.einsum("pac,pbc->pab", A.curl, B.curl) * K[q].sum(1)[:, None, None])
        elif kind == "efie":
            L = (torch.einsum("pn,pnac,pnbc->pab", K[q], f, g),
                 (K[q].sum(1) / (A.area * B.area))[:, None, None].expand(-1, 3, 3))
        else:
            d = (x - y)[:, :, None]
            L = torch.einsum("pn,pnac,pnbc->pab", H[q], f, torch.linalg.cross(d.expand_as(g), g))
        out.append(L)
    return _combine(op, out)


def _combine(op, parts):
    re, im = parts
    if isinstance(re, tuple):
        return complex(op.alpha) * torch.complex(re[0], im[0]) + complex(op.beta) * torch.complex(
            re[1].contiguous(), im[1].contiguous())
    return complex(op.alpha) * torch.complex(re, im)


def _pair_kernel(A, B, la, lb, wt, k):
    """Weighted G and G'/R at matching points of pairs: ((re, im), (re, im)), each [pair, point]."""
    x, y = torch.einsum("na,pac->pnc", la, A.v), torch.einsum("na,pac->pnc", lb, B.v)
    r2 = ((x - y) ** 2).sum(-1)
    R, gr, gi = _green(r2, k)
    w = wt * (4 * A.area * B.area)[:, None]
    gr, gi = gr * w, gi * w
    # G' / R = -(1/R + i k) G / R
    return (gr, gi), ((-(gr / R - k * gi)) / R, (-(gi / R + k * gr)) / R)


def _ss_points(cls, n):
    """Sauter-Schwab rule of a class (1 vertex, 2 edge, 3 face): chart points of both triangles as
    barycentrics of their reordered vertices, and weights."""
    q, w = _gauss(n)
    h1, h2, h3, xi = (a.ravel() for a in np.meshgrid(q, q, q, q, indexing="ij"))
    wt = np.prod(np.meshgrid(w, w, w, w, indexing="ij"), axis=0).ravel() * xi ** 3
    if cls == 1:
        a, b = (1 - xi, xi * h1), (1 - xi * h2, xi * h2 * h3)
        regions = [(a, b, wt * h2), (b, a, wt * h2)]
    elif cls == 2:
        m, m5 = wt * h1 ** 2 * h2, wt * h1 ** 2
        x1 = xi * h1
        e = (1 - xi * (1 - h1 * h2 * h3), x1 * h2 * (1 - h3))
        regions = [((1 - xi, x1), e, m), ((1 - xi * (1 - h1 * h2), x1 * (1 - h2)), (1 - xi, x1 * h2 * h3), m),
                   (e, (1 - xi, x1), m), ((1 - xi * (1 - h1 * h2 * h3), x1 * (1 - h2 * h3)), (1 - xi, x1 * h2), m),
                   ((1 - xi, x1 * h3), (1 - xi * (1 - h1 * h2), x1 * (1 - h2)), m5)]
    else:
        m, x1 = wt * h1 ** 2 * h2, xi * h1
        a, b, c = xi - x1 + x1 * h2, 1 - xi + x1 * h2 * h3, xi - x1
        d, e, f, g = x1 * (1 - h2 + h2 * h3), 1 - xi + x1 * h2, x1 * (1 - h2), x1 * (1 - h2 * h3)
        regions = [((1 - xi, a), (b, c), m), ((b, c), (1 - xi, a), m), ((1 - xi, d), (e, f), m),
                   ((e, f), (1 - xi, d), m), ((b, g), (1 - xi, f), m), ((1 - xi, f), (b, g), m)]

    def bary(which):
        u = np.concatenate([r[which][0] for r in regions])
        v = np.concatenate([r[which][1] for r in regions])
        return torch.tensor(np.stack([u, v, 1 - u - v], 1), dtype=F8, device=DEV)

    return bary(0), bary(1), torch.tensor(np.concatenate([r[2] for r in regions]), dtype=F8, device=DEV)


def _orders(cls, same):
    """Vertex orders of both triangles that put the shared vertices where the rule wants them; `same`
    [pair, 3, 3] marks coinciding vertices (test, trial)."""
    n = same.shape[0]
    i = torch.arange(3, device=DEV)
    if cls == 3:
        return i.expand(n, 3).contiguous(), same.to(torch.int64).argmax(2)
    flat = same.reshape(n, 9).to(torch.int64)
    hit = (flat * torch.arange(9, 0, -1, device=DEV)).topk(cls, dim=1).indices.sort(1).values  # in (i, j) order
    out = []
    for s in (hit // 3, hit % 3):
        if cls == 1:  # shared, then the lower and the higher other
            a = s[:, 0]
            b = torch.where(a == 0, 1, 0)
            out.append(torch.stack([a, b, 3 - a - b], 1))
        else:  # second shared, the vertex off the edge, first shared
            a, b = s[:, 0], s[:, 1]
            out.append(torch.stack([b, 3 - a - b, a], 1))
    return out


def _back(L, pa, pb):
    """L of reordered triangles, in the triangles' own orders."""
    out = torch.zeros_like(L)
    p = torch.arange(L.shape[0], device=DEV)[:, None, None]
    out[p, pa[:, :, None], pb[:, None, :]] = L
    return out


def _potentials(T, x):
    """Closed-form integrals over flat triangles at points x [pair, point, 3]: of 1/R, R, d/R^3 and of
    (y - rho) times 1/R, R, 1/R^3 (rho the foot of x, d its height)."""
    n = T.n[:, None]
    d = (n * (x - T.v[:, 2][:, None])).sum(-1)
    rho = x - d[..., None] * n
    tf, tk = torch.zeros_like(d), torch.zeros_like(d)
    jm1, j1, jm3 = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
    for e in range(3):
        a, b = T.v[:, e][:, None], T.v[:, (e + 1) % 3][:, None]
        l = (b - a) / (b - a).norm(dim=-1, keepdim=True)
        m = torch.linalg.cross(l, n.expand_as(l))
        sp, sm, t0 = ((b - rho) * l).sum(-1), ((a - rho) * l).sum(-1), ((a - rho) * m).sum(-1)
        rp, rm = (x - b).norm(dim=-1), (x - a).norm(dim=-1)
        r02 = t0 * t0 + d * d
        f = torch.where((sp < 0) & (sm < 0), torch.log((rm - sm) / (rp - sp)),
                        torch.where(sm >= 0, torch.log((rp + sp) / (rm + sm)),
                                    torch.log((rp + sp) * (rm - sm) / r02)))
        k1 = 0.5 * (sp * rp - sm * rm + r02 * f)
        k3 = 0.25 * (sp * rp ** 3 - sm * rm ** 3) + 0.75 * r02 * k1
        tf, tk = tf + t0 * f, tk + t0 * k1
        jm1, j1, jm3 = jm1 + m * k1[..., None], j1 + m * (k3 / 3)[..., None], jm3 - m * f[..., None]
    q = T.v[:, None] - x[:, :, None]
    r = q.norm(dim=-1)
    q0, q1, q2 = q.unbind(2)
    trip = (q0 * torch.linalg.cross(q1, q2)).sum(-1)
    den = (r.prod(-1) + (q0 * q1).sum(-1) * r[..., 2] + (q0 * q2).sum(-1) * r[..., 1] + (q1 * q2).sum(-1) * r[..., 0])
    om = -2 * torch.atan2(trip, den)
    im1 = tf - d * om
    i1 = (d * d * im1 + tk) / 3
    return d, rho, im1, i1, om, jm1, j1, jm3


def _near(kind, op, A, B, k, outer=12, inner=13):
    """Near pairs: 1/R - i k - k^2 R / 2 over the trial triangle in closed form at the outer rule's points,
    the smooth rest by the double rule."""
    if kind == "hh_dlt":  # the double layer seen from the trial side
        return _near("hh_dl", op, B, A, k, inner, outer).transpose(1, 2)
    lo, wo = _rule(outer)
    li, wi = _rule(inner)
    # the rest: G_r = (e^-z - 1 + z - z^2/2) / (4 pi R), G_r'/R = -(z e2 + e3) / (4 pi R^3), z = i k R
    la, lb = lo.repeat_interleave(inner, 0), li.repeat(outer, 1)
    wt = (wo[:, None] * wi[None]).reshape(-1) / 4
    x, y = torch.einsum("na,pac->pnc", la, A.v), torch.einsum("na,pac->pnc", lb, B.v)
    R = (x - y).norm(dim=-1)
    z = torch.complex(torch.zeros_like(R), k * R)
    series = torch.ones_like(z)
    for n in range(24, 3, -1):
        series = 1 + series * (-z) / n
    e3 = torch.where(z.abs() < 1, (-z) ** 3 / 6 * series, torch.exp(-z) - 1 + z - z * z / 2)
    e2 = e3 + z * z / 2
    w = wt * (4 * A.area * B.area)[:, None]
    g, h = e3 * w / (4 * math.pi * R), -(z * e2 + e3) * w / (4 * math.pi * R ** 3)
    L = _contract(kind, op, A, B, la, lb, (g.real, g.imag), (h.real, h.imag))
    # the singular terms
    x = torch.einsum("na,pac->pnc", lo, A.v)
    w = wo * A.area[:, None]
    d, rho, im1, i1, om, jm1, j1, jm3 = _potentials(B, x)
    gam, g2h = 1j * k, -k * k / 2
    cen = B.v.mean(1)[:, None]
    c4 = 1 / (4 * math.pi)
    s0 = (im1 - gam * B.area[:, None] + g2h * i1) * c4
    sv = (jm1 - gam * B.area[:, None, None] * (cen - rho) + g2h * j1) * c4
    grad = torch.linalg.cross(B.n[:, None].expand(-1, 3, -1), B.v[:, [2, 0, 1]] - B.v[:, [1, 2, 0]])
    grad = grad / (2 * B.area)[:, None, None]
    hat = 1 / 3 + torch.einsum("pjc,pnc->pnj", grad, rho - cen)
    gc = grad.to(torch.complex128)
    alpha, beta = complex(op.alpha), complex(op.beta)
    if kind in ("hh_sl", "hh_hs", "hh_dl"):
        a0, av = s0, sv
        if kind == "hh_dl":
            a0 = (om - g2h * d * im1) * c4
            av = (d[..., None] * jm3 - g2h * d[..., None] * jm1) * c4
        inner_j = a0[..., None] * hat + torch.einsum("pjc,pnc->pnj", gc, av.to(torch.complex128))
        S = torch.einsum("pn,na,pnj->paj", w.to(torch.complex128), lo.to(torch.complex128), inner_j)
        if kind != "hh_hs":
            return L + alpha * S
        cc = torch.einsum("pac,pbc->pab", A.curl, B.curl)
        return L + alpha * S * (A.n * B.n).sum(-1)[:, None, None] + beta * cc * (w * s0).sum(1)[:, None, None]
    f = (x[:, :, None] - A.v[:, None]) / (2 * A.area)[:, None, None, None]
    if kind == "efie":
        gj = (sv[:, :, None] + s0[..., None, None] * (rho[:, :, None] - B.v[:, None])) / (2 * B.area)[:, None, None, None]
        S = torch.einsum("pn,pnac,pnbc->pab", w.to(torch.complex128), f.to(torch.complex128), gj)
        return L + alpha * S + beta * ((w * s0).sum(1) / (A.area * B.area))[:, None, None]
    n = B.n[:, None]
    gv = (jm3 - n * om[..., None] + g2h * (d[..., None] * n * im1[..., None] - jm1)) * c4
    xw = (x[:, :, None] - B.v[:, None]) / (2 * B.area)[:, None, None, None]
    cr = torch.linalg.cross(gv[:, :, None].expand_as(xw), xw)
    return L + alpha * torch.einsum("pn,pnac,pnbc->pab", w, f, cr)


def _far_rows(kind, op, A, B, k, qt, qb, nonfar):
    """Far-rule local matrices [T, S, 3, 3] of the test triangles A against all of B; pairs in `nonfar`
    [T, S] are zero."""
    lt, wt = _rule(qt)
    lb, wb = _rule(qb)
    x, y = torch.einsum("na,tac->tnc", lt, A.v), torch.einsum("na,sac->snc", lb, B.v)
    T, S = x.shape[0], y.shape[0]
    d = x.reshape(T, qt, 1, 1, 3) - y.reshape(1, 1, S, qb, 3)
    r2 = (d * d).sum(-1)
    w = (wt[None] * A.area[:, None])[:, :, None, None] * (wb[None] * B.area[:, None])[None, None]
    w = w * (~nonfar)[:, None, :, None]
    R, gr, gi = _green(torch.where(nonfar[:, None, :, None], torch.ones_like(r2), r2), k)
    K = [gr * w, gi * w]
    if kind in ("hh_dl", "hh_dlt", "mfie"):
        K = [-(K[0] / R - k * K[1]) / R, -(K[1] / R + k * K[0]) / R]
        if kind == "hh_dl":
            rn = -torch.einsum("tisjc,sc->tisj", d, B.n)
        elif kind == "hh_dlt":
            rn = torch.einsum("tisjc,tc->tisj", d, A.n)
        if kind != "mfie":
            K = [q * rn for q in K]
    del d, r2, w
    out = []
    if kind.startswith("hh"):
        for q in K:
            L = torch.einsum("tisb,ia->tsab", torch.einsum("tisj,jb->tisb", q, lb), lt)
            if kind == "hh_hs":
                nn = torch.einsum("tc,sc->ts", A.n, B.n)
                L = (L * nn[..., None, None],
                     torch.einsum("tac,sbc->tsab", A.curl, B.curl) * q.sum((1, 3))[..., None, None])
            out.append(L)
        return _combine(op, out)
    f = (x[:, :, None] - A.v[:, None]) / (2 * A.area)[:, None, None, None]  # [t, i, a, c]
    g = (y[:, :, None] - B.v[:, None]) / (2 * B.area)[:, None, None, None]  # [s, j, b, c]
    if kind == "efie":
        for q in K:
            L = torch.einsum("tisbc,tiac->tsab", torch.einsum("tisj,sjbc->tisbc", q, g), f)
            D = q.sum((1, 3)) / (A.area[:, None] * B.area[None])
            out.append((L, D[..., None, None].expand(-1, -1, 3, 3)))
        return _combine(op, out)
    # f . ((x - y) x g) = g . (f x x) - f . (y x g), coordinates from the block's centre
    o = x.mean((0, 1))
    fx = torch.linalg.cross(f, (x - o)[:, :, None].expand_as(f))
    yg = torch.linalg.cross((y - o)[:, :, None].expand_as(g), g)
    for q in K:
        L = torch.einsum("tisbc,tiac->tsab", torch.einsum("tisj,sjbc->tisbc", q, g), fx)
        out.append(L - torch.einsum("tisbc,tiac->tsab", torch.einsum("tisj,sjbc->tisbc", q, yg), f))
    return _combine(op, out)


def _supports(space):
    """Padded supports of every function: positions in the flattened (cell, local) axis and coefficients."""
    idx = torch.as_tensor(space.fn_index.astype(np.int64)).reshape(-1)
    coef = torch.as_tensor(space.fn_coef).reshape(-1)
    where = torch.nonzero(idx >= 0)[:, 0]
    f = idx[where]
    order = torch.argsort(f, stable=True)
    where, f = where[order], f[order]
    count = torch.bincount(f, minlength=space.nfun)
    start = torch.cumsum(count, 0) - count
    slot = torch.arange(f.numel()) - start[f]
    width = int(count.max())
    pos = torch.zeros((space.nfun, width), dtype=torch.int64)
    c = torch.zeros((space.nfun, width), dtype=F8)
    pos[f, slot] = where
    c[f, slot] = coef[where]
    return pos.to(DEV), c.to(DEV)


def _exact_triangles(op, kind, X, qs):
    m = X.mesh
    v = torch.as_tensor(m.vertices, device=DEV)
    tri = torch.as_tensor(m.triangles.astype(np.int64), device=DEV)
    T = _Tri(v[tri])
    k = op.wavenumber
    nt, nf = m.nt, X.nfun
    pos, coef = _supports(X)
    Z = torch.zeros((nf, nf), dtype=torch.complex128, device=DEV)
    fidx = torch.as_tensor(X.fn_index.astype(np.int64), device=DEV)
    fcoef = torch.as_tensor(X.fn_coef, device=DEV)
    far_pts = qs.far_test * qs.far_trial
    step = max(1, int(1.2e9 / (nt * far_pts * 8 * 3)))
    nonfar = []
    for t0 in range(0, nt, step):
        t1 = min(nt, t0 + step)
        hits = torch.zeros((t1 - t0, nt), dtype=torch.int64, device=DEV)
        dmin2 = torch.full((t1 - t0, nt), math.inf, dtype=F8, device=DEV)
        for a in range(3):
            for b in range(3):
                hits += tri[t0:t1, a][:, None] == tri[:, b][None]
                dmin2 = torch.minimum(dmin2, ((T.v[t0:t1, a][:, None] - T.v[:, b][None]) ** 2).sum(-1))
        near = (hits == 0) & (torch.maximum(dmin2 * k * k, dmin2 / (16 * T.area[None])) < 0.04)
        special = (hits > 0) | near
        p = torch.nonzero(special)
        nonfar.append((p[:, 0] + t0, p[:, 1], torch.where(near, 4, hits)[p[:, 0], p[:, 1]]))
        L = _far_rows(kind, op, T.at(slice(t0, t1)), T, k, qs.far_test, qs.far_trial, special)
        L = L.permute(0, 2, 1, 3).reshape((t1 - t0) * 3, nt * 3)
        H = torch.zeros((L.shape[0], nf), dtype=L.dtype, device=DEV)
        for s in range(pos.shape[1]):
            H += L[:, pos[:, s]] * coef[:, s]
        rows, c = fidx[t0:t1].reshape(-1), fcoef[t0:t1].reshape(-1)
        ok = rows >= 0
        Z.index_add_(0, rows[ok], H[ok] * c[ok][:, None])
        del L, H
    ti, si, cls = (torch.cat(q) for q in zip(*nonfar))
    for code in (1, 2, 3, 4):
        sel = torch.nonzero(cls == code)[:, 0]
        if code < 4:
            la, lb, wt = _ss_points(code, (0, qs.ss_cv, qs.ss_ce, qs.ss_cf)[code])
        for p0 in range(0, sel.numel(), 8192):
            q = sel[p0:p0 + 8192]
            t, s = ti[q], si[q]
            if code == 4:
                L = _near(kind, op, T.at(t), T.at(s), k, qs.near_test, qs.near_trial)
            elif code == 3 and kind in ("hh_dl", "hh_dlt", "mfie"):
                continue  # vanishes on a flat triangle
            else:
                pa, pb = _orders(code, tri[t][:, :, None] == tri[s][:, None, :])
                A, B = T.at(t, pa), T.at(s, pb)
                K, H = _pair_kernel(A, B, la, lb, wt, k)
                L = _back(_contract(kind, op, A, B, la, lb, K, H), pa, pb)
            rows, cols = fidx[t][:, :, None].expand(-1, 3, 3), fidx[s][:, None, :].expand(-1, 3, 3)
            val = L * (fcoef[t][:, :, None] * fcoef[s][:, None, :])
            ok = (rows >= 0) & (cols >= 0)
            Z.index_put_((rows[ok], cols[ok]), val[ok], accumulate=True)
    return Z


def _bessel_series(z, order):
    """J and Y of order 0 or 1 for z < 2 from the power series (Abramowitz & Stegun 9.1.10-9.1.13)."""
    q = -z * z / 4
    term = torch.ones_like(z) if order == 0 else z / 2
    digamma = -0.5772156649015329 * 2 + (0.0 if order == 0 else 1.0)  # psi(k + 1) + psi(k + order + 1)
    J, S = torch.zeros_like(z), torch.zeros_like(z)
    for k in range(16):
        J, S = J + term, S + term * digamma
        term = term * q / ((k + 1) * (k + 1 + order))
        digamma += 1 / (k + 1) + 1 / (k + 1 + order)
    Y = (2 * torch.log(z / 2) * J - S) / math.pi
    return J, Y if order == 0 else Y - 2 / (math.pi * z)


def _bessel_recurrence(z, order):
    """The same for 2 <= z < 25: downward recurrence with sum rule, Y by Neumann's series (9.1.46, 9.1.88-89)."""
    top = 78
    up, cur = torch.zeros_like(z), torch.full_like(z, 1e-290)
    norm, S, J = torch.zeros_like(z), torch.zeros_like(z), {}
    for n in range(top, -1, -1):  # cur is J_n up to the common factor
        if n % 2 == 0:
            norm = norm + cur * (1 if n == 0 else 2)
        k = (n - order) // 2
        if (n - order) % 2 == 0 and k >= 1:
            S = S + cur * ((-1) ** k * (1 / k if order == 0 else (2 * k + 1) / (k * (k + 1))))
        if n < 2:
            J[n] = cur
        up, cur = cur, 2 * n / z * cur - up
    lead = torch.log(z / 2) + 0.5772156649015329 - order
    if order == 0:
        return J[0] / norm, (2 * lead * J[0] - 4 * S) / (math.pi * norm)
    return J[1] / norm, (2 * lead * J[1] - 2 * S - 2 * J[0] / z) / (math.pi * norm)


def _bessel_asymptotic(z, order):
    """The same for z >= 25: Hankel's expansion (9.2.5-9.2.10)."""
    mu, p, q, term = 4.0 * order, torch.ones_like(z), torch.zeros_like(z), torch.ones_like(z)
    for k in range(1, 24):
        term = term * ((mu - (2 * k - 1) ** 2) / k) / (8 * z)
        if k % 2:
            q = q + term * (-1) ** (k // 2)
        else:
            p = p + term * (-1) ** (k // 2)
    c, s = torch.cos(z), torch.sin(z)
    # cos and sin of z - pi/4 (order 0) or z - 3 pi/4 (order 1), both times sqrt(2)
    cc, ss = (c + s, s - c) if order == 0 else (s - c, -s - c)
    a = 1 / torch.sqrt(math.pi * z)
    return a * (p * cc - q * ss), a * (p * ss + q * cc)


def _hankel(z, order):
    """J and Y of order 0 or 1."""
    J, Y = torch.empty_like(z), torch.empty_like(z)
    for part, fn in ((z < 2, _bessel_series), ((z >= 2) & (z < 25), _bessel_recurrence), (z >= 25, _bessel_asymptotic)):
        if bool(part.any()):
            J[part], Y[part] = fn(z[part], order)
    return J, Y


def _curve_local(kind, op, A, B, s, t, r, wt):
    """2 x 2 local matrices of segment pairs: chart parameters s, t and weights wt [point] or [pair, point],
    separations r = x - y [pair, point, 2]; A, B = (length, normal)."""
    k = op.wavenumber
    R = r.norm(dim=-1)
    w = wt * (A[0] * B[0])[:, None]
    if kind in ("dl", "dlt"):
        n = B[1] if kind == "dl" else A[1]
        rn = (r * n[:, None]).sum(-1) * (-1 if kind == "dl" else 1)
        j, y = _hankel(k * R, 1)
        K = [q * (k / 4) / R * rn * w for q in (y, j)]
    else:
        j, y = _hankel(k * R, 0)
        K = [-q / 4 * w for q in (y, j)]
    f, g = torch.stack([1 - s, s], -1), torch.stack([1 - t, t], -1)
    n = "pn" if s.dim() == 2 else "n"
    P = torch.complex(*(torch.einsum(f"pn,{n}a,{n}b->pab", q, f, g) for q in K))
    if kind != "hs":
        return complex(op.alpha) * P
    M = torch.complex(K[0].sum(1), K[1].sum(1))
    sign = torch.tensor([[1.0, -1.0], [-1.0, 1.0]], dtype=F8, device=DEV)
    nn = (A[1] * B[1]).sum(-1)[:, None, None]
    return complex(op.alpha) * P * nn + complex(op.beta) * M[:, None, None] * sign / (A[0] * B[0])[:, None, None]


def _piece_distance(p0, p1, q0, q1):
    """Distance of straight pieces p0-p1 and q0-q1 that do not cross."""
    def d2(x, a, b):
        e = b - a
        t = (((x - a) * e).sum(-1) / (e * e).sum(-1)).clamp(0.0, 1.0)
        return ((a + t[:, None] * e - x) ** 2).sum(-1)

    return torch.stack([d2(p0, q0, q1), d2(p1, q0, q1), d2(q0, p0, p1), d2(q1, p0, p1)]).amin(0).sqrt()


def _graded(n, levels):
    gx, gw = _gauss(n)
    ends = [0.0] + [0.35 ** lev for lev in range(levels, -1, -1)]
    x = np.concatenate([a + (b - a) * gx for a, b in zip(ends, ends[1:])])
    w = np.concatenate([(b - a) * gw for a, b in zip(ends, ends[1:])])
    return x, w


def _exact_curve(op, kind, X, qs):
    m = X.mesh
    v = torch.as_tensor(m.vertices, device=DEV)
    seg = torch.as_tensor(m.segments.astype(np.int64), device=DEV)
    p, d = v[seg[:, 0]], v[seg[:, 1]] - v[seg[:, 0]]
    ln = d.norm(dim=1)
    nrm = torch.stack([d[:, 1], -d[:, 0]], 1) / ln[:, None]
    ns, nf, k = m.ns, X.nfun, op.wavenumber
    Z = torch.zeros((nf, nf), dtype=torch.complex128, device=DEV)
    fidx = torch.as_tensor(X.fn_index.astype(np.int64), device=DEV)

    def add(ti, si, L):
        rows, cols = fidx[ti][:, :, None].expand(-1, 2, 2), fidx[si][:, None, :].expand(-1, 2, 2)
        ok = (rows >= 0) & (cols >= 0)
        Z.index_put_((rows[ok], cols[ok]), L[ok], accumulate=True)

    def tensor(a):
        return torch.tensor(np.asarray(a), dtype=F8, device=DEV)

    gs, gw = _gauss(qs.far_test)
    ht, hw = _gauss(qs.far_trial)
    S, T = (tensor(a.ravel()) for a in np.meshgrid(gs, ht, indexing="ij"))
    W = tensor(np.outer(gw, hw).ravel())
    near_pairs = []
    for t0 in range(0, ns, 128):
        ti = torch.arange(t0, min(ns, t0 + 128), device=DEV)
        hits = sum((seg[ti, a][:, None] == seg[:, b][None]).to(torch.int64) for a in range(2) for b in range(2))
        ends = torch.stack([((v[seg[ti, a]][:, None] - v[seg[:, b]][None]) ** 2).sum(-1)
                            for a in range(2) for b in range(2)]).amin(0)
        near = (hits == 0) & (torch.maximum(ends * k * k, ends / (16 * ln[None])) < 0.04)
        close = torch.nonzero(near)
        near_pairs.append(torch.stack([ti[close[:, 0]], close[:, 1]], 1))
        far = torch.nonzero((hits == 0) & ~near)
        a, b = ti[far[:, 0]], far[:, 1]
        r = (p[a][:, None] + S[:, None] * d[a][:, None]) - (p[b][:, None] + T[:, None] * d[b][:, None])
        add(a, b, _curve_local(kind, op, (ln[a], nrm[a]), (ln[b], nrm[b]), S, T, r, W))
    # near pairs: the longer piece halved until the pieces are as far apart as the longer is long
    gx, gwx = _gauss(qs.near)
    U, V = (tensor(a.ravel()) for a in np.meshgrid(gx, gx, indexing="ij"))
    Wn = tensor(np.outer(gwx, gwx).ravel())
    pair = torch.cat(near_pairs)
    box = tensor([[0.0, 1.0, 0.0, 1.0]]).expand(pair.shape[0], 4)
    for depth in range(17):
        a, b = pair[:, 0], pair[:, 1]
        la, lb = (box[:, 1] - box[:, 0]) * ln[a], (box[:, 3] - box[:, 2]) * ln[b]
        split = _piece_distance(p[a] + box[:, :1] * d[a], p[a] + box[:, 1:2] * d[a], p[b] + box[:, 2:3] * d[b],
                                p[b] + box[:, 3:] * d[b]) < torch.maximum(la, lb)
        leaf = torch.nonzero(~split if depth < 16 else split | ~split)[:, 0]
        for q0 in range(0, leaf.numel(), 1 << 15):
            i = leaf[q0:q0 + (1 << 15)]
            x, hs, ht = box[i], (box[i, 1] - box[i, 0])[:, None], (box[i, 3] - box[i, 2])[:, None]
            s, t = x[:, :1] + hs * U, x[:, 2:3] + ht * V
            r = (p[a[i]][:, None] + s[..., None] * d[a[i]][:, None]) - (p[b[i]][:, None] + t[..., None] * d[b[i]][:, None])
            add(a[i], b[i], _curve_local(kind, op, (ln[a[i]], nrm[a[i]]), (ln[b[i]], nrm[b[i]]), s, t, r, Wn * hs * ht))
        rest = torch.nonzero(split)[:, 0]
        if depth == 16 or rest.numel() == 0:
            break
        first, second, by_s = box[rest].clone(), box[rest].clone(), (la >= lb)[rest]
        mid = torch.where(by_s, (first[:, 0] + first[:, 1]) / 2, (first[:, 2] + first[:, 3]) / 2)
        first[by_s, 1], second[by_s, 0] = mid[by_s], mid[by_s]
        first[~by_s, 3], second[~by_s, 2] = mid[~by_s], mid[~by_s]
        pair, box = pair[rest].repeat(2, 1), torch.cat([first, second])
    # pairs with a common vertex: graded towards it, in two triangles of the chart square
    n = qs.singular
    gx, gwx = _gauss(n)
    z, wz = _graded(n, (3 * n) // 2)
    Zg, Wg = (a.ravel() for a in np.meshgrid(z, gx, indexing="ij"))
    wt = np.outer(wz * z, gwx).ravel()
    xi, eta = tensor(np.concatenate([Zg, Zg * Wg])), tensor(np.concatenate([Zg * Wg, Zg]))
    wt = tensor(np.concatenate([wt, wt]))
    for ma in range(2):
        for mb in range(2):
            same = {int(x): i for i, x in enumerate(seg[:, ma].tolist())}
            pairs = [(same[int(x)], i) for i, x in enumerate(seg[:, mb].tolist()) if int(x) in same and same[int(x)] != i]
            for q0 in range(0, len(pairs), 2048):
                q = torch.tensor(pairs[q0:q0 + 2048], device=DEV)
                a, b = q[:, 0], q[:, 1]
                da, db = (d[a] if ma == 0 else -d[a]), (d[b] if mb == 0 else -d[b])
                r = xi[:, None] * da[:, None] - eta[:, None] * db[:, None]
                s, t = (xi if ma == 0 else 1 - xi), (eta if mb == 0 else 1 - eta)
                add(a, b, _curve_local(kind, op, (ln[a], nrm[a]), (ln[b], nrm[b]), s, t, r, wt))
    if kind in ("sl", "hs"):  # coincident segments (double layers vanish on them)
        z, wz = _graded(n, 3 * n)
        Zg, Wg = (a.ravel() for a in np.meshgrid(z, gx, indexing="ij"))
        wt = np.outer(wz * (1 - z), gwx).ravel()
        lo = (1 - Zg) * Wg
        s, t = tensor(np.concatenate([Zg + lo, lo])), tensor(np.concatenate([lo, Zg + lo]))
        st, wt = tensor(np.concatenate([Zg, -Zg])), tensor(np.concatenate([wt, wt]))
        for a0 in range(0, ns, 1024):
            a = torch.arange(a0, min(ns, a0 + 1024), device=DEV)
            add(a, a, _curve_local(kind, op, (ln[a], nrm[a]), (ln[a], nrm[a]), s, t, st[:, None] * d[a][:, None], wt))
    return Z


def exact(case, seed):
    problems, qs = _inputs(case, seed)
    out = []
    for op, X in problems:
        Z = _exact_curve(op, case["op"], X, qs) if case["mesh"] == "curve" else _exact_triangles(op, case["op"], X, qs)
        out.append(Z)
    if case["mesh"] == "ellipsoids":
        return out
    return out[0][case["row0"]:case["row0"] + case["nrows"]] if case["nrows"] else out[0]
