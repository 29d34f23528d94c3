"""Far pairs whose points nearly meet: small triangles at the inside of large ones, pair by pair against the oracle.

The error of a kernel value is the points' own: each coordinate of x - y carries a few roundings eps of the largest
coordinate, relative to the distance R.  A squared distance formed from terms of size R0^2 (R0: the centroid distance)
would carry eps (R0 / R)^2 instead, which these pairs would show."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

OPS = {"efie": (bg.Maxwell3D.singlelayer, bg.raviartthomas), "mfie": (bg.Maxwell3D.doublelayer, bg.raviartthomas),
       "hh": (bg.Helmholtz3D.singlelayer, bg.lagrangec0d1), "dl": (bg.Helmholtz3D.doublelayer, bg.lagrangec0d1),
       "dlt": (bg.Helmholtz3D.doublelayer_transposed, bg.lagrangec0d1), "hs": (bg.Helmholtz3D.hypersingular, bg.lagrangec0d1)}
RULES = {3: [(2 / 3, 1 / 6), (1 / 6, 2 / 3), (1 / 6, 1 / 6)], 4: [(1 / 3, 1 / 3), (0.6, 0.2), (0.2, 0.6), (0.2, 0.2)]}
EPS = 2.0 ** -53


N = 4  # small triangles per large one


def meshes(swap):
    """Large triangles, and small ones of any orientation of which a rule point is 1e-4 to 1e-6 from a rule point of
    the large one."""
    rng = np.random.default_rng(7)
    a = bg.icosphere(0)
    n = N * a.nt
    va = np.repeat(a.vertices[a.triangles], N, axis=0)
    qa, qb = (4, 3) if swap else (3, 4)
    vb = 0.02 * rng.uniform(-1, 1, (n, 3, 3))
    x, y = points(va, qa), points(vb, qb)
    i, j = rng.integers(1 if swap else 0, qa, n), rng.integers(0, qb, n)  # not the centroid of the large one
    gap = rng.standard_normal((n, 3))
    gap *= (10.0 ** rng.uniform(-6, -4, n) / np.linalg.norm(gap, axis=1))[:, None]
    p = np.arange(n)
    vb += (x[p, i] - y[p, j] + gap)[:, None]
    b = bg.Mesh(vb.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3))
    return (b, a) if swap else (a, b)


def pairs(a, b):
    p = np.arange(max(a.nt, b.nt), dtype=np.int32)
    return (p, p // N) if a.nt > b.nt else (p // N, p)


def points(v, q):
    return np.stack([u * v[:, 0] + w * v[:, 1] + (1 - u - w) * v[:, 2] for u, w in RULES[q]], axis=1)


def distances(a, b):
    """R0 / R and 1 / R of the closest points of each pair."""
    t, s = pairs(a, b)
    va, vb = a.vertices[a.triangles[t]], b.vertices[b.triangles[s]]
    R = np.linalg.norm(points(va, 3)[:, :, None] - points(vb, 4)[:, None], axis=-1).min(axis=(1, 2))
    return np.linalg.norm(va.mean(axis=1) - vb.mean(axis=1), axis=-1) / R, 1 / R


@pytest.mark.parametrize("swap", [False, True])
def test_pairs_can_tell(swap):
    ratio, inv = distances(*meshes(swap))
    # with squared distances of size R0^2 most pairs would be off by more than the bound below
    assert (0.5 * ratio ** 2 > 96 * inv).sum() >= 40


def every_shape(make_space, m):  # a function per local shape
    s = make_space(m)
    return bg.Space(m, s.refspace, np.arange(3 * m.nt, dtype=np.int32).reshape(-1, 3), np.ones((m.nt, 3)), 3 * m.nt)


@pytest.mark.gpu
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("k", [2.0, 20.0])  # phases from series and from sincos
@pytest.mark.parametrize("name", sorted(OPS))
def test_local_matrices_fp64(name, k, swap):
    make_op, make_space = OPS[name]
    a, b = meshes(swap)
    X, Y = every_shape(make_space, a), every_shape(make_space, b)
    inv = distances(a, b)[1]
    t, s = pairs(a, b)
    op = make_op(wavenumber=k)
    ref, cls = oracle.local_matrices(op, X, Y, bg.QuadStrat(), t, s)
    assert not cls.any()
    Z = bg.assemble_gpu(op, X, Y, bg.GPUConfiguration())
    got = np.stack([Z[3 * p:3 * p + 3, 3 * q:3 * q + 3] for p, q in zip(t, s)])
    err = np.linalg.norm((got - ref).reshape(-1, 9), axis=1)
    size = np.linalg.norm(ref.reshape(-1, 9), axis=1)
    # 8 roundings of a coordinate (up to 1) in x - y, on both sides, at most to the power 3 in the kernel: 48 / R,
    # doubled; a pair's entries may nearly cancel: against the typical size at least
    assert (err <= 96 * EPS * inv * np.maximum(size, np.median(size))).all()
