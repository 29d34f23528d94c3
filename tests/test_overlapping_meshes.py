"""Test and trial spaces on two meshes of one surface that share few vertices: far pairs of triangles that lie on each
other, with equal centroids (a triangle and the middle one of its refinement)."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

OPS = {"efie": (bg.Maxwell3D.singlelayer, bg.raviartthomas), "mfie": (bg.Maxwell3D.doublelayer, bg.raviartthomas),
       "hh": (bg.Helmholtz3D.singlelayer, bg.lagrangec0d1), "dl": (bg.Helmholtz3D.doublelayer, bg.lagrangec0d1),
       "dlt": (bg.Helmholtz3D.doublelayer_transposed, bg.lagrangec0d1), "hs": (bg.Helmholtz3D.hypersingular, bg.lagrangec0d1)}


def centroids(mesh):
    v = mesh.vertices[mesh.triangles]
    return (v[:, 0] + v[:, 1] + v[:, 2]) / 3.0


def cubes(swap=False):
    pair = bg.meshcuboid(1, 1, 1, 0.5), bg.meshcuboid(1, 1, 1, 0.25)
    return pair[::-1] if swap else pair


def test_cubes_have_far_pairs_with_equal_centroids():
    a, b = cubes()
    equal = (centroids(a)[:, None] == centroids(b)[None]).all(-1)
    far = oracle.classify_block(bg.lagrangec0d1(a), bg.lagrangec0d1(b), 1.0) == 0
    assert (equal & far).sum() == 48


@pytest.mark.gpu
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("name", sorted(OPS))
def test_equal_centroids_fp64(name, swap):
    make_op, make_space = OPS[name]
    X, Y = (make_space(m) for m in cubes(swap))
    op = make_op(wavenumber=1.0)
    ref = oracle.assemble(op, X, Y, bg.QuadStrat())
    Z = bg.assemble_gpu(op, X, Y, bg.GPUConfiguration())
    # points of the pairs are at least ~R0 / 4 apart: a few hundred roundings of 1.1e-16, as for other FP64 matrices
    assert np.linalg.norm(Z - ref) <= 1e-12 * np.linalg.norm(ref)
    b = bg.Batch([(op, X, Y)], bg.GPUConfiguration(), autotune=False)
    got = b.outputs[0].cpu().numpy()
    b.close()
    np.testing.assert_array_equal(got, Z)


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [(3, 4), (4, 6)])
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("name", sorted(OPS))
def test_equal_centroids_mixed(name, swap, rule):
    make_op, make_space = OPS[name]
    X, Y = (make_space(m) for m in cubes(swap))
    op, qs = make_op(wavenumber=1.0), bg.QuadStrat(far_test=rule[0], far_trial=rule[1])
    ref = oracle.assemble(op, X, Y, qs)
    # FP32 rounding (6e-8) of R^2 relative to R0^2, (R0 / R)^2 <= 16, in a few terms: below 1e-5
    for shift in (0.0, 1e-9):  # the second: centroids that differ below FP32 only
        T = make_space(bg.Mesh(X.mesh.vertices + shift, X.mesh.triangles))
        Z = bg.assemble_gpu(op, T, Y, bg.GPUConfiguration(precision="mixed"), quadstrat=qs)
        assert np.linalg.norm(Z - (ref if shift == 0.0 else oracle.assemble(op, T, Y, qs))) <= 1e-5 * np.linalg.norm(ref)


def thirds(n):
    """A square of n segments a side, and the same square with each segment cut in three."""
    def square(m):
        c = np.array([[0.0, 0.0], [3.0, 0.0], [3.0, 3.0], [0.0, 3.0]])
        v = np.concatenate([c[i] + (c[(i + 1) % 4] - c[i]) * np.arange(m)[:, None] / m for i in range(4)])
        i = np.arange(4 * m, dtype=np.int32)
        return bg.CurveMesh(v, np.stack([i, (i + 1) % (4 * m)], axis=1))
    return square(n), square(3 * n)


def test_squares_have_far_pairs_with_equal_midpoints():
    a, b = thirds(2)
    mid = [m.vertices[m.segments].mean(axis=1) for m in (a, b)]
    equal = (mid[0][:, None] == mid[1][None]).all(-1)
    far = oracle.classify_block_curve(bg.curve_lagrangec0d1(a), bg.curve_lagrangec0d1(b), 4.0) == 0
    assert (equal & far).sum() == 8


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [(4, 4), (4, 6)])
@pytest.mark.parametrize("name", ["singlelayer", "doublelayer", "doublelayer_transposed", "hypersingular"])
def test_equal_midpoints_curve(name, rule):
    a, b = thirds(2)
    op, qs = getattr(bg.Helmholtz2D, name)(wavenumber=2.0), bg.QuadStrat2D(far_test=rule[0], far_trial=rule[1])
    for m, n in ((a, b), (b, a)):
        X, Y = bg.curve_lagrangec0d1(m), bg.curve_lagrangec0d1(n)
        ref = oracle.assemble_rows_curve(op, X, Y, qs, np.arange(X.nfun, dtype=np.int32))
        for prec, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
            Z = bg.assemble_gpu(op, X, Y, bg.GPUConfiguration(precision=prec), quadstrat=qs)
            assert np.linalg.norm(Z - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [(4, 3), (1, 1), (4, 1), (1, 3)])
@pytest.mark.parametrize("name", sorted(OPS))
def test_trial_vertex_in_a_test_point(name, rule):
    """The centroid of a triangle, a test point of these rules, is a vertex of the mesh that cuts its edges in three:
    no rule point lies there, so every entry is finite."""
    make_op, make_space = OPS[name]
    a, b = bg.plate(1, 0, 0), bg.plate(3, 0, 0)
    d = np.linalg.norm(centroids(a)[:, None] - b.vertices[None], axis=-1)
    assert (d < 1e-15).any(axis=1).all()
    def every_shape(m):  # a function per local shape
        s = make_space(m)
        return bg.Space(m, s.refspace, np.arange(3 * m.nt, dtype=np.int32).reshape(-1, 3), np.ones((m.nt, 3)), 3 * m.nt)
    X, Y = every_shape(a), every_shape(b)
    op, qs = make_op(wavenumber=1.0), bg.QuadStrat(far_test=rule[0], far_trial=rule[1])
    ref = oracle.assemble(op, X, Y, qs)
    Z = bg.assemble_gpu(op, X, Y, bg.GPUConfiguration(precision="mixed"), quadstrat=qs)
    assert np.isfinite(ref).all() and np.isfinite(Z).all()
    if name in ("efie", "hh", "hs"):  # (the double layers vanish on a plane)
        assert np.linalg.norm(Z - ref) <= 1e-5 * np.linalg.norm(ref)
