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
