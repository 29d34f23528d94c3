"""Chunk spheres 32 at a time in the classifier, and the FP64 gather's supports with and without unit coefficients."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

pytestmark = pytest.mark.gpu


def part(mesh, n, seed=None):
    tri = mesh.triangles if seed is None else mesh.triangles[np.random.default_rng(seed).permutation(mesh.nt)]
    return bg.Mesh(mesh.vertices, tri[:n])


@pytest.mark.parametrize("shuffled", [False, True])  # shuffled: chunk spheres as wide as the mesh
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 1057, 1250])
def test_class_counts_around_32_chunks(n, shuffled):
    mesh = bg.plate(25, 0.04, 2)  # 1,250 triangles
    X = bg.lagrangec0d1(mesh)
    Y = bg.lagrangec0d1(part(mesh, n, 3 if shuffled else None))
    if Y.nfun == 0:
        Y = bg.Space(Y.mesh, Y.refspace, np.arange(3 * n, dtype=np.int32).reshape(n, 3), np.ones((n, 3)), 3 * n)
    c = oracle.classify_block(X, Y, 1.0)
    _, st = bg.assemble_gpu(bg.Helmholtz3D.singlelayer(wavenumber=1.0), X, Y, bg.GPUConfiguration(precision="mixed"),
                            return_stats=True)
    assert list(st["pairs_class"]) == [int((c == k).sum()) for k in range(5)]


@pytest.mark.parametrize("coefs", [(1.0,), (1.0, -0.5, 2.0), (0.25, -3.0)])
def test_fp64_gather_coefficients(coefs):
    X = bg.lagrangec0d1(bg.ellipsoid(1, (1.0, 0.7, 0.9)))
    cf = np.random.default_rng(2).choice(coefs, size=X.fn_coef.shape)
    Y = bg.Space(X.mesh, X.refspace, X.fn_index, cf, X.nfun)
    op = bg.Helmholtz3D.singlelayer(wavenumber=3.0)
    ref = oracle.assemble(op, Y, Y, bg.QuadStrat())
    Z = bg.assemble_gpu(op, Y, Y, bg.GPUConfiguration())
    assert np.linalg.norm(Z - ref) <= 1e-12 * np.linalg.norm(ref)
    b = bg.Batch([(op, Y, Y)], bg.GPUConfiguration(), autotune=False)
    got = b.outputs[0].cpu().numpy()
    b.close()
    np.testing.assert_array_equal(got, Z)
