"""FP64 double layers of meshes far from the coordinate origin.

The vertices are multiples of 2^-20 and the shift a multiple of 2^-20 too, so the moved mesh is the same mesh exactly
and the oracle's values at the origin are its values as well."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

OPS = {"dl": bg.Helmholtz3D.doublelayer, "dlt": bg.Helmholtz3D.doublelayer_transposed,
       "hs": lambda wavenumber: bg.Helmholtz3D.hypersingular(wavenumber=wavenumber, beta=0.0)}
U = 2.0 ** -53
SHIFT = np.array([256.0, -192.0, 224.0])


def meshes():
    """Two spheres of ~0.02 edges, about 2 apart."""
    v = bg.icosphere(1).vertices
    v = np.round(v / 32 * 2 ** 20) / 2 ** 20
    t = bg.icosphere(1).triangles
    return bg.Mesh(v + [1.0, 0.0, 0.0], t), bg.Mesh(v - [0.75, 0.5, 0.25], t)


def moved(m):
    v = m.vertices + SHIFT
    assert (v - SHIFT == m.vertices).all()
    return bg.Mesh(v, m.triangles)


def every_shape(m):  # a function per local shape
    s = bg.lagrangec0d1(m)
    return bg.Space(m, s.refspace, np.arange(3 * m.nt, dtype=np.int32).reshape(-1, 3), np.ones((m.nt, 3)), 3 * m.nt)


@pytest.mark.gpu
@pytest.mark.parametrize("rule", [(3, 4), (4, 6)])
@pytest.mark.parametrize("name", sorted(OPS))
def test_double_layers_far_from_the_origin(name, rule):
    a, b = meshes()
    op, qs = OPS[name](wavenumber=1.0), bg.QuadStrat(far_test=rule[0], far_trial=rule[1])
    ref = oracle.assemble(op, every_shape(a), every_shape(b), qs)
    Z = bg.assemble_gpu(op, every_shape(moved(a)), every_shape(moved(b)), bg.GPUConfiguration(), quadstrat=qs)
    # Coordinates up to C = 257: a centroid is off by up to 2.7 C U in each (two sums, a division), the points of both
    # sides by as much, |x - y| by 2 x 2.7 sqrt(3) C U = 9.3 C U.  At R = 1.8 and k = 1 the kernels change by at most
    # 3 / R of that relative to the largest value: 16 C U.  Normals from edges add a few U; a normal from offsets whose
    # sum is off by 3 x 2.7 C U would add up to 300 C U (4 |error| / edge, edge 0.02).
    assert np.abs(Z - ref).max() <= 16 * 257 * U * np.abs(ref).max()
