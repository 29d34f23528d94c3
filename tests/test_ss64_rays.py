"""FP64 Sauter-Schwab integrals summed along the rays from the shared vertex (plain path; mixed path for the
operators without a double-float kernel): assembled matrices, whose entries between neighbouring functions are
sums of singular pairs only, against the oracle for series of every length, the point-by-point sums (large
theta, lossy wave numbers), other rule orders, and vertices that coincide within the tolerance only."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

pytestmark = pytest.mark.gpu

OPS = {"efie": (bg.Maxwell3D.singlelayer, bg.raviartthomas), "mfie": (bg.Maxwell3D.doublelayer, bg.raviartthomas),
       "hh": (bg.Helmholtz3D.singlelayer, bg.lagrangec0d1), "dl": (bg.Helmholtz3D.doublelayer, bg.lagrangec0d1),
       "dlt": (bg.Helmholtz3D.doublelayer_transposed, bg.lagrangec0d1), "hs": (bg.Helmholtz3D.hypersingular, bg.lagrangec0d1)}
TOL = 1e-12


def check(op, X, qs=bg.QuadStrat()):
    ref = oracle.assemble(op, X, X, qs)
    Z = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(), quadstrat=qs)
    assert np.linalg.norm(Z - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("name", sorted(OPS))
@pytest.mark.parametrize("gamma", [1e-3j, 0.3j, 1.5j, 4j, 30j, -2j, 0.4 + 2j, 0.8])
def test_wave_numbers(name, gamma):
    # edges ~0.6: k (|X| + |Y|) from 1e-3 to 36, i.e. 1 to 13 series terms and the direct sums
    make_op, make_space = OPS[name]
    check(make_op(gamma=gamma), make_space(bg.ellipsoid(1, (1.0, 0.8, 1.2))))


@pytest.mark.parametrize("name", ["efie", "dl"])
@pytest.mark.parametrize("orders", [(1, 1, 1), (2, 3, 5), (7, 6, 4)])
def test_rule_orders(name, orders):
    make_op, make_space = OPS[name]
    qs = bg.QuadStrat(ss_cf=orders[0], ss_ce=orders[1], ss_cv=orders[2])
    X = make_space(bg.plate(3, 0.3, 4) if name == "efie" else bg.icosphere(1))
    check(make_op(wavenumber=2.0), X, qs)
    check(make_op(wavenumber=2.0), X)  # the tables follow the orders of the call


@pytest.mark.parametrize("name", sorted(OPS))
def test_vertices_equal_within_the_tolerance(name):
    """Two icospheres of which the second is a copy moved by rounding: every triangle meets its copy in three
    vertices 1e-14 apart or bit-equal, its neighbours' copies in two or one."""
    make_op, make_space = OPS[name]
    a, b = bg.icosphere(1), bg.icosphere(1)
    rng = np.random.default_rng(3)
    v = b.vertices + 1e-14 * rng.integers(-1, 2, b.vertices.shape)
    X, Y = make_space(a), make_space(bg.Mesh(v, b.triangles))
    op = make_op(wavenumber=1.7)
    ref = oracle.assemble(op, X, Y, bg.QuadStrat())
    Z = bg.assemble_gpu(op, X, Y, bg.GPUConfiguration())
    assert np.linalg.norm(Z - ref) <= TOL * np.linalg.norm(ref)
    B = bg.Batch([(op, X, Y)], bg.GPUConfiguration(), autotune=False)
    got = B.outputs[0].cpu().numpy()
    B.close()
    np.testing.assert_array_equal(got, Z)
