"""Mixed far pairs of the rules other than 3 x 4: trial points two at a time (odd rules padded with a zero weight),
trial records staged per chunk.  Every rule size against the oracle, tile shapes bit-identical.

Bound: FP32 rounding (6e-8) of the kernel values, their phases (k R up to ~10: below 3e-7) and sums of at most 169
terms of one magnitude: below 1e-6 of the matrix's norm, checked at 3e-6.
"""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle
from beastgpu_gb300.meshes import merge

pytestmark = pytest.mark.gpu

OPS = {"efie": (bg.Maxwell3D.singlelayer, bg.raviartthomas), "mfie": (bg.Maxwell3D.doublelayer, bg.raviartthomas),
       "hh": (bg.Helmholtz3D.singlelayer, bg.lagrangec0d1), "dl": (bg.Helmholtz3D.doublelayer, bg.lagrangec0d1),
       "dlt": (bg.Helmholtz3D.doublelayer_transposed, bg.lagrangec0d1),
       "hs": (bg.Helmholtz3D.hypersingular, bg.lagrangec0d1)}
TOL = 3e-6


def check(name, rule, mesh, **k):
    make_op, make_space = OPS[name]
    op, X = make_op(**k), make_space(mesh)
    qs = bg.QuadStrat(far_test=rule[0], far_trial=rule[1])
    ref = oracle.assemble(op, X, X, qs)
    Z = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(precision="mixed"), quadstrat=qs)
    assert np.linalg.norm(Z - ref) <= TOL * np.linalg.norm(ref)
    return op, X, qs, Z


@pytest.mark.parametrize("name", sorted(OPS))
@pytest.mark.parametrize("rule", [(1, 1), (4, 3), (3, 3), (6, 7), (7, 6), (12, 13), (13, 1)])
def test_rules(name, rule):
    mesh = bg.ellipsoid(2, (1.0, 0.8, 1.1)) if max(rule) < 12 else bg.ellipsoid(1, (1.0, 0.7, 0.9))
    check(name, rule, mesh, wavenumber=5.0)


@pytest.mark.parametrize("name", sorted(OPS))
def test_lossy_and_reduced_phase(name):
    check(name, (6, 7), bg.ellipsoid(1, (1.0, 0.8, 1.1)), gamma=0.7 + 4.0j)
    check(name, (7, 4), bg.ellipsoid(1, (1.0, 0.8, 1.1)), wavenumber=9.0)  # k (r + r') > pi on the coarse mesh


@pytest.mark.parametrize("name", ["efie", "mfie", "hh"])
def test_tiles_and_batch_bit_identical(name):
    mesh = merge([bg.ellipsoid(2, (1.0, 0.7, 0.9)), bg.plate(5, 0.2, 2)])
    op, X, qs, ref = check(name, (6, 7), mesh, wavenumber=5.0)
    for tile in (7, 13, 18, 22, 19):
        Z = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(precision="mixed", tile_config=tile), quadstrat=qs)
        np.testing.assert_array_equal(Z, ref)
    b = bg.Batch([(op, X, X)], bg.GPUConfiguration(precision="mixed"), quadstrat=qs, autotune=False)
    got = b.outputs[0].cpu().numpy()
    b.close()
    np.testing.assert_array_equal(got, ref)
