"""The plain FP64 far stage of single assemblies: local matrices of panels of pairs, then the gather.

The result must not depend on the panels (sized by the HBM budget), the tiles or their chunks, nor on
the path (a batch computes the pairs inside its tiles): bit-identical, and within 1e-12 of the oracle.
"""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle
from beastgpu_gb300.meshes import merge

pytestmark = pytest.mark.gpu

OPS = {"efie": (bg.Maxwell3D.singlelayer, bg.raviartthomas), "mfie": (bg.Maxwell3D.doublelayer, bg.raviartthomas),
       "hh": (bg.Helmholtz3D.singlelayer, bg.lagrangec0d1), "dlt": (bg.Helmholtz3D.doublelayer_transposed, bg.lagrangec0d1),
       "hs": (bg.Helmholtz3D.hypersingular, bg.lagrangec0d1)}
TOL = 1e-12  # of the Frobenius norm, as for every FP64 kernel (a few hundred roundings of 1.1e-16 per entry)


def spaces(name, ragged=False):
    make_op, make_space = OPS[name]
    mesh = merge([bg.ellipsoid(1, (1.0, 0.7, 0.9)), bg.plate(5, 0.2, 2)]) if ragged else bg.ellipsoid(2, (1.0, 0.8, 1.1))
    return make_op(wavenumber=5.0), make_space(mesh)


@pytest.mark.parametrize("name", sorted(OPS))
@pytest.mark.parametrize("rule", [(3, 4), (4, 6)])
def test_panels_tiles_and_batch_bit_identical(name, rule):
    op, X = spaces(name, ragged=True)
    qs = bg.QuadStrat(far_test=rule[0], far_trial=rule[1])
    ref = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(), quadstrat=qs)
    o = oracle.assemble(op, X, X, qs)
    assert np.linalg.norm(ref - o) <= TOL * np.linalg.norm(o)
    nt = X.mesh.nt
    for panel_cols in (1, 7, 40):  # a budget of that many columns of local matrices (at least one tile)
        cfg = bg.GPUConfiguration(total_GPU_budget=144 * nt * panel_cols)
        Z = bg.assemble_gpu(op, X, X, cfg, quadstrat=qs, out="device")
        np.testing.assert_array_equal(Z.cpu().numpy(), ref)
    # RWG tile 0: chunks of 16 triangles do not fit twice, narrower ones are used
    for tile in (0, 7, 13, 18, 22) if X.refspace == 1 and rule == (3, 4) else (7, 13, 18, 22):
        Z = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(tile_config=tile), quadstrat=qs)
        np.testing.assert_array_equal(Z, ref)
    b = bg.Batch([(op, X, X)], bg.GPUConfiguration(), quadstrat=qs, autotune=False)
    got = b.outputs[0].cpu().numpy()
    b.close()
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("name", ["efie", "hh"])
def test_row_windows_and_functions_without_supports(name):
    op, X = spaces(name)
    ref = bg.assemble_gpu(op, X, X, bg.GPUConfiguration())
    for r0, n in ((0, 1), (X.nfun - 1, 1), (5, 33), (17, X.nfun - 17)):
        Z = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(total_GPU_budget=1 << 16), rows=(r0, n))
        np.testing.assert_array_equal(Z, ref[r0:r0 + n])
    # two more functions that no triangle carries: zero rows and columns
    Y = bg.Space(X.mesh, X.refspace, X.fn_index, X.fn_coef, X.nfun + 2)
    Z = bg.assemble_gpu(op, Y, Y, bg.GPUConfiguration())
    np.testing.assert_array_equal(Z[:-2, :-2], ref)
    assert not Z[-2:].any() and not Z[:, -2:].any()
