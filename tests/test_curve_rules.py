"""The curve path's unrolled 4 x 4 far rule against the runtime rule loops, its near and singular sums for every
operator and space, at sizes around the blocks of 128 test segments: whole matrices against the oracle."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

pytestmark = pytest.mark.gpu

OPS = {"sl": bg.Helmholtz2D.singlelayer, "dl": bg.Helmholtz2D.doublelayer,
       "dlt": bg.Helmholtz2D.doublelayer_transposed, "hs": bg.Helmholtz2D.hypersingular}


@pytest.mark.parametrize("name", sorted(OPS))
@pytest.mark.parametrize("n", [3, 127, 129, 260])
@pytest.mark.parametrize("rule", [(4, 4), (4, 3), (6, 4)])
def test_far_rules_and_block_edges(name, n, rule):
    X = bg.curve_lagrangec0d1(bg.ellipse(n, 1.0, 0.5, jitter=0.2, seed=n))
    qs = bg.QuadStrat2D(far_test=rule[0], far_trial=rule[1])
    for k in (0.0, 0.7, 0.04 * n):
        op = OPS[name](wavenumber=k)
        ref = oracle.assemble_rows_curve(op, X, X, qs, np.arange(X.nfun, dtype=np.int32))
        scale = np.linalg.norm(ref)
        if scale == 0.0:
            continue
        assert np.linalg.norm(bg.assemble_gpu(op, X, X, bg.GPUConfiguration(), quadstrat=qs) - ref) <= 1e-12 * scale
        M = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(precision="mixed"), quadstrat=qs)
        assert np.linalg.norm(M - ref) <= 1e-5 * scale


def test_constants_on_the_test_side():
    m = bg.ellipse(150, 1.0, 0.5, jitter=0.2, seed=1)
    X, Y = bg.curve_lagrangecxd0(m), bg.curve_lagrangec0d1(m)
    for T, S in ((X, Y), (Y, X), (X, X)):
        op = bg.Helmholtz2D.singlelayer(wavenumber=5.0)
        ref = oracle.assemble_rows_curve(op, T, S, bg.QuadStrat2D(), np.arange(T.nfun, dtype=np.int32))
        for prec, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
            Z = bg.assemble_gpu(op, T, S, bg.GPUConfiguration(precision=prec))
            assert np.linalg.norm(Z - ref) <= tol * np.linalg.norm(ref)
