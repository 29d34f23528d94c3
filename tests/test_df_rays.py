"""Double-float Sauter-Schwab integrals (mixed path) along the rays: every singular local matrix within 1e-12
of the FP64 oracle, pair by pair, from one series term to the point-by-point sums, for several rule orders."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

pytestmark = pytest.mark.gpu

OPS = {"efie": (bg.Maxwell3D.singlelayer, bg.raviartthomas), "mfie": (bg.Maxwell3D.doublelayer, bg.raviartthomas),
       "hh": (bg.Helmholtz3D.singlelayer, bg.lagrangec0d1)}


def check(op, X, qs=bg.QuadStrat()):
    t, s = np.nonzero(oracle.classify_block(X, X, op.wavenumber ** 2))
    ref, _ = oracle.local_matrices(op, X, X, qs, t, s)
    got, cls = bg.local_matrices(op, X, X, t, s, precision="mixed", quadstrat=qs)
    assert set(np.unique(cls)) == {1, 2, 3}
    err = np.linalg.norm((got - ref).reshape(-1, 9), axis=1)
    size = np.linalg.norm(ref.reshape(-1, 9), axis=1)
    # 48-bit operations: a few hundred roundings of 3.6e-15; pairs that nearly vanish against the largest
    assert (err <= 1e-12 * np.maximum(size, 1e-2 * size.max())).all()


@pytest.mark.parametrize("name", sorted(OPS))
@pytest.mark.parametrize("k", [1e-3, 0.4, 2.0, 3.3, 4.5, 20.0])
def test_wave_numbers(name, k):
    make_op, make_space = OPS[name]  # edges ~0.6: k (|X| + |Y|) from 1e-3 to 24; series up to 3
    check(make_op(wavenumber=k), make_space(bg.ellipsoid(1, (1.0, 0.8, 1.2))))


@pytest.mark.parametrize("name", sorted(OPS))
@pytest.mark.parametrize("orders", [(1, 2, 1), (6, 5, 7)])
def test_rule_orders(name, orders):
    make_op, make_space = OPS[name]
    qs = bg.QuadStrat(ss_cf=orders[0], ss_ce=orders[1], ss_cv=orders[2])
    check(make_op(wavenumber=2.0), make_space(bg.icosphere(1)), qs)


def test_forced_singular_class_of_a_separate_pair():
    X = bg.raviartthomas(bg.icosphere(1))
    op = bg.Maxwell3D.singlelayer(wavenumber=2.0)
    t, s = np.nonzero(oracle.classify_block(X, X, 4.0) == 0)
    t, s = t[:64], s[:64]
    got, _ = bg.local_matrices(op, X, X, t, s, precision="mixed", force_class=1)
    ref, _ = bg.local_matrices(op, X, X, t, s, precision="fp64", force_class=1)
    np.testing.assert_array_equal(got, ref)
