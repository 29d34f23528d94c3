"""Double-float singular pairs of hats (mixed path): rounding errors of sums of positive terms, class by class."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

pytestmark = pytest.mark.gpu

U = 2.0 ** -48


@pytest.mark.parametrize("k", [0.5, 2.0, 8.0])
@pytest.mark.parametrize("mesh", ["ellipsoid", "plate"])
def test_rounding_of_hats(mesh, k):
    X = bg.lagrangec0d1(bg.ellipsoid(2, (1.0, 0.4, 1.3)) if mesh == "ellipsoid" else bg.plate(8, 0.3, 3))
    op = bg.Helmholtz3D.singlelayer(wavenumber=k)
    t, s = np.nonzero(oracle.classify_block(X, X, k * k))
    ref, _ = oracle.local_matrices(op, X, X, bg.QuadStrat(), t, s)
    got, cls = bg.local_matrices(op, X, X, t, s, precision="mixed")
    err = np.linalg.norm((got - ref).reshape(-1, 9), axis=1) / np.linalg.norm(ref.reshape(-1, 9), axis=1)
    for c in (1, 2, 3):
        # a term passes about 12 roundings of U/2 at most (0.3 U rms each), its sum and the constant factors as many
        # again: 2 U rms, doubled.  Entries from sums that cancel (moments of 1, alpha xi, beta xi) come to 5 - 7 U.
        assert np.sqrt(np.mean(err[cls == c] ** 2)) <= 4 * U
