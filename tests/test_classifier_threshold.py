"""Vertices whose distance is next to the tolerance of the classifier: the GPU's classes are the oracle's, which takes
the root of the squared distance."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle

DTOL = 2.220446049250313e-16 * 1.0e3


def offsets():
    """Vertex offsets of lengths around DTOL: along an axis, and with both or all three coordinates within an ulp or two
    of a vector of that length."""
    out = [(DTOL, 0, 0), (np.nextafter(DTOL, 0), 0, 0), (0, np.nextafter(DTOL, 1), 0), (0, 0, -DTOL)]
    for u in ((0.6, 0.8, 0.0), (2 / 3, 1 / 3, -2 / 3)):
        base = DTOL * np.array(u)
        for i in range(-2, 3):
            for j in range(-2, 3):
                v = base.copy()
                v[0] += i * np.spacing(v[0])
                v[1] += j * np.spacing(v[1])
                out.append(tuple(v))
    return np.array(out)


def spaces():
    d = offsets()
    a = bg.Mesh(np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]]), np.array([[0, 1, 2]], dtype=np.int32))
    v = np.stack([d, np.tile([-1.0, 0.25, 0.5], (len(d), 1)), np.tile([-1.0, -0.5, 0.75], (len(d), 1))], axis=1)
    b = bg.Mesh(v.reshape(-1, 3), np.arange(3 * len(d), dtype=np.int32).reshape(-1, 3))
    return every_shape(a), every_shape(b)


def every_shape(m):  # a function per local shape
    s = bg.lagrangec0d1(bg.icosphere(0))
    return bg.Space(m, s.refspace, np.arange(3 * m.nt, dtype=np.int32).reshape(-1, 3), np.ones((m.nt, 3)), 3 * m.nt)


def test_offsets_are_on_both_sides():
    cls = oracle.classify_block(*spaces(), 1.0)[0]
    assert cls[0] != 1 and cls[1] == 1 and cls[2] != 1 and cls[3] != 1
    assert (cls[4:29] == 1).any() and (cls[4:29] != 1).any() and (cls[29:] == 1).any() and (cls[29:] != 1).any()


@pytest.mark.gpu
def test_classes_are_the_oracles():
    X, Y = spaces()
    ref = oracle.classify_block(X, Y, 1.0)
    np.testing.assert_array_equal(bg.classify(X, Y, 1.0), ref)
    np.testing.assert_array_equal(bg.classify(Y, X, 1.0).T, oracle.classify_block(Y, X, 1.0).T)
    _, cls = bg.local_matrices(bg.Helmholtz3D.singlelayer(wavenumber=1.0), X, Y, np.zeros(Y.mesh.nt, dtype=np.int32),
                               np.arange(Y.mesh.nt, dtype=np.int32))
    np.testing.assert_array_equal(cls, ref[0])
