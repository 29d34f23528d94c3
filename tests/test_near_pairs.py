"""Near pairs (singularity extraction) of both precisions: every operator on jittered and folded plates, whole
matrices against the oracle, for lossless and lossy wave numbers on both sides of |gamma R| = 1 (series and
exponential), in one device block, in host output blocks and in a batch."""
import numpy as np
import pytest

import beastgpu_gb300 as bg
import oracle
from test_ss64_rays import OPS

pytestmark = pytest.mark.gpu


def folded(n, seed):
    m = bg.two_plates(n, 0.3, seed, 0.01)
    v = m.vertices.copy()
    up = v[:, 0] > 1.005
    x = v[up, 0] - 1.01
    v[up, 0], v[up, 2] = 1.01 + x * np.cos(np.pi / 6), x * np.sin(np.pi / 6)
    return bg.Mesh(v, m.triangles)


@pytest.mark.parametrize("name", sorted(OPS))
@pytest.mark.parametrize("gamma", [0j, 2j, 9j, 0.5 + 3j])
def test_matrices_with_near_pairs(name, gamma):
    make_op, make_space = OPS[name]
    X = make_space(folded(7, 2))
    if gamma == 0 and name in ("efie", "hs"):
        op = make_op(gamma=0j, alpha=1.0, beta=0.5)
    else:
        op = make_op(gamma=gamma)
    near = oracle.classify_block(X, X, abs(gamma) ** 2) == 4
    assert near.sum() > 20 and near.sum(1).max() > 3  # several near partners of one triangle
    ref = oracle.assemble(op, X, X, bg.QuadStrat())
    scale = np.linalg.norm(ref)
    Z = bg.assemble_gpu(op, X, X, bg.GPUConfiguration())
    assert np.linalg.norm(Z - ref) <= 1e-12 * scale
    M = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(precision="mixed"))
    assert np.linalg.norm(M - ref) <= 1e-5 * scale
    blocks = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(total_GPU_budget=4 * 16 * X.nfun * 11))
    np.testing.assert_array_equal(blocks, Z)
    b = bg.Batch([(op, X, X), (op, X, X)], bg.GPUConfiguration(), autotune=False)
    got = [o.cpu().numpy() for o in b.outputs]
    b.close()
    for o in got:
        np.testing.assert_array_equal(o, Z)
