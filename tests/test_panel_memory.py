"""Device memory of plain FP64 calls: within the HBM budget, also where not even one output tile's panel of local
matrices fits, and given back on request; the matrix is the same bit for bit."""
import numpy as np
import pytest

import beastgpu_gb300 as bg

pytestmark = pytest.mark.gpu

MIB = 1 << 20
SLACK = 16 * MIB  # triangle records, index tables and tile plans of 5,120 triangles, in the allocator's 2 MiB pages


def used():
    """Device memory that is not torch's."""
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free - torch.cuda.memory_reserved()


@pytest.fixture(scope="module")
def case():
    X = bg.lagrangec0d1(bg.icosphere(4))  # 737 KB of local matrices per trial triangle
    op = bg.Helmholtz3D.singlelayer(wavenumber=3.0)
    return op, X, bg.assemble_gpu(op, X, X, bg.GPUConfiguration())


# 16 and 96 MiB: less than a tile's panel (twice, beside three staging buffers of 24 MiB); 600 MiB: a few tiles
@pytest.mark.parametrize("out,mib", [("device", 16), ("device", 200), (None, 96), (None, 600)])
def test_budget_holds(case, out, mib):
    op, X, ref = case
    cfg = dict(total_GPU_budget=mib * MIB)
    bg.assemble_gpu(op, X, X, bg.GPUConfiguration(precision="mixed", **cfg), out="device")  # the handle's other buffers
    before = used()
    Z = bg.assemble_gpu(op, X, X, bg.GPUConfiguration(**cfg), **({"out": out} if out else {}))
    assert used() - before <= mib * MIB + SLACK
    np.testing.assert_array_equal(Z.cpu().numpy() if out else Z, ref)


def test_release(case):
    op, X, ref = case
    bg.assemble_gpu(op, X, X, bg.GPUConfiguration(), out="device")
    before = used()
    bg.release_memory()
    assert before - used() >= 144 * X.mesh.nt ** 2 // 2
    np.testing.assert_array_equal(bg.assemble_gpu(op, X, X, bg.GPUConfiguration()), ref)
