"""A program that holds many small direct FP64 systems: their matrices together stay
within 16 GiB, the systems beyond that answer as well (to the rounding of
test_gpu_near64.py), and closing systems gives the memory back."""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def held(torch, before):
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


def test_many_systems(gpu):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    g = np.stack(np.meshgrid(*[np.arange(11.0)] * 3, indexing="ij"), -1).reshape(-1, 3)[:1024]
    xyz = 4.0 * (g + rng.uniform(-0.2, 0.2, g.shape))
    a6 = np.zeros((1024, 6))
    a6[:, [0, 3, 5]] = rng.uniform(2.0, 6.0, (1024, 1))
    ptr, idx = np.zeros(1025, np.int32), np.zeros(1, np.int32)
    v = rng.normal(size=3 * 1024)
    torch.cuda.init()
    before = torch.cuda.mem_get_info()[0]
    systems, out = [], []
    for _ in range(280):  # 20.6 GiB of matrices
        systems.append(cabi.System(xyz, a6, ptr, idx))
        out.append(systems[-1].apply(v))
    assert 15 * GIB < held(torch, before) < 18 * GIB
    for o in out:
        assert np.linalg.norm(o - out[0]) < 4e-15 * np.linalg.norm(out[0])
    # the last system solves as the first
    F = 0.05 * rng.normal(size=3 * 1024)
    a, b = (s.solve(F) for s in (systems[0], systems[-1]))
    assert a[1] == b[1]
    np.testing.assert_allclose(a[0], b[0], rtol=0, atol=1e-10)
    for s in systems:
        s.close()
    assert held(torch, before) < GIB
    s = cabi.System(xyz, a6, ptr, idx)
    s.apply(v)
    assert held(torch, before) > 70 << 20  # a matrix again
    s.close()
