"""The double-float operator of small FMM systems, whose launch leaves room for the far
field (up to 2,432 work items), and beyond; the same launch in a batch of one
right-hand side, where a graph holds it.

Tolerance: the operator's documented 5e-12 of its result against FP64.
"""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("damp", [True, False])
@pytest.mark.parametrize("waters,order", [(60, 5), (400, 6), (640, 5), (2000, 5), (6000, 6)])
def test_apply(gpu, waters, order, damp):
    from cppe_gb300 import synthetic
    b = synthetic.water_box(waters, seed=waters)
    v = np.random.default_rng(1).normal(size=3 * b.n)
    s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, summation=cabi.FMM, order=order, damp=damp)
    want = s.apply(v)
    assert np.linalg.norm(s.apply(v, dd=True) - want) < 5e-12 * np.linalg.norm(want)
    s.close()


def test_batch_of_one_right_hand_side(gpu):
    from cppe_gb300 import synthetic
    boxes = [synthetic.water_box(w, seed=w) for w in (400, 640)]
    rng = np.random.default_rng(2)
    rhs = [0.05 * rng.normal(size=3 * b.n) for b in boxes]
    batch = cabi.Batch(boxes, 1, direct_below=100, damp=True, thresh=1e-8, precision=cabi.MIXED,
                       summation=cabi.FMM)
    for _ in range(2):
        mu = batch.solve(np.concatenate(rhs))[0]
    at = 0
    for b, f in zip(boxes, rhs):
        s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, summation=cabi.FMM, damp=True)
        assert np.linalg.norm(s.apply(mu[at:at + 3 * b.n]) - f) < 1.01e-8
        at += 3 * b.n
        s.close()
