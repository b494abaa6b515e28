"""The one-block solver of the smallest systems takes limits of up to 1,024 iterations:
with a larger one, which a solve that does not converge would spend in one kernel
(with a pinned norm per iteration), the solve is a loop of launches."""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu


def test_large_iteration_limit(gpu):
    from cppe_gb300 import synthetic
    b = synthetic.water_box(6, seed=1)
    F = 0.05 * np.random.default_rng(2).normal(size=3 * b.n)
    out = []
    for maxiter in (50, 1024, 1025, 1000000):
        s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, maxiter=maxiter)
        s.solve(F)
        k = cabi.launch_count()
        mu, it, hist, _ = s.solve(F)
        launches = cabi.launch_count() - k
        assert launches == 1 if maxiter <= 1024 else launches > it
        out.append((mu, it, hist))
        s.close()
    for mu, it, hist in out[1:]:
        assert it == out[0][1]
        # tolerances as test_gpu_dense.py's
        np.testing.assert_allclose(mu, out[0][0], rtol=0, atol=1e-10)
        np.testing.assert_allclose(hist, out[0][2], rtol=1e-6, atol=1e-14)
