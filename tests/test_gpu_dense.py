"""Small direct FP64 systems: the dense operator (up to 1,024 sites) and the
one-block solver (up to 53) against the oracle, at the sizes where they begin
and end; asymmetric exclusions; guesses; non-convergence.

Tolerances: the apply as test_gpu_near64.py (4e-15 in norm); solves take the
oracle's iterations, so their norms agree to rounding amplified by the
iteration (1e-6, the bound of the other solve tests) and mu to 1e-10.
"""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu


def system(n, seed):
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(11.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    xyz = 4.0 * (g[rng.permutation(g.shape[0])[:n]] + rng.uniform(-0.2, 0.2, (n, 3)))
    alpha6 = np.zeros((n, 6))
    alpha6[:, [0, 3, 5]] = rng.uniform(2.0, 8.0, (n, 3))
    alpha6[:, [1, 2, 4]] = rng.uniform(-0.3, 0.3, (n, 3))
    excl = [sorted(rng.choice(n, min(n, int(rng.integers(0, 4))), replace=False)) for _ in range(n)]
    ptr = np.concatenate([[0], np.cumsum([len(e) for e in excl])]).astype(np.int32)
    idx = np.array([j for e in excl for j in e], np.int32)
    if idx.size == 0:
        idx = np.zeros(1, np.int32)
    return xyz, alpha6, ptr, idx, rng


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("n", [1, 2, 16, 42, 53, 54, 129, 1024, 1025])
def test_apply_and_solve(gpu, port, n, damp):
    xyz, alpha6, ptr, idx, rng = system(n, n)
    damping = 2.1304 if damp else 0.0
    s = cabi.System(xyz, alpha6, ptr, idx, damp=damp)
    v = rng.normal(size=3 * n)
    ref = port.bmatrix_apply(xyz, alpha6, ptr, idx, v, fmm=0, damping=damping)
    assert np.linalg.norm(s.apply(v) - ref) < 4e-15 * np.linalg.norm(ref)
    F = 0.05 * rng.normal(size=3 * n)
    mu_o, it_o, hist_o, ok = port.solve(xyz, alpha6, ptr, idx, F, fmm=0, damping=damping)
    assert ok
    mu, it, hist, _ = s.solve(F)
    assert it == it_o
    np.testing.assert_allclose(hist, hist_o, rtol=1e-6, atol=1e-14)
    np.testing.assert_allclose(mu, mu_o, rtol=0, atol=1e-10)
    assert s.stats()["fp64_applies"] == it + 1
    # from a guess and from zero: the same answer
    for kw in (dict(guess=0.9 * mu, make_guess=False), dict(make_guess=False)):
        got, _, _, _ = s.solve(F, **kw)
        np.testing.assert_allclose(got, mu, rtol=0, atol=1e-6)
        assert np.linalg.norm(F - s.apply(got)) < 1e-8
    assert np.array_equal(s.solve(F)[0], mu)
    s.close()


@pytest.mark.parametrize("n", [18, 60])
def test_not_converged(gpu, n):
    xyz, alpha6, ptr, idx, rng = system(n, 3)
    s = cabi.System(xyz, alpha6, ptr, idx, maxiter=2)
    F = rng.normal(size=3 * n)
    mu, it, hist, rc = s.solve(F, allow_not_converged=True)
    assert rc == cabi.NOT_CONVERGED and it == 2 and (hist > 1e-8).all()
    assert s.solve(np.zeros(3 * n), allow_not_converged=True)[3] == cabi.NOT_CONVERGED
    s.close()
