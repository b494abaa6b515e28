"""The double-float operator where its offset sums could go wrong: moments over nine
orders of magnitude, sites far closer than a bond, odd tiles and partial warps,
and several right-hand sides of very different size in one batch."""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu

# A run adds at most 32 products, each rounded a few times at 2^-48 of an offset of
# 8.2 sum |m| R^-3 (3e-12 of that sum), and a separation known to 2^-41 enters R^-5.
TOL = 1e-11


def _sites(n, seed, close):
    rng = np.random.default_rng(seed)
    g = int(np.ceil(n ** (1 / 3)))
    xyz = np.stack(np.meshgrid(*[np.arange(g)] * 3), -1).reshape(-1, 3)[:n] * 3.1 + rng.uniform(-.4, .4, (n, 3))
    if close and n > 1:
        xyz[1] = xyz[0] + [0.3, 0.0, -0.4]
    alpha = np.zeros((n, 6))
    alpha[:, [0, 3, 5]] = rng.uniform(3, 8, (n, 1))
    return xyz, alpha


def _scale(xyz, alpha, v, damp):
    """Per site: sum of |T| |m| bounds and alpha^-1 |m|."""
    m = np.abs(v).sum(1)
    s = alpha[:, 0] ** (-1 / 6)
    out = m / alpha[:, 0]
    for i in range(len(xyz)):
        r = np.linalg.norm(xyz - xyz[i], axis=1)
        r[i] = np.inf
        cube = r ** -3.0
        if damp:
            cube = np.minimum(cube, (2.1304 * s[i] * s) ** 3 / 6)
        out[i] += 3 * (cube * m).sum()
    return out


@pytest.mark.parametrize("damp", [True, False])
@pytest.mark.parametrize("n,close", [(1, False), (2, True), (33, False), (515, True), (1500, False)])
def test_double_float_apply(gpu, n, close, damp):
    xyz, alpha = _sites(n, n, close)
    rng = np.random.default_rng(3)
    v = rng.standard_normal((n, 3)) * 10.0 ** rng.uniform(-6, 3, (n, 1))
    s = cabi.System(xyz, alpha, damp=damp, damping=2.1304)
    want = s.apply(v.ravel()).reshape(n, 3)
    got = s.apply(v.ravel(), dd=True).reshape(n, 3)
    assert np.all(np.abs(got - want).max(1) <= TOL * _scale(xyz, alpha, v, damp))


@pytest.mark.parametrize("nrhs", [3, 8, 9])
def test_batch_with_right_hand_sides_of_very_different_size(gpu, nrhs):
    from cppe_gb300 import synthetic
    boxes = [synthetic.water_box(w, seed=40 + w) for w in (31, 200)]
    rng = np.random.default_rng(7)
    rhs = [rng.standard_normal(3 * b.n) * 0.01 * 10.0 ** (-1.5 * (r % 4)) for b in boxes for r in range(nrhs)]
    thresh = 1e-10
    batch = cabi.Batch(boxes, nrhs, damp=True, damping=2.1304, thresh=thresh, precision=cabi.MIXED)
    mu = np.asarray(batch.solve(np.concatenate(rhs))[0])
    at = 0
    for k, b in enumerate(boxes):
        s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, damp=True, damping=2.1304)
        for r in range(nrhs):
            f = rhs[k * nrhs + r]
            m = mu[at:at + 3 * b.n]
            at += 3 * b.n
            res = np.linalg.norm(s.apply(m) - f)
            # the stopping rule, and the double-float residual's own error
            assert res <= 1.5 * thresh + 1e-11 * np.linalg.norm(f)
