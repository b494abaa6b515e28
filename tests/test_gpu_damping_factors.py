"""Thole damping with factors at the ends of their range: zero, so small that the
argument damping s_i s_j R of every pair is below any limit a kernel compares it
with (that of the source which fills an odd tile's last pair, too), and negative.

Tolerances: a damped term is the undamped one times 1 - c with c rounded to
2^-53, so errors are measured against the undamped sums: 4e-15 of an apply
(alpha^-1 v is most of it) and 4e-14 of a static field, as in test_gpu_near64.py.
"""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu
TOL = 4e-15


def sites(b, order):
    from oracle import oracle as O
    return O.Sites(xyz=b.xyz, elements=b.elements, q=b.q, mu=b.mu, quad=b.quad, max_order=order,
                   alpha6=b.alpha6, polarizable=np.ones(b.n, np.int32), excl_ptr=b.excl_ptr,
                   excl_idx=b.excl_idx)


def free(b):
    """The box without its exclusions (the undamped sums that set the scale hold
    every pair)."""
    import copy
    c = copy.copy(b)
    c.excl_ptr, c.excl_idx = np.zeros(b.n + 1, np.int32), np.zeros(1, np.int32)
    return c


@pytest.mark.parametrize("factor", [0.0, 1e-12, 1e-5])
@pytest.mark.parametrize("waters,fmm,ncrit", [(343, False, 64), (511, False, 64), (900, True, 16),
                                              (901, True, 64)])
def test_apply(gpu, port, waters, fmm, ncrit, factor):
    from cppe_gb300 import synthetic
    b = synthetic.water_box(waters, seed=waters)
    v = np.random.default_rng(1).normal(size=3 * b.n)
    s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, damp=True, damping=factor, order=5,
                    ncrit=ncrit, summation=cabi.FMM if fmm else cabi.DIRECT)
    ref = port.bmatrix_apply(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, v, fmm=int(fmm),
                             ncrit=ncrit, order=5, damping=factor)
    assert np.linalg.norm(s.apply(v) - ref) < TOL * np.linalg.norm(ref)
    s.close()


@pytest.mark.parametrize("factor", [0.0, 1e-12, 1e-5])
@pytest.mark.parametrize("waters,fmm", [(1, False), (11, False), (101, False), (343, False),
                                        (65, True), (901, True)])
def test_static_fields(gpu, port, waters, fmm, factor):
    from cppe_gb300 import synthetic
    b = synthetic.water_box(waters, seed=waters)
    one = np.ones(b.n, np.int32)
    scale = np.linalg.norm(port.multipole_fields(sites(free(b), 2), fmm=fmm, order=6, damping=0.0))
    for order in (1, 2):
        ref = port.multipole_fields(sites(b, order), fmm=fmm, order=6, damping=factor)
        got = cabi.multipole_fields(b.xyz, b.q, b.mu, b.quad, order, one, b.alpha_iso, b.excl_ptr,
                                    b.excl_idx, fmm=fmm, order=6, damp=True, damping=factor)
        assert np.linalg.norm(got - ref) < 10 * TOL * scale


def test_one_site(gpu):
    # the smallest odd tile: nothing but the site itself
    one = np.ones(1)
    for factor in (0.0, 1e-12, 1e-5, 2.1304):
        got = cabi.multipole_fields(np.zeros((1, 3)), one, np.ones((1, 3)), np.ones((1, 6)), 2,
                                    np.ones(1, np.int32), one, np.zeros(2, np.int32),
                                    np.zeros(1, np.int32), damp=True, damping=factor)
        assert np.abs(got).max() < 1e-30


def test_batch(gpu):
    from cppe_gb300 import synthetic
    boxes = [synthetic.water_box(w, seed=w) for w in (11, 101, 343)]
    rhs = np.concatenate([0.01 * np.random.default_rng(b.n).normal(size=6 * b.n) for b in boxes])
    mu = [cabi.Batch(boxes, 2, thresh=1e-9, **kw).solve(rhs)[0]
          for kw in (dict(damp=True, damping=0.0), dict(damp=False))]
    np.testing.assert_allclose(mu[0], mu[1], rtol=0, atol=1e-8)


@pytest.mark.parametrize("factor", [0.0, -2.1304, -1e-3, float("nan")])
@pytest.mark.parametrize("waters,fmm", [(11, False), (343, False), (901, True)])
def test_factors_that_damp_nothing(gpu, port, waters, fmm, factor):
    """A factor that is not positive: the undamped operator in every arithmetic, and
    the undamped fields."""
    from cppe_gb300 import synthetic
    b = synthetic.water_box(waters, seed=waters)
    v = np.random.default_rng(1).normal(size=3 * b.n)
    opts = dict(order=5, summation=cabi.FMM if fmm else cabi.DIRECT)
    s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, damp=True, damping=factor, **opts)
    u = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, damp=False, **opts)
    ref = port.bmatrix_apply(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, v, fmm=int(fmm), order=5)
    assert np.linalg.norm(s.apply(v) - ref) < TOL * np.linalg.norm(ref)
    for kw in (dict(fp32=True), dict(dd=True)):
        assert np.array_equal(s.apply(v, **kw), u.apply(v, **kw))
    one = np.ones(b.n, np.int32)
    args = (b.xyz, b.q, b.mu, b.quad, 2, one, b.alpha_iso, b.excl_ptr, b.excl_idx)
    got = cabi.multipole_fields(*args, fmm=fmm, damp=True, damping=factor)
    want = cabi.multipole_fields(*args, fmm=fmm)
    assert np.linalg.norm(got - want) <= 10 * TOL * np.linalg.norm(want)
    s.close(), u.close()


@pytest.mark.parametrize("factor", [1e-6, 1e-15])
def test_sites_without_a_damping_partner(gpu, port, factor):
    """Half of the sites take no part in the damping: their pairs stay undamped
    whatever the factor."""
    from cppe_gb300 import synthetic
    from oracle import oracle as O
    b = free(synthetic.water_box(343, seed=3))
    pol = (np.arange(b.n) % 2).astype(np.int32)
    a6 = b.alpha6 * pol[:, None]
    for order in (1, 2):
        site = O.Sites(xyz=b.xyz, elements=b.elements, q=b.q, mu=b.mu, quad=b.quad,
                       max_order=order, alpha6=a6, polarizable=pol, excl_ptr=b.excl_ptr,
                       excl_idx=b.excl_idx)
        und = port.multipole_fields(site, fmm=False, order=5, damping=0.0)
        ref = port.multipole_fields(site, fmm=False, order=5, damping=factor)
        got = cabi.multipole_fields(b.xyz, b.q, b.mu, b.quad, order, pol, b.alpha_iso, b.excl_ptr,
                                    b.excl_idx, damp=True, damping=factor)
        assert np.linalg.norm(got - ref) < 10 * TOL * np.linalg.norm(und)
