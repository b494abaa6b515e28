"""The FP64 dipole operator's near field (far pairs in double-float, near pairs
in FP64) against the oracle, at the sizes and inputs where its split can go
wrong: one chunk and its edges, the staged tile's edges (304 sources), leaves
of more than 128 sites, every pair near, every pair far, excluded far pairs,
moments at the ends of the FP64 range, and systems too large for the split.

Tolerance: a sum of n terms in FP64 (the oracle's and the kernel's) rounds to
about sqrt(n) 2^-53 of its largest terms; far terms carry 5e-14 of themselves
at most and are below 2 / 24^3 = 1.5e-4 of a unit moment against
alpha^-1 >= 0.17, i.e. 4e-17 of the result each.  4e-15 in norm covers n <=
3,000 with a factor of two.
"""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu
DAMPING = 2.1304
TOL = 4e-15


def close(a, ref, tol=TOL):
    assert np.linalg.norm(a - ref) < tol * np.linalg.norm(ref)


def check_dipole_field(port, xyz, alpha, ptr, idx, v, damp):
    from oracle import oracle as O
    n = xyz.shape[0]
    a6 = np.zeros((n, 6))
    a6[:, [0, 3, 5]] = alpha[:, None]
    mu, one = v.reshape(n, 3), np.ones(n, np.int32)
    sites = O.Sites(xyz=xyz, elements=["O"] * n, q=np.zeros(n), mu=mu, quad=np.zeros((n, 6)),
                    max_order=1, alpha6=a6, polarizable=one, excl_ptr=ptr, excl_idx=idx)
    ref = port.multipole_fields(sites, fmm=False, order=5, damping=DAMPING if damp else 0.0)

    def run(m):
        return cabi.multipole_fields(xyz, np.zeros(n), m, np.zeros((n, 6)), 1, one, alpha, ptr, idx,
                                     damp=damp)
    got = run(mu)
    # (no alpha^-1 term beside the field: measured against the dipoles' own size)
    assert np.linalg.norm(got - ref) < TOL * (np.linalg.norm(ref) + 0.1 * np.linalg.norm(v))
    for e in (-900, 900):
        assert np.array_equal(run(mu * 2.0 ** e), got * 2.0 ** e)


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("waters", [1, 10, 11, 22, 43, 101, 102, 333, 700])
def test_direct_sizes(gpu, port, waters, damp):
    from cppe_gb300 import synthetic
    b = synthetic.water_box(waters, seed=waters)
    s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, damp=damp)
    v = np.random.default_rng(1).normal(size=3 * b.n)
    ref = port.bmatrix_apply(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, v, fmm=0,
                             damping=DAMPING if damp else 0.0)
    close(s.apply(v), ref)
    # powers of two scale the result exactly
    for e in (-900, 900):
        assert np.array_equal(s.apply(v * 2.0 ** e), s.apply(v) * 2.0 ** e)
    s.close()
    # the same pairs through the static field of dipoles (the pair kernel at
    # every size; the operator itself is a dense matrix up to 1,024 sites)
    check_dipole_field(port, b.xyz, b.alpha_iso, b.excl_ptr, b.excl_idx, v, damp)


@pytest.mark.parametrize("ncrit", [16, 64, 300])
def test_fmm_leaf_sizes(gpu, port, ncrit):
    from cppe_gb300 import synthetic
    b = synthetic.water_box(900, seed=5)
    s = cabi.System(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, damp=True, summation=cabi.FMM,
                    order=5, ncrit=ncrit)
    v = np.random.default_rng(2).normal(size=3 * b.n)
    ref = port.bmatrix_apply(b.xyz, b.alpha6, b.excl_ptr, b.excl_idx, v, fmm=1, ncrit=ncrit,
                             order=5, theta=0.5, damping=DAMPING)
    close(s.apply(v), ref)
    s.close()


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("spacing", [1.5, 24.0, 40.0, 3.0e4])
def test_distance_classes(gpu, port, spacing, damp):
    """A jittered lattice of 343 sites with random (near and far) exclusions:
    all near, around the 24-bohr limit, all far, and 2^18 bohr across."""
    rng = np.random.default_rng(7)
    g = np.stack(np.meshgrid(*[np.arange(7.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    xyz = spacing * (g + rng.uniform(-0.1, 0.1, g.shape))
    n = xyz.shape[0]
    alpha6 = np.zeros((n, 6))
    alpha6[:, [0, 3, 5]] = rng.uniform(1.0, 12.0, (n, 1))
    excl = [sorted(rng.choice(n, rng.integers(0, 9), replace=False)) for _ in range(n)]
    ptr = np.concatenate([[0], np.cumsum([len(e) for e in excl])]).astype(np.int32)
    idx = np.array([j for e in excl for j in e], np.int32)
    s = cabi.System(xyz, alpha6, ptr, idx, damp=damp)
    v = rng.normal(size=3 * n)
    v[: 3 * (n // 2)] *= 1e-30  # a range of moments within the tiles
    ref = port.bmatrix_apply(xyz, alpha6, ptr, idx, v, fmm=0, damping=DAMPING if damp else 0.0)
    close(s.apply(v), ref)
    s.close()
    v = rng.normal(size=3 * n)
    check_dipole_field(port, xyz, alpha6[:, 0], ptr, idx, v, damp)


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("fmm", [False, True])
@pytest.mark.parametrize("waters", [1, 32, 33, 64, 700])
def test_static_fields(gpu, port, waters, fmm, damp):
    """Charges, dipoles and quadrupoles together; 192 sources a tile for the
    quadrupoles (waters 32, 33, 64).  The static fields cancel to a tenth of
    their terms: ten times the tolerance."""
    from cppe_gb300 import synthetic
    from oracle import oracle as O
    b = synthetic.water_box(waters, seed=waters)
    one = np.ones(b.n, np.int32)
    sites = O.Sites(xyz=b.xyz, elements=b.elements, q=b.q, mu=b.mu, quad=b.quad, max_order=2,
                    alpha6=b.alpha6, polarizable=one, excl_ptr=b.excl_ptr, excl_idx=b.excl_idx)
    ref = port.multipole_fields(sites, fmm=fmm, order=6, damping=DAMPING if damp else 0.0)
    got = cabi.multipole_fields(b.xyz, b.q, b.mu, b.quad, 2, one, b.alpha_iso, b.excl_ptr,
                                b.excl_idx, fmm=fmm, order=6, damp=damp)
    if waters == 1:
        assert np.abs(got).max() < 1e-14  # every pair is excluded
    else:
        close(got, ref, 10 * TOL)
