"""FP64 static fields and applies over sparse, wide and mixed systems: where the far
pairs are most of the field they have to be as accurate as near ones.

The sums in extended precision are numpy longdoubles (64 or 113 bits of mantissa).
Tolerance: a term takes about ten FP64 roundings, of 3e-16 together at random, and
the fields here have few terms of their size: 1.5e-15 of the field's norm is four
times that.  Double-float far pairs carry 2e-14.
"""
import numpy as np
import pytest

import cabi

pytestmark = pytest.mark.gpu
DAMPING = 2.1304
L = np.longdouble


def lattice(k, spacing, seed=7, jitter=0.1):
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(float(k))] * 3, indexing="ij"), -1).reshape(-1, 3)
    return spacing * (g + rng.uniform(-jitter, jitter, g.shape)), rng


def field(xyz, mom, order, alpha, damp):
    """The static field of dipoles or quadrupoles at every site."""
    n, X = len(xyz), xyz.astype(L)
    out = np.zeros((n, 3), L)
    s = alpha.astype(L) ** (L(-1) / 6)
    for i in range(n):
        ok = np.arange(n) != i
        d, m = (X[i] - X)[ok], mom[ok].astype(L)
        r = np.sqrt((d * d).sum(1))
        fE = fT = fD = L(1)
        if damp:
            v = L(DAMPING) * s[i] * s[ok] * r
            e = np.exp(-v)
            fE = 1 - (1 + v + v * v / 2) * e
            fT = fE - v ** 3 / 6 * e
            fD = fT - v ** 4 / 30 * e
        if order == 1:
            f = d * ((d * m).sum(1) * 3 * fT / r ** 5)[:, None] - m * (fE / r ** 3)[:, None]
        else:
            T = m[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(-1, 3, 3)
            Td = (T * d[:, None, :]).sum(2)
            f = d * (7.5 * fD / r ** 7 * (d * Td).sum(1) -
                     1.5 * fT / r ** 5 * (m[:, 0] + m[:, 3] + m[:, 5]))[:, None] - \
                Td * (3 * fT / r ** 5)[:, None]
        out[i] = f.sum(0)
    return out


def static(xyz, mom, order, alpha, damp, ptr=None, idx=None):
    n = len(xyz)
    zero3, zero6 = np.zeros((n, 3)), np.zeros((n, 6))
    ptr = np.zeros(n + 1, np.int32) if ptr is None else ptr
    idx = np.zeros(1, np.int32) if idx is None else idx
    return cabi.multipole_fields(xyz, np.zeros(n), mom if order == 1 else zero3,
                                 mom if order == 2 else zero6, order, np.ones(n, np.int32), alpha,
                                 ptr, idx, damp=damp).reshape(n, 3)


def norm(a):
    return float(np.sqrt((a * a).sum()))


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("spacing", [3.0, 12.0, 40.0, 1.0e3, 3.0e4])
def test_sparse_fields(gpu, spacing, order, damp):
    xyz, rng = lattice(6, spacing)
    mom = rng.normal(size=(len(xyz), 3 * order))
    alpha = rng.uniform(1, 12, len(xyz))
    ref = field(xyz, mom, order, alpha, damp)
    got = static(xyz, mom, order, alpha, damp)
    # (a dipole's field is returned with the sign of the others)
    assert min(norm(got - ref), norm(got + ref)) < 1.5e-15 * norm(ref)


@pytest.mark.parametrize("damp", [False, True])
def test_dense_lattice_with_far_exclusions(gpu, port, damp):
    """Near and far pairs and exclusions of both kinds beside each other (a dense
    lattice, 33 bohr across), against the oracle with the tolerances of
    test_gpu_near64.py."""
    from oracle import oracle as O
    xyz, rng = lattice(11, 3.0)
    n = len(xyz)
    alpha = rng.uniform(0.5, 1.5, n)
    a6 = np.zeros((n, 6))
    a6[:, [0, 3, 5]] = alpha[:, None]
    excl = [sorted(rng.choice(n, rng.integers(0, 9), replace=False)) for _ in range(n)]
    ptr = np.concatenate([[0], np.cumsum([len(e) for e in excl])]).astype(np.int32)
    idx = np.array([j for e in excl for j in e], np.int32)
    f = DAMPING if damp else 0.0
    v = rng.normal(size=3 * n)
    s = cabi.System(xyz, a6, ptr, idx, damp=damp)
    ref = port.bmatrix_apply(xyz, a6, ptr, idx, v, fmm=0, damping=f)
    assert np.linalg.norm(s.apply(v) - ref) < 4e-15 * np.linalg.norm(ref)
    s.close()
    for order in (1, 2):
        mom = rng.normal(size=(n, 3 * order))
        zero = np.zeros((n, 6))
        sites = O.Sites(xyz=xyz, elements=["O"] * n, q=np.zeros(n),
                        mu=mom if order == 1 else zero[:, :3], quad=mom if order == 2 else zero,
                        max_order=order, alpha6=a6, polarizable=np.ones(n, np.int32), excl_ptr=ptr,
                        excl_idx=idx)
        want = port.multipole_fields(sites, fmm=False, order=5, damping=f)
        got = static(xyz, mom, order, alpha, damp, ptr, idx).ravel()
        assert np.linalg.norm(got - want) < 4e-14 * np.linalg.norm(want)


@pytest.mark.parametrize("damp", [False, True])
def test_wide_system(gpu, port, damp):
    """Half extent 3.5e5 bohr: the coordinate grid (1/8 bohr) is too coarse for the
    distance classes and the all-FP64 kernel serves dipoles and quadrupoles, with every
    exclusion subtracted afterwards.  Eight dense clusters with exclusions inside and
    between them, against the oracle with the tolerances of test_gpu_near64.py."""
    from oracle import oracle as O
    one, rng = lattice(6, 3.0)
    corners = 7.0e5 * np.stack(np.meshgrid(*[[0.0, 1.0]] * 3, indexing="ij"), -1).reshape(-1, 3)
    xyz = np.concatenate([one + c for c in corners])
    n = len(xyz)
    alpha = rng.uniform(0.5, 1.5, n)
    a6 = np.zeros((n, 6))
    a6[:, [0, 3, 5]] = alpha[:, None]
    excl = [sorted({int(j) for j in rng.choice(n, rng.integers(0, 5))} |
                   {int(j) for j in 216 * (i // 216) + rng.choice(216, rng.integers(0, 5))})
            for i in range(n)]
    ptr = np.concatenate([[0], np.cumsum([len(e) for e in excl])]).astype(np.int32)
    idx = np.array([j for e in excl for j in e], np.int32)
    f = DAMPING if damp else 0.0
    v = rng.normal(size=3 * n)
    s = cabi.System(xyz, a6, ptr, idx, damp=damp)
    ref = port.bmatrix_apply(xyz, a6, ptr, idx, v, fmm=0, damping=f)
    assert np.linalg.norm(s.apply(v) - ref) < 4e-15 * np.linalg.norm(ref)
    s.close()
    for order in (1, 2):
        mom = rng.normal(size=(n, 3 * order))
        zero = np.zeros((n, 6))
        sites = O.Sites(xyz=xyz, elements=["O"] * n, q=np.zeros(n),
                        mu=mom if order == 1 else zero[:, :3], quad=mom if order == 2 else zero,
                        max_order=order, alpha6=a6, polarizable=np.ones(n, np.int32), excl_ptr=ptr,
                        excl_idx=idx)
        want = port.multipole_fields(sites, fmm=False, order=5, damping=f)
        got = static(xyz, mom, order, alpha, damp, ptr, idx).ravel()
        assert np.linalg.norm(got - want) < 4e-14 * np.linalg.norm(want)


def cluster_and_outlier(distance):
    """A dense cluster (every sum over its sites is one of near pairs) and a site far
    from it, whose field is one of far pairs only."""
    xyz, rng = lattice(6, 3.0)
    return np.concatenate([xyz, [[distance, 0.3 * distance, 0.2 * distance]]]), rng


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("distance", [1.0e3, 7.0e3, 1.0e4, 3.0e4, 1.0e5, 1.0e6])
def test_far_site(gpu, distance, order):
    """The far pairs' accuracy does not fall with the distance: 2e-14 a pair and the
    terms' cancellation, 2e-13 of the outlier's own field."""
    xyz, rng = cluster_and_outlier(distance)
    mom = rng.normal(size=(len(xyz), 3 * order))
    mom[-1] = 0
    alpha = rng.uniform(1, 12, len(xyz))
    ref = field(xyz, mom, order, alpha, False)[-1]
    got = static(xyz, mom, order, alpha, False)[-1]
    assert min(norm(got - ref), norm(got + ref)) < 2e-13 * norm(ref)


@pytest.mark.parametrize("damp", [False, True])
@pytest.mark.parametrize("order", [1, 2])
def test_no_source_no_field(gpu, order, damp):
    """One site; a molecule whose pairs are all excluded: exactly zero."""
    from cppe_gb300 import synthetic
    rng = np.random.default_rng(3)
    assert not static(np.zeros((1, 3)), rng.normal(size=(1, 3 * order)), order, np.ones(1),
                      damp).any()
    b = synthetic.water_box(1, seed=1)
    assert not static(b.xyz, rng.normal(size=(3, 3 * order)), order, b.alpha_iso, damp, b.excl_ptr,
                      b.excl_idx).any()


@pytest.mark.parametrize("order", [1, 2])
def test_a_moment_that_is_not_a_number(gpu, order):
    """reaches the field of every other molecule, near and far."""
    from cppe_gb300 import synthetic
    b = synthetic.water_box(700, seed=2)
    mom = np.random.default_rng(3).normal(size=(b.n, 3 * order))
    mom[999] = np.nan
    got = static(b.xyz, mom, order, b.alpha_iso, False, b.excl_ptr, b.excl_idx)
    others = np.arange(b.n) // 3 != 333
    assert np.isnan(got[others]).all()


@pytest.mark.parametrize("distance", [1e-60, 1e-20, 1e-3, 1e10, 3e19, 1e25, 1e100])
def test_two_charges(gpu, distance):
    """q / R^2 over the range in which R^2 and R^-2 are FP64 numbers."""
    xyz = np.array([[0.0, 0, 0], [distance, 0, 0]])
    got = cabi.multipole_fields(xyz, np.array([2.0, 3.0]), np.zeros((2, 3)), np.zeros((2, 6)), 0,
                                np.ones(2, np.int32), np.ones(2), np.zeros(3, np.int32),
                                np.zeros(1, np.int32)).reshape(2, 3)
    want = np.array([[-3.0, 0, 0], [2.0, 0, 0]]) / distance ** 2
    np.testing.assert_allclose(got, want, rtol=1e-15, atol=0)
