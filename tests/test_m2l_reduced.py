"""The harmonic-reduced M2L of gen_m2l.py against the full translation, in FP64
on the CPU: folded multipoles, the reduced terms and the unfolded local
expansion give the full contraction (rounding of up to 840 terms: 1e-12 of
the largest coefficient).  And the double-float rows' positions (m2l_fixed.cuh:
order o from sum of 2q + 2) cover every reduced coefficient once."""
import os
import sys

import numpy as np
import pytest

import cabi


def gen():
    sys.path.insert(0, os.path.join(cabi.LIB_PATH.rsplit(os.sep, 1)[0], "csrc"))
    import gen_m2l
    return gen_m2l


@pytest.mark.parametrize("m,p", [(1, 5), (1, 6), (0, 4), (2, 6)])
def test_reduced_translation_matches_full(m, p):
    g = gen()
    rng = np.random.default_rng(10 * m + p)
    mi = g.multi_indices(p)
    at = {t: j for j, t in enumerate(mi)}
    nt, moff = g.nterms(p), g.nterms(m - 1)
    x = rng.normal(size=3) * 3.0
    D = np.zeros(nt)
    D[0] = (x @ x) ** -0.5
    down = lambda n, i, k: at[tuple(c - (k if q == i else 0) for q, c in enumerate(n))]
    for j, n in enumerate(mi[1:], 1):
        o = sum(n)
        s = sum((2 * o - 1) * n[i] * x[i] * D[down(n, i, 1)] for i in range(3) if n[i] > 0)
        s += sum((o - 1) * n[i] * (n[i] - 1) * D[down(n, i, 2)] for i in range(3) if n[i] > 1)
        D[j] = -s / (x @ x) / o
    M = rng.normal(size=nt - moff)
    L = np.zeros(g.nterms(p - m))
    for k in range(moff, nt):
        for n in range(g.nterms(p - sum(mi[k]))):
            L[n] += D[at[tuple(a + b for a, b in zip(mi[n], mi[k]))]] * M[k - moff]
    Mr = [sum(f * M[k] for k, f in row) for row in g.fold_rows(m, p)]
    Dr = [D[at[t]] for t in mi if t[2] <= 2]
    Lr = np.zeros(len(g.reduced(0, p - m)))
    for k, n, w in g.reduced_terms(m, p):
        Lr[n] += Dr[w] * Mr[k]
    got = np.array([sum(f * Lr[n] for n, f in row) for row in g.unfold_rows(m, p)])
    np.testing.assert_allclose(got, L, rtol=0, atol=1e-12 * np.abs(L).max())


@pytest.mark.parametrize("p", [5, 6])
def test_double_float_rows(p):
    g = gen()
    pos, k = [], 0
    for o in range(1, p + 1):
        off = sum(2 * q + 2 for q in range(1, o))
        pos += [off + i for i in range(2 * o + 1)]
        assert off % 2 == 0
    assert len(pos) == len(set(pos)) == len(g.reduced(1, p))
