"""The generated translations as they are compiled (csrc/m2l_gen.cuh, built here for
the host): for every order emitted, the derivative recurrence, the straight-line
translation, the same from a tabulated tensor, the loop form's table of tensor
entries and the folding and unfolding tables, against the full contraction
L_n = sum_k D_{n+k} M_k with the tensor from its defining recurrence.

Tolerance: sums of up to 840 terms of either sign in FP64, 1e-12 of the largest
coefficient (test_m2l_reduced.py).
"""
import os
import subprocess

import numpy as np
import pytest

import cabi

CSRC = os.path.join(cabi.LIB_PATH.rsplit(os.sep, 1)[0], "csrc")
MAIN = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>
#define __device__
#define __constant__
#define __forceinline__ inline
#define __restrict__
using std::fma;
template <typename T> T crat(int n, int d) { return T(n) / T(d); }
template <typename T> T cinv(int d) { return T(1) / T(d); }
static double rsqrt_t(double x) { return 1.0 / std::sqrt(x); }
#include "m2l_gen.cuh"
static int nred(int p) { return p < 0 ? 0 : (p + 1) * (p + 1); }
static void print(const char* what, const double* v, int n) {
  printf("%s", what);
  for (int i = 0; i < n; ++i) printf(" %.17g", v[i]);
  printf("\n");
}
// standard input: m p x y z and the multipole; output: tensor, local expansions
int main() {
  int m, p;
  double x, y, z;
  if (scanf("%d %d %lf %lf %lf", &m, &p, &x, &y, &z) != 5) return 1;
  std::vector<double> M;
  for (double v; scanf("%lf", &v) == 1;) M.push_back(v);
#define RUN(MM, PP, NAME, NT, LS, MS, FW, UW, FLS)                                          \
  if (m == MM && p == PP) {                                                                 \
    double Mr[MS] = {}, D[NT], L[3][LS] = {};                                               \
    for (int r = 0; r < MS; ++r)                                                            \
      for (int i = 0; i < FW; ++i)                                                          \
        Mr[r] += m2l_fold_##NAME[r][i][1] * M[m2l_fold_##NAME[r][i][0]];                    \
    dtensor_##NAME<double>(x, y, z, D);                                                     \
    m2l_##NAME<double>(x, y, z, Mr, L[0]);                                                  \
    m2l_##NAME##_pre<double>(D, Mr, L[1]);                                                  \
    int t = 0, c = 0;                                                                       \
    for (int o = MM; o <= PP; ++o)                                                          \
      for (int k = 0; k < nred(o) - nred(o - 1); ++k, ++c)                                  \
        for (int n = 0; n < nred(PP - o); ++n) L[2][n] += D[m2l_w_##NAME[t++]] * Mr[c];     \
    if (t != (int)sizeof(m2l_w_##NAME) || c != MS) return 2;                                \
    print("D", D, NT);                                                                      \
    for (int f = 0; f < 3; ++f) {                                                           \
      double F[FLS] = {};                                                                   \
      for (int r = 0; r < FLS; ++r)                                                         \
        for (int i = 0; i < UW; ++i)                                                        \
          F[r] += m2l_unfold_##NAME[r][i][1] * L[f][m2l_unfold_##NAME[r][i][0]];            \
      print("L", F, FLS);                                                                   \
    }                                                                                       \
  }
  CPPE_M2L_REDUCED(RUN)
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("m2l")
    (d / "main.cc").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O0", "-w", "-I", CSRC, "-o", str(d / "m2l"),
                    str(d / "main.cc")], check=True, capture_output=True)
    return str(d / "m2l")


def indices(p):
    import sys
    sys.path.insert(0, CSRC)
    import gen_m2l
    return gen_m2l.multi_indices(p)


@pytest.mark.parametrize("m,p", [(1, 5), (1, 6), (0, 5), (0, 6), (2, 5), (2, 6)])
def test_compiled_translation(program, m, p):
    mi = indices(p)
    at = {t: j for j, t in enumerate(mi)}
    moff = sum(1 for t in mi if sum(t) < m)
    rng = np.random.default_rng(10 * m + p)
    for _ in range(3):
        x = rng.normal(size=3) * 3.0
        D = np.zeros(len(mi))
        D[0] = (x @ x) ** -0.5
        for j, n in enumerate(mi[1:], 1):
            o, s = sum(n), 0.0
            for i in range(3):
                lower = lambda k: D[at[tuple(c - k * (q == i) for q, c in enumerate(n))]]
                if n[i] > 0:
                    s += (2 * o - 1) * n[i] * x[i] * lower(1)
                if n[i] > 1:
                    s += (o - 1) * n[i] * (n[i] - 1) * lower(2)
            D[j] = -s / (x @ x) / o
        M = rng.normal(size=len(mi) - moff)
        want = np.zeros(sum(1 for t in mi if sum(t) <= p - m))
        for k in range(moff, len(mi)):
            for n, tn in enumerate(mi):
                if sum(tn) + sum(mi[k]) <= p:
                    want[n] += D[at[tuple(a + b for a, b in zip(tn, mi[k]))]] * M[k - moff]
        given = f"{m} {p} " + " ".join(repr(float(v)) for v in (*x, *M))
        out = subprocess.run([program], input=given, text=True, capture_output=True,
                             check=True).stdout.split("\n")
        rows = [(r[0], np.array(r[1:].split(), float)) for r in out if r]
        assert [r[0] for r in rows] == ["D", "L", "L", "L"]
        Dr = np.array([D[at[t]] for t in mi if t[2] <= 2])
        np.testing.assert_allclose(rows[0][1], Dr, rtol=0, atol=1e-12 * np.abs(Dr).max())
        for _, got in rows[1:]:
            np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(want).max())
