// Host-side octree + interaction lists (reference semantics) and the
// level-/leaf-contiguous layout uploaded to the GPU.
//
// Semantics kept from the reference (src/core/fmm/tree.cc, calculate.cc):
//  * root centre = mean site position, half-width 1.001 * max |x - mean|
//    over the three axes, rmax = sqrt(3 r^2)                   (tree.cc:158-188)
//  * sites are inserted in input order; a cell whose count reaches ncrit is
//    split at once, its ncrit sites re-inserted in their stored order, and a
//    split cell keeps counting arrivals                         (tree.cc:189-209, :111-132)
//  * octant = (x > cx) + 2 (y > cy) + 4 (z > cz); child centre = parent
//    centre +- r/2 per axis                                     (tree.cc:94-109)
//  * dual-tree walk from (root, root): R theta > rmax_A + rmax_B -> M2L(B->A);
//    both leaves -> P2P(A<-B); else split A if B is a leaf or (rmax_A >=
//    rmax_B and A is not a leaf), otherwise split B            (calculate.cc:74-127)
//  * the M2L list is ordered by source cell                    (tree.cc:224-227)
// This file must be compiled without floating-point contraction
// (-ffp-contract=off): the acceptance distance sits exactly on the theta
// boundary for cells offset by (4,4,4) half-widths, and the reference's golden
// FMM errors are reproduced by the uncontracted evaluation only.
#include "tree.h"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace cg {

namespace {

struct Builder {
  const double* xyz;
  int ncrit;
  RefTree& t;

  int add_cell(double x, double y, double z, double r, int parent, int level) {
    int c = (int)t.x.size();
    t.x.push_back(x), t.y.push_back(y), t.z.push_back(z), t.r.push_back(r);
    t.rmax.push_back(std::sqrt(3 * r * r));
    t.parent.push_back(parent), t.level.push_back(level);
    t.nleaf.push_back(0), t.nchild.push_back(0u);
    t.child.insert(t.child.end(), 8, 0);
    t.head.push_back(-1), t.tail.push_back(-1);
    return c;
  }

  int octant(int i, int c) const {
    return (xyz[3 * i] > t.x[c]) + ((xyz[3 * i + 1] > t.y[c]) << 1) +
           ((xyz[3 * i + 2] > t.z[c]) << 2);
  }

  int child_of(int p, int o) {
    if (!(t.nchild[p] & (1u << o))) {
      const double h = t.r[p] / 2.0;
      int c          = add_cell(t.x[p] + h * ((o & 1) * 2 - 1), t.y[p] + h * ((o & 2) - 1),
                                t.z[p] + h * ((o & 4) / 2 - 1), h, p, t.level[p] + 1);
      t.child[8 * p + o] = c;
      t.nchild[p] |= (1u << o);
    }
    return t.child[8 * p + o];
  }

  // Appends site i to cell c and splits c when it becomes full.
  bool place(int c, int i, int depth) {
    t.next[i] = -1;
    (t.tail[c] < 0 ? t.head[c] : t.next[t.tail[c]]) = i;
    t.tail[c] = i;
    t.nleaf[c] += 1;
    if (t.nleaf[c] < ncrit) return true;
    if (depth > 96) return false;
    for (int s = t.head[c], k = 0; k < ncrit; ++k) {
      const int nx = t.next[s];
      int ch       = child_of(c, octant(s, c));
      if (!place(ch, s, depth + 1)) return false;
      s = nx;
    }
    t.head[c] = t.tail[c] = -1;
    return true;
  }

  bool insert(int i) {
    int c = 0, depth = 0;
    while (t.nleaf[c] >= ncrit) {
      t.nleaf[c] += 1;
      c = child_of(c, octant(i, c));
      if (++depth > 96) return false;
    }
    return place(c, i, depth);
  }
};

enum Step { STEP_M2L, STEP_P2P, STEP_SPLIT_A, STEP_SPLIT_B };

// The walk's decision for the cell pair (A, B).
Step walk_step(const RefTree& t, int A, int B, double theta, int ncrit) {
  const double dx = t.x[A] - t.x[B];
  const double dy = t.y[A] - t.y[B];
  const double dz = t.z[A] - t.z[B];
  const double R  = std::sqrt(dx * dx + dy * dy + dz * dz);
  if (R * theta > t.rmax[A] + t.rmax[B]) return STEP_M2L;
  const bool leafA = t.nchild[A] == 0, leafB = t.nchild[B] == 0;
  if (leafA && leafB)  // (a full leaf is unreachable for well-formed trees)
    return t.nleaf[B] >= ncrit ? STEP_M2L : STEP_P2P;
  return leafB || (t.rmax[A] >= t.rmax[B] && !leafA) ? STEP_SPLIT_A : STEP_SPLIT_B;
}

void walk(const RefTree& t, int A, int B, double theta, int ncrit, RefTree::Pairs& m2l,
          RefTree::Pairs& p2p) {
  switch (walk_step(t, A, B, theta, ncrit)) {
    case STEP_M2L: m2l.emplace_back(B, A); break;
    case STEP_P2P: p2p.emplace_back(A, B); break;
    case STEP_SPLIT_A:
      for (int o = 0; o < 8; ++o)
        if (t.nchild[A] & (1u << o)) walk(t, t.child[8 * A + o], B, theta, ncrit, m2l, p2p);
      break;
    case STEP_SPLIT_B:
      for (int o = 0; o < 8; ++o)
        if (t.nchild[B] & (1u << o)) walk(t, A, t.child[8 * B + o], theta, ncrit, m2l, p2p);
  }
}

// The walk from (root, root): expanded in order to a few hundred cell pairs,
// which threads then walk in contiguous shares; the shares in sequence are the
// recursion's order.  (100,002 sites on 16 host cores: tree and lists 61 -> 14 ms, 300,000 sites 600 -> 75 ms.)
void walk_all(RefTree& t, int n) {
  std::vector<std::pair<int, int>> at{{0, 0}}, nx;
  const int threads = host_threads(n, 4096);
  for (int round = 0; round < 12 && threads > 1 && at.size() < 64u * threads; ++round) {
    nx.clear();
    bool any = false;
    for (const auto& p : at) {
      const Step st = walk_step(t, p.first, p.second, t.theta, t.ncrit);
      if (st == STEP_M2L || st == STEP_P2P) {
        nx.push_back(p);  // its own walk emits it in place
        continue;
      }
      any         = true;
      const int c = st == STEP_SPLIT_A ? p.first : p.second;
      for (int o = 0; o < 8; ++o)
        if (t.nchild[c] & (1u << o)) {
          const int ch = t.child[8 * c + o];
          nx.emplace_back(st == STEP_SPLIT_A ? ch : p.first, st == STEP_SPLIT_A ? p.second : ch);
        }
    }
    at.swap(nx);
    if (!any) break;
  }
  // more shares than threads, taken in turn, so that uneven ones even out
  const int shares = threads > 1 ? (int)std::min<size_t>(at.size(), 16u * threads) : 1;
  t.m2l.assign(shares, {}), t.p2p.assign(shares, {});
  host_parallel(threads, threads, [&](int th, long, long) {
    for (int s = th; s < shares; s += threads) {
      const size_t b = at.size() * s / shares, e = at.size() * (s + 1) / shares;
      for (size_t k = b; k < e; ++k)
        walk(t, at[k].first, at[k].second, t.theta, t.ncrit, t.m2l[s], t.p2p[s]);
    }
  });
  for (const auto& v : t.m2l) t.nm2l += (long)v.size();
  for (const auto& v : t.p2p) t.np2p += (long)v.size();
}

// Groups the pairs of `parts` by key(pair) into CSR rows, each row in walk order:
// out[ptr[k]..) = value(pair).  Threads take contiguous shares of the parts.
template <class Key, class Value>
void group_pairs(const std::vector<RefTree::Pairs>& parts, long total, int nkeys, Key key,
                 Value value, std::vector<int>& ptr, std::vector<int>& out) {
  const int threads =
        std::min(host_threads(total, 1 << 15), (int)std::max<size_t>(1, parts.size()));
  std::vector<std::vector<int>> pos(threads);
  host_parallel(threads, (long)parts.size(), [&](int th, long b, long e) {
    pos[th].assign(nkeys, 0);
    for (long q = b; q < e; ++q)
      for (const auto& p : parts[q]) pos[th][key(p)]++;
  });
  ptr.assign(nkeys + 1, 0);
  int at = 0;
  for (int k = 0; k < nkeys; ++k) {
    ptr[k] = at;
    for (int th = 0; th < threads; ++th) {
      const int c = pos[th][k];
      pos[th][k]  = at;
      at += c;
    }
  }
  ptr[nkeys] = at;
  out.resize(total);
  host_parallel(threads, (long)parts.size(), [&](int th, long b, long e) {
    for (long q = b; q < e; ++q)
      for (const auto& p : parts[q]) out[pos[th][key(p)]++] = value(p);
  });
}

}  // namespace

bool build_ref_tree(int n, const double* xyz, int ncrit, double theta, RefTree& t,
                    std::string& err) {
  t       = RefTree();
  t.ncrit = ncrit;
  t.theta = theta;
  if (n <= 0) {
    err = "empty system";
    return false;
  }
  if (ncrit < 1) {
    err = "tree_ncrit must be >= 1";
    return false;
  }
  double xa = 0, ya = 0, za = 0;
  for (int i = 0; i < n; ++i) {
    if (!std::isfinite(xyz[3 * i]) || !std::isfinite(xyz[3 * i + 1]) ||
        !std::isfinite(xyz[3 * i + 2])) {
      err = "non-finite site position " + std::to_string(i);
      return false;
    }
    xa += xyz[3 * i], ya += xyz[3 * i + 1], za += xyz[3 * i + 2];
  }
  xa /= n, ya /= n, za /= n;
  double xm = 0, ym = 0, zm = 0;
  for (int i = 0; i < n; ++i) {
    xm = std::max(xm, std::abs(xyz[3 * i] - xa));
    ym = std::max(ym, std::abs(xyz[3 * i + 1] - ya));
    zm = std::max(zm, std::abs(xyz[3 * i + 2] - za));
  }
  double r = (xm > ym ? (xm > zm ? xm : zm) : (ym > zm ? ym : zm)) * 1.001;
  Builder b{xyz, ncrit, t};
  t.next.assign(n, -1);
  b.add_cell(xa, ya, za, r, 0, 0);
  for (int i = 0; i < n; ++i)
    if (!b.insert(i)) {
      err = "octree depth limit reached: sites coincide (at least " + std::to_string(ncrit) +
            " sites at one position)";
      return false;
    }
  walk_all(t, n);
  return true;
}

RefTree::Pairs RefTree::p2p_flat() const {
  Pairs out;
  out.reserve(np2p);
  for (const auto& v : p2p) out.insert(out.end(), v.begin(), v.end());
  return out;
}

RefTree::Pairs RefTree::m2l_by_source() const {
  Pairs out;
  out.reserve(nm2l);
  for (const auto& v : m2l) out.insert(out.end(), v.begin(), v.end());
  std::stable_sort(out.begin(), out.end(),
                   [](const std::pair<int, int>& a, const std::pair<int, int>& b) {
                     return a.first < b.first;
                   });
  return out;
}

void make_layout(const RefTree& t, int n, TreeLayout& L) {
  const int nc = (int)t.x.size();
  L        = TreeLayout();
  L.n      = n;
  L.ncells = nc;
  // Renumber cells by (level, creation index).
  int maxl = 0;
  for (int c = 0; c < nc; ++c) maxl = std::max(maxl, t.level[c]);
  L.nlevels = maxl + 1;
  L.level_start.assign(L.nlevels + 1, 0);
  for (int c = 0; c < nc; ++c) L.level_start[t.level[c] + 1]++;
  for (int l = 0; l < L.nlevels; ++l) L.level_start[l + 1] += L.level_start[l];
  std::vector<int> fill(L.level_start.begin(), L.level_start.end() - 1);
  std::vector<int> new_of_old(nc);
  L.old_of_new.resize(nc);
  for (int c = 0; c < nc; ++c) {
    int k           = fill[t.level[c]]++;
    new_of_old[c]   = k;
    L.old_of_new[k] = c;
  }
  L.center.resize(4 * (size_t)nc);
  L.parent.resize(nc);
  L.is_leaf.assign(nc, 0);
  L.child_ptr.assign(nc + 1, 0);
  for (int k = 0; k < nc; ++k) {
    int c               = L.old_of_new[k];
    L.center[4 * k]     = t.x[c];
    L.center[4 * k + 1] = t.y[c];
    L.center[4 * k + 2] = t.z[c];
    L.center[4 * k + 3] = t.r[c];
    L.parent[k]         = c == 0 ? -1 : new_of_old[t.parent[c]];
    L.is_leaf[k]        = t.nleaf[c] < t.ncrit ? 1 : 0;
    for (int o = 0; o < 8; ++o)
      if (t.nchild[c] & (1u << o)) L.child_idx.push_back(new_of_old[t.child[8 * c + o]]);
    L.child_ptr[k + 1] = (int)L.child_idx.size();
  }
  // Leaves in renumbered order; particles leaf-contiguous.
  L.leaf_of_cell.assign(nc, -1);
  L.leaf_start.push_back(0);
  L.perm.reserve(n);
  for (int k = 0; k < nc; ++k) {
    if (!L.is_leaf[k]) continue;
    int c                = L.old_of_new[k];
    L.leaf_of_cell[k]    = (int)L.leaf_cell.size();
    L.leaf_cell.push_back(k);
    for (int q = t.head[c]; q >= 0; q = t.next[q]) L.perm.push_back(q);
    L.leaf_start.push_back((int)L.perm.size());
  }
  L.nleaves = (int)L.leaf_cell.size();
  L.inv_perm.assign(n, -1);
  for (int k = 0; k < (int)L.perm.size(); ++k) L.inv_perm[L.perm[k]] = k;
  // M2L grouped by target, each target's sources in the reference's order (the
  // list sorted by source: creation order), renumbered.
  group_pairs(t.m2l, t.nm2l, nc, [&](const std::pair<int, int>& p) { return new_of_old[p.second]; },
              [](const std::pair<int, int>& p) { return p.first; }, L.m2l_ptr, L.m2l_src);
  host_parallel(host_threads(t.nm2l, 1 << 13), nc, [&](int, long c0, long c1) {
    for (long k = c0; k < c1; ++k) {
      int *q0 = L.m2l_src.data() + L.m2l_ptr[k], *q1 = L.m2l_src.data() + L.m2l_ptr[k + 1];
      if (!std::is_sorted(q0, q1)) std::sort(q0, q1);
      for (int* q = q0; q < q1; ++q) *q = new_of_old[*q];
    }
  });
  // P2P grouped by target leaf (walk order).
  group_pairs(t.p2p, t.np2p, L.nleaves,
              [&](const std::pair<int, int>& p) { return L.leaf_of_cell[new_of_old[p.first]]; },
              [&](const std::pair<int, int>& p) { return L.leaf_of_cell[new_of_old[p.second]]; },
              L.p2p_ptr, L.p2p_src);
  for (int a = 0; a < L.nleaves; ++a) {
    const long na = L.leaf_start[a + 1] - L.leaf_start[a];
    for (int q = L.p2p_ptr[a]; q < L.p2p_ptr[a + 1]; ++q)
      L.p2p_pairs += na * (L.leaf_start[L.p2p_src[q] + 1] - L.leaf_start[L.p2p_src[q]]);
  }
}

}  // namespace cg
