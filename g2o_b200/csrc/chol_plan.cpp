// chol_plan.cpp -- see chol_plan.h.
#include "chol_plan.h"

#include <algorithm>
#include <climits>
#include <cstddef>
#include <numeric>
#include <utility>

namespace g2oc {
namespace {

// ------------------------------------------------------- nested dissection
// Order of elimination for a sparse block graph: separators found by
// breadth-first level structures (George 1973; George and Liu 1978), each cut
// between two levels reduced to a minimum vertex cover of its edges (Konig),
// then thinned by moving vertices. A narrow band order (Cuthill-McKee) makes
// every tile step wait for the one before; the dissection's tree leaves the
// subtrees independent, so the chain of steps is about the separators of one
// path from a leaf to the root.
struct Dissector {
  const std::vector<int>& ptr;
  const std::vector<int>& adj;
  int leaf;                              // blocks of one tile
  std::vector<std::vector<int>> groups;  // elimination order: children before their separator
  std::vector<int> tag;                  // region of a vertex in the recursion
  std::vector<int> dist, match, seen;
  std::vector<int> place;                // of a vertex in the breadth-first order under way
  int ntags = 1, stamp = 0;

  Dissector(const std::vector<int>& p, const std::vector<int>& a, int nv, int leaf_blocks)
      : ptr(p), adj(a), leaf(leaf_blocks), tag(nv, 0), dist(nv, -1), match(nv, -1), seen(nv, 0),
        place(nv, 0) {}

  // breadth-first order of the region t from s; dist gets the levels
  void bfs(int s, int t, std::vector<int>& order) {
    order.clear();
    order.push_back(s);
    dist[s] = 0;
    for (size_t h = 0; h < order.size(); ++h) {
      const int u = order[h];
      for (int e = ptr[u]; e < ptr[u + 1]; ++e) {
        const int v = adj[e];
        if (tag[v] == t && dist[v] < 0) {
          dist[v] = dist[u] + 1;
          order.push_back(v);
        }
      }
    }
  }
  void clear(const std::vector<int>& vs) {
    for (int v : vs) dist[v] = -1;
  }

  // augmenting path of the bipartite matching between side 0 (dist <= cut)
  // and side 1 of the cut's edges
  bool augment(int u, int t, int cut) {
    for (int e = ptr[u]; e < ptr[u + 1]; ++e) {
      const int v = adj[e];
      if (tag[v] != t || dist[v] != cut + 1 || seen[v] == stamp) continue;
      seen[v] = stamp;
      if (match[v] < 0 || augment(match[v], t, cut)) {
        match[v] = u;
        match[u] = v;
        return true;
      }
    }
    return false;
  }

  // A cut of a region: side[] (0 / 1 / 2 = separator) of its vertices in
  // breadth-first order, their numbers, and the range of the separator's places
  struct Cut {
    std::vector<signed char> side;
    int cnt[3], lo, hi;
  };

  // Minimum vertex cover of the edges between level `cut` and level cut + 1;
  // below: vertices below a level. Looks at the two levels only.
  void cover(const std::vector<int>& order, const std::vector<int>& below, int t, int cut, Cut& C) {
    const int a = below[cut], b = below[cut + 1], c = below[cut + 2], m = (int)order.size();
    for (int i = a; i < b; ++i) {
      ++stamp;
      augment(order[i], t, cut);
    }
    // reached from the unmatched left vertices by alternating paths
    ++stamp;
    std::vector<int> q;
    for (int i = a; i < b; ++i)
      if (match[order[i]] < 0) {
        seen[order[i]] = stamp;
        q.push_back(order[i]);
      }
    for (size_t h = 0; h < q.size(); ++h)
      for (int e = ptr[q[h]]; e < ptr[q[h] + 1]; ++e) {
        const int v = adj[e];
        if (tag[v] != t || dist[v] != cut + 1 || seen[v] == stamp) continue;
        seen[v] = stamp;
        if (match[v] >= 0 && seen[match[v]] != stamp) {
          seen[match[v]] = stamp;
          q.push_back(match[v]);
        }
      }
    C.side.assign(m, 1);
    std::fill(C.side.begin(), C.side.begin() + b, 0);
    C.cnt[0] = b;
    C.cnt[1] = m - b;
    C.cnt[2] = 0;
    C.lo = m;
    C.hi = -1;
    for (int i = a; i < c; ++i) {
      const int u = order[i];
      if (match[u] < 0) continue;
      if (i < b ? seen[u] != stamp : seen[u] == stamp) {
        --C.cnt[C.side[i]];
        C.side[i] = 2;
        ++C.cnt[2];
        C.lo = std::min(C.lo, i);
        C.hi = i;
      }
      match[u] = -1;
    }
    // (a matched vertex is in one of the two levels, and so is its mate)
  }

  // one region (connected): cut it or make it one group
  void region(std::vector<int>& vs, int t) {
    const int m = (int)vs.size();
    if (m <= leaf) {
      groups.push_back(vs);
      return;
    }
    // Every look at a cut costs the edges of its separator and every
    // breadth-first order those of the region. Where a vertex has more than 16
    // neighbours fewer are tried: the plan of 4,000 poses with 200 neighbours
    // each took 150 ms, as long as all else that a first solve does
    long long edges = 0;
    for (int v : vs) edges += ptr[v + 1] - ptr[v];
    const bool thick = edges > 16ll * m;
    // pseudo-peripheral start
    std::vector<int> order;
    int s = vs[0], ecc = -1;
    for (int sweep = 0; sweep < (thick ? 2 : 6); ++sweep) {
      bfs(s, t, order);
      const int e = dist[order.back()];
      // a vertex of the last level with the fewest neighbours
      int far = order.back();
      for (size_t i = order.size(); i-- > 0 && dist[order[i]] == e;)
        if (ptr[order[i] + 1] - ptr[order[i]] < ptr[far + 1] - ptr[far]) far = order[i];
      clear(order);
      if (e <= ecc) break;
      ecc = e;
      s = far;
    }
    if (ecc <= 1) {  // every vertex next to every other
      groups.push_back(vs);
      return;
    }
    const int tries = thick ? 1 : 3;
    std::vector<int> orders[3];
    Cut C;
    std::vector<signed char> best_side;
    int best_try = -1;
    double best = 1e300;
    std::vector<int> cand;
    for (int k = 0; k < tries; ++k) {
      std::vector<int>& order = orders[k];
      bfs(s, t, order);
      for (int i = 0; i < m; ++i) place[order[i]] = i;
      const int e = dist[order.back()];
      std::vector<int> count(e + 2, 0), below(e + 2, 0);
      for (int u : order) ++count[dist[u]];
      for (int l = 0; l <= e; ++l) below[l + 1] = below[l] + count[l];
      cand.clear();
      for (int l = 0; l < e; ++l) {
        const double f = (double)below[l + 1] / m;
        // a cut through wide levels is no separator, and costly to cover
        if (f >= 0.2 && f <= 0.8 && std::min(count[l], count[l + 1]) <= m / 4 + leaf) cand.push_back(l);
      }
      if (cand.empty()) {  // the level that crosses the middle
        int l = 0;
        while (l + 1 < e && below[l + 1] * 2 < m) ++l;
        if (e > 0 && std::min(count[l], count[l + 1]) <= m / 4 + leaf) cand.push_back(l);
      }
      // the narrowest first; where few are looked at, for what the cut takes off
      // the larger part
      auto width = [&](int l) {
        const int w = std::min(count[l], count[l + 1]);
        return thick ? (double)w / std::min(below[l + 1], m - below[l + 1]) : (double)w;
      };
      std::sort(cand.begin(), cand.end(), [&](int a, int b) {
        const double wa = width(a), wb = width(b);
        return wa < wb || (wa == wb && a < b);
      });
      const size_t most = thick ? std::max(1ll, 128ll * m / edges) : 8;
      if (cand.size() > most) cand.resize(most);
      for (int l : cand) {
        cover(order, below, t, l, C);
        thin(order, t, C);
        const double sc = score(C.cnt);
        if (sc < best) {
          best = sc;
          best_side = C.side;
          best_try = k;
        }
      }
      // the next try starts from a vertex of the middle level
      const int mid = order[m / 2];
      const int next = order.back();
      clear(order);
      s = k == 0 ? mid : next;
    }
    if (best >= 1e299) {
      if (!hubs(vs, t)) groups.push_back(vs);
      return;
    }
    std::vector<int> part[3];
    for (int i = 0; i < m; ++i) part[best_side[i]].push_back(orders[best_try][i]);
    std::vector<signed char>().swap(best_side);
    std::vector<signed char>().swap(C.side);
    for (auto& o : orders) std::vector<int>().swap(o);
    for (int p = 0; p < 2; ++p) {
      const int nt = ntags++;
      for (int v : part[p]) tag[v] = nt;
      // separator vertices leave the regions
    }
    for (int v : part[2]) tag[v] = -1;
    for (int p = 0; p < 2; ++p)
      if (!part[p].empty()) components(part[p]);
    std::sort(part[2].begin(), part[2].end());
    groups.push_back(part[2]);
  }

  // A region that no cut between levels shortens, since some vertices are
  // next to a large part of it: those with eight times the median number of
  // neighbours become its separator, and what is left is dissected by itself.
  // A pose that 19,999 others are measured from (137 million tile products as
  // one dense group) leaves a graph without edges.
  bool hubs(const std::vector<int>& vs, int t) {
    const int m = (int)vs.size();
    if (m <= 2 * leaf) return false;
    std::vector<int> deg(m, 0);
    for (int i = 0; i < m; ++i)
      for (int e = ptr[vs[i]]; e < ptr[vs[i] + 1]; ++e) deg[i] += tag[adj[e]] == t;
    std::vector<int> sorted(deg);
    std::nth_element(sorted.begin(), sorted.begin() + m / 2, sorted.end());
    const int least = std::max(leaf, 8 * sorted[m / 2]);
    std::vector<int> sep, rest;
    for (int i = 0; i < m; ++i) (deg[i] >= least ? sep : rest).push_back(vs[i]);
    if (sep.empty() || (int)sep.size() > m / 8) return false;
    const int nt = ntags++;
    for (int v : rest) tag[v] = nt;
    for (int v : sep) tag[v] = -1;
    components(rest);
    std::sort(sep.begin(), sep.end());
    groups.push_back(sep);
    return true;
  }

  // tiles a set of k blocks fills
  double tiles(int k) const { return (double)((k + leaf - 1) / leaf); }

  // how good a cut is: the chain through the separator and the larger part,
  // in tiles, with the parts taken to shrink by the same ratio; a cut that
  // does not shorten the chain is no cut
  double score(const int cnt[3]) const {
    const int m = cnt[0] + cnt[1] + cnt[2];
    if (cnt[0] == 0 || cnt[1] == 0) return 1e300;
    const int big = std::max(cnt[0], cnt[1]);
    if (tiles(cnt[2]) + tiles(big) >= tiles(m) + (tiles(m) > 2 ? 0 : 1)) return 1e300;
    // separator size against the share of vertices taken off the larger part
    return (double)(cnt[2] + 1) / (double)(m - big) * (double)m;
  }

  // thin the separator: vertices with neighbours on one side only join it;
  // then moves of one vertex to a side that bring in at most as many as leave
  void thin(const std::vector<int>& order, int t, Cut& C) {
    std::vector<signed char>& side = C.side;
    int(&cnt)[3] = C.cnt;
    for (int pass = 0; pass < 8; ++pass) {
      bool moved = false;
      for (int i = C.lo; i <= C.hi; ++i) {
        if (side[i] != 2) continue;
        const int u = order[i];
        int nb[2] = {0, 0};
        for (int e = ptr[u]; e < ptr[u + 1]; ++e)
          if (tag[adj[e]] == t && side[place[adj[e]]] != 2) ++nb[side[place[adj[e]]]];
        // move u to side p: its neighbours on the other side enter
        for (int q = 0; q < 2; ++q) {
          const int p = cnt[0] <= cnt[1] ? q : 1 - q;
          const int in = nb[1 - p];
          const bool to_small = cnt[p] < cnt[1 - p];
          if (in == 0 || (in == 1 && to_small && pass < 6 && cnt[1 - p] - cnt[p] > 2)) {
            side[i] = (signed char)p;
            ++cnt[p];
            --cnt[2];
            if (in)
              for (int e = ptr[u]; e < ptr[u + 1]; ++e) {
                const int v = place[adj[e]];
                if (tag[adj[e]] == t && side[v] == 1 - p) {
                  side[v] = 2;
                  --cnt[1 - p];
                  ++cnt[2];
                  C.lo = std::min(C.lo, v);
                  C.hi = std::max(C.hi, v);
                }
              }
            moved = true;
            break;
          }
        }
      }
      if (!moved) break;
    }
  }

  // the connected components of a set that already has its own tag; small
  // ones share a group
  void components(std::vector<int>& vs) {
    const int t = tag[vs[0]];
    std::vector<std::vector<int>> big;
    std::vector<int> small, order;
    for (int v : vs) {
      if (dist[v] >= 0) continue;
      bfs(v, t, order);
      if ((int)order.size() <= leaf / 2) {
        if ((int)(small.size() + order.size()) > leaf) {
          groups.push_back(small);
          small.clear();
        }
        small.insert(small.end(), order.begin(), order.end());
      } else {
        big.push_back(order);
      }
    }
    clear(vs);
    std::vector<int>().swap(vs);
    if (!small.empty()) groups.push_back(small);
    for (auto& b : big) {
      int nt = t;
      if (big.size() > 1 || !small.empty()) {
        nt = ntags++;
        for (int v : b) tag[v] = nt;
      }
      region(b, nt);
    }
  }
};

}  // namespace

// the fill of the pattern below the diagonal (tile rows by column) and its
// slots; false: more of them, or of the products, than the plan may have
static bool plan_slots(CholSymbolic& P, std::vector<std::vector<int>>& col, long long max_tiles) {
  const int nt = P.nt;
  long long tiles = nt, products = 0;
  // fill: the rows of a column join its parent's (the first row below it)
  P.col_ptr.assign(nt + 1, 0);
  for (int k = 0; k < nt; ++k) {
    std::vector<int>& l = col[k];
    std::sort(l.begin(), l.end());
    l.erase(std::unique(l.begin(), l.end()), l.end());
    if (!l.empty() && l.size() > 1) {
      std::vector<int>& p = col[l[0]];
      p.insert(p.end(), l.begin() + 1, l.end());
    }
    const long long rows = (long long)l.size();
    tiles += 1 + rows;
    products += rows * (rows + 1) / 2;
    if (tiles > std::min<long long>(max_tiles, INT_MAX) || products > INT_MAX) return false;
    P.col_ptr[k + 1] = P.col_ptr[k] + 1 + (int)rows;
  }
  const int ns = P.col_ptr[nt];
  P.row.resize(ns);
  P.col.resize(ns);
  for (int k = 0; k < nt; ++k) {
    int s = P.col_ptr[k];
    P.row[s] = k;
    P.col[s++] = k;
    for (int i : col[k]) {
      P.row[s] = i;
      P.col[s++] = k;
    }
  }
  return true;
}

// update lists, hand-out order and substitution lists of the slots
static void plan_lists(CholSymbolic& P) {
  const int nt = P.nt, ns = P.col_ptr[nt];
  // updates, by target slot (columns ascending within a target)
  P.upd_ptr.assign(ns + 1, 0);
  auto each_update = [&](auto&& f) {
    for (int j = 0; j < nt; ++j) {
      const int s0 = P.col_ptr[j] + 1, s1 = P.col_ptr[j + 1];
      for (int b = s0; b < s1; ++b) {
        // targets in tile column row[b]: its rows are a superset of row[b..]
        const int k = P.row[b];
        int s = P.col_ptr[k];
        for (int a = b; a < s1; ++a) {
          while (P.row[s] != P.row[a]) ++s;
          f(s, a, b);
        }
      }
    }
  };
  each_update([&](int s, int, int) { ++P.upd_ptr[s + 1]; });
  for (int s = 0; s < ns; ++s) P.upd_ptr[s + 1] += P.upd_ptr[s];
  P.upd.resize(2 * (size_t)P.upd_ptr[ns]);
  {
    std::vector<int> at(P.upd_ptr.begin(), P.upd_ptr.end() - 1);
    each_update([&](int s, int a, int b) {
      const size_t o = 2 * (size_t)at[s]++;
      P.upd[o] = a;
      P.upd[o + 1] = b;
    });
  }
  // hand-out order: list scheduling with estimated times (a product, the
  // diagonal tile's factorization, a panel's product with the inverse). A
  // slot's updates are taken as their operands finish; the slot is handed
  // out early enough to have all but the last done by then, but after every
  // slot it needs (so that a wait is always for a tile that some CTA has).
  constexpr float kGemm = 2.5f, kPotrf = 20.f, kPanel = 6.f, kEps = 1e-3f;
  std::vector<float> fin(ns, 0.f), key(ns, 0.f);
  std::vector<std::pair<float, int>> order;
  std::vector<int> tmp;
  for (int s = 0; s < ns; ++s) {
    const int u0 = P.upd_ptr[s], u1 = P.upd_ptr[s + 1];
    order.clear();
    float kmin = 0.f;
    for (int u = u0; u < u1; ++u) {
      const int a = P.upd[2 * (size_t)u], b = P.upd[2 * (size_t)u + 1];
      order.push_back({std::max(fin[a], fin[b]), u});
      kmin = std::max(kmin, std::max(key[a], key[b]) + kEps);
    }
    float t = 0.f;
    if (!std::is_sorted(order.begin(), order.end())) {  // it is where the columns form a chain
      std::sort(order.begin(), order.end());
      tmp.clear();
      for (auto& o : order) {
        tmp.push_back(P.upd[2 * (size_t)o.second]);
        tmp.push_back(P.upd[2 * (size_t)o.second + 1]);
      }
      std::copy(tmp.begin(), tmp.end(), P.upd.begin() + 2 * (size_t)u0);
    }
    for (auto& o : order) t = std::max(t, o.first) + kGemm;
    float start = order.empty() ? 0.f : order.back().first - kGemm * (order.size() - 1);
    if (s != P.col_ptr[P.col[s]]) {
      const int d = P.col_ptr[P.col[s]];
      kmin = std::max(kmin, key[d] + kEps);
      if (order.empty()) start = fin[d];
      t = std::max(t, fin[d]) + kPanel;
      start = std::max(start, std::min(fin[d], t) - kGemm * (order.size() + 1));
    } else {
      t += kPotrf;
    }
    fin[s] = t;
    key[s] = std::max(std::max(start, 0.f), kmin);
  }
  P.task.resize(ns);
  std::iota(P.task.begin(), P.task.end(), 0);
  std::stable_sort(P.task.begin(), P.task.end(), [&](int a, int b) { return key[a] < key[b]; });
  // substitutions
  P.fwd_ptr.assign(nt + 1, 0);
  for (int s = 0; s < ns; ++s)
    if (P.row[s] != P.col[s]) ++P.fwd_ptr[P.row[s] + 1];
  for (int k = 0; k < nt; ++k) P.fwd_ptr[k + 1] += P.fwd_ptr[k];
  P.fwd.resize(P.fwd_ptr[nt]);
  {
    std::vector<int> at(P.fwd_ptr.begin(), P.fwd_ptr.end() - 1);
    for (int s = 0; s < ns; ++s)
      if (P.row[s] != P.col[s]) P.fwd[at[P.row[s]]++] = s;
  }
  // by depth from the leaves of the column tree
  std::vector<int> depth(nt, 0);
  for (int k = 0; k < nt; ++k)
    for (int s = P.col_ptr[k] + 1; s < P.col_ptr[k + 1]; ++s) depth[P.row[s]] = std::max(depth[P.row[s]], depth[k] + 1);
  P.solve_order.resize(nt);
  std::iota(P.solve_order.begin(), P.solve_order.end(), 0);
  std::stable_sort(P.solve_order.begin(), P.solve_order.end(), [&](int a, int b) { return depth[a] < depth[b]; });
}

bool chol_symbolic(CholSymbolic& P, int nb, int bs, const std::vector<int>& brow, const std::vector<int>& bcol,
                   bool reorder, const std::vector<int32_t>* extra, long long max_tiles) {
  P = CholSymbolic();
  P.nb = nb;
  P.bs = bs;
  P.n = nb * bs;
  const int nnzb = (int)brow.size();
  // positions: the groups of the elimination order start on tile boundaries
  P.pos.assign(nb, 0);
  if (reorder) {
    std::vector<int> ptr(nb + 1, 0), adj;
    for (int k = 0; k < nnzb; ++k)
      if (brow[k] != bcol[k]) ++ptr[brow[k] + 1], ++ptr[bcol[k] + 1];
    for (int i = 0; i < nb; ++i) ptr[i + 1] += ptr[i];
    adj.resize(ptr[nb]);
    std::vector<int> at(ptr.begin(), ptr.end() - 1);
    for (int k = 0; k < nnzb; ++k)
      if (brow[k] != bcol[k]) {
        adj[at[brow[k]]++] = bcol[k];
        adj[at[bcol[k]]++] = brow[k];
      }
    Dissector D(ptr, adj, nb, std::max(1, kTile / bs));
    std::vector<int> all(nb);
    std::iota(all.begin(), all.end(), 0);
    D.components(all);
    int p = 0;
    for (auto& g : D.groups) {
      for (int v : g) {
        P.pos[v] = p;
        p += bs;
      }
      p = (p + kTile - 1) / kTile * kTile;
    }
    P.nt = p / kTile;
  } else {
    for (int i = 0; i < nb; ++i) P.pos[i] = i * bs;
    P.nt = (P.n + kTile - 1) / kTile;
  }
  const int nt = P.nt;
  P.orig.assign((size_t)nt * kTile, -1);
  for (int i = 0; i < nb; ++i)
    for (int a = 0; a < bs; ++a) P.orig[P.pos[i] + a] = i * bs + a;
  P.width.assign(nt, 0);
  for (int t = 0; t < nt; ++t)
    for (int a = 0; a < kTile; ++a)
      if (P.orig[(size_t)t * kTile + a] >= 0) P.width[t] = a + 1;
  // the first and the last tile that a block's unknowns are in
  struct Tiles {
    int first, last;
  };
  std::vector<Tiles> tiles(nb);
  for (int i = 0; i < nb; ++i) tiles[i] = Tiles{P.pos[i] / kTile, (P.pos[i] + bs - 1) / kTile};
  // pattern of the tiles below the diagonal, by column
  std::vector<std::vector<int>> col(nt);
  auto mark = [&](int r, int c) {
    const Tiles a = tiles[r], b = tiles[c];
    for (int ti = a.first; ti <= a.last; ++ti)
      for (int tj = b.first; tj <= b.last; ++tj)
        if (ti != tj) {
          std::vector<int>& l = col[std::min(ti, tj)];
          const int i = std::max(ti, tj);
          if (l.empty() || l.back() != i) l.push_back(i);
        }
  };
  for (int k = 0; k < nnzb; ++k) mark(brow[k], bcol[k]);
  if (extra)
    for (size_t k = 0; k < extra->size() / 2; ++k) mark((*extra)[2 * k], (*extra)[2 * k + 1]);
  if (!plan_slots(P, col, max_tiles)) return false;
  const int ns = P.col_ptr[nt];
  auto slot = [&](int i, int k) {
    if (i == k) return P.col_ptr[k];
    const auto b = P.row.begin() + P.col_ptr[k] + 1, e = P.row.begin() + P.col_ptr[k + 1];
    return (int)(std::lower_bound(b, e, i) - P.row.begin());
  };
  // assembly: a block's tiles in order; the blocks of a row follow one another,
  // so a tile's slot mostly is that of the last one in its tile column (a row
  // has at most two of those) or the next
  P.asm_ptr.assign(ns + 1, 0);
  struct Last {
    int i, j, slot;
  } lasts[2] = {{-1, -1, 0}, {-1, -1, 0}};
  auto each_entry = [&](auto&& f) {
    for (int k = 0; k < nnzb; ++k) {
      // the tile holds the block with the larger position as the row
      const bool tr = P.pos[brow[k]] < P.pos[bcol[k]];
      const Tiles a = tiles[tr ? bcol[k] : brow[k]], b = tiles[tr ? brow[k] : bcol[k]];
      for (int ti = a.first; ti <= a.last; ++ti)
        for (int tj = b.first; tj <= b.last; ++tj) {
          if (ti < tj) continue;
          Last& l = lasts[tj & 1];
          if (tj != l.j || ti != l.i) {
            const bool next = tj == l.j && l.slot + 1 < P.col_ptr[tj + 1] && P.row[l.slot + 1] == ti;
            l = Last{ti, tj, next ? l.slot + 1 : slot(ti, tj)};
          }
          f(l.slot, k);
        }
    }
  };
  each_entry([&](int s, int) { ++P.asm_ptr[s + 1]; });
  for (int s = 0; s < ns; ++s) P.asm_ptr[s + 1] += P.asm_ptr[s];
  P.asm_ent.resize(P.asm_ptr[ns]);
  std::vector<int> at(P.asm_ptr.begin(), P.asm_ptr.end() - 1);
  each_entry([&](int s, int k) { P.asm_ent[at[s]++] = k; });
  plan_lists(P);
  return true;
}

bool chol_dense_batch(CholSymbolic& P, const std::vector<int>& first, std::vector<int>& window,
                      std::vector<int>& index, long long max_tiles) {
  P = CholSymbolic();
  const int nw = (int)first.size() - 1;
  P.n = first[nw];
  std::vector<int> order(nw);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return first[a + 1] - first[a] > first[b + 1] - first[b]; });
  window.clear();
  index.clear();
  std::vector<std::vector<int>> col;
  for (int w : order) {
    const int n = first[w + 1] - first[w], t = (n + kTile - 1) / kTile, k0 = (int)col.size();
    for (int k = 0; k < t; ++k) {
      window.push_back(w);
      index.push_back(k);
      col.emplace_back();
      for (int i = k + 1; i < t; ++i) col.back().push_back(k0 + i);
      P.width.push_back(std::min(kTile, n - k * kTile));
      for (int a = 0; a < kTile; ++a) P.orig.push_back(k * kTile + a < n ? first[w] + k * kTile + a : -1);
    }
  }
  P.nt = (int)col.size();
  if (!plan_slots(P, col, max_tiles)) return false;
  P.asm_ptr.assign(P.row.size() + 1, 0);
  plan_lists(P);
  return true;
}

}  // namespace g2oc
