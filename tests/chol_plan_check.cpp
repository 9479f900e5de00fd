// Host-side check of the tiled Cholesky's plan (g2o_b200/csrc/chol_plan.cpp):
// chol_plan_check <kind> <blocks> <block size> <reorder> builds the plan of a
// pattern, checks it against its definition where it is small enough and prints
// "tile columns, stored tiles, tile products, longest chain".
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "chol_plan.h"

using namespace g2oc;

static int fail(const char* what) {
  std::printf("wrong: %s\n", what);
  return 1;
}

// blocks (row <= column), row by row
static std::vector<std::pair<int, int>> pattern(const std::string& kind, int nb) {
  std::vector<std::vector<int>> up(nb);
  unsigned seed = 12345u + nb;
  auto rnd = [&](int n) {
    seed = seed * 1664525u + 1013904223u;
    return (int)((seed >> 8) % (unsigned)n);
  };
  auto add = [&](int a, int b) {
    if (a != b) up[std::min(a, b)].push_back(std::max(a, b));
  };
  if (kind == "chain" || kind == "hubchain")
    for (int i = 1; i + 1 < nb; ++i) add(i, i + 1);
  if (kind == "star" || kind == "hubchain")
    for (int i = 1; i < nb; ++i) add(0, i);
  if (kind == "hubs")  // a chain, and each vertex next to one of 20 hubs
    for (int i = 20; i < nb; ++i) add(rnd(20), i), add(i, std::min(i + 1, nb - 1));
  if (kind == "starloops")  // random loops over a star
    for (int i = 1; i < nb; ++i) add(0, i), add(i, std::min(nb - 1, i + 1 + rnd(200)));
  if (kind == "random")
    for (int i = 0; i < 2 * nb; ++i) add(rnd(nb), rnd(nb));
  if (kind == "grid")
    for (int i = 0; i < nb; ++i) {
      if (i % 40 != 39 && i + 1 < nb) add(i, i + 1);
      if (i + 40 < nb) add(i, i + 40);
    }
  if (kind == "full")
    for (int i = 0; i < nb; ++i)
      for (int j = i + 1; j < nb; ++j) up[i].push_back(j);
  std::vector<std::pair<int, int>> out;
  for (int i = 0; i < nb; ++i) {
    std::sort(up[i].begin(), up[i].end());
    up[i].erase(std::unique(up[i].begin(), up[i].end()), up[i].end());
    out.push_back({i, i});
    for (int j : up[i]) out.push_back({i, j});
  }
  return out;
}

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  const int nb = std::atoi(argv[2]), bs = std::atoi(argv[3]);
  const bool reorder = std::atoi(argv[4]) != 0;
  std::vector<int> brow, bcol;
  for (auto& p : pattern(argv[1], nb)) brow.push_back(p.first), bcol.push_back(p.second);
  CholSymbolic P;
  if (!chol_symbolic(P, nb, bs, brow, bcol, reorder, nullptr)) {
    std::printf("refused\n");
    return 3;
  }
  const int nt = P.nt, ns = (int)P.row.size();
  // positions: every unknown once
  std::vector<char> seen((size_t)nb * bs, 0);
  for (int o : P.orig)
    if (o >= 0 && seen[o]++) return fail("position");
  if (std::count(seen.begin(), seen.end(), 1) != nb * bs) return fail("positions");
  // tasks: every stored tile once, after the ones it needs
  std::vector<int> at(ns, -1);
  for (size_t t = 0; t < P.task.size(); ++t) {
    const int s = P.task[t];
    if (s < 0 || s >= ns || at[s] >= 0) return fail("task");
    for (int u = P.upd_ptr[s]; u < P.upd_ptr[s + 1]; ++u)
      if (at[P.upd[2 * (size_t)u]] < 0 || at[P.upd[2 * (size_t)u + 1]] < 0) return fail("order of products");
    if (P.row[s] != P.col[s] && at[P.col_ptr[P.col[s]]] < 0) return fail("order of the diagonal tile");
    at[s] = (int)t;
  }
  if ((int)P.task.size() != ns) return fail("tasks");
  // products and assembly lists by their definition
  if (nt <= 120) {
    std::vector<int> slot((size_t)nt * nt, -1);
    for (int s = 0; s < ns; ++s) slot[(size_t)P.row[s] * nt + P.col[s]] = s;
    for (int s = 0; s < ns; ++s) {
      const int i = P.row[s], k = P.col[s];
      std::set<std::pair<int, int>> want, have;
      for (int j = 0; j < k; ++j)
        if (slot[(size_t)i * nt + j] >= 0 && slot[(size_t)k * nt + j] >= 0)
          want.insert({slot[(size_t)i * nt + j], slot[(size_t)k * nt + j]});
      for (int u = P.upd_ptr[s]; u < P.upd_ptr[s + 1]; ++u)
        have.insert({P.upd[2 * (size_t)u], P.upd[2 * (size_t)u + 1]});
      if (want != have || (int)have.size() != P.upd_ptr[s + 1] - P.upd_ptr[s]) return fail("products");
    }
    for (int i = 0; i < nt; ++i)  // fill
      for (int k = 0; k < i; ++k)
        for (int j = 0; j < k; ++j)
          if (slot[(size_t)i * nt + j] >= 0 && slot[(size_t)k * nt + j] >= 0 && slot[(size_t)i * nt + k] < 0)
            return fail("fill");
    std::vector<std::vector<int>> where(brow.size());
    for (int s = 0; s < ns; ++s)
      for (int e = P.asm_ptr[s]; e < P.asm_ptr[s + 1]; ++e) {
        const int k = P.asm_ent[e];
        if (k < 0 || k >= (int)brow.size()) return fail("assembly entry");
        where[k].push_back(s);
      }
    for (size_t k = 0; k < brow.size(); ++k) {
      const int a = P.pos[brow[k]], b = P.pos[bcol[k]];
      std::set<int> want;
      for (int x = 0; x < bs; ++x)
        for (int y = 0; y < bs; ++y) {
          const int i = std::max(a + x, b + y) / kTile, j = std::min(a + x, b + y) / kTile;
          want.insert(slot[(size_t)i * nt + j]);
        }
      if (std::set<int>(where[k].begin(), where[k].end()) != want || where[k].size() != want.size())
        return fail("assembly list");
    }
  }
  std::vector<int> depth(nt, 1);
  int chain = 0;
  for (int k = 0; k < nt; ++k) {
    chain = std::max(chain, depth[k]);
    for (int s = P.col_ptr[k] + 1; s < P.col_ptr[k + 1]; ++s) depth[P.row[s]] = std::max(depth[P.row[s]], depth[k] + 1);
  }
  std::printf("%d %d %zu %d\n", nt, ns, P.upd.size() / 2, chain);
  return 0;
}
