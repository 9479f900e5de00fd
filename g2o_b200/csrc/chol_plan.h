// chol_plan.h -- host-side plan of the tiled sparse Cholesky (cholesky.cuh):
// elimination order, tile-level symbolic factorization, the assembly and
// update lists of every stored tile and the order in which the tiles are
// computed. Pure host code: no CUDA types.
#pragma once

#include <cstdint>
#include <vector>

namespace g2oc {

constexpr int kTile = 64;  // scalar rows and columns of a tile

struct CholSymbolic {
  int nb = 0, bs = 0, n = 0;
  int nt = 0;                // tile columns; positions 0 .. nt * kTile - 1, some of them padding
  std::vector<int> pos;      // per block: position of its first unknown (the others follow)
  std::vector<int> orig;     // per position: the unknown there, or -1 (padding: identity)
  std::vector<int> width;    // per tile column: positions up to its last unknown
  // stored tiles of L ("slots"), column by column, the diagonal tile first,
  // then the rows below it ascending
  std::vector<int> col_ptr;  // nt + 1
  std::vector<int> row;      // per slot: tile row
  std::vector<int> col;      // per slot: tile column
  // blocks of the matrix (of the row-ordered list) in each slot; one that
  // straddles tiles is in several
  std::vector<int> asm_ptr;  // slots + 1
  std::vector<int> asm_ent;
  // updates of each slot (i, k): the slots (i, j), (k, j) of every earlier
  // column j that has both, the ones expected to be finished first in front
  std::vector<int> upd_ptr;  // slots + 1
  std::vector<int> upd;      // 2 per entry
  std::vector<int> task;     // the slots in the order in which they are handed out
  // substitutions: tile columns by the order of the forward pass; backward
  // takes them in reverse. fwd lists: per tile row i its slots (i, j), j < i
  std::vector<int> solve_order;
  std::vector<int> fwd_ptr, fwd;  // per tile row: slots left of the diagonal, columns ascending
};

// rc: (row, col) pairs of the upper blocks, row-ordered list index = position
// in brow / bcol; extra: further block pairs the pattern has to hold.
// reorder: nested dissection, else the given order. False, before any list is
// made, where the factor has more than max_tiles tiles or more tile products
// than an int counts (dense, 150,000 unknowns).
bool chol_symbolic(CholSymbolic& P, int nb, int bs, const std::vector<int>& brow, const std::vector<int>& bcol,
                   bool reorder, const std::vector<int32_t>* extra, long long max_tiles = 1ll << 31);

// The plan of a batch of dense matrices: matrix w has the unknowns first[w] ..
// first[w + 1] - 1. The largest come first, so that their chains start first.
// window, index: per tile column its matrix and its place in it. No assembly
// lists: the tiles are read from the matrices. The order of a matrix's sums
// does not depend on the others.
bool chol_dense_batch(CholSymbolic& P, const std::vector<int>& first, std::vector<int>& window,
                      std::vector<int>& index, long long max_tiles = 1ll << 31);

}  // namespace g2oc
