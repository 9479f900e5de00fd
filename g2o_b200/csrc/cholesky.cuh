// cholesky.cuh -- LinearSolverCudaCholesky: FP64 tiled Cholesky of the
// (reduced) block system, the role of LinearSolverEigen's SimplicialLLT and
// LinearSolverDense's LDLT (g2o/solvers/eigen/linear_solver_eigen.h:94-191,
// g2o/solvers/dense/linear_solver_dense.h:57-105).
//
// Plan (once per pattern, on the host, chol_plan.cpp): nested-dissection
// order for sparse systems (the given order for the reduced camera systems),
// the symbolic factorization at the level of 64 x 64 tiles and, per stored
// tile, the blocks it is assembled from and the tile products it takes.
// Numeric (every solve, on the device): one launch computes every tile of L
// (chol_factor_dag), handing the tiles out in an order in which each only
// needs tiles handed out before it; a second one substitutes backward. A
// pivot that is zero to working precision, or a direction that is (see
// kRankTol), sets the info flag (G2OC_ERR_NOT_PD at the boundary); nothing
// traps.
#pragma once

#include <algorithm>
#include <climits>
#include <exception>
#include <vector>

#include "chol_plan.h"
#include "g2oc_internal.h"
#include "pcg_kernels.cuh"
#include "reduce.cuh"
#include "tile_potrf.cuh"

namespace g2oc {

constexpr int kTileElems = kTile * kTile;
constexpr int kTileBuf = kTile * kLd;  // doubles per tile in shared memory
// polls of one wait before a CTA gives up and the call returns
// G2OC_ERR_TIMEOUT (each poll is an L2 round trip: a few seconds in all; the
// longest legitimate wait is the factorization itself)
constexpr unsigned kCholSpinLimit = 1u << 22;

// Hand-out state of one kind of launch: tickets of the current launch, CTAs
// that have left it, and the count of finished launches. A tile is ready when
// its flag holds the current launch's number, so no flag is ever cleared; the
// last CTA to leave resets the ticket and advances the number, so a launch
// replayed from a graph starts like any other.
struct CholTickets {
  unsigned next, left, epoch, pad;
};

// Rank of a matrix in a dissected order. A pivot there is what its unknown
// has left when all others are known only through the separators above it:
// for a pose in the middle of 40,000 it is 7e-11 of the largest diagonal entry
// in a definite system, while the pivot of a part that may turn about its
// hinge, zero but for rounding, is 1e-11 of it already at 10,000 poses. The
// pivot's size does not tell them apart; its direction does. With u = L^-T e_k
// (u'Au = 1), 1 / sum_i a_ii u_i^2 is the pivot's share of what rounding the
// entries of A can change: at most 2 eps for systems with a free direction (2D
// graphs of 4 to 20,000 poses: chains, grids, cliques, random loops, a hub),
// at least 788 eps for definite ones (the least for a straight corridor of
// 10,000 odometry edges). Pivots that kept less than kSuspect of their diagonal
// entry are looked at together, u = L^-T (ones at them): the sum's inverse is
// then no larger than the smallest share. The system is refused when it is
// below kRankTol. u rides along in the backward pass, and only if a pivot is
// suspect: none is in a graph of some thousand poses; 20,000 odometry edges
// without a closure pay 6% of a solve (520 to 550 us).
constexpr double kSuspect = 1e-6, kRankTol = 4 * 2.220446049250313e-16;

struct CholState {
  CholTickets factor, forward, backward;
  int info;  // a pivot was not positive
  int err;   // a wait ran out
  int suspect, pad;  // a pivot is small beside its diagonal entry (kSuspect)
  unsigned long long max_diag;  // bits of the largest |diagonal entry| (chol_floor), back to 0 after a factorization
};

// device side of the plan
struct CholDev {
  int n, nt, ns, ntask;  // unknowns, tile columns, slots, tasks of the factorization
  const int *col_ptr, *row, *col, *width, *orig;
  const int* asm_ptr;
  const int4* asm_ent;  // offset (low, high) and stride of the block's entries, packed place
  const int* upd_ptr;
  const int2* upd;
  const int *task, *solve_order, *fwd_ptr, *fwd;
  double *L, *W;   // tiles row-major, kTileElems each: per slot, per tile column (W(k) = L(k,k)^-1)
  double *y, *x;   // nt * kTile: forward and backward substituted vectors
  bool dissected;  // the rank is decided by kRankTol, with the vectors below
  double *adiag, *suspect, *u;  // nt * kTile: diagonal of the matrix, ones at the suspect pivots, L^-T of those
  double* uu;      // per tile column its part of sum_i a_ii u_i^2
  unsigned *flag, *yflag, *xflag;
  CholState* st;
};

// int arrays of a plan, laid end to end (16-byte aligned) so that a plan is
// one device allocation and one copy
struct CholInts {
  std::vector<int> v;
  size_t add(const int* p, size_t n) {
    const size_t at = v.size();
    v.insert(v.end(), p, p + n);
    v.resize((v.size() + 3) & ~(size_t)3);
    return at;
  }
  size_t add(const std::vector<int>& a) { return add(a.data(), a.size()); }
};

struct CholPlan {
  CholSymbolic S;
  DBuf<int> ints;
  DBuf<int4> places;
  DBuf<double> vals;    // L, W, y, x
  DBuf<unsigned> flags;
  DBuf<CholState> state;
  CholDev d{};
  bool smem_raised = false;  // the kernels may use their shared memory
  const int *pos = nullptr, *asm_ent = nullptr;  // device copies of S.pos and S.asm_ent
  int sms = 0;
  // the selected inverse: its lists (device; made on first use) and tiles
  DBuf<int> inv_ints;
  DBuf<unsigned> inv_flag;
  DBuf<double> inv_sigma;
  size_t inv_at[3] = {0, 0, 0};
  // the bounded-wait tests: flags are compared with a number that is never
  // reached, in every launch, in the next factorization and solve alone, or in
  // the solves with a kept factor
  unsigned extra = 0, extra_once = 0, extra_kept = 0;
  const CholDev& dev() const { return d; }
};

// The symbolic part of a plan by make(max_tiles), which says whether the plan
// may be: no more tiles than fit on the device, so that what cannot be solved
// costs no lists (up to 32,768 unknowns they are few, and the device is not
// asked). No exception leaves it (its callers are C entries).
template <typename F>
static int chol_plan_symbolic(long long n, F&& make) {
  size_t free_bytes = 0, total = (size_t)1 << 60;
  if (n > 32768) G2OC_CUDA_TRY(cudaMemGetInfo(&free_bytes, &total));
  try {
    if (make((long long)(total / (kTileElems * sizeof(double))))) return G2OC_OK;
    set_error("cholesky: the factor does not fit on the device, or has more than %d tile products", INT_MAX);
  } catch (const std::exception& e) {
    set_error("cholesky plan: %s", e.what());
  }
  return G2OC_ERR_NOT_SUPPORTED;
}

// device arrays of the plan whose symbolic part is made
static int chol_plan_alloc(CholPlan& P, bool dissected, cudaStream_t st) {
  CholSymbolic& S = P.S;
  const size_t ns = S.row.size(), nt = (size_t)S.nt;
  CholInts I;
  I.v.reserve(S.asm_ent.size() + S.upd.size() + 8 * (ns + nt) + nt * kTile + S.pos.size() + 64);
  const size_t o[] = {I.add(S.col_ptr), I.add(S.row), I.add(S.col), I.add(S.width), I.add(S.orig), I.add(S.asm_ptr),
                      I.add(S.asm_ent), I.add(S.upd_ptr), I.add(S.upd), I.add(S.task), I.add(S.solve_order),
                      I.add(S.fwd_ptr), I.add(S.fwd), I.add(S.pos)};
  std::vector<int>().swap(S.asm_ent);
  std::vector<int>().swap(S.upd);
  I.v.resize(I.v.size() + 4, 0);
  G2OC_TRY(P.ints.upload(I.v, st));
  G2OC_TRY(P.places.alloc(S.asm_ptr.back()));
  const size_t vec = nt * kTile;
  G2OC_TRY(P.vals.alloc((ns + nt) * kTileElems + 5 * vec + nt));
  G2OC_TRY(P.flags.alloc(ns + 2 * nt));
  G2OC_TRY(P.state.alloc(1));
  G2OC_CUDA_TRY(cudaMemsetAsync(P.vals.p, 0, P.vals.bytes(), st));  // the parts without unknowns stay zero
  G2OC_CUDA_TRY(cudaMemsetAsync(P.flags.p, 0, P.flags.bytes(), st));
  G2OC_CUDA_TRY(cudaMemsetAsync(P.state.p, 0, P.state.bytes(), st));
  const int* q = P.ints.p;
  double* L = P.vals.p;
  double* W = L + ns * kTileElems;
  double* y = W + nt * kTileElems;
  P.d = CholDev{S.n, S.nt, (int)ns, (int)S.task.size(), q + o[0], q + o[1], q + o[2], q + o[3], q + o[4], q + o[5],
                P.places.p, q + o[7], reinterpret_cast<const int2*>(q + o[8]), q + o[9],
                q + o[10], q + o[11], q + o[12], L, W, y, y + vec, dissected, y + 2 * vec, y + 3 * vec, y + 4 * vec, y + 5 * vec,
                P.flags.p, P.flags.p + ns, P.flags.p + ns + nt, P.state.p};
  P.pos = q + o[13];
  P.asm_ent = q + o[6];
  int dev = 0;
  G2OC_CUDA_TRY(cudaGetDevice(&dev));
  G2OC_CUDA_TRY(cudaDeviceGetAttribute(&P.sms, cudaDevAttrMultiProcessorCount, dev));
  G2OC_CUDA_TRY(cudaStreamSynchronize(st));  // the copied host array goes out of scope
  return G2OC_OK;
}

// Where the entries of a slot's blocks are (values of block p of row r at
// rptr[r] bs^2 + e nblk + (p - rptr[r])) and where they go: the row and column
// of the block's first entry in the tile, negative or beyond the tile for a
// block that straddles tiles. One CTA per slot, once per plan: the list of
// blocks is a quarter of it, which is what the host makes and sends.
static __global__ void chol_places(CholDev P, const int* asm_ent, const int* brow, const int* rcol, const int* rptr,
                                   const int* pos, int bs, int4* places) {
  const int s = blockIdx.x, i0 = P.row[s] * kTile, j0 = P.col[s] * kTile;
  for (int q = P.asm_ptr[s] + threadIdx.x; q < P.asm_ptr[s + 1]; q += blockDim.x) {
    const int k = asm_ent[q], r = brow[k], c = rcol[k], rb = rptr[r];
    const bool tr = pos[r] < pos[c];  // the tile holds it with the larger position as the row
    const long long off = (long long)rb * bs * bs + (k - rb);
    const int i = pos[tr ? c : r] - i0 + kTile, j = pos[tr ? r : c] - j0 + kTile;
    places[q] = make_int4((int)(off & 0xffffffffll), (int)(off >> 32), rptr[r + 1] - rb, i | (j << 8) | ((tr ? 1 : 0) << 16));
  }
}

// brow, bcol: the blocks of the matrix, row by row, and d_brow, d_rcol, d_rptr
// its lists on the device (SysDev); extra: further (row, col) block pairs whose
// entries the plan must hold (the blocks a selected inverse is asked for),
// treated as structural nonzeros of the matrix so that the symbolic fill covers
// them
static int chol_plan_build(CholPlan& P, int nb, int bs, const std::vector<int>& brow, const std::vector<int>& bcol,
                           const int* d_brow, const int* d_rcol, const int* d_rptr, bool reorder, cudaStream_t st,
                           const std::vector<int32_t>* extra = nullptr) {
  G2OC_TRY(chol_plan_symbolic((long long)nb * bs, [&](long long max_tiles) {
    return chol_symbolic(P.S, nb, bs, brow, bcol, reorder, extra, max_tiles);
  }));
  G2OC_TRY(chol_plan_alloc(P, reorder, st));
  chol_places<<<P.d.ns, 128, 0, st>>>(P.dev(), P.asm_ent, d_brow, d_rcol, d_rptr, P.pos, bs, P.places.p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("cholesky plan launch: %s", cudaGetErrorString(e));
    return G2OC_ERR_CUDA;
  }
  return G2OC_OK;
}

// asynchronous 16-byte global -> shared copies past L1 (tiles written by
// other CTAs of the same launch)
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ unsigned chol_load_flag(const unsigned* f) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
  return v;
}
__device__ __forceinline__ void chol_store_flag(unsigned* f, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(f), "r"(v) : "memory");
}

// wait of one thread for a tile's flag; false when the wait ran out here or
// elsewhere
__device__ __forceinline__ bool chol_wait(const unsigned* f, unsigned want, int* err) {
  for (unsigned spins = 0; chol_load_flag(f) != want; ++spins) {
    if ((spins & 255u) == 255u && *(volatile int*)err) return false;
    if (spins >= kCholSpinLimit) {
      atomicExch(err, 1);
      return false;
    }
  }
  return true;
}

// next ticket for the CTA (a barrier on both sides)
__device__ __forceinline__ int chol_ticket(CholTickets* t, int* sh) {
  __syncthreads();
  if (threadIdx.x == 0) *sh = (int)atomicAdd(&t->next, 1u);
  __syncthreads();
  return *sh;
}
// the last CTA to leave also runs `end`, with all its threads
template <typename F>
__device__ __forceinline__ void chol_leave(CholTickets* t, F&& end) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicInc(&t->left, gridDim.x - 1) == gridDim.x - 1;  // left is back at 0 then
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  if (threadIdx.x == 0) {
    t->next = 0;
    t->epoch += 1;
  }
  end();
}

// The largest |diagonal entry| of the matrix (the pivot floor is a multiple
// of it) and the outcome of the last factorization cleared: one thread per
// diagonal entry, a maximum has no order. m: this thread's entry
__device__ __forceinline__ void chol_floor_max(double m, CholState* st) {
  __shared__ double red[32];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->info = 0;
    st->err = 0;
    st->suspect = 0;
  }
  block_max(m, red);
  if (threadIdx.x == 0 && red[0] > 0.0) atomicMax(&st->max_diag, (unsigned long long)__double_as_longlong(red[0]));
}

template <typename Real>
__global__ void chol_floor(SysDev<Real> S, int bs, CholState* st) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0.0;
  if (t < S.nb * bs) {
    const int i = t / bs, a = t % bs;
    const int rb = S.rptr[i], nblk = S.rptr[i + 1] - rb;
    m = fabs((double)S.val[(size_t)rb * bs * bs + (size_t)a * (bs + 1) * nblk + (S.diag[i] - rb)]);
  }
  chol_floor_max(m, st);
}

// sys_gather_damped and chol_floor in one pass: the damped pose-graph system
// and its largest diagonal entry
template <typename Real, int BS>
__global__ void chol_gather_damped(const Real* src, const int* perm, const int* brow, const int* rptr,
                                   const int* rcol, int nnzb, double lambda, Real* dst, CholState* st) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0.0;
  if (t < (long long)nnzb * BS * BS) {
    const int k = (int)(t / (BS * BS)), e = (int)(t % (BS * BS));
    const int r = brow[k], rb = rptr[r], nblk = rptr[r + 1] - rb;
    double v = (double)src[(size_t)perm[k] * BS * BS + e];
    const bool diag = rcol[k] == r && e % (BS + 1) == 0;
    if (diag) v += lambda;
    const Real d = (Real)v;
    dst[sys_offset<BS>(rb, nblk, k - rb, e)] = d;
    if (diag) m = fabs((double)d);
  }
  chol_floor_max(m, st);
}

// Products of tiles in 16 x 16 blocks: only the blocks of the tiles' leading
// parts that hold unknowns are formed (the groups of a dissection seldom fill
// their last tile), of a symmetric product only the lower ones. Block b of
// the nblk blocks goes to warp b % 8; a warp's (at most two) blocks are in
// acc[b / 8], as 2 x 2 fragments of 8 x 8.
struct CholBlocks {
  int mb, n;   // block rows, blocks
  bool lower;  // only bi >= bj
  __device__ __forceinline__ CholBlocks(int rows, int cols, bool low) : mb((rows + 15) >> 4), lower(low) {
    const int nb = (cols + 15) >> 4;
    n = low ? mb * (mb + 1) / 2 : mb * nb;
  }
  __device__ __forceinline__ bool at(int q, int& bi, int& bj) const {
    int b = (threadIdx.x >> 5) + 8 * q;
    if (b >= n) return false;
    if (lower) {
      bj = 0;
      while (b >= mb - bj) b -= mb - bj++;
      bi = bj + b;
    } else {
      bj = b / mb;
      bi = b - bj * mb;
    }
    return true;
  }
};
using CholAcc = double[2][2][2][2];  // [block][fragment row][fragment column][element]

// acc += X Y^T over k < K (a multiple of 4); X(i, k) at X[i * kLd + k] or, with
// XK, at X[k * kLd + i], likewise Y. TRI: Y(j, k) is zero for k > j.
template <bool XK, bool YK, bool TRI = false>
__device__ __forceinline__ void chol_mma(const CholBlocks& B, const double* X, const double* Y, int K, CholAcc& acc) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    int bi, bj;
    if (!B.at(q, bi, bj)) continue;
    const double* x = XK ? X + t * kLd + 16 * bi + g : X + (16 * bi + g) * kLd + t;
    const double* y = YK ? Y + t * kLd + 16 * bj + g : Y + (16 * bj + g) * kLd + t;
    const int k1 = TRI ? min(K, 16 * bj + 16) : K;
#pragma unroll 4
    for (int k0 = 0; k0 < k1; k0 += 4) {
      const int kx = XK ? k0 * kLd : k0, ky = YK ? k0 * kLd : k0;
      double fa[2], fb[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        fa[u] = x[kx + (XK ? 8 * u : 8 * u * kLd)];
        fb[u] = y[ky + (YK ? 8 * u : 8 * u * kLd)];
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v)
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                       : "+d"(acc[q][u][v][0]), "+d"(acc[q][u][v][1])
                       : "d"(fa[u]), "d"(fb[v]));
    }
  }
}

// f(row, column, the two accumulators of row and column, column + 1)
template <typename F>
__device__ __forceinline__ void chol_each_frag(const CholBlocks& B, CholAcc& acc, F&& f) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    int bi, bj;
    if (!B.at(q, bi, bj)) continue;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) f(16 * bi + 8 * u + g, 16 * bj + 8 * v + 2 * t, acc[q][u][v]);
  }
}
__device__ __forceinline__ void chol_clear(CholAcc& acc) {
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) acc[q][u][v][0] = acc[q][u][v][1] = 0.0;
}

// the leading rows x cols (rounded up to 16, and to 16, 32 or 64) of a tile of
// global memory (row-major) into shared memory
__device__ __forceinline__ void chol_load_tile(const double* src, double* dst, int rows, int cols) {
  const int sh = cols <= 16 ? 3 : cols <= 32 ? 4 : 5;  // 16-byte pieces per row
  const int n = ((rows + 15) & ~15) << sh;
  for (int i = threadIdx.x; i < n; i += 256) {
    const int r = i >> sh, c = 2 * (i & ((1 << sh) - 1));
    cp_async16(dst + r * kLd + c, src + r * kTile + c);
  }
}
__device__ __forceinline__ void chol_load_tile(const double* src, double* dst) { chol_load_tile(src, dst, kTile, kTile); }

// shared memory of chol_factor_dag: three stages of two operand tiles, a
// vector per stage and the right-hand side
constexpr int kFactorStages = 3;
constexpr int kFactorSmem = kFactorStages * (2 * kTileBuf + kTile) * (int)sizeof(double) + kTile * (int)sizeof(double);

// How many of the products from u on (at most 16, in list order) have both
// operand tiles ready: one round trip for all of them. One warp.
__device__ __forceinline__ int chol_ready(const CholDev& P, const int2* upd, int u, int nu, unsigned want) {
  const int lane = threadIdx.x & 31, q = u + (lane >> 1);
  bool ok = false;
  if (q < nu) {
    const int2 ab = upd[q];
    ok = chol_load_flag(P.flag + ((lane & 1) ? ab.y : ab.x)) == want;
  }
  const unsigned m = __ballot_sync(0xffffffffu, ok), missing = ~(m & (m >> 1)) & 0x55555555u;
  return missing ? (__ffs(missing) - 1) >> 1 : 16;
}

// The blocks of a slot into a tile of shared memory (256 threads; identity on
// the padding of a diagonal tile); a barrier is needed before and after.
template <typename Real>
__device__ __forceinline__ void chol_assemble(const SysDev<Real>& S, int bs, const CholDev& P, int s, double* As) {
  const int k = P.col[s];
  const bool diag = P.row[s] == k;
  for (int e = threadIdx.x; e < kTileElems; e += 256) {
    const int r = e >> 6, c = e & 63;
    As[r * kLd + c] = diag && r == c && P.orig[(size_t)k * kTile + r] < 0 ? 1.0 : 0.0;
  }
  __syncthreads();
  const int bs2 = bs * bs, e0 = P.asm_ptr[s], ne = (P.asm_ptr[s + 1] - e0) * bs2;
  for (int q = threadIdx.x; q < ne; q += 256) {
    const int b = q / bs2, e = q - b * bs2;
    const int4 en = P.asm_ent[e0 + b];
    const size_t off = ((size_t)(unsigned)en.x | ((size_t)(unsigned)en.y << 32)) + (size_t)e * en.z;
    const int bi = e / bs, bj = e - bi * bs;
    const bool tr = (en.w >> 16) != 0;
    const int r = (en.w & 255) - kTile + (tr ? bj : bi), c = ((en.w >> 8) & 255) - kTile + (tr ? bi : bj);
    if ((unsigned)r < (unsigned)kTile && (unsigned)c < (unsigned)kTile) As[r * kLd + c] = (double)S.val[off];
  }
}

// fragments <- -tile and tile <- -fragments
__device__ __forceinline__ void chol_frags_from(const CholBlocks& B, const double* T, CholAcc& acc) {
  chol_each_frag(B, acc, [&](int r, int c, double (&a)[2]) {
    a[0] = -T[r * kLd + c];
    a[1] = -T[r * kLd + c + 1];
  });
}
__device__ __forceinline__ void chol_frags_to(const CholBlocks& B, double* T, CholAcc& acc) {
  chol_each_frag(B, acc, [&](int r, int c, double (&a)[2]) {
    T[r * kLd + c] = -a[0];
    T[r * kLd + c + 1] = -a[1];
  });
}

// What chol_factor_dag factors: a block-sparse matrix (the tiles' entries by
// the plan's assembly lists). A source has
//   scale    the magnitude that the pivot floor is relative to (0: any
//            positive pivot passes)
//   skip     whether the tile column k is left out of this launch
//   begin    called by thread 0 before the first pivot of a tile column
//   info     where a pivot that is too small is noted
//   ranked   whether the rank is decided by kRankTol
template <typename Real>
struct CholSystem {
  SysDev<Real> S;
  int bs;
  __device__ __forceinline__ double scale(const CholDev& P) const {
    return __longlong_as_double((long long)P.st->max_diag);
  }
  __device__ __forceinline__ bool skip(const CholDev&, int) const { return false; }
  __device__ __forceinline__ void begin(const CholDev&, int) const {}
  __device__ __forceinline__ int* info(const CholDev& P, int) const { return &P.st->info; }
  __device__ __forceinline__ bool ranked(const CholDev& P) const { return P.dissected; }
  __device__ __forceinline__ void assemble(const CholDev& P, int s, double* As) const {
    chol_assemble(S, bs, P, s, As);
  }
};

// The whole factorization, one persistent CTA of 256 threads per SM. Tiles
// are handed out by ticket in the plan's order (estimated start times, always
// after every tile they need), so a wait is for a tile that some CTA is
// already working on: no grid barrier, and no assumption on how many CTAs
// run. Per tile (i, k): assemble A(i, k) from its blocks, subtract
// L(i, j) L(k, j)^T for the plan's list of columns j as their tiles become
// ready (the next product's operands are fetched while one runs), then factor
// (i == k: L and W = L^-1 in shared memory, W kept) or multiply by W(k)^T.
// The forward substitution rides along: the diagonal task has every L(k, j)
// in shared memory and forms y(k) = W(k) (rhs(k) - sum_j L(k, j) y(j)).
// The sums' orders are the plan's: results do not depend on the timing.
//
// Bound by the chain of tiles from the leaves to the root of the elimination
// tree, not by memory or FLOPs: a 3,500-pose 2D graph has 1,200 tiles of 32 KB
// and 1,600 products, which 148 SMs pass in some 20 us, but a chain of 11
// diagonal tiles. What counts is the time of a tile of that chain: the
// diagonal factorization (tile_potrf_inv64) and the hand-over through L2.
// A task near the root has up to 40 products in its list, nearly all of them
// long ready when it starts: the flags of 16 products are read in one round
// trip and the operands of two are on their way while one is multiplied.
// Measured per solve, factorization and both substitutions: a 3,500-pose 2D
// graph (n = 10,497, 11 levels) 0.20 ms, against 10.1 ms for a reverse
// Cuthill-McKee band (165 strictly sequential tile steps in one CTA); a
// 2,500-pose 3D graph (n = 14,994) 0.27 ms, against 19.7 ms. With one flag
// per round trip, one product's operands ahead and whole 64 x 64 products
// they took 0.27 and 0.34 ms. Computing the tile below the diagonal in the
// diagonal's task (W(k) then need not travel) gained 4% where that task had
// few products and lost 15% where it had many.
template <typename Source>
__global__ void __launch_bounds__(256, 1) chol_factor_dag(Source A, CholDev P, const double* rhs, unsigned extra) {
  extern __shared__ __align__(16) double sm_chol[];
  __shared__ int sh_ticket, sh_ready;
  // stage q: operand tiles at 2 q and 2 q + 1
  auto buf = [&](int q) { return sm_chol + q * kTileBuf; };
  double* yb = sm_chol + 2 * kFactorStages * kTileBuf;
  double* vb = yb + kFactorStages * kTile;
  const int tid = threadIdx.x;
  const unsigned want = P.st->factor.epoch + 1;  // the flag value of this launch
  const unsigned wait_for = want + extra;
  const double scale = A.scale(P);
  int* err = &P.st->err;
  for (;;) {
    const int tk = chol_ticket(&P.st->factor, &sh_ticket);
    if (tk >= P.ntask) break;
    const int s = P.task[tk];
    const int k = P.col[s];
    const bool diag = P.row[s] == k;
    if (A.skip(P, k)) {
      if (tid == 0) chol_store_flag(P.flag + s, want);
      continue;
    }
    const int wk = P.width[k], wi = P.width[P.row[s]];
    const CholBlocks B(wi, wk, diag);
    CholAcc acc;
    chol_clear(acc);
    const int2* upd = P.upd + P.upd_ptr[s];
    const int nu = P.upd_ptr[s + 1] - P.upd_ptr[s];
    if (tid < 32) {
      const int n = chol_ready(P, upd, 0, nu, wait_for);
      if (tid == 0) sh_ready = n;
    }
    A.assemble(P, s, buf(0));
    if (diag && tid == 0) A.begin(P, k);
    if (diag && tid < kTile) {
      const int o = rhs ? P.orig[(size_t)k * kTile + tid] : -1;
      vb[tid] = o >= 0 ? rhs[o] : 0.0;
    }
    __syncthreads();
    const double akk = diag && tid < kTile ? buf(0)[tid * (kLd + 1)] : 0.0;
    int ready = sh_ready;  // products below are known to have their operands
    chol_frags_from(B, buf(0), acc);
    __syncthreads();
    // updates L(i, j) L(k, j)^T: the operands of the next two are fetched while
    // one is multiplied, as far as they are known to be ready
    double ysum = 0.0;
    auto issue = [&](int u) {
      const int2 ab = upd[u];
      const int q = u % kFactorStages, K = P.width[P.col[ab.x]];
      chol_load_tile(P.L + (size_t)ab.x * kTileElems, buf(2 * q), wi, K);
      if (!diag) chol_load_tile(P.L + (size_t)ab.y * kTileElems, buf(2 * q + 1), wk, K);
      if (diag && tid < kTile / 2)
        cp_async16(yb + q * kTile + 2 * tid, P.y + (size_t)P.col[ab.x] * kTile + 2 * tid);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int issued = 0, terms = wk;  // terms: a bound on the entries of L in a row of the tile
    bool ok = true;
    for (int u = 0; u < nu; ++u) {
      if (u >= ready) {
        __syncthreads();  // sh_ready has been read
        if (tid < 32) {
          int n = 0;
          unsigned spins = 0;
          while ((n = chol_ready(P, upd, u, nu, wait_for)) == 0) {
            if ((spins & 255u) == 255u && __any_sync(0xffffffffu, *(volatile int*)err != 0)) break;
            if (spins++ >= kCholSpinLimit) {
              if (tid == 0) atomicExch(err, 1);
              break;
            }
          }
          if (tid == 0) sh_ready = u + n;
        }
        __syncthreads();
        ready = sh_ready;
        ok = ready > u;
        if (!ok) break;
      }
      if (issued <= u) {
        issue(u);
        issued = u + 1;
      }
      if (issued - u == 1) asm volatile("cp.async.wait_group 0;" ::: "memory");
      else asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      while (issued < nu && issued < ready && issued < u + kFactorStages) issue(issued++);
      const int2 ab = upd[u];
      const int q = u % kFactorStages;
      const double *X = buf(2 * q), *Y = diag ? X : buf(2 * q + 1);
      const int wj = P.width[P.col[ab.x]], K = (wj + 3) & ~3;
      terms += wj;
      chol_mma<false, false>(B, X, Y, K, acc);
      if (diag) {
        const int r = tid >> 2;
        const double* yv = yb + q * kTile;
        if (r < wk)
          for (int c = tid & 3; c < K; c += 4) ysum += X[r * kLd + c] * yv[c];
      }
    }
    if (!ok) break;
    __syncthreads();
    double *T = buf(0), *Ws = buf(1);  // the tile after its updates; W(k)
    chol_frags_to(B, T, acc);
    if (diag) {
      ysum += __shfl_xor_sync(0xffffffffu, ysum, 1);
      ysum += __shfl_xor_sync(0xffffffffu, ysum, 2);
      if ((tid & 3) == 0) vb[tid >> 2] -= ysum;
      // what does not exceed the rounding of the sums that a pivot is made of
      // is taken for zero: n terms in the given order; in a dissected one the
      // terms of the tile's rows, and the rank is decided by kRankTol (n in
      // their place refuses definite systems whose root is weakly tied to the
      // fixed vertices)
      const bool ranked = A.ranked(P);
      const double floor = 4.0 * (ranked ? terms : P.n) * 2.220446049250313e-16 * scale;
      tile_potrf_inv64(T, Ws, buf(2), wk, floor, A.info(P, k));
      if (ranked && tid < kTile) {
        const double w = Ws[tid * (kLd + 1)];  // 1 / sqrt(pivot)
        const bool small = kSuspect * akk * w * w >= 1.0;
        P.adiag[(size_t)k * kTile + tid] = akk;
        P.suspect[(size_t)k * kTile + tid] = small ? 1.0 : 0.0;
        if (small) P.st->suspect = 1;
      }
      double* Wg = P.W + (size_t)k * kTileElems;
#pragma unroll
      for (int q = 0; q < kTileElems / 2 / 256; ++q) {
        const int e = 2 * (tid + 256 * q);
        *reinterpret_cast<double2*>(Wg + e) = *reinterpret_cast<const double2*>(Ws + (e >> 6) * kLd + (e & 63));
      }
      const int r = tid >> 2, q = tid & 3;
      double yv = 0.0;
#pragma unroll
      for (int c = 0; c < 16; ++c) yv += Ws[r * kLd + 4 * c + q] * vb[4 * c + q];
      yv += __shfl_xor_sync(0xffffffffu, yv, 1);
      yv += __shfl_xor_sync(0xffffffffu, yv, 2);
      if (q == 0) P.y[(size_t)k * kTile + r] = yv;
    } else {
      if (tid == 0) sh_ready = chol_wait(P.flag + P.col_ptr[k], wait_for, err);
      __syncthreads();
      if (sh_ready == 0) break;
      chol_load_tile(P.W + (size_t)k * kTileElems, Ws, wk, wk);
      cp_async_wait_all();
      __syncthreads();
      chol_clear(acc);
      chol_mma<false, false, true>(B, T, Ws, (wk + 3) & ~3, acc);  // W(j, t): lower triangular
      double* Lg = P.L + (size_t)s * kTileElems;
      chol_each_frag(B, acc, [&](int r, int c, double (&a)[2]) {
        *reinterpret_cast<double2*>(Lg + r * kTile + c) = make_double2(a[0], a[1]);
      });
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      chol_store_flag(P.flag + s, want);
    }
  }
  chol_leave(&P.st->factor, [&]() {
    if (tid == 0) P.st->max_diag = 0;
  });
}

// Substitutions: tile columns handed out by ticket, one CTA of 256 threads
// each at a time; the tile of the next product is fetched before the wait
// for the part of the vector that it multiplies. Bound, as the
// factorization, by the chain of the elimination tree.
//
// y(k) = W(k) (rhs(k) - sum_j L(k, j) y(j)): needed only where a right-hand
// side other than the factorization's is solved for (refinement)
static __global__ void __launch_bounds__(256) chol_forward_dag(CholDev P, const double* rhs, unsigned extra) {
  __shared__ int sh_ticket, sh_ok;
  __shared__ double v[kTile];
  const int tid = threadIdx.x, r = tid >> 2, q = tid & 3;
  const unsigned want = P.st->forward.epoch + 1, wait_for = want + extra;
  int* err = &P.st->err;
  for (;;) {
    const int tk = chol_ticket(&P.st->forward, &sh_ticket);
    if (tk >= P.nt) break;
    const int k = P.solve_order[tk];
    const int f0 = P.fwd_ptr[k], nf = P.fwd_ptr[k + 1] - f0;
    double2 w[8], t[8];
    auto fetch = [&](const double* tile, double2 (&d)[8]) {
#pragma unroll
      for (int c = 0; c < 8; ++c) d[c] = *reinterpret_cast<const double2*>(tile + r * kTile + 8 * c + 2 * q);
    };
    auto dot = [&](const double2 (&d)[8]) {
      double a = 0.0;
#pragma unroll
      for (int c = 0; c < 8; ++c) a += d[c].x * v[8 * c + 2 * q] + d[c].y * v[8 * c + 2 * q + 1];
      return a;
    };
    fetch(P.W + (size_t)k * kTileElems, w);
    double sum = 0.0;
    bool ok = true;
    for (int f = 0; f < nf; ++f) {
      const int s = P.fwd[f0 + f], j = P.col[s];
      fetch(P.L + (size_t)s * kTileElems, t);
      if (tid == 0) sh_ok = chol_wait(P.yflag + j, wait_for, err);
      __syncthreads();
      ok = sh_ok != 0;
      if (!ok) break;
      if (tid < kTile) v[tid] = __ldcg(P.y + (size_t)j * kTile + tid);
      __syncthreads();
      sum += dot(t);
    }
    if (!ok) break;
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    __syncthreads();
    if (q == 0) {
      const int o = P.orig[(size_t)k * kTile + r];
      v[r] = (o >= 0 ? rhs[o] : 0.0) - sum;
    }
    __syncthreads();
    double y = dot(w);
    y += __shfl_xor_sync(0xffffffffu, y, 1);
    y += __shfl_xor_sync(0xffffffffu, y, 2);
    if (q == 0) P.y[(size_t)k * kTile + r] = y;
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      chol_store_flag(P.yflag + k, want);
    }
  }
  chol_leave(&P.st->forward, []() {});
}

// x(k) = W(k)^T (y(k) - sum_i L(i, k)^T x(i)), written in the caller's order;
// sc != nullptr gets the outcome of the solve. A source's columns may have no
// solution (dead: x is zero there); solved is called by thread 0 per column.
// Decides the rank of a factorization with suspect pivots (kRankTol); xout ==
// nullptr: does only that.
struct CholAlive {
  __device__ __forceinline__ bool ranked(const CholDev& P) const { return P.dissected; }
  __device__ __forceinline__ bool dead(const CholDev&, int) const { return false; }
  __device__ __forceinline__ void solved(const CholDev&, int) const {}
  __device__ __forceinline__ void end(const CholDev& P, DevScalars* sc) const {
    if (!sc) return;
    sc->solve_ok = P.st->info == 0;
    if (P.st->err) sc->chol_error = 1;
  }
};
template <typename Source>
__global__ void __launch_bounds__(256) chol_backward_dag(Source A, CholDev P, double* xout, DevScalars* sc,
                                                         unsigned extra) {
  __shared__ int sh_ticket, sh_ok;
  __shared__ double v[kTile], vu[kTile], part[4][kTile];
  const int tid = threadIdx.x, c = tid & 63, q = tid >> 6;
  const bool ranked = A.ranked(P) && P.st->suspect != 0;
  if (!xout && !ranked) return;
  const unsigned want = P.st->backward.epoch + 1, wait_for = want + extra;
  int* err = &P.st->err;
  for (;;) {
    const int tk = chol_ticket(&P.st->backward, &sh_ticket);
    if (tk >= P.nt) break;
    const int k = P.solve_order[P.nt - 1 - tk];
    if (tid == 0) A.solved(P, k);
    if (A.dead(P, k)) {
      if (tid < kTile) {
        const int o = P.orig[(size_t)k * kTile + tid];
        if (o >= 0) xout[o] = 0.0;
      }
      if (tid == 0) chol_store_flag(P.xflag + k, want);
      continue;
    }
    double w[16], t[16];
    auto fetch = [&](const double* tile, double (&d)[16]) {
#pragma unroll
      for (int a = 0; a < 16; ++a) d[a] = tile[(16 * q + a) * kTile + c];
    };
    auto dot = [&](const double (&d)[16], const double* z) {
      double a = 0.0;
#pragma unroll
      for (int b = 0; b < 16; ++b) a += d[b] * z[16 * q + b];
      return a;
    };
    fetch(P.W + (size_t)k * kTileElems, w);
    const double yk = tid < kTile ? P.y[(size_t)k * kTile + tid] : 0.0;
    double sum = 0.0, sumu = 0.0;
    bool ok = true;
    for (int s = P.col_ptr[k + 1] - 1; s > P.col_ptr[k]; --s) {
      const int i = P.row[s];
      fetch(P.L + (size_t)s * kTileElems, t);
      if (tid == 0) sh_ok = chol_wait(P.xflag + i, wait_for, err);
      __syncthreads();
      ok = sh_ok != 0;
      if (!ok) break;
      if (tid < kTile) v[tid] = __ldcg(P.x + (size_t)i * kTile + tid);
      if (ranked && tid < kTile) vu[tid] = __ldcg(P.u + (size_t)i * kTile + tid);
      __syncthreads();
      sum += dot(t, v);
      if (ranked) sumu += dot(t, vu);
    }
    if (!ok) break;
    // W(k)^T (y - sum), to thread tid < kTile
    auto finish = [&](double s, double y, double* z) {
      part[q][c] = s;
      __syncthreads();
      if (tid < kTile) z[tid] = y - (((part[0][tid] + part[1][tid]) + part[2][tid]) + part[3][tid]);
      __syncthreads();
      part[q][c] = dot(w, z);
      __syncthreads();
      return tid < kTile ? ((part[0][tid] + part[1][tid]) + part[2][tid]) + part[3][tid] : 0.0;
    };
    const double x = finish(sum, yk, v);
    if (tid < kTile) {
      P.x[(size_t)k * kTile + tid] = x;
      const int o = P.orig[(size_t)k * kTile + tid];
      if (o >= 0 && xout) xout[o] = x;
    }
    if (ranked) {
      __syncthreads();  // part is read
      const size_t at = (size_t)k * kTile + tid;
      const double u = finish(sumu, tid < kTile ? P.suspect[at] : 0.0, vu);
      double uu = 0.0;
      if (tid < kTile) {
        P.u[at] = u;
        uu = P.adiag[at] * u * u;
      }
      uu = warp_sum(uu);
      __syncthreads();
      if (tid == 32) part[0][0] = uu;
      __syncthreads();
      if (tid == 0) P.uu[k] = uu + part[0][0];
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      chol_store_flag(P.xflag + k, want);
    }
  }
  chol_leave(&P.st->backward, [&]() {
    if (ranked) {
      double uu = 0.0;
      for (int k = tid; k < P.nt; k += 256) uu += __ldcg(P.uu + k);
      uu = warp_sum(uu);
      if ((tid & 31) == 0) part[0][tid >> 5] = uu;
      __syncthreads();
      if (tid == 0) {
        for (int w = 1; w < 8; ++w) uu += part[0][w];
        if (!(kRankTol * uu < 1.0)) P.st->info = 1;
        P.st->suspect = 0;  // decided: not again for a further right-hand side
      }
    }
    if (tid == 0) A.end(P, sc);
  });
}

static int chol_launch_check(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s launch: %s", what, cudaGetErrorString(e));
    return G2OC_ERR_CUDA;
  }
  return G2OC_OK;
}

// factor S: the plan holds L (tiles below the diagonal), W, the pivot flag
// and, for rhs != nullptr, the forward-substituted vector. have_floor: the
// largest diagonal entry is in the state already (chol_gather_damped)
template <typename Real>
static int chol_factor(CholPlan& P, cudaStream_t st, const SysDev<Real>& S, const double* rhs, long long* nl,
                       bool have_floor = false) {
  const int ntask = (int)P.S.task.size();
  if (!P.smem_raised) {
    G2OC_CUDA_TRY(
        cudaFuncSetAttribute(chol_factor_dag<CholSystem<double>>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFactorSmem));
    G2OC_CUDA_TRY(
        cudaFuncSetAttribute(chol_factor_dag<CholSystem<float>>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFactorSmem));
    P.smem_raised = true;
  }
  if (!have_floor) {
    chol_floor<Real><<<(P.S.n + 255) / 256, 256, 0, st>>>(S, P.S.bs, P.state.p);
    *nl += 1;
  }
  chol_factor_dag<<<std::min(P.sms, ntask), 256, kFactorSmem, st>>>(CholSystem<Real>{S, P.S.bs}, P.dev(), rhs, P.extra);
  *nl += 1;
  return chol_launch_check("cholesky");
}

// backward substitution of the vector the plan holds
static int chol_backward(CholPlan& P, cudaStream_t st, double* xout, long long* nl, DevScalars* sc = nullptr,
                         unsigned extra = 0) {
  chol_backward_dag<<<std::min(2 * P.sms, P.S.nt), 256, 0, st>>>(CholAlive{}, P.dev(), xout, sc, P.extra + extra);
  *nl += 1;
  return chol_launch_check("cholesky solve");
}

// forward and backward substitution with the factor the plan holds (a
// refinement's correction solve reuses it). Its waits are bounded too: one
// that ran out goes to sc->chol_error, which the end of the trial reads
static int chol_resolve(CholPlan& P, cudaStream_t st, const double* rhs, double* xout, long long* nlaunch,
                        DevScalars* sc) {
  long long nl = 1;
  chol_forward_dag<<<std::min(2 * P.sms, P.S.nt), 256, 0, st>>>(P.dev(), rhs, P.extra + P.extra_kept);
  G2OC_TRY(chol_launch_check("cholesky solve"));
  G2OC_TRY(chol_backward(P, st, xout, &nl, sc, P.extra_kept));
  if (nlaunch) *nlaunch += nl;
  return G2OC_OK;
}

// factor and solve, all queued on the stream; the outcome stays in P.state
// and, for sc != nullptr, goes to sc->solve_ok / chol_error
template <typename Real>
static int chol_solve_async(CholPlan& P, cudaStream_t st, const SysDev<Real>& S, const double* rhs, double* xout,
                            long long* nlaunch, DevScalars* sc = nullptr, bool have_floor = false) {
  long long nl = 0;
  P.extra += P.extra_once;
  const int rc = chol_factor<Real>(P, st, S, rhs, &nl, have_floor);
  const int rb = rc == G2OC_OK ? chol_backward(P, st, xout, &nl, sc) : rc;
  P.extra -= P.extra_once;
  P.extra_once = 0;
  if (rb != G2OC_OK) return rb;
  if (nlaunch) *nlaunch += nl;
  return G2OC_OK;
}

// wait for the queued factorization and read its outcome
static int chol_outcome(CholPlan& P, cudaStream_t st, int* ok) {
  CholState h;
  G2OC_CUDA_TRY(cudaMemcpyAsync(&h, P.state.p, sizeof(CholState), cudaMemcpyDeviceToHost, st));
  G2OC_CUDA_TRY(cudaStreamSynchronize(st));
  if (h.err) {
    set_error("cholesky: a wait for a tile ran out");
    return G2OC_ERR_TIMEOUT;
  }
  *ok = h.info == 0;
  return G2OC_OK;
}

template <typename Real>
static int chol_solve(CholPlan& P, cudaStream_t st, const SysDev<Real>& S, const double* rhs, double* xout, int* ok,
                      long long* nlaunch) {
  G2OC_TRY(chol_solve_async<Real>(P, st, S, rhs, xout, nlaunch));
  return chol_outcome(P, st, ok);
}

// ------------------------------------------------------------------------
// Selected inverse (the marginal covariances of
// LinearSolver::solvePattern, g2o/core/linear_solver.h:78-90, which g2o's
// Cholesky solvers compute with MarginalCovarianceCholesky,
// g2o/core/linear_solver.h:165-173 and g2o/core/marginal_covariance_cholesky.h:42-106). From H = L L^T
// and L^T Sigma = L^-1 (upper-triangular right side), for tile column J
// taken from last to first with S_J = {I > J : L(I,J) != 0},
// W = L(J,J)^-1 and Lh(I,J) = L(I,J) W:
//   Sigma(K,J) = - sum_{I in S_J} Sigma(K,I) Lh(I,J)          (K in S_J)
//   Sigma(J,J) = W^T W - sum_{I in S_J} Lh(I,J)^T Sigma(I,J)
// Every Sigma(K,I) needed lies in the filled tile pattern (S_J is a clique
// of it), so only the pattern's tiles are computed: the tile form of the
// Takahashi recurrences. Sigma has the slots of L (lower tiles, full diagonal
// tiles); L's tiles are overwritten by Lh. The tiles run by ticket from the
// root of the elimination tree downwards, as chol_factor_dag runs upwards.

// Lh(I,J) = L(I,J) W(J), in place, one CTA per stored tile
static __global__ void __launch_bounds__(256) selinv_panel(CholDev P) {
  extern __shared__ __align__(16) double sm_sp[];
  const int s = blockIdx.x, J = P.col[s];
  if (P.row[s] == J) return;
  double* X = sm_sp;
  double* Y = sm_sp + kTileBuf;
  double* Lg = P.L + (size_t)s * kTileElems;
  chol_load_tile(Lg, X);
  chol_load_tile(P.W + (size_t)J * kTileElems, Y);
  cp_async_wait_all();
  __syncthreads();
  const CholBlocks B(P.width[P.row[s]], P.width[J], false);
  CholAcc acc;
  chol_clear(acc);
  chol_mma<false, true>(B, X, Y, (P.width[J] + 3) & ~3, acc);
  chol_each_frag(B, acc, [&](int r, int c, double (&a)[2]) {
    *reinterpret_cast<double2*>(Lg + r * kTile + c) = make_double2(a[0], a[1]);
  });
}

// products of a tile of Sigma: (slot of Sigma, slot of Lh, the Sigma tile is
// used transposed, K)
struct SelinvDev {
  const int* ptr;
  const int4* ent;
  const int* task;
  unsigned* flag;
  double* sigma;
};

static __global__ void __launch_bounds__(256) selinv_dag(CholDev P, SelinvDev Q, unsigned extra) {
  extern __shared__ __align__(16) double sm_sv[];
  __shared__ int sh_ticket, sh_ok;
  double* buf[2][2] = {{sm_sv, sm_sv + kTileBuf}, {sm_sv + 2 * kTileBuf, sm_sv + 3 * kTileBuf}};
  const int tid = threadIdx.x;
  // runs between a factorization and the next: the forward pass' tickets are free
  const unsigned want = P.st->forward.epoch + 1, wait_for = want + extra;
  int* err = &P.st->err;
  for (;;) {
    const int tk = chol_ticket(&P.st->forward, &sh_ticket);
    if (tk >= P.ns) break;
    const int s = Q.task[tk], J = P.col[s];
    const bool diag = P.row[s] == J;
    const CholBlocks B(P.width[P.row[s]], P.width[J], false);
    CholAcc acc;
    chol_clear(acc);
    if (diag) {
      chol_load_tile(P.W + (size_t)J * kTileElems, buf[0][0]);
      cp_async_wait_all();
      __syncthreads();
      chol_mma<true, true>(B, buf[0][0], buf[0][0], kTile, acc);  // W is zero above the diagonal and beyond the width
      chol_each_frag(B, acc, [](int, int, double (&a)[2]) {
        a[0] = -a[0];
        a[1] = -a[1];
      });
      __syncthreads();
    }
    const int q0 = Q.ptr[s], nq = Q.ptr[s + 1] - q0;
    auto issue = [&](int4 e, int stage) {
      chol_load_tile(Q.sigma + (size_t)e.x * kTileElems, buf[stage][0]);
      chol_load_tile(P.L + (size_t)e.y * kTileElems, buf[stage][1]);
    };
    bool issued = false, ok = true;
    int4 en = nq > 0 ? Q.ent[q0] : make_int4(0, 0, 0, 0);
    for (int q = 0; q < nq; ++q) {
      const int stage = q & 1;
      const int4 nx = q + 1 < nq ? Q.ent[q0 + q + 1] : make_int4(0, 0, 0, 0);
      if (!issued) {
        if (tid == 0) sh_ok = chol_wait(Q.flag + en.x, wait_for, err);
        __syncthreads();
        ok = sh_ok != 0;
        if (!ok) break;
        issue(en, stage);
      }
      cp_async_wait_all();
      int ready = 0;
      if (tid == 0 && q + 1 < nq) ready = chol_load_flag(Q.flag + nx.x) == wait_for;
      issued = __syncthreads_or(ready) != 0;
      if (issued) issue(nx, stage ^ 1);
      if (diag) chol_mma<true, true>(B, buf[stage][1], buf[stage][0], en.w, acc);
      else if (en.z) chol_mma<true, true>(B, buf[stage][0], buf[stage][1], en.w, acc);
      else chol_mma<false, true>(B, buf[stage][0], buf[stage][1], en.w, acc);
      en = nx;
    }
    if (!ok) break;
    double* Sg = Q.sigma + (size_t)s * kTileElems;
    if (diag) {
      double* T = buf[0][0];
      __syncthreads();
      chol_frags_to(B, T, acc);
      __syncthreads();
      const int w = 16 * B.mb;
      for (int e = tid; e < kTileElems; e += 256) {
        const int r = e >> 6, c = e & 63;
        if (r < w && c < w) Sg[e] = 0.5 * (T[r * kLd + c] + T[c * kLd + r]);
      }
    } else {
      chol_each_frag(B, acc, [&](int r, int c, double (&a)[2]) {
        *reinterpret_cast<double2*>(Sg + r * kTile + c) = make_double2(-a[0], -a[1]);
      });
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      chol_store_flag(Q.flag + s, want);
    }
  }
  chol_leave(&P.st->forward, []() {});
}

// requested blocks (row, col) of H^-1, row-major bs x bs each
static __global__ void selinv_gather(CholDev P, const double* sigma, const int* pos, int bs, const int2* req,
                                     int nreq, double* out) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int per = bs * bs;
  if (t >= (long long)nreq * per) return;
  const int q = (int)(t / per), e = (int)(t % per);
  int i = pos[req[q].x] + e / bs, j = pos[req[q].y] + e % bs;
  if (i / kTile < j / kTile) {  // the transposed tile is stored
    const int m = i;
    i = j;
    j = m;
  }
  const int ti = i / kTile, tj = j / kTile;
  int lo = P.col_ptr[tj], hi = P.col_ptr[tj + 1] - 1;  // rows ascending, the diagonal first
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (P.row[mid] < ti) lo = mid + 1;
    else hi = mid;
  }
  out[t] = sigma[(size_t)lo * kTileElems + (i % kTile) * kTile + j % kTile];
}

// the lists of the selected inverse, which are the plan's alone
static int chol_inverse_plan(CholPlan& P, cudaStream_t st) {
  if (P.inv_ints.p) return G2OC_OK;
  const CholSymbolic& Y = P.S;
  const int ns = (int)Y.row.size(), nt = Y.nt;
  auto slot = [&](int i, int k) {
    if (i == k) return Y.col_ptr[k];
    return (int)(std::lower_bound(Y.row.begin() + Y.col_ptr[k] + 1, Y.row.begin() + Y.col_ptr[k + 1], i) -
                 Y.row.begin());
  };
  std::vector<int> ptr(ns + 1, 0), task(ns), depth(nt, 0);
  std::vector<int4> ent;
  for (int J = 0; J < nt; ++J) {
    const int s0 = Y.col_ptr[J], s1 = Y.col_ptr[J + 1];
    for (int s = s0; s < s1; ++s) {
      for (int a = s0 + 1; a < s1; ++a) {
        const int I = Y.row[a], K = Y.row[s], kw = (Y.width[I] + 3) & ~3;
        if (s == s0) ent.push_back(make_int4(a, a, 0, kw));
        else ent.push_back(make_int4(K >= I ? slot(K, I) : slot(I, K), a, K < I, kw));
      }
      ptr[s + 1] = (int)ent.size();
    }
  }
  for (int J = nt - 1; J >= 0; --J)
    for (int s = Y.col_ptr[J] + 1; s < Y.col_ptr[J + 1]; ++s) depth[J] = std::max(depth[J], depth[Y.row[s]] + 1);
  for (int s = 0; s < ns; ++s) task[s] = s;
  std::stable_sort(task.begin(), task.end(), [&](int a, int b) {
    const int ka = 2 * depth[Y.col[a]] + (Y.row[a] == Y.col[a]), kb = 2 * depth[Y.col[b]] + (Y.row[b] == Y.col[b]);
    return ka < kb;
  });
  CholInts I;
  P.inv_at[0] = I.add(ptr);
  P.inv_at[1] = I.add(task);
  P.inv_at[2] = I.add(reinterpret_cast<const int*>(ent.data()), 4 * ent.size());
  I.v.resize(I.v.size() + 4, 0);
  G2OC_TRY(P.inv_flag.alloc(ns));
  G2OC_TRY(P.inv_ints.upload(I.v, st));
  G2OC_CUDA_TRY(cudaStreamSynchronize(st));  // the copied host array goes out of scope
  return G2OC_OK;
}

// The tiles of the inverse stay with the plan up to this size (some 2,000 of
// them, a 5,000-pose 2D graph), as making them anew is a good part of a small
// call; larger ones, as large as the factor, would take the memory of whatever
// the program does next.
constexpr size_t kInverseKept = 64u << 20;

// whether the plan's pattern holds the block (r, c)
static bool chol_covers(const CholPlan& P, int r, int c) {
  const CholSymbolic& Y = P.S;
  const int i0 = Y.pos[r], j0 = Y.pos[c];
  for (int a = 0; a < Y.bs; a += std::max(Y.bs - 1, 1))
    for (int b = 0; b < Y.bs; b += std::max(Y.bs - 1, 1)) {
      const int i = std::max(i0 + a, j0 + b) / kTile, j = std::min(i0 + a, j0 + b) / kTile;
      if (!std::binary_search(Y.row.begin() + Y.col_ptr[j], Y.row.begin() + Y.col_ptr[j + 1], i)) return false;
    }
  return true;
}

// the requested blocks of S^-1 (pairs (row, col) of block indices, covered by
// the plan's extra pairs) into out (device, nreq * bs * bs)
template <typename Real>
static int chol_selected_inverse(CholPlan& P, cudaStream_t st, const SysDev<Real>& S, const int2* d_req, int nreq,
                                 double* d_out, int* ok, long long* nlaunch) {
  long long nl = 0;
  G2OC_TRY(chol_factor<Real>(P, st, S, nullptr, &nl));
  G2OC_TRY(chol_backward(P, st, nullptr, &nl));  // the rank
  G2OC_TRY(chol_inverse_plan(P, st));
  const int ns = (int)P.S.row.size(), bs = P.S.bs;
  if (!P.inv_sigma.p) {
    G2OC_TRY(P.inv_sigma.alloc((size_t)ns * kTileElems));
    G2OC_CUDA_TRY(cudaMemsetAsync(P.inv_sigma.p, 0, P.inv_sigma.bytes(), st));  // the parts without unknowns stay zero
  }
  G2OC_CUDA_TRY(cudaMemsetAsync(P.inv_flag.p, 0, P.inv_flag.bytes(), st));
  const int* q = P.inv_ints.p;
  const SelinvDev Q{q + P.inv_at[0], reinterpret_cast<const int4*>(q + P.inv_at[2]), q + P.inv_at[1], P.inv_flag.p,
                    P.inv_sigma.p};
  constexpr int kSmem = 4 * kTileBuf * (int)sizeof(double);
  G2OC_CUDA_TRY(cudaFuncSetAttribute(selinv_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem / 2));
  G2OC_CUDA_TRY(cudaFuncSetAttribute(selinv_dag, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  selinv_panel<<<ns, 256, kSmem / 2, st>>>(P.dev());
  selinv_dag<<<std::min(P.sms, ns), 256, kSmem, st>>>(P.dev(), Q, P.extra);
  nl += 2;
  const long long work = (long long)nreq * bs * bs;
  if (work > 0) {
    selinv_gather<<<(int)((work + 255) / 256), 256, 0, st>>>(P.dev(), P.inv_sigma.p, P.pos, bs, d_req, nreq, d_out);
    nl += 1;
  }
  G2OC_TRY(chol_launch_check("selected inverse"));
  if (nlaunch) *nlaunch += nl;
  const int rc = chol_outcome(P, st, ok);
  if (P.inv_sigma.bytes() > kInverseKept) P.inv_sigma.release();
  return rc;
}

}  // namespace g2oc
