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
// non-positive pivot sets the info flag (G2OC_ERR_NOT_PD at the boundary);
// nothing traps.
#pragma once

#include <algorithm>
#include <vector>

#include "chol_plan.h"
#include "g2oc_internal.h"
#include "pcg_kernels.cuh"
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
struct CholState {
  CholTickets factor, forward, backward;
  int info;  // a pivot was not positive
  int err;   // a wait ran out
  double floor;  // smallest accepted pivot of the current factorization
};

// device side of the plan
struct CholDev {
  int nt, ns;
  const int *col_ptr, *row, *col, *width, *orig;
  const int* asm_ptr;
  const int4* asm_ent;  // offset (low, high) and stride of the block's entries, packed place
  const int* upd_ptr;
  const int2* upd;
  const int *task, *solve_order, *fwd_ptr, *fwd;
  double *L, *W;   // tiles row-major, kTileElems each: per slot, per tile column (W(k) = L(k,k)^-1)
  double *y, *x;   // nt * kTile: forward and backward substituted vectors
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
  DBuf<double> vals;    // L, W, y, x
  DBuf<unsigned> flags;
  DBuf<CholState> state;
  CholDev d{};
  const int* pos = nullptr;  // device copy of S.pos
  int sms = 0;
  unsigned extra = 0;  // the bounded-wait test: flags are compared with a number that is never reached
  const CholDev& dev() const { return d; }
};

// brow, bcol: the blocks of the matrix, row by row; extra: further (row,
// col) block pairs whose entries the plan must hold (the blocks a selected
// inverse is asked for), treated as structural nonzeros of the matrix so that
// the symbolic fill covers them
static int chol_plan_build(CholPlan& P, int nb, int bs, const std::vector<int>& brow, const std::vector<int>& bcol,
                           bool reorder, cudaStream_t st, const std::vector<int32_t>* extra = nullptr) {
  CholSymbolic& S = P.S;
  chol_symbolic(S, nb, bs, brow, bcol, reorder, extra);
  const size_t ns = S.row.size(), nt = (size_t)S.nt;
  // entries of block p of row r at rptr[r] * bs^2 + e * nblk + (p - rptr[r])
  std::vector<int> rptr(nb + 1, 0);
  for (int r : brow) ++rptr[r + 1];
  for (int i = 0; i < nb; ++i) rptr[i + 1] += rptr[i];
  for (size_t q = 0; q < S.asm_ent.size() / 4; ++q) {
    int* a = S.asm_ent.data() + 4 * q;
    const int r = brow[a[0]];
    const long long off = (long long)rptr[r] * bs * bs + (a[0] - rptr[r]);
    const int place = (a[1] + kTile) | ((a[2] + kTile) << 8) | (a[3] << 16);
    a[0] = (int)(off & 0xffffffffll);
    a[1] = (int)(off >> 32);
    a[2] = rptr[r + 1] - rptr[r];
    a[3] = place;
  }
  CholInts I;
  const size_t o[] = {I.add(S.col_ptr), I.add(S.row), I.add(S.col), I.add(S.width), I.add(S.orig), I.add(S.asm_ptr),
                      I.add(S.asm_ent), I.add(S.upd_ptr), I.add(S.upd), I.add(S.task), I.add(S.solve_order),
                      I.add(S.fwd_ptr), I.add(S.fwd), I.add(S.pos)};
  std::vector<int>().swap(S.asm_ent);
  std::vector<int>().swap(S.upd);
  I.v.resize(I.v.size() + 4, 0);
  G2OC_TRY(P.ints.upload(I.v, st));
  G2OC_TRY(P.vals.alloc((ns + nt) * kTileElems + 2 * nt * kTile));
  G2OC_TRY(P.flags.alloc(ns + 2 * nt));
  G2OC_TRY(P.state.alloc(1));
  G2OC_CUDA_TRY(cudaMemsetAsync(P.flags.p, 0, P.flags.bytes(), st));
  G2OC_CUDA_TRY(cudaMemsetAsync(P.state.p, 0, P.state.bytes(), st));
  const int* q = P.ints.p;
  double* L = P.vals.p;
  double* W = L + ns * kTileElems;
  double* y = W + nt * kTileElems;
  P.d = CholDev{S.nt, (int)ns, q + o[0], q + o[1], q + o[2], q + o[3], q + o[4], q + o[5],
                reinterpret_cast<const int4*>(q + o[6]), q + o[7], reinterpret_cast<const int2*>(q + o[8]), q + o[9],
                q + o[10], q + o[11], q + o[12], L, W, y, y + nt * kTile, P.flags.p, P.flags.p + ns,
                P.flags.p + ns + nt, P.state.p};
  P.pos = q + o[13];
  int dev = 0;
  G2OC_CUDA_TRY(cudaGetDevice(&dev));
  G2OC_CUDA_TRY(cudaDeviceGetAttribute(&P.sms, cudaDevAttrMultiProcessorCount, dev));
  G2OC_CUDA_TRY(cudaStreamSynchronize(st));  // the copied host array goes out of scope
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
__device__ __forceinline__ void chol_leave(CholTickets* t) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicInc(&t->left, gridDim.x - 1) == gridDim.x - 1) {  // the last one; left is back at 0
      t->next = 0;
      t->epoch += 1;
      __threadfence();
    }
  }
}

// The pivot floor of a factorization: 4 n eps times the largest diagonal
// entry of the matrix, and the info flag cleared. One CTA of 1024 threads
// (fixed tree).
template <typename Real>
__global__ void __launch_bounds__(1024) chol_begin(SysDev<Real> S, int bs, CholState* st) {
  __shared__ double red[32];
  const int n = S.nb * bs;
  double m = 0.0;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int i = t / bs, a = t % bs;
    const int rb = S.rptr[i], nblk = S.rptr[i + 1] - rb;
    m = fmax(m, fabs((double)S.val[(size_t)rb * bs * bs + (size_t)a * (bs + 1) * nblk + (S.diag[i] - rb)]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r = fmax(r, red[w]);
    st->floor = 4.0 * (double)n * 2.220446049250313e-16 * r;
    st->info = 0;
    st->err = 0;
  }
}

// One tile product: acc += X Y^T over k < K (a multiple of 4), X and Y tiles
// in shared memory (row-major, kLd, k contiguous); the fragments as
// tile_dmma64 deals them to the eight warps.
template <bool XK, bool YK>
__device__ __forceinline__ void chol_mma(const double* Xs, const double* Ys, int K, double (&acc)[2][4][2]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int i0 = 16 * (w & 3), j0 = 32 * (w >> 2);
#pragma unroll 4
  for (int k0 = 0; k0 < K; k0 += 4) {
    double fa[2], fb[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) fa[u] = XK ? Xs[(k0 + t) * kLd + i0 + 8 * u + g] : Xs[(i0 + 8 * u + g) * kLd + k0 + t];
#pragma unroll
    for (int v = 0; v < 4; ++v) fb[v] = YK ? Ys[(k0 + t) * kLd + j0 + 8 * v + g] : Ys[(j0 + 8 * v + g) * kLd + k0 + t];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                     : "+d"(acc[u][v][0]), "+d"(acc[u][v][1])
                     : "d"(fa[u]), "d"(fb[v]));
  }
}

// f(row, column, value pair) over this thread's fragment elements
template <typename F>
__device__ __forceinline__ void chol_each_frag(F&& f) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int i0 = 16 * (w & 3), j0 = 32 * (w >> 2);
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) f(i0 + 8 * u + g, j0 + 8 * v + 2 * t, u, v);
}

// a tile of global memory (row-major) into shared memory
__device__ __forceinline__ void chol_load_tile(const double* src, double* dst) {
#pragma unroll
  for (int q = 0; q < kTileElems / 2 / 256; ++q) {
    const int e = 2 * (threadIdx.x + 256 * q);
    cp_async16(dst + (e >> 6) * kLd + (e & 63), src + e);
  }
}

// shared memory of chol_factor_dag: two stages of two operand tiles, a
// vector per stage and the right-hand side
constexpr int kFactorSmem = (4 * kTileBuf + 3 * kTile) * (int)sizeof(double);

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
// Measured on a 3,500-pose 2D graph (n = 10,497, 11 levels): factorization and
// both substitutions 0.28 ms per solve, against 10.1 ms for the reverse
// Cuthill-McKee band (165 strictly sequential tile steps in one CTA); on a
// 2,500-pose 3D graph (n = 14,994) 0.35 ms against 19.7 ms.
template <typename Real>
__global__ void __launch_bounds__(256) chol_factor_dag(SysDev<Real> S, int bs, CholDev P, const double* rhs,
                                                       unsigned extra) {
  extern __shared__ __align__(16) double sm_chol[];
  __shared__ int sh_ticket, sh_ok;
  double* buf[2][2] = {{sm_chol, sm_chol + kTileBuf}, {sm_chol + 2 * kTileBuf, sm_chol + 3 * kTileBuf}};
  double* yb = sm_chol + 4 * kTileBuf;
  double* vb = yb + 2 * kTile;
  const int tid = threadIdx.x;
  const unsigned want = P.st->factor.epoch + 1;  // the flag value of this launch
  const unsigned wait_for = want + extra;
  const double floor = P.st->floor;
  int* err = &P.st->err;
  for (;;) {
    const int tk = chol_ticket(&P.st->factor, &sh_ticket);
    if (tk >= P.ns) break;
    const int s = P.task[tk];
    const int i = P.row[s], k = P.col[s];
    const bool diag = i == k;
    // A(i, k)
    double* As = buf[0][0];
    for (int e = tid; e < kTileElems; e += 256) {
      const int r = e >> 6, c = e & 63;
      As[r * kLd + c] = diag && r == c && P.orig[(size_t)k * kTile + r] < 0 ? 1.0 : 0.0;
    }
    if (diag && tid < kTile) {
      const int o = rhs ? P.orig[(size_t)k * kTile + tid] : -1;
      vb[tid] = o >= 0 ? rhs[o] : 0.0;
    }
    __syncthreads();
    const int bs2 = bs * bs, e0 = P.asm_ptr[s], ne = (P.asm_ptr[s + 1] - e0) * bs2;
    for (int q = tid; q < ne; q += 256) {
      const int b = q / bs2, e = q - b * bs2;
      const int4 en = P.asm_ent[e0 + b];
      const size_t off = ((size_t)(unsigned)en.x | ((size_t)(unsigned)en.y << 32)) + (size_t)e * en.z;
      const int bi = e / bs, bj = e - bi * bs;
      const bool tr = (en.w >> 16) != 0;
      const int r = (en.w & 255) - kTile + (tr ? bj : bi), c = ((en.w >> 8) & 255) - kTile + (tr ? bi : bj);
      if ((unsigned)r < (unsigned)kTile && (unsigned)c < (unsigned)kTile) As[r * kLd + c] = (double)S.val[off];
    }
    __syncthreads();
    double acc[2][4][2];
    chol_each_frag([&](int r, int c, int u, int v) {
      acc[u][v][0] = -As[r * kLd + c];
      acc[u][v][1] = -As[r * kLd + c + 1];
    });
    __syncthreads();
    // updates
    const int u0 = P.upd_ptr[s], nu = P.upd_ptr[s + 1] - u0;
    double ysum = 0.0;
    auto issue = [&](int2 ab, int stage) {
      chol_load_tile(P.L + (size_t)ab.x * kTileElems, buf[stage][0]);
      if (ab.y != ab.x) chol_load_tile(P.L + (size_t)ab.y * kTileElems, buf[stage][1]);
      if (diag && tid < kTile / 2)
        cp_async16(yb + stage * kTile + 2 * tid, P.y + (size_t)P.col[ab.x] * kTile + 2 * tid);
    };
    bool issued = false, ok = true;
    int2 ab = nu > 0 ? P.upd[u0] : make_int2(0, 0);
    for (int u = 0; u < nu; ++u) {
      const int stage = u & 1;
      const int2 nx = u + 1 < nu ? P.upd[u0 + u + 1] : make_int2(0, 0);
      if (!issued) {
        if (tid == 0)
          sh_ok = chol_wait(P.flag + ab.x, wait_for, err) && (ab.y == ab.x || chol_wait(P.flag + ab.y, wait_for, err));
        __syncthreads();
        ok = sh_ok != 0;
        if (!ok) break;
        issue(ab, stage);
      }
      cp_async_wait_all();
      int ready = 0;
      if (tid == 0 && u + 1 < nu) ready = chol_load_flag(P.flag + nx.x) == wait_for && chol_load_flag(P.flag + nx.y) == wait_for;
      issued = __syncthreads_or(ready) != 0;
      if (issued) issue(nx, stage ^ 1);
      const double* X = buf[stage][0];
      const double* Y = ab.y == ab.x ? X : buf[stage][1];
      const int K = (P.width[P.col[ab.x]] + 3) & ~3;
      chol_mma<false, false>(X, Y, K, acc);
      if (diag) {
        const int r = tid >> 2, q = tid & 3;
        const double* yv = yb + stage * kTile;
#pragma unroll
        for (int c = 0; c < 16; ++c) ysum += X[r * kLd + 4 * c + q] * yv[4 * c + q];
      }
      ab = nx;
    }
    if (!ok) break;
    __syncthreads();
    const int wk = P.width[k];
    if (diag) {
      double* T = buf[0][0];
      double* Ws = buf[0][1];
      chol_each_frag([&](int r, int c, int u, int v) {
        T[r * kLd + c] = -acc[u][v][0];
        T[r * kLd + c + 1] = -acc[u][v][1];
      });
      ysum += __shfl_xor_sync(0xffffffffu, ysum, 1);
      ysum += __shfl_xor_sync(0xffffffffu, ysum, 2);
      if ((tid & 3) == 0) vb[tid >> 2] -= ysum;
      tile_potrf_inv64(T, Ws, buf[1][0], wk, floor, &P.st->info);
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
      double* X = buf[0][0];
      double* Ws = buf[1][0];
      chol_each_frag([&](int r, int c, int u, int v) {
        X[r * kLd + c] = -acc[u][v][0];
        X[r * kLd + c + 1] = -acc[u][v][1];
        acc[u][v][0] = acc[u][v][1] = 0.0;
      });
      if (tid == 0) sh_ok = chol_wait(P.flag + P.col_ptr[k], wait_for, err);
      __syncthreads();
      if (sh_ok == 0) break;
      chol_load_tile(P.W + (size_t)k * kTileElems, Ws);
      cp_async_wait_all();
      __syncthreads();
      chol_mma<false, false>(X, Ws, (wk + 3) & ~3, acc);  // Y(j, t) = W(j, t)
      double* Lg = P.L + (size_t)s * kTileElems;
      chol_each_frag([&](int r, int c, int u, int v) {
        *reinterpret_cast<double2*>(Lg + r * kTile + c) = make_double2(acc[u][v][0], acc[u][v][1]);
      });
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      chol_store_flag(P.flag + s, want);
    }
  }
  chol_leave(&P.st->factor);
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
  chol_leave(&P.st->forward);
}

// x(k) = W(k)^T (y(k) - sum_i L(i, k)^T x(i)), written in the caller's order
static __global__ void __launch_bounds__(256) chol_backward_dag(CholDev P, double* xout, unsigned extra) {
  __shared__ int sh_ticket, sh_ok;
  __shared__ double v[kTile], part[4][kTile];
  const int tid = threadIdx.x, c = tid & 63, q = tid >> 6;
  const unsigned want = P.st->backward.epoch + 1, wait_for = want + extra;
  int* err = &P.st->err;
  for (;;) {
    const int tk = chol_ticket(&P.st->backward, &sh_ticket);
    if (tk >= P.nt) break;
    const int k = P.solve_order[P.nt - 1 - tk];
    double w[16], t[16];
    auto fetch = [&](const double* tile, double (&d)[16]) {
#pragma unroll
      for (int a = 0; a < 16; ++a) d[a] = tile[(16 * q + a) * kTile + c];
    };
    auto dot = [&](const double (&d)[16]) {
      double a = 0.0;
#pragma unroll
      for (int b = 0; b < 16; ++b) a += d[b] * v[16 * q + b];
      return a;
    };
    fetch(P.W + (size_t)k * kTileElems, w);
    const double yk = tid < kTile ? P.y[(size_t)k * kTile + tid] : 0.0;
    double sum = 0.0;
    bool ok = true;
    for (int s = P.col_ptr[k + 1] - 1; s > P.col_ptr[k]; --s) {
      const int i = P.row[s];
      fetch(P.L + (size_t)s * kTileElems, t);
      if (tid == 0) sh_ok = chol_wait(P.xflag + i, wait_for, err);
      __syncthreads();
      ok = sh_ok != 0;
      if (!ok) break;
      if (tid < kTile) v[tid] = __ldcg(P.x + (size_t)i * kTile + tid);
      __syncthreads();
      sum += dot(t);
    }
    if (!ok) break;
    part[q][c] = sum;
    __syncthreads();
    if (tid < kTile) v[tid] = yk - (((part[0][tid] + part[1][tid]) + part[2][tid]) + part[3][tid]);
    __syncthreads();
    part[q][c] = dot(w);
    __syncthreads();
    if (tid < kTile) {
      const double x = ((part[0][tid] + part[1][tid]) + part[2][tid]) + part[3][tid];
      P.x[(size_t)k * kTile + tid] = x;
      const int o = P.orig[(size_t)k * kTile + tid];
      if (o >= 0) xout[o] = x;
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      chol_store_flag(P.xflag + k, want);
    }
  }
  chol_leave(&P.st->backward);
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
// and, for rhs != nullptr, the forward-substituted vector
template <typename Real>
static int chol_factor(CholPlan& P, cudaStream_t st, const SysDev<Real>& S, const double* rhs, long long* nl) {
  const int ns = (int)P.S.row.size();
  G2OC_CUDA_TRY(
      cudaFuncSetAttribute(chol_factor_dag<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFactorSmem));
  chol_begin<Real><<<1, 1024, 0, st>>>(S, P.S.bs, P.state.p);
  chol_factor_dag<Real><<<std::min(P.sms, ns), 256, kFactorSmem, st>>>(S, P.S.bs, P.dev(), rhs, P.extra);
  *nl += 2;
  return chol_launch_check("cholesky");
}

// backward substitution of the vector the plan holds
static int chol_backward(CholPlan& P, cudaStream_t st, double* xout, long long* nl) {
  chol_backward_dag<<<std::min(2 * P.sms, P.S.nt), 256, 0, st>>>(P.dev(), xout, P.extra);
  *nl += 1;
  return chol_launch_check("cholesky solve");
}

// forward and backward substitution with the factor the plan holds (a
// refinement's correction solve reuses it)
static int chol_resolve(CholPlan& P, cudaStream_t st, const double* rhs, double* xout, long long* nlaunch) {
  long long nl = 1;
  chol_forward_dag<<<std::min(2 * P.sms, P.S.nt), 256, 0, st>>>(P.dev(), rhs, P.extra);
  G2OC_TRY(chol_launch_check("cholesky solve"));
  G2OC_TRY(chol_backward(P, st, xout, &nl));
  if (nlaunch) *nlaunch += nl;
  return G2OC_OK;
}

// factor and solve, all queued on the stream; the outcome stays in P.state
template <typename Real>
static int chol_solve_async(CholPlan& P, cudaStream_t st, const SysDev<Real>& S, const double* rhs, double* xout,
                            long long* nlaunch) {
  long long nl = 0;
  G2OC_TRY(chol_factor<Real>(P, st, S, rhs, &nl));
  G2OC_TRY(chol_backward(P, st, xout, &nl));
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
  double acc[2][4][2] = {};
  chol_mma<false, true>(X, Y, (P.width[J] + 3) & ~3, acc);
  chol_each_frag([&](int r, int c, int u, int v) {
    *reinterpret_cast<double2*>(Lg + r * kTile + c) = make_double2(acc[u][v][0], acc[u][v][1]);
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
    double acc[2][4][2] = {};
    if (diag) {
      chol_load_tile(P.W + (size_t)J * kTileElems, buf[0][0]);
      cp_async_wait_all();
      __syncthreads();
      chol_mma<true, true>(buf[0][0], buf[0][0], kTile, acc);  // W is zero above the diagonal and beyond the width
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v][0] = -acc[u][v][0], acc[u][v][1] = -acc[u][v][1];
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
      if (diag) chol_mma<true, true>(buf[stage][1], buf[stage][0], en.w, acc);
      else if (en.z) chol_mma<true, true>(buf[stage][0], buf[stage][1], en.w, acc);
      else chol_mma<false, true>(buf[stage][0], buf[stage][1], en.w, acc);
      en = nx;
    }
    if (!ok) break;
    double* Sg = Q.sigma + (size_t)s * kTileElems;
    if (diag) {
      double* T = buf[0][0];
      __syncthreads();
      chol_each_frag([&](int r, int c, int u, int v) {
        T[r * kLd + c] = -acc[u][v][0];
        T[r * kLd + c + 1] = -acc[u][v][1];
      });
      __syncthreads();
      for (int e = tid; e < kTileElems; e += 256) {
        const int r = e >> 6, c = e & 63;
        Sg[e] = 0.5 * (T[r * kLd + c] + T[c * kLd + r]);
      }
    } else {
      chol_each_frag([&](int r, int c, int u, int v) {
        *reinterpret_cast<double2*>(Sg + r * kTile + c) = make_double2(-acc[u][v][0], -acc[u][v][1]);
      });
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      chol_store_flag(Q.flag + s, want);
    }
  }
  chol_leave(&P.st->forward);
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

// the requested blocks of S^-1 (pairs (row, col) of block indices, covered by
// the plan's extra pairs) into out (device, nreq * bs * bs)
template <typename Real>
static int chol_selected_inverse(CholPlan& P, cudaStream_t st, const SysDev<Real>& S, const int2* d_req, int nreq,
                                 double* d_out, int* ok, long long* nlaunch) {
  long long nl = 0;
  G2OC_TRY(chol_factor<Real>(P, st, S, nullptr, &nl));
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
  const size_t o[] = {I.add(ptr), I.add(task), I.add(reinterpret_cast<const int*>(ent.data()), 4 * ent.size())};
  I.v.resize(I.v.size() + 4, 0);
  DBuf<int> ints;
  DBuf<unsigned> flag;
  DBuf<double> sigma;
  G2OC_TRY(ints.upload(I.v, st));
  G2OC_TRY(flag.alloc(ns));
  G2OC_TRY(sigma.alloc((size_t)ns * kTileElems));
  G2OC_CUDA_TRY(cudaMemsetAsync(flag.p, 0, flag.bytes(), st));
  G2OC_TRY(chol_outcome(P, st, ok));
  if (!*ok) return G2OC_OK;
  const SelinvDev Q{ints.p + o[0], reinterpret_cast<const int4*>(ints.p + o[2]), ints.p + o[1], flag.p, sigma.p};
  constexpr int kSmem = 4 * kTileBuf * (int)sizeof(double);
  G2OC_CUDA_TRY(cudaFuncSetAttribute(selinv_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem / 2));
  G2OC_CUDA_TRY(cudaFuncSetAttribute(selinv_dag, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  selinv_panel<<<ns, 256, kSmem / 2, st>>>(P.dev());
  selinv_dag<<<std::min(P.sms, ns), 256, kSmem, st>>>(P.dev(), Q, P.extra);
  nl += 2;
  const long long work = (long long)nreq * Y.bs * Y.bs;
  if (work > 0) {
    selinv_gather<<<(int)((work + 255) / 256), 256, 0, st>>>(P.dev(), sigma.p, P.pos, Y.bs, d_req, nreq, d_out);
    nl += 1;
  }
  G2OC_TRY(chol_launch_check("selected inverse"));
  int fine = 0;
  G2OC_TRY(chol_outcome(P, st, &fine));
  if (nlaunch) *nlaunch += nl;
  return G2OC_OK;
}

}  // namespace g2oc
