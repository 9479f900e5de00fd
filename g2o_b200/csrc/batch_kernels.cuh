// batch_kernels.cuh -- many independent local bundle adjustments (windows)
// in one packed graph: the linearization, Schur complement and
// back-substitution kernels run over all windows at once (the packed Hessian
// is block-diagonal by window), while the Levenberg-Marquardt control of
// OptimizationAlgorithmLevenberg::solve (g2o/core/optimization_algorithm_levenberg.cpp:60-153)
// runs per window on the device: each round every unfinished window makes one
// trial with its own lambda, accepts or rejects it (restoring only its own
// vertices) and advances its own iteration count. Each window's reduced
// camera system is solved by a dense FP64 Cholesky (LinearSolverDense,
// g2o/solvers/dense/linear_solver_dense.h:57-105), tile by tile over all windows.
#pragma once

#include "../../include/g2o_cuda.h"
#include "ba_kernels.cuh"
#include "cholesky.cuh"
#include "pcg_kernels.cuh"
#include "reduce.cuh"

namespace g2oc {

struct WinState {
  double chi2_init;   // robust chi2 before the first iteration
  double chi2_cur;    // currentChi of the window's iteration
  double chi2_temp;   // tempChi after the trial
  double lambda;
  double ni;
  double scale;       // computeScale() + 1e-3
  double rho;
  double max_diag;
  int iteration;      // completed iterations
  int qmax;           // trials in the current iteration
  int trials;         // trials in all
  int done;           // finished (iteration limit or Terminate)
  int accept;         // the last trial was accepted
  int result;         // G2OC_RESULT_* of the last iteration
  int solve_ok;       // the last factorization succeeded
  int not_pd;         // a pivot of the factorization under way was not positive
};

// ranges of window w: free cameras [cam[w], cam[w+1]) and landmarks
// [lm[w], lm[w+1]) in Hessian order, device edges [edge[w], edge[w+1]),
// vertices (caller order) poses [pose[w], pose[w+1]) and points
// [point[w], point[w+1])
struct WinDev {
  int nw;
  const int* cam;
  const int* lm;
  const int* edge;
  const int* pose;
  const int* point;
  const long long* mat;  // offset of the window's dense n x n matrix in the scratch
};

// robust chi2 per window (activeRobustChi2) into chi2_cur (which = 0, windows
// at the start of an iteration) or chi2_temp (which = 1), over edge chunks of
// at most kWinChi2Chunk edges so that the largest windows do not set the
// launch's tail: per chunk a CTA's sum, then per window the chunk sums in
// chunk order (win_chi2_finish).
constexpr int kWinChi2Chunk = 2048;
template <int THREADS>
__global__ void __launch_bounds__(THREADS) win_chi2_chunks(BAEdges E, BAVertices V, WinDev W, const int* chunk_w,
                                                          const int* chunk_e0, const WinState* ws, int which,
                                                          double* partial) {
  const int ch = blockIdx.x, w = chunk_w[ch];
  const WinState& s = ws[w];
  if (s.done || (which == 0 && s.qmax != 0)) return;
  const int k1 = min(chunk_e0[ch] + kWinChi2Chunk, W.edge[w + 1]);
  double r = 0.0;
  for (int k = chunk_e0[ch] + threadIdx.x; k < k1; k += THREADS) {
    double e[2], Xc[3], chi2, wt;
    const double4 om = ba_om(E, k);
    ba_edge_error(V, E.v[k], E.z[k], om, e, Xc, chi2, wt);
    if (om.w > 0.0) {
      double rho[3];
      huber(chi2, om.w, rho);
      r += rho[0];
    } else {
      r += chi2;
    }
  }
  r = block_sum1(r);
  if (threadIdx.x == 0) partial[ch] = r;
}

static __global__ void win_chi2_finish(const int* win_chunk_ptr, int nw, const double* partial, WinState* ws,
                                       int which) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  WinState& s = ws[w];
  if (s.done || (which == 0 && s.qmax != 0)) return;
  double r = 0.0;
  for (int c = win_chunk_ptr[w]; c < win_chunk_ptr[w + 1]; ++c) r += partial[c];
  if (which == 0) {
    s.chi2_cur = r;
    if (s.iteration == 0) s.chi2_init = r;
  } else {
    s.chi2_temp = r;
  }
}

// computeLambdaInit for windows starting their first iteration: lambda =
// tau * max |diag H| over the window's free cameras and landmarks, ni = 2
template <typename Real, int THREADS>
__global__ void __launch_bounds__(THREADS) win_lambda_init(const Real* hpp, const Real* hll, WinDev W, WinState* ws,
                                                            double user_lambda, double tau) {
  const int w = blockIdx.x;
  WinState& s = ws[w];
  if (s.done || s.iteration != 0 || s.qmax != 0) return;
  double m = 0.0;
  const int c0 = W.cam[w], nc = (W.cam[w + 1] - c0) * 6;
  for (int t = threadIdx.x; t < nc; t += THREADS) {
    const int h = c0 + t / 6, d = t % 6;
    m = fmax(m, fabs((double)hpp[(size_t)h * 36 + d * 7]));  // BA: Hpp block h is camera h's diagonal
  }
  const int l0 = W.lm[w], nl = (W.lm[w + 1] - l0) * 3;
  for (int t = threadIdx.x; t < nl; t += THREADS) {
    const int l = l0 + t / 3, d = t % 3;
    m = fmax(m, fabs((double)hll[(size_t)l * 6 + (d == 0 ? 0 : d == 1 ? 3 : 5)]));
  }
  __shared__ double sm[THREADS / 32];
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0.0;
    for (int i = 0; i < THREADS / 32; ++i) x = fmax(x, sm[i]);
    s.max_diag = x;
    s.lambda = user_lambda > 0.0 ? user_lambda : tau * x;
    s.ni = 2.0;
  }
}

// the window's lambda on each of its free cameras and landmarks
static __global__ void win_spread_lambda(const int* win_of_cam, int Cf, const int* win_of_lm, int Pf,
                                         const WinState* ws, double* lam_c, double* lam_l) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < Cf) lam_c[t] = ws[win_of_cam[t]].lambda;
  else if (t < Cf + Pf) lam_l[t - Cf] = ws[win_of_lm[t - Cf]].lambda;
}

// Largest number of free camera unknowns of a window: what the interface has
// promised since one CTA held a panel of a window's matrix in shared memory.
// The tiles below know no such limit; a larger window is a bundle adjustment of
// its own (g2oc_optimize).
constexpr int kWinMaxUnknowns = 837;

// The windows' dense reduced camera systems as one batch for the tiled
// Cholesky (LinearSolverDense: LLT of the damped Schur complement, then the
// two triangular solves): the tiles of all windows are tasks of one launch, so
// a large window is worked on by several SMs and small ones fill the rest.
// With a CTA per window the launch took as long as its largest window: 96
// windows of 8 to 58 free cameras (n = 48 to 348) 480 us a round, against
// 122 us for both launches here.
// The matrices (n x n, row-major, lower triangle) are as the Schur rows wrote
// them and stay so. Any positive pivot passes; a window with another one gets
// solve_ok = 0 and x = 0. Finished windows are left out.
struct CholWindows {
  const double* M;
  const long long* mat;
  const int* cam;
  const int2* tile;  // per tile column: window, place in it
  WinState* ws;
  __device__ __forceinline__ double scale(const CholDev&) const { return 0.0; }
  __device__ __forceinline__ bool ranked(const CholDev&) const { return false; }
  __device__ __forceinline__ bool skip(const CholDev&, int k) const { return ws[tile[k].x].done != 0; }
  __device__ __forceinline__ void begin(const CholDev&, int k) const {
    if (tile[k].y == 0) ws[tile[k].x].not_pd = 0;
  }
  __device__ __forceinline__ int* info(const CholDev&, int k) const { return &ws[tile[k].x].not_pd; }
  __device__ __forceinline__ void assemble(const CholDev& P, int s, double* As) const {
    const int k = P.col[s], i = P.row[s], wk = P.width[k], wi = P.width[i];
    const int2 t = tile[k];
    const int n = 6 * (cam[t.x + 1] - cam[t.x]);  // even: rows and columns start on 16 bytes
    const double* src = M + mat[t.x] + (size_t)(t.y + i - k) * kTile * n + t.y * kTile;
    for (int e = threadIdx.x; e < kTileElems / 2; e += 256) {
      const int r = e >> 5, c = 2 * (e & 31);
      double2 v = make_double2(0.0, 0.0);
      if (r < wi && c < wk) v = *reinterpret_cast<const double2*>(src + (size_t)r * n + c);
      if (i == k) {
        if (c > r) v.x = 0.0;
        if (c + 1 > r) v.y = 0.0;
        if (r >= wk && c == r) v.x = 1.0;
        if (r >= wk && c + 1 == r) v.y = 1.0;
      }
      *reinterpret_cast<double2*>(As + r * kLd + c) = v;
    }
  }
  __device__ __forceinline__ bool dead(const CholDev&, int k) const {
    const WinState& s = ws[tile[k].x];
    return s.done || s.not_pd;
  }
  __device__ __forceinline__ void solved(const CholDev&, int k) const {
    WinState& s = ws[tile[k].x];
    if (tile[k].y == 0 && !s.done) s.solve_ok = !s.not_pd;
  }
  __device__ __forceinline__ void end(const CholDev& P, DevScalars* sc) const {
    if (P.st->err) sc->chol_error = 1;
  }
};

// zero the step of finished windows (their vertices stay as they are)
static __global__ void win_mask_step(const int* win_of_cam, int Cf, const int* win_of_lm, int Pf, const WinState* ws,
                                     double* x) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < Cf * 6) {
    if (ws[win_of_cam[t / 6]].done) x[t] = 0.0;
  } else if (t < Cf * 6 + Pf * 3) {
    if (ws[win_of_lm[(t - Cf * 6) / 3]].done) x[t] = 0.0;
  }
}

// computeScale per window: x . (lambda x + b) over its Hessian range, + 1e-3
template <int THREADS>
__global__ void __launch_bounds__(THREADS) win_scale(const double* x, const double* b, int Cf, WinDev W,
                                                      WinState* ws) {
  const int w = blockIdx.x;
  WinState& s = ws[w];
  if (s.done) return;
  const double lambda = s.lambda;
  double acc = 0.0;
  const int c0 = W.cam[w] * 6, c1 = W.cam[w + 1] * 6;
  for (int i = c0 + threadIdx.x; i < c1; i += THREADS) acc += x[i] * (lambda * x[i] + b[i]);
  const int l0 = Cf * 6 + W.lm[w] * 3, l1 = Cf * 6 + W.lm[w + 1] * 3;
  for (int i = l0 + threadIdx.x; i < l1; i += THREADS) acc += x[i] * (lambda * x[i] + b[i]);
  acc = block_sum1(acc);
  if (threadIdx.x == 0) s.scale = acc + 1e-3;
}

// One trial's decision per window (lm_decide), then the trial loop and
// iteration bookkeeping of OptimizationAlgorithmLevenberg::solve and
// SparseOptimizer::optimize: the trial loop continues while rho < 0 and
// fewer than max_trials trials were made; it ends in Terminate when
// max_trials is reached, rho == 0 or lambda is not finite.
static __global__ void win_decide(WinState* ws, int nw, int max_trials, int max_iterations, int* active) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  WinState& s = ws[w];
  if (s.done) return;
  const bool ok2 = s.solve_ok != 0;
  double tempChi = s.chi2_temp;
  if (!ok2) tempChi = 1.79769313486231570815e+308;
  double rho = s.chi2_cur - tempChi;
  rho /= ok2 ? s.scale : 1.0;
  if (rho > 0 && isfinite(tempChi) && ok2) {
    double alpha = 1. - pow((2 * rho - 1), 3);
    alpha = fmin(alpha, 2. / 3.);
    s.lambda *= fmax(1. / 3., alpha);
    s.ni = 2;
    s.chi2_cur = tempChi;
    s.accept = 1;
  } else {
    s.lambda *= s.ni;
    s.ni *= 2;
    s.accept = 0;
  }
  s.rho = rho;
  s.qmax++;
  s.trials++;
  const bool more = rho < 0 && s.qmax < max_trials && isfinite(s.lambda);
  if (more) {
    atomicAdd(active, 1);
    return;
  }
  // the iteration is over
  if (s.qmax == max_trials || rho == 0 || !isfinite(s.lambda)) {
    s.result = G2OC_RESULT_TERMINATE;
    s.done = 1;
  } else {
    s.result = G2OC_RESULT_OK;
  }
  s.iteration++;
  s.qmax = 0;
  if (s.iteration >= max_iterations) s.done = 1;
  if (!s.done) atomicAdd(active, 1);
}

// restore the vertices of windows whose trial was rejected (pop), one thread
// per vertex record
static __global__ void win_pop(const int* win_of_pose, int C, const int* win_of_point, int P, const WinState* ws,
                               const double* pose_bak, double* pose, const double* point_bak, double* point) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < C * 8) {
    const WinState& s = ws[win_of_pose[t / 8]];
    if (!s.accept) pose[t] = pose_bak[t];
  } else if (t < C * 8 + P * 4) {
    const int u = t - C * 8;
    const WinState& s = ws[win_of_point[u / 4]];
    if (!s.accept) point[u] = point_bak[u];
  }
}

}  // namespace g2oc
