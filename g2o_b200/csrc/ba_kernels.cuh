// ba_kernels.cuh -- device kernels of the bundle-adjustment path
// (EdgeProjectXYZ2UV between VertexPointXYZ landmarks, marginalized, and
// VertexSE3Expmap cameras). Real is the storage/accumulation type of the
// Jacobians, Hessian blocks and Schur products (double: FP64 path; float:
// mixed path). Errors, chi2, the gradient b and the solution x are FP64 in
// both paths.
//
// Every sum is a fixed-order reduction (per-thread loop, fixed shuffle tree,
// fixed shared-memory tree, partials summed in index order), so results are
// bit-identical run to run; no floating-point atomics.
#pragma once

#include <type_traits>

#include "g2o_math.cuh"
#include "g2oc_internal.h"
#include "reduce.cuh"

namespace g2oc {

// two entries of the storage type in one access
template <typename Real>
struct Vec2;
template <>
struct Vec2<double> {
  using T = double2;
};
template <>
struct Vec2<float> {
  using T = float2;
};

struct BAEdges {
  int n;                  // active edges
  const int2* v;          // (point index, pose index), point-major device order
  const double2* z;       // measurement
  const double4* om;      // (Omega00, Omega01, Omega11, Huber delta; <= 0: none)
  const int* hpl;         // Hpl block per edge or -1
  // om == nullptr: every edge has the information and Huber delta om_const
  // (a uniform graph reads no per-edge record)
  double4 om_const = {0.0, 0.0, 0.0, 0.0};
  // stereo edges (stereo_kernels.cuh) instead of z / om: (u, v, u_right,
  // Huber delta), (O00, O01, O02, O11), (O12, O22)
  const double4* z3 = nullptr;
  const double4* oa3 = nullptr;
  const double2* ob3 = nullptr;
};

struct BACamEdges {       // camera-major copy of the edges of free cameras
  const int* ptr;         // Cf + 1
  const int2* v;
  const double2* z;
  const double4* om;
  const double4* z3 = nullptr;  // stereo, as BAEdges
  double4 om_const = {0.0, 0.0, 0.0, 0.0};  // om == nullptr: as BAEdges
  const double4* oa3 = nullptr;
  const double2* ob3 = nullptr;
};

struct BAVertices {
  double* cam;            // C x 8: qx qy qz qw tx ty tz pad (SE3Quat)
  double* pt;             // P x 4: x y z pad
  const int* free_pose;   // Cf: pose index of Hessian row h
  const int* free_point;  // Pf: point index of landmark l
  double fx, fy, cx, cy;  // EdgeProjectXYZ2UV: fx = fy = focal_length
  double bf = 0.0;        // EdgeStereoSE3ProjectXYZ::bf
};

// the information record of edge k (per edge, or the graph's uniform one)
__device__ __forceinline__ double4 ba_om(const BAEdges& E, int k) { return E.om ? E.om[k] : E.om_const; }
__device__ __forceinline__ double4 ba_om(const BACamEdges& E, int k) { return E.om ? E.om[k] : E.om_const; }

// Per-edge residual, robust weight and weighted error in FP64.
// robust weight = rho'(e^T Omega e) (BaseEdge::robustInformation keeps rho'
// only, g2o/core/base_edge.h:156-162); we = -rho' Omega e
// (BaseFixedSizedEdge::constructQuadraticForm, base_fixed_sized_edge.hpp:48-63).
__device__ __forceinline__ void ba_edge_error(const BAVertices& V, int2 v, double2 z, double4 om,
                                              double e[2], double Xc[3], double& chi2, double& w) {
  const double* cam = V.cam + (size_t)v.y * 8;
  const double* X = V.pt + (size_t)v.x * 4;
  ba_transform(cam, X, Xc);
  e[0] = z.x - (Xc[0] / Xc[2] * V.fx + V.cx);
  e[1] = z.y - (Xc[1] / Xc[2] * V.fy + V.cy);
  const double t0 = om.x * e[0] + om.y * e[1];
  const double t1 = om.y * e[0] + om.z * e[1];
  chi2 = e[0] * t0 + e[1] * t1;
  w = 1.0;
  if (om.w > 0.0) {
    double rho[3];
    huber(chi2, om.w, rho);
    w = rho[1];
  }
}

// computeActiveErrors + activeChi2 / activeRobustChi2
// (g2o/core/sparse_optimizer.cpp:78-130): partials[2*block] = (chi2, robust)
static __global__ void ba_chi2_kernel(BAEdges E, BAVertices V, double* partials, GridSum G) {
  double c = 0.0, r = 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < E.n; k += gridDim.x * blockDim.x) {
    double e[2], Xc[3], chi2, w;
    const double4 om = ba_om(E, k);
    ba_edge_error(V, E.v[k], E.z[k], om, e, Xc, chi2, w);
    c += chi2;
    if (om.w > 0.0) {
      double rho[3];
      huber(chi2, om.w, rho);
      r += rho[0];
    } else {
      r += chi2;
    }
  }
  block_sum2(c, r, partials + 2 * blockIdx.x);
  grid_sum2(partials, G);
}

// ------------------------------------------------------- structure only
// StructureOnlySolver<3>::calc (g2o/solvers/structure_only/structure_only_solver.h:66-215)
// for every free landmark, the cameras held fixed: each landmark runs its own
// small Levenberg-Marquardt on its 3x3 system (mu = 0.01, nu = 2; stop when
// |b| < 0.001 or after num_max_trials rejected steps), with robust chi2
// rho[0] and the rho'-weighted quadratic form. Landmarks are independent: one
// thread each, its edges the landmark's contiguous device range.
__device__ __forceinline__ double so_robust_chi2(const BAEdges& E, const BAVertices& V, int k0, int k1) {
  double s = 0.0;
  for (int k = k0; k < k1; ++k) {
    double e[2], Xc[3], chi2, w;
    const double4 om = ba_om(E, k);
    ba_edge_error(V, E.v[k], E.z[k], om, e, Xc, chi2, w);
    if (om.w > 0.0) {
      double rho[3];
      huber(chi2, om.w, rho);
      s += rho[0];
    } else {
      s += chi2;
    }
  }
  return s;
}

static __global__ void ba_structure_only(BAEdges E, BAVertices V, const int* l_ptr, int Pf, int num_iters,
                                         int num_max_trials) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= Pf) return;
  double* X = V.pt + (size_t)V.free_point[l] * 4;
  const int k0 = l_ptr[l], k1 = l_ptr[l + 1];
  double chi2 = so_robust_chi2(E, V, k0, k1);
  double mu = 0.01, nu = 2.0;
  bool stop = false;
  for (int ig = 0; ig < num_iters; ++ig) {
    double H[6] = {0, 0, 0, 0, 0, 0};  // 00 01 02 11 12 22
    double b[3] = {0, 0, 0};
    for (int k = k0; k < k1; ++k) {
      double e[2], Xc[3], c2, w;
      const int2 v = E.v[k];
      const double4 om = ba_om(E, k);
      ba_edge_error(V, v, E.z[k], om, e, Xc, c2, w);
      double Jp[6], Jc[12];
      ba_jacobians_from_xc(V.cam + (size_t)v.y * 8, Xc, V.fx, V.fy, Jp, Jc);
      // weightedOmega = rho' Omega, omega_r = -rho' Omega e (constructQuadraticForm)
      const double w00 = w * om.x, w01 = w * om.y, w11 = w * om.z;
      const double r0 = -(om.x * e[0] + om.y * e[1]) * w, r1 = -(om.y * e[0] + om.z * e[1]) * w;
      double WJ[6];  // (rho' Omega) Jp, 2x3
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        WJ[c] = w00 * Jp[c] + w01 * Jp[3 + c];
        WJ[3 + c] = w01 * Jp[c] + w11 * Jp[3 + c];
      }
      H[0] += Jp[0] * WJ[0] + Jp[3] * WJ[3];
      H[1] += Jp[0] * WJ[1] + Jp[3] * WJ[4];
      H[2] += Jp[0] * WJ[2] + Jp[3] * WJ[5];
      H[3] += Jp[1] * WJ[1] + Jp[4] * WJ[4];
      H[4] += Jp[1] * WJ[2] + Jp[4] * WJ[5];
      H[5] += Jp[2] * WJ[2] + Jp[5] * WJ[5];
#pragma unroll
      for (int c = 0; c < 3; ++c) b[c] += Jp[c] * r0 + Jp[3 + c] * r1;
    }
    if (sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]) < 0.001) break;
    int trial = 0;
    do {
      // LDL^T of H + mu I
      const double a00 = H[0] + mu, a11 = H[3] + mu, a22 = H[5] + mu;
      const double d0 = a00;
      const double l10 = H[1] / d0, l20 = H[2] / d0;
      const double d1 = a11 - l10 * l10 * d0;
      const double l21 = (H[4] - l20 * l10 * d0) / d1;
      const double d2 = a22 - l20 * l20 * d0 - l21 * l21 * d1;
      bool good = false;
      if (d0 > 0.0 && d1 > 0.0 && d2 > 0.0) {
        const double y0 = b[0], y1 = b[1] - l10 * y0, y2 = b[2] - l20 * y0 - l21 * y1;
        const double z2 = y2 / d2, z1 = y1 / d1 - l21 * z2, z0 = y0 / d0 - l10 * z1 - l20 * z2;
        const double old[3] = {X[0], X[1], X[2]};
        X[0] += z0;
        X[1] += z1;
        X[2] += z2;
        const double new_chi2 = so_robust_chi2(E, V, k0, k1);
        if (chi2 - new_chi2 > 0.0 && isfinite(new_chi2)) {
          good = true;
          chi2 = new_chi2;
        } else {
          X[0] = old[0];
          X[1] = old[1];
          X[2] = old[2];
        }
      }
      if (good) {
        mu *= 1.0 / 3.0;
        nu = 2.0;
        break;
      }
      mu *= nu;
      nu *= 2.0;
      if (++trial >= num_max_trials) stop = true;
    } while (!stop);
    if (stop) break;
  }
}

// per-edge errors (parity hook)
static __global__ void ba_errors_kernel(BAEdges E, BAVertices V, double* err) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= E.n) return;
  double e[2], Xc[3], chi2, w;
  ba_edge_error(V, E.v[k], E.z[k], ba_om(E, k), e, Xc, chi2, w);
  err[2 * k] = e[0];
  err[2 * k + 1] = e[1];
}

// per-edge Jacobians in FP64 (parity hook): Jp 2x3, Jc 2x6
static __global__ void ba_jacobians_kernel(BAEdges E, BAVertices V, double* jp, double* jc) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= E.n) return;
  const int2 v = E.v[k];
  const double* cam = V.cam + (size_t)v.y * 8;
  double Xc[3];
  ba_transform(cam, V.pt + (size_t)v.x * 4, Xc);
  double Jp[6], Jc[12];
  ba_jacobians_from_xc(cam, Xc, V.fx, V.fy, Jp, Jc);
  for (int i = 0; i < 6; ++i) jp[6 * k + i] = Jp[i];
  for (int i = 0; i < 12; ++i) jc[12 * k + i] = Jc[i];
}

// place of entry (r, c) of a 6 x 3 Hpl block in its 18 stored values: the
// first two components of every row in pairs, then the third ones, as
// schur_rows reads them
__host__ __device__ constexpr int hpl_at(int r, int c) { return c < 2 ? 2 * r + c : 12 + r; }

// Landmark pass of BlockSolver::buildSystem (block_solver.hpp:492-565) for the
// landmark side: one thread per free landmark walks its edges (contiguous in
// the point-major order), accumulates H_ll = sum Jp^T Om' Jp and
// b_l = sum Jp^T we, and writes each Hpl block Jc^T Om' Jp (the transposed
// mapping of block_solver.hpp:210-216). Edges sharing a (camera, landmark)
// block are adjacent and summed in order.
template <typename Real>
__global__ void ba_landmark_pass(BAEdges E, BAVertices V, const int* l_ptr, int Pf, Real* hll, Real* hpl,
                                 double* b_l) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= Pf) return;
  Real H[6] = {0, 0, 0, 0, 0, 0};
  double bl[3] = {0, 0, 0};
  Real B[18];
  int cur = -1;
  const int k1 = l_ptr[l + 1];
  for (int k = l_ptr[l]; k < k1; ++k) {
    const int2 v = E.v[k];
    const double4 om = ba_om(E, k);
    double e[2], Xc[3], chi2, w;
    ba_edge_error(V, v, E.z[k], om, e, Xc, chi2, w);
    const double* cam = V.cam + (size_t)v.y * 8;
    double Jpd[6], Jcd[12];
    ba_jacobians_from_xc(cam, Xc, V.fx, V.fy, Jpd, Jcd);
    Real Jp[6], Jc[12];
#pragma unroll
    for (int i = 0; i < 6; ++i) Jp[i] = (Real)Jpd[i];
#pragma unroll
    for (int i = 0; i < 12; ++i) Jc[i] = (Real)Jcd[i];
    const double we0 = -w * (om.x * e[0] + om.y * e[1]);
    const double we1 = -w * (om.y * e[0] + om.z * e[1]);
    const Real o00 = (Real)(w * om.x), o01 = (Real)(w * om.y), o11 = (Real)(w * om.z);
    // AtO = Jp^T Om' (3x2)
    Real A0[3], A1[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      A0[i] = Jp[i] * o00 + Jp[3 + i] * o01;
      A1[i] = Jp[i] * o01 + Jp[3 + i] * o11;
    }
    H[0] += A0[0] * Jp[0] + A1[0] * Jp[3];
    H[1] += A0[0] * Jp[1] + A1[0] * Jp[4];
    H[2] += A0[0] * Jp[2] + A1[0] * Jp[5];
    H[3] += A0[1] * Jp[1] + A1[1] * Jp[4];
    H[4] += A0[1] * Jp[2] + A1[1] * Jp[5];
    H[5] += A0[2] * Jp[2] + A1[2] * Jp[5];
#pragma unroll
    for (int i = 0; i < 3; ++i) bl[i] += Jpd[i] * we0 + Jpd[3 + i] * we1;
    const int blk = E.hpl[k];
    if (blk >= 0) {
      if (blk != cur) {
        if (cur >= 0) {
#pragma unroll
          for (int i = 0; i < 18; ++i) hpl[(size_t)cur * 18 + i] = B[i];
        }
#pragma unroll
        for (int i = 0; i < 18; ++i) B[i] = Real(0);
        cur = blk;
      }
      // B(6x3) += Jc^T (Om' Jp) = Jc^T (AtO)^T
#pragma unroll
      for (int r = 0; r < 6; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) B[hpl_at(r, c)] += Jc[r] * A0[c] + Jc[6 + r] * A1[c];
    }
  }
  if (cur >= 0) {
#pragma unroll
    for (int i = 0; i < 18; ++i) hpl[(size_t)cur * 18 + i] = B[i];
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) hll[(size_t)l * 6 + i] = H[i];
#pragma unroll
  for (int i = 0; i < 3; ++i) b_l[(size_t)l * 3 + i] = bl[i];
}

// Landmark pass, edge-parallel form (graphs whose landmarks have at most 32
// edges and whose (camera, landmark) pairs are unique): one warp per chunk of
// whole landmarks (at most 32 edges, packed on the host), one lane per edge.
// Edge loads are coalesced. The Hpl blocks of a chunk's edges are one
// contiguous range (one block per edge of a free camera, numbered in edge
// order): each lane puts its block in shared memory and the warp stores the
// range with coalesced pair stores. H_ll and b_l are summed by a segmented
// warp scan keyed by landmark (fixed shuffle order), written by the segment's
// last lane. Launched with 256 threads (8 warps).
template <typename Real>
__global__ void __launch_bounds__(256) ba_landmark_warp(BAEdges E, BAVertices V, const int* chunk_ptr, int nchunks, const int* e_lm,
                                 Real* hll, Real* hpl, double* b_l) {
  using R2 = typename Vec2<Real>::T;
  __shared__ R2 stage[8][32 * 9];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ch = blockIdx.x * (blockDim.x >> 5) + wid;
  if (ch >= nchunks) return;
  const int e0 = chunk_ptr[ch], e1 = chunk_ptr[ch + 1];
  const int k = e0 + lane;
  const bool act = k < e1;
  Real H[6] = {0, 0, 0, 0, 0, 0};
  double bl[3] = {0, 0, 0};
  int key = -1 - lane;  // distinct for idle lanes
  const int blk = act ? E.hpl[k] : -1;
  const unsigned has = __ballot_sync(0xffffffffu, blk >= 0);
  const int blk0 = (int)__reduce_min_sync(0xffffffffu, blk >= 0 ? (unsigned)blk : 0x7fffffffu);
  if (act) {
    key = e_lm[k];
    const int2 v = E.v[k];
    const double4 om = ba_om(E, k);
    double e[2], Xc[3], chi2, w;
    ba_edge_error(V, v, E.z[k], om, e, Xc, chi2, w);
    double Jpd[6], Jcd[12];
    ba_jacobians_from_xc(V.cam + (size_t)v.y * 8, Xc, V.fx, V.fy, Jpd, Jcd);
    Real Jp[6], Jc[12];
#pragma unroll
    for (int i = 0; i < 6; ++i) Jp[i] = (Real)Jpd[i];
#pragma unroll
    for (int i = 0; i < 12; ++i) Jc[i] = (Real)Jcd[i];
    const double we0 = -w * (om.x * e[0] + om.y * e[1]);
    const double we1 = -w * (om.y * e[0] + om.z * e[1]);
    const Real o00 = (Real)(w * om.x), o01 = (Real)(w * om.y), o11 = (Real)(w * om.z);
    Real A0[3], A1[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      A0[i] = Jp[i] * o00 + Jp[3 + i] * o01;
      A1[i] = Jp[i] * o01 + Jp[3 + i] * o11;
    }
    H[0] = A0[0] * Jp[0] + A1[0] * Jp[3];
    H[1] = A0[0] * Jp[1] + A1[0] * Jp[4];
    H[2] = A0[0] * Jp[2] + A1[0] * Jp[5];
    H[3] = A0[1] * Jp[1] + A1[1] * Jp[4];
    H[4] = A0[1] * Jp[2] + A1[1] * Jp[5];
    H[5] = A0[2] * Jp[2] + A1[2] * Jp[5];
#pragma unroll
    for (int i = 0; i < 3; ++i) bl[i] = Jpd[i] * we0 + Jpd[3 + i] * we1;
    if (blk >= 0) {
      Real hb[18];
#pragma unroll
      for (int r = 0; r < 6; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) hb[hpl_at(r, c)] = Jc[r] * A0[c] + Jc[6 + r] * A1[c];
      R2* o = &stage[wid][(blk - blk0) * 9];
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        R2 t;
        t.x = hb[2 * q];
        t.y = hb[2 * q + 1];
        o[q] = t;
      }
    }
  }
  // segmented inclusive scan by landmark
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int ko = __shfl_up_sync(0xffffffffu, key, off);
    Real Ho[6];
    double bo[3];
#pragma unroll
    for (int i = 0; i < 6; ++i) Ho[i] = __shfl_up_sync(0xffffffffu, H[i], off);
#pragma unroll
    for (int i = 0; i < 3; ++i) bo[i] = __shfl_up_sync(0xffffffffu, bl[i], off);
    if (lane >= off && ko == key) {
#pragma unroll
      for (int i = 0; i < 6; ++i) H[i] += Ho[i];
#pragma unroll
      for (int i = 0; i < 3; ++i) bl[i] += bo[i];
    }
  }
  const int knext = __shfl_down_sync(0xffffffffu, key, 1);
  if (act && (lane == 31 || knext != key)) {
#pragma unroll
    for (int i = 0; i < 6; ++i) hll[(size_t)key * 6 + i] = H[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) b_l[(size_t)key * 3 + i] = bl[i];
  }
  // the chunk's Hpl range (8-byte aligned in FP32, 16 in FP64), coalesced
  __syncwarp();
  const int npair = __popc(has) * 9;
  if (npair > 0) {
    R2* out = reinterpret_cast<R2*>(hpl + (size_t)blk0 * 18);
    for (int i = lane; i < npair; i += 32) out[i] = stage[wid][i];
  }
}

// Camera pass: one CTA per free camera sums H_pp = sum Jc^T Om' Jc (21 unique)
// and b_p = sum Jc^T we over the camera's edges with a fixed-order block
// reduction, and writes the full 6x6 block.
template <typename Real, int THREADS>
__global__ void __launch_bounds__(THREADS) ba_camera_pass(BACamEdges CE, BAVertices V, Real* hpp, double* b_p) {
  const int h = blockIdx.x;
  Real H[21];
  double bp[6];
#pragma unroll
  for (int i = 0; i < 21; ++i) H[i] = Real(0);
#pragma unroll
  for (int i = 0; i < 6; ++i) bp[i] = 0.0;
  const int j1 = CE.ptr[h + 1];
  // the next edge's record is loaded while this one's point is
  int j = CE.ptr[h] + threadIdx.x;
  int2 vn = make_int2(0, 0);
  double2 zn = make_double2(0.0, 0.0);
  double4 omn = make_double4(0.0, 0.0, 0.0, 0.0);
  if (j < j1) {
    vn = CE.v[j];
    zn = CE.z[j];
    omn = ba_om(CE, j);
  }
  for (; j < j1; j += THREADS) {
    const int2 v = vn;
    const double2 z = zn;
    const double4 om = omn;
    if (j + THREADS < j1) {
      vn = CE.v[j + THREADS];
      zn = CE.z[j + THREADS];
      omn = ba_om(CE, j + THREADS);
    }
    double e[2], Xc[3], chi2, w;
    ba_edge_error(V, v, z, om, e, Xc, chi2, w);
    const double* cam = V.cam + (size_t)v.y * 8;
    double Jpd[6], Jcd[12];
    ba_jacobians_from_xc(cam, Xc, V.fx, V.fy, Jpd, Jcd);
    Real Jc[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) Jc[i] = (Real)Jcd[i];
    const double we0 = -w * (om.x * e[0] + om.y * e[1]);
    const double we1 = -w * (om.y * e[0] + om.z * e[1]);
    const Real o00 = (Real)(w * om.x), o01 = (Real)(w * om.y), o11 = (Real)(w * om.z);
    Real A0[6], A1[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      A0[i] = Jc[i] * o00 + Jc[6 + i] * o01;
      A1[i] = Jc[i] * o01 + Jc[6 + i] * o11;
    }
    int t = 0;
#pragma unroll
    for (int r = 0; r < 6; ++r)
#pragma unroll
      for (int c = r; c < 6; ++c) H[t++] += A0[r] * Jc[c] + A1[r] * Jc[6 + c];
#pragma unroll
    for (int i = 0; i < 6; ++i) bp[i] += Jcd[i] * we0 + Jcd[6 + i] * we1;
  }
  __shared__ double red[THREADS / 32][27];
  block_sum_array<Real, 21, THREADS>(H, &red[0][0]);
  block_sum_array<double, 6, THREADS>(bp, &red[0][0]);
  if (threadIdx.x == 0) {
    Real* out = hpp + (size_t)h * 36;
    int t = 0;
    for (int r = 0; r < 6; ++r)
      for (int c = r; c < 6; ++c) {
        out[r * 6 + c] = H[t];
        out[c * 6 + r] = H[t];
        ++t;
      }
    for (int i = 0; i < 6; ++i) b_p[(size_t)h * 6 + i] = bp[i];
  }
}

// ---------------------------------------------------------------- Schur
// Landmark step of the Schur loop (block_solver.hpp:359-378):
// Dinv = (H_ll + lambda I)^-1 of every landmark.
template <typename Real>
__global__ void schur_landmark(const Real* hll, int Pf, double lambda_all, const double* lambda_of, Real* dinv,
                               int* nonfinite) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= Pf) return;
  const double lambda = lambda_of ? lambda_of[l] : lambda_all;  // per landmark (batched windows)
  const Real* h = hll + (size_t)l * 6;
  double A[9] = {(double)h[0] + lambda, (double)h[1], (double)h[2],
                 (double)h[1], (double)h[3] + lambda, (double)h[4],
                 (double)h[2], (double)h[4], (double)h[5] + lambda};
  double Di[9];
  if (!inverse3(A, Di)) *nonfinite = 1;
#pragma unroll
  for (int i = 0; i < 9; ++i) dinv[(size_t)l * 9 + i] = (Real)Di[i];
}

// One 6 x 3 Hpl block (18 values, hpl_at order) into registers. FP32 blocks are
// 72 bytes at a 72-byte stride: a block starts on a 16-byte boundary when its
// index is even (four 16-byte loads, then 8 bytes) and on an 8-byte one when
// odd (8 bytes, then four 16-byte loads): five loads instead of nine. FP64
// blocks (144 bytes) are nine 16-byte loads.
__device__ __forceinline__ void ldg_block18(const float* hpl, int blk, float (&b)[18]) {
  const float* base = hpl + (size_t)blk * 18;
  const bool odd = blk & 1;
  const int o4 = odd ? 2 : 0;
  const float4 u0 = __ldg(reinterpret_cast<const float4*>(base + o4));
  const float4 u1 = __ldg(reinterpret_cast<const float4*>(base + o4 + 4));
  const float4 u2 = __ldg(reinterpret_cast<const float4*>(base + o4 + 8));
  const float4 u3 = __ldg(reinterpret_cast<const float4*>(base + o4 + 12));
  const float2 w = __ldg(reinterpret_cast<const float2*>(base + (odd ? 0 : 16)));
  const float q[18] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w, u2.x,
                       u2.y, u2.z, u2.w, u3.x, u3.y, u3.z, u3.w, w.x,  w.y};
#pragma unroll
  for (int t = 0; t < 18; ++t) b[t] = odd ? (t < 2 ? q[16 + t] : q[t - 2]) : q[t];
}
__device__ __forceinline__ void ldg_block18(const double* hpl, int blk, double (&b)[18]) {
  const double2* B2 = reinterpret_cast<const double2*>(hpl + (size_t)blk * 18);
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    const double2 v = __ldg(B2 + t);
    b[2 * t] = v.x;
    b[2 * t + 1] = v.y;
  }
}

// Dense output of the Schur rows for batched windows: each camera row belongs
// to one window, whose reduced system is a dense FP64 matrix (n x n,
// row-major, at M + mat[w]). Only the lower triangle is written: the diagonal blocks whole, each upper block
// (r, c) transposed into block (c, r).
struct DenseOut {
  const int* win_of_cam;  // window of each camera row
  const int* cam;         // first camera row of each window (nw + 1)
  const long long* mat;   // offset of each window's matrix in M
  double* M;              // nullptr: no dense output
};

// Where the Schur complement goes: the row-SoA layout of sys_offset (S);
// tiles != nullptr: straight into the dense tiles of the tile PCG (block k at
// tile_off[k], scalar rows 96 apart; an off-diagonal block inside a diagonal
// tile also into its transposed place); dn.M != nullptr: into the windows'
// dense matrices.
template <typename Real>
struct SchurOut {
  Real* S;
  Real* tiles;
  const int* tile_off;
  DenseOut dn;
};

// The camera's part of a Schur row, by the CTA that has the row: BD_a =
// B_a Dinv_l of the camera's Hpl blocks, one thread per block, into BDw (shared
// memory, or the camera's part of the scratch); with B_a still in registers,
// its diagonal-block term BD_a B_a^T (upper 21 entries) and its
// right-hand-side term BD_a b_l. The sums over the blocks give S(r, r) =
// Hpp(r) + lambda I - sum_a BD_a B_a^T and, with bs != nullptr, bs_r = b_r -
// sum_a BD_a b_l(a). They are those of LANES threads (blocks LANES apart, warp
// sums, the warps in order) however many the CTA has: a row has the same bits
// whether it is formed here by schur_rows or by schur_cameras, which depends on
// the other cameras of the graph. Ends with a barrier that publishes BDw.
template <typename Real, int THREADS, int LANES = THREADS>
__device__ __forceinline__ void schur_camera(int r, const int* hc_ptr, const int* hc_blk, const int* hc_col,
                                             const Real* hpl, const Real* dinv, Real* BDw, const int* rptr,
                                             const int* s_hpp, const Real* hpp, double lambda,
                                             const SchurOut<Real>& out, const double* b_p, const double* b_l,
                                             double* bs, double (*red)[36]) {
  constexpr int TS = kTileBlocks * 6;  // scalar row stride of a tile
  const int a0 = hc_ptr[r], na = hc_ptr[r + 1] - a0;
  const int lane = threadIdx.x & 31;
  for (int first = threadIdx.x; first < LANES; first += THREADS) {
    if (THREADS < LANES && first - lane >= na) {  // no blocks for this warp: its sums are zero
      red[first >> 5][lane] = 0.0;
      continue;
    }
    Real dacc[21];
    double racc[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int u = 0; u < 21; ++u) dacc[u] = 0;
    // the next block's indices are loaded while this one's Hpl and Dinv are
    int a_next = 0, l_next = 0;
    if (first < na) {
      a_next = hc_blk[a0 + first];
      l_next = hc_col[a0 + first];
    }
    for (int t = first; t < na; t += LANES) {
      const int a = a_next, l = l_next;
      if (t + LANES < na) {
        a_next = hc_blk[a0 + t + LANES];
        l_next = hc_col[a0 + t + LANES];
      }
      const Real* Dl = dinv + (size_t)l * 9;
      Real b[18], D[9], bd[18];
      ldg_block18(hpl, a, b);
#pragma unroll
      for (int q = 0; q < 9; ++q) D[q] = Dl[q];
      Real* o = BDw + (size_t)t * 18;
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          bd[hpl_at(i, c)] = b[hpl_at(i, 0)] * D[c] + b[hpl_at(i, 1)] * D[3 + c] + b[hpl_at(i, 2)] * D[6 + c];
          o[hpl_at(i, c)] = bd[hpl_at(i, c)];
        }
      int u = 0;
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int c = i; c < 6; ++c, ++u)
          dacc[u] += bd[hpl_at(i, 0)] * b[hpl_at(c, 0)] + bd[hpl_at(i, 1)] * b[hpl_at(c, 1)] +
                     bd[hpl_at(i, 2)] * b[hpl_at(c, 2)];
      if (bs) {
        const double* bl = b_l + (size_t)l * 3;
#pragma unroll
        for (int q = 0; q < 6; ++q)
          racc[q] += (double)bd[hpl_at(q, 0)] * bl[0] + (double)bd[hpl_at(q, 1)] * bl[1] +
                     (double)bd[hpl_at(q, 2)] * bl[2];
      }
    }
    double acc[32];
#pragma unroll
    for (int u = 0; u < 21; ++u) acc[u] = (double)dacc[u];
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[21 + q] = racc[q];
#pragma unroll
    for (int u = 27; u < 32; ++u) acc[u] = 0.0;
    red[first >> 5][lane] = warp_sums32(acc);
  }
  __threadfence_block();
  __syncthreads();
  const int u = threadIdx.x;
  if (u >= 27) return;
  double sum = red[0][u];
#pragma unroll
  for (int w = 1; w < LANES / 32; ++w) sum += red[w][u];
  if (u >= 21) {
    if (bs) bs[(size_t)r * 6 + (u - 21)] = b_p[(size_t)r * 6 + (u - 21)] - sum;
    return;
  }
  int i = 0, c = u;  // u -> (i, c), i <= c, row by row
  while (c >= 6 - i) {
    c -= 6 - i;
    ++i;
  }
  c += i;
  const int rb = rptr[r], nblk = rptr[r + 1] - rb, hb = s_hpp[rb];
  double v = -sum + (i == c ? lambda : 0.0), w = -sum;
  if (hb >= 0) {
    v += (double)hpp[(size_t)hb * 36 + i * 6 + c];
    w += (double)hpp[(size_t)hb * 36 + c * 6 + i];
  }
  if (out.tiles) {
    Real* Td = out.tiles + out.tile_off[rb];
    Td[i * TS + c] = (Real)v;
    if (c != i) Td[c * TS + i] = (Real)w;
  } else if (out.dn.M) {
    const int wi = out.dn.win_of_cam[r], h0 = out.dn.cam[wi], n = 6 * (out.dn.cam[wi + 1] - h0);
    double* Dd = out.dn.M + out.dn.mat[wi] + (size_t)(r - h0) * 6 * n + (r - h0) * 6;
    Dd[(size_t)i * n + c] = (double)(Real)v;
    if (c != i) Dd[(size_t)c * n + i] = (double)(Real)w;
  } else {
    Real* Sr = out.S + (size_t)rb * 36;
    Sr[(size_t)(i * 6 + c) * nblk] = (Real)v;
    if (c != i) Sr[(size_t)(c * 6 + i) * nblk] = (Real)w;
  }
}

// An off-diagonal block S(r, cc) = [Hpp(r, cc)] - sum BD_a B_b^T (block j of
// row r), lane (g, t) = (lane / 4, lane % 4) holding the sum's entries (g, 2 t)
// and (g, 2 t + 1)
template <typename Real>
__device__ __forceinline__ void schur_store(const SchurOut<Real>& out, int r, int rb, int nblk, int j, int cc, int off,
                                            const Real* hpp, double acc0, double acc1) {
  constexpr int TS = kTileBlocks * 6;
  using R2 = typename Vec2<Real>::T;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (g >= 6 || t > 2) return;
  double w0 = -acc0, w1 = -acc1;
  if (hpp) {
    w0 += (double)hpp[g * 6 + 2 * t];
    w1 += (double)hpp[g * 6 + 2 * t + 1];
  }
  if (out.tiles) {
    R2 pr;
    pr.x = (Real)w0;
    pr.y = (Real)w1;
    __stcs(reinterpret_cast<R2*>(out.tiles + off + g * TS + 2 * t), pr);
    if (r / kTileBlocks == cc / kTileBlocks) {
      Real* base = out.tiles + (size_t)(off / (TS * TS)) * (TS * TS);
      Real* m = base + ((cc % kTileBlocks) * 6 + 2 * t) * TS + (r % kTileBlocks) * 6 + g;
      __stcs(m, pr.x);
      __stcs(m + TS, pr.y);
    }
  } else if (out.dn.M) {
    // block (r, cc) transposed into the lower triangle of the window's matrix
    const int wi = out.dn.win_of_cam[r], h0 = out.dn.cam[wi], n = 6 * (out.dn.cam[wi + 1] - h0);
    double* D = out.dn.M + out.dn.mat[wi] + ((size_t)(cc - h0) * 6 + 2 * t) * n + (r - h0) * 6 + g;
    D[0] = (double)(Real)w0;
    D[n] = (double)(Real)w1;
  } else {
    Real* Sr = out.S + (size_t)rb * 36;
    __stcs(Sr + (size_t)(g * 6 + 2 * t) * nblk + j, (Real)w0);
    __stcs(Sr + (size_t)(g * 6 + 2 * t + 1) * nblk + j, (Real)w1);
  }
}

// Schur complement by camera rows (block_solver.hpp:343-433): one CTA per
// free camera r of `rows` (the ones with the most pairs first). schur_camera
// stages the camera's BD_a blocks and forms the diagonal block and the reduced
// right-hand side; each off-diagonal block S(r, c) = [Hpp(r, c)] -
// sum BD_a B_b^T is summed by a warp over its co-observing pairs.
// pose_blocks: some off-diagonal blocks have an Hpp part (a pose edge set).
//
// A warp takes four pairs per FP64 tensor-core step (m8n8k4): the product
// sum over pairs of BD_a B_b^T is one over k = (pair, component), and the
// components of a pair can go into different steps, so lane (g, t) holds row
// g of pair t and step m takes component m: two loads per four pairs for each
// operand, of runs of 96 and 48 bytes (hpl_at). Sums are FP64 for both storage
// types, in the order of the pair list by fours: a fixed order. Rows with
// fewer blocks than a CTA has warps cut each block's pairs over two or four
// warps (sums in warp order).
//
// Bound by latency: the gathers (one Hpl block per pair, from L2 and DRAM),
// the chain of a step, and the camera's part, during which no gather is under
// way. On the 1000-camera graph in FP64 (3.7 M pairs, 7.5 per block) it takes
// 0.33 ms (0.35 with vector FMAs, two lanes per block); on windows of 10 to 60
// cameras (longer lists, few rows) 96 windows take 342 against 431 us, and one
// launch serves every list length, where the lanes per block had to be chosen
// by it (123 cameras: 42 us in one launch against 109 in three).
template <typename Real, int THREADS, bool STAGE>
__global__ void __launch_bounds__(THREADS, sizeof(Real) == 4 ? 2 : 1)
    schur_rows(const int* rows, const int* hc_ptr, const int* hc_blk, const int* hc_col, const Real* hpl,
               const Real* dinv, Real* bdc, const int* rptr, const int* rcol, const int* pair_ptr,
               const int2* pairs, const int* s_hpp, const Real* hpp, double lambda_all, const double* lambda_of,
               SchurOut<Real> out, const double* b_p, const double* b_l, double* bs, bool pose_blocks) {
  constexpr int WARPS = THREADS / 32;
  using R2 = typename Vec2<Real>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[WARPS][36];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = rows[blockIdx.x];
  const int rb = rptr[r], nblk = rptr[r + 1] - rb, noff = nblk - 1;
  // the row's pair list comes into L2 while the camera's blocks are staged
  if (noff > 0) {
    const char* p0 = reinterpret_cast<const char*>(pairs + pair_ptr[rb + 1]);
    const char* p1 = reinterpret_cast<const char*>(pairs + pair_ptr[rb + nblk]);
    for (const char* p = p0 + 128 * threadIdx.x; p < p1; p += 128 * THREADS)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  }
  Real* const BDw = STAGE ? reinterpret_cast<Real*>(smem_raw) : bdc + (size_t)hc_ptr[r] * 18;
  schur_camera<Real, THREADS>(r, hc_ptr, hc_blk, hc_col, hpl, dinv, BDw, rptr, s_hpp, hpp,
                              lambda_of ? lambda_of[r] : lambda_all, out, b_p, b_l, bs, red);
  const int g = lane >> 2, t = lane & 3;
  const bool in = g < 6;  // the fragment's rows 6 and 7 are empty
  auto gather = [&](int blk, bool valid, Real (&b)[3]) {
    const Real* B = hpl + (size_t)blk * 18;
    R2 u;
    u.x = u.y = Real(0);
    b[2] = Real(0);
    if (valid && in) {
      u = __ldg(reinterpret_cast<const R2*>(B) + g);
      b[2] = __ldg(B + 12 + g);
    }
    b[0] = u.x;
    b[1] = u.y;
  };
  auto product = [&](int a, const Real (&b)[3], double (&acc)[2]) {
    double x[3] = {0.0, 0.0, 0.0};
    if (a >= 0 && in) {
      const Real* D = BDw + (size_t)a * 18;
      const R2 u = *(reinterpret_cast<const R2*>(D) + g);
      x[0] = (double)u.x;
      x[1] = (double)u.y;
      x[2] = (double)D[12 + g];
    }
#pragma unroll
    for (int m = 2; m >= 0; --m)
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                   : "+d"(acc[0]), "+d"(acc[1])
                   : "d"(x[m]), "d"((double)b[m]));
  };
  auto store = [&](int j, double acc0, double acc1, int hb, int off, int cc) {
    schur_store(out, r, rb, nblk, j, cc, off, hb >= 0 ? hpp + (size_t)hb * 36 : nullptr, acc0, acc1);
  };
  const int split = noff * 4 <= WARPS ? 4 : noff * 2 <= WARPS ? 2 : 1;
  if (split > 1) {
    const int j = 1 + warp / split, sub = warp % split;
    double acc[2] = {0.0, 0.0};
    if (j < nblk) {
      const int p1 = pair_ptr[rb + j + 1];
      int p = pair_ptr[rb + j] + 4 * sub + t;
      int2 nx = p < p1 ? __ldcs(pairs + p) : make_int2(-1, 0);
      for (; p - t < p1; p += 4 * split) {
        const bool valid = p < p1;
        const int2 pr = nx;
        if (p + 4 * split < p1) nx = __ldcs(pairs + p + 4 * split);
        Real b[3];
        gather(pr.y, valid, b);
        product(valid ? pr.x : -1, b, acc);
      }
    }
    __syncthreads();  // red is read above
    if (in && t < 3) {
      red[warp][g * 6 + 2 * t] = acc[0];
      red[warp][g * 6 + 2 * t + 1] = acc[1];
    }
    __syncthreads();
    if (j < nblk && sub == 0 && in && t < 3) {
      for (int w = 1; w < split; ++w) {
        acc[0] += red[warp + w][g * 6 + 2 * t];
        acc[1] += red[warp + w][g * 6 + 2 * t + 1];
      }
      const int k = rb + j;
      store(j, acc[0], acc[1], pose_blocks ? s_hpp[k] : -1, out.tiles ? out.tile_off[k] : 0, rcol[k]);
    }
    return;
  }
  // This warp's blocks are j = 1 + warp + WARPS i; lane i % 32 loads what
  // belongs to block i (its pairs' range, its column and place), so that a
  // warp waits for it once in 32 blocks and not at each. A step is up to
  // eight pairs of one block; the pair indices of step n + 3 and the blocks of
  // step n + 2 are on their way while step n is multiplied (four stages,
  // unrolled so that no register waiting for a load is moved).
  struct Step {
    int i, p, p1;  // block of the batch (>= mine: none), first pair, the block's end
  };
  for (int i0 = 0; 1 + warp + WARPS * i0 < nblk; i0 += 32) {
    const int mine = min(32, (nblk - 2 - warp - WARPS * i0) / WARPS + 1);
    const int jl = 1 + warp + WARPS * (i0 + lane);
    int m_p0 = 0, m_p1 = 0, m_col = 0, m_off = 0, m_hb = -1;
    if (lane < mine) {
      m_p0 = pair_ptr[rb + jl];
      m_p1 = pair_ptr[rb + jl + 1];
      m_col = rcol[rb + jl];
      if (out.tiles) m_off = out.tile_off[rb + jl];
      if (pose_blocks) m_hb = s_hpp[rb + jl];
    }
    auto open = [&](int i) {
      return Step{i, __shfl_sync(0xffffffffu, m_p0, i & 31), __shfl_sync(0xffffffffu, m_p1, i & 31)};
    };
    auto after = [&](const Step& st) {
      if (st.i < mine && st.p + 8 < st.p1) return Step{st.i, st.p + 8, st.p1};
      return open(st.i + 1);
    };
    auto index = [&](const Step& st, int2 (&pr)[2]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int p = st.p + 4 * h + t;
        pr[h] = st.i < mine && p < st.p1 ? __ldcs(pairs + p) : make_int2(-1, -1);
      }
    };
    auto blocks = [&](const int2 (&pr)[2], Real (&b)[2][3]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) gather(max(pr[h].y, 0), pr[h].y >= 0, b[h]);
    };
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};  // the two halves of the steps: independent chains of products
    int2 ix[4][2];
    Real bv[4][2][3];
    Step s0 = open(0);
    index(s0, ix[0]);
    Step s1 = after(s0);
    index(s1, ix[1]);
    Step s2 = after(s1);
    index(s2, ix[2]);
    blocks(ix[0], bv[0]);
    blocks(ix[1], bv[1]);
    auto stage = [&](auto cur) {
      constexpr int C = decltype(cur)::value;
      if (s0.i >= mine) return false;
      const Step s3 = after(s2);
      index(s3, ix[(C + 3) & 3]);
      blocks(ix[(C + 2) & 3], bv[(C + 2) & 3]);
      product(ix[C][0].x, bv[C][0], acc[0]);
      if (s0.p + 4 < s0.p1) product(ix[C][1].x, bv[C][1], acc[1]);
      if (s1.i != s0.i) {
        const int hb = __shfl_sync(0xffffffffu, m_hb, s0.i), off = __shfl_sync(0xffffffffu, m_off, s0.i);
        const int cc = __shfl_sync(0xffffffffu, m_col, s0.i);
        store(1 + warp + WARPS * (i0 + s0.i), acc[0][0] + acc[1][0], acc[0][1] + acc[1][1], hb, off, cc);
        acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = 0.0;
      }
      s0 = s1;
      s1 = s2;
      s2 = s3;
      return true;
    };
    while (stage(std::integral_constant<int, 0>()) && stage(std::integral_constant<int, 1>()) &&
           stage(std::integral_constant<int, 2>()) && stage(std::integral_constant<int, 3>())) {
    }
  }
}

// Warps of a CTA of schur_rows on FP64 values: the sums of the two launches
// below are those of that many
constexpr int kSchurWarps = 16;

// The two parts of schur_rows as two launches, for graphs with a camera whose
// blocks do not fit in shared memory: the BD_a go through global memory anyway,
// and the blocks no longer wait for their camera's part nor a camera for the
// blocks of the one before it.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
    schur_cameras(const int* rows, const int* hc_ptr, const int* hc_blk, const int* hc_col, const double* hpl,
                  const double* dinv, double* bdc, const int* rptr, const int* s_hpp, const double* hpp, double lambda_all,
                  const double* lambda_of, SchurOut<double> out, const double* b_p, const double* b_l, double* bs) {
  __shared__ double red[kSchurWarps][36];
  const int r = rows[blockIdx.x];
  schur_camera<double, THREADS, 32 * kSchurWarps>(r, hc_ptr, hc_blk, hc_col, hpl, dinv, bdc + (size_t)hc_ptr[r] * 18, rptr, s_hpp,
                                       hpp, lambda_of ? lambda_of[r] : lambda_all, out, b_p, b_l, bs, red);
}

// A warp per off-diagonal block, whose fours of pairs go to two sums in turn;
// the blocks of rows that schur_rows cuts over four warps (quads, nquad of
// them) take four warps here too, in CTAs of their own, the last ones (4% of
// both launches less than as the first ones). The sums are those of schur_rows.
// Bound by the gathers of both operands. 96 windows of 10 to 60 cameras (2 M
// edges, Hpl 290 MB in FP64): schur_cameras and schur_blocks 271 us together
// (580 MB in the first), against 335 us for schur_rows, which has 16 warps per
// SM to hide the gathers with and none during a camera's part.
static __global__ void __launch_bounds__(256, 3)
    schur_blocks(int nnzb, const int* quads, int nquad, const int* brow, const int* hc_ptr, const double* hpl,
                 const double* bdc, const int* rptr, const int* rcol, const int* pair_ptr, const int2* pairs,
                 const int* s_hpp, const double* hpp, SchurOut<double> out, bool pose_blocks) {
  __shared__ double red[8][36];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = lane & 3, g = lane >> 2;
  const bool in = g < 6;
  const int plain_ctas = (nnzb + 7) / 8;
  const bool quad = (int)blockIdx.x >= plain_ctas;
  int k = (int)blockIdx.x * 8 + warp;
  if (quad) {
    const int q = ((int)blockIdx.x - plain_ctas) * 2 + (warp >> 2);
    k = q < nquad ? quads[q] : nnzb;
  }
  if (!quad && k >= nnzb) return;
  int r = 0, rb = 0, nblk = 0, j = 0, p = 0, p1 = 0;
  const double* BD = bdc;
  if (k < nnzb) {
    r = brow[k];
    rb = rptr[r];
    nblk = rptr[r + 1] - rb;
    j = k - rb;
    p = pair_ptr[k];
    p1 = pair_ptr[k + 1];
    BD = bdc + (size_t)hc_ptr[r] * 18;
  }
  auto index = [&](int p) { return p + t < p1 ? __ldcs(pairs + p + t) : make_int2(-1, -1); };
  auto gather = [&](const double* base, int blk, double (&b)[3]) {
    double2 u = make_double2(0.0, 0.0);
    b[2] = 0.0;
    if (blk >= 0 && in) {
      const double* B = base + (size_t)blk * 18;
      u = __ldg(reinterpret_cast<const double2*>(B) + g);
      b[2] = __ldg(B + 12 + g);
    }
    b[0] = u.x;
    b[1] = u.y;
  };
  auto product = [&](const double (&x)[3], const double (&b)[3], double (&c)[2]) {
#pragma unroll
    for (int m = 2; m >= 0; --m)
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                   : "+d"(c[0]), "+d"(c[1])
                   : "d"(x[m]), "d"(b[m]));
  };
  // fours of pairs, two at a time, into one sum or two; the indices of the step
  // after next and the operands of the next are on their way
  auto sums = [&](auto second, auto step, auto& acc) {
    constexpr int H = decltype(second)::value, STEP = decltype(step)::value, N = sizeof(acc) / sizeof(acc[0]);
    int2 i0[2] = {index(p), index(p + H)}, i1[2] = {index(p + STEP), index(p + STEP + H)};
    double x[2][3], b[2][3];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      gather(BD, i0[h].x, x[h]);
      gather(hpl, i0[h].y, b[h]);
    }
    for (; p < p1; p += STEP) {
      const int2 i2[2] = {index(p + 2 * STEP), index(p + 2 * STEP + H)};
      double xn[2][3], bn[2][3];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        gather(BD, i1[h].x, xn[h]);
        gather(hpl, i1[h].y, bn[h]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) product(x[h], b[h], acc[h % N]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        i1[h] = i2[h];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          x[h][m] = xn[h][m];
          b[h][m] = bn[h][m];
        }
      }
    }
  };
  double s0, s1;
  if (quad) {
    double acc[1][2] = {{0.0, 0.0}};
    p += 4 * (warp & 3);
    sums(std::integral_constant<int, 16>(), std::integral_constant<int, 32>(), acc);
    if (in && t < 3) {
      red[warp][g * 6 + 2 * t] = acc[0][0];
      red[warp][g * 6 + 2 * t + 1] = acc[0][1];
    }
    __syncthreads();
    if ((warp & 3) || k >= nnzb || !in || t > 2) return;
    s0 = acc[0][0];
    s1 = acc[0][1];
    for (int w = 1; w < 4; ++w) {
      s0 += red[warp + w][g * 6 + 2 * t];
      s1 += red[warp + w][g * 6 + 2 * t + 1];
    }
  } else {
    if (j == 0 || (nblk - 1) * 4 <= kSchurWarps) return;  // schur_cameras; the last CTAs
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    sums(std::integral_constant<int, 4>(), std::integral_constant<int, 8>(), acc);
    s0 = acc[0][0] + acc[1][0];
    s1 = acc[0][1] + acc[1][1];
  }
  const int hb = pose_blocks ? s_hpp[k] : -1;
  schur_store(out, r, rb, nblk, j, rcol[k], out.tiles ? out.tile_off[k] : 0,
              hb >= 0 ? hpp + (size_t)hb * 36 : nullptr, s0, s1);
}

// FP32 rows with short pair lists: the off-diagonal blocks by two lanes each
// (lane parity = rows 0-2 or 3-5, 18 FP32 accumulators each) over their pairs
// in landmark order, two gathers in flight per lane. FP32 FMAs need no
// conversion to FP64 fragments: 228 us per pass of the 1000-camera graph (7.5
// pairs per block) against 245 for schur_rows; lists of 12 and more pairs
// leave too few lanes busy here.
template <int THREADS, bool STAGE>
__global__ void __launch_bounds__(THREADS, 2)
    schur_rows_short(const int* rows, const int* hc_ptr, const int* hc_blk, const int* hc_col, const float* hpl,
                     const float* dinv, float* bdc, const int* rptr, const int* rcol, const int* pair_ptr,
                     const int2* pairs, const int* s_hpp, const float* hpp, double lambda_all,
                     const double* lambda_of, SchurOut<float> out, const double* b_p, const double* b_l, double* bs,
                     bool pose_blocks) {
  constexpr int TS = kTileBlocks * 6;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[THREADS / 32][36];
  const int r = rows[blockIdx.x];
  const int rb = rptr[r], nblk = rptr[r + 1] - rb;
  float* const BDw = STAGE ? reinterpret_cast<float*>(smem_raw) : bdc + (size_t)hc_ptr[r] * 18;
  schur_camera<float, THREADS>(r, hc_ptr, hc_blk, hc_col, hpl, dinv, BDw, rptr, s_hpp, hpp,
                               lambda_of ? lambda_of[r] : lambda_all, out, b_p, b_l, bs, red);
  const int half = threadIdx.x & 1;
  for (int j = 1 + (int)threadIdx.x / 2; j < nblk; j += THREADS / 2) {
    const int k = rb + j;
    float acc[18];
#pragma unroll
    for (int t = 0; t < 18; ++t) acc[t] = 0.f;
    // two pairs per step: their index and Hpl loads are independent;
    // accumulation stays in pair order. The pair list and S are touched once
    // per pass: streamed, so the L2 lines go to the Hpl blocks gathered again
    auto accum = [&](int a, const float (&b)[18]) {
      const float* D = BDw + (size_t)a * 18;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int q = half * 3 + i;
        const float d0 = D[2 * q], d1 = D[2 * q + 1], d2 = D[12 + q];
#pragma unroll
        for (int c = 0; c < 6; ++c)
          acc[i * 6 + c] += d0 * b[hpl_at(c, 0)] + d1 * b[hpl_at(c, 1)] + d2 * b[hpl_at(c, 2)];
      }
    };
    int p = pair_ptr[k];
    const int p1 = pair_ptr[k + 1];
    // the next step's pair indices are loaded while this step's blocks are
    int2 na2 = make_int2(0, 0), nb2 = make_int2(0, 0);
    if (p < p1) na2 = __ldcs(pairs + p);
    if (p + 1 < p1) nb2 = __ldcs(pairs + p + 1);
    for (; p + 1 < p1; p += 2) {
      const int2 pa = na2, pb = nb2;
      if (p + 2 < p1) na2 = __ldcs(pairs + p + 2);
      if (p + 3 < p1) nb2 = __ldcs(pairs + p + 3);
      float ba[18], bb[18];
      ldg_block18(hpl, pa.y, ba);
      ldg_block18(hpl, pb.y, bb);
      accum(pa.x, ba);
      accum(pb.x, bb);
    }
    if (p < p1) {
      float ba[18];
      ldg_block18(hpl, na2.y, ba);
      accum(na2.x, ba);
    }
    const int hb = pose_blocks ? s_hpp[k] : -1, cc = rcol[k];
    float v[18];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        double w = -(double)acc[i * 6 + c];
        if (hb >= 0) w += (double)hpp[(size_t)hb * 36 + (half * 3 + i) * 6 + c];
        v[i * 6 + c] = (float)w;
      }
    if (out.tiles) {
      // this lane's three scalar rows of the block, in pairs (8-byte aligned)
      const int off = out.tile_off[k];
      float* T = out.tiles + off + half * 3 * TS;
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 6; c += 2)
          __stcs(reinterpret_cast<float2*>(T + i * TS + c), make_float2(v[i * 6 + c], v[i * 6 + c + 1]));
      if (r / kTileBlocks == cc / kTileBlocks) {
        float* base = out.tiles + (size_t)(off / (TS * TS)) * (TS * TS);
        const int lr = (r % kTileBlocks) * 6 + half * 3, lc = (cc % kTileBlocks) * 6;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < 6; ++c) __stcs(base + (lc + c) * TS + lr + i, v[i * 6 + c]);
      }
    } else if (out.dn.M) {
      const int wi = out.dn.win_of_cam[r], h0 = out.dn.cam[wi], n = 6 * (out.dn.cam[wi + 1] - h0);
      double* D = out.dn.M + out.dn.mat[wi] + (size_t)(cc - h0) * 6 * n + (r - h0) * 6 + half * 3;
#pragma unroll
      for (int c = 0; c < 6; ++c)
#pragma unroll
        for (int i = 0; i < 3; ++i) D[(size_t)c * n + i] = (double)v[i * 6 + c];
    } else {
      float* Sr = out.S + (size_t)rb * 36;
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 6; ++c) __stcs(Sr + (size_t)((half * 3 + i) * 6 + c) * nblk + j, v[i * 6 + c]);
    }
  }
}

// db_l = Dinv_l r_l
template <typename Real>
__global__ void schur_db(const Real* dinv, const double* r_l, int Pf, double* db) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= Pf) return;
  const Real* D = dinv + (size_t)l * 9;
  const double* rl = r_l + (size_t)l * 3;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    db[(size_t)l * 3 + i] = (double)D[i * 3] * rl[0] + (double)D[i * 3 + 1] * rl[1] + (double)D[i * 3 + 2] * rl[2];
}

// Reduced right-hand side for a given (r_p, r_l) (block_solver.hpp:366-392,
// 429-433): one CTA per free camera, bs = r_p - sum_a B_a db_l(a), threads
// over the camera's Hpl blocks (camera-major lists), fixed-order reduction.
template <typename Real, int THREADS>
__global__ void __launch_bounds__(THREADS) schur_rhs(const int* hc_ptr, const int* hc_blk, const int* hc_col,
                                                     const Real* hpl, const double* db, const double* r_p,
                                                     double* bs) {
  const int h = blockIdx.x;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  const int e1 = hc_ptr[h + 1];
  for (int p = hc_ptr[h] + threadIdx.x; p < e1; p += THREADS) {
    const double* d = db + (size_t)hc_col[p] * 3;
    const Real* B = hpl + (size_t)hc_blk[p] * 18;
#pragma unroll
    for (int q = 0; q < 6; ++q)
      acc[q] += (double)B[hpl_at(q, 0)] * d[0] + (double)B[hpl_at(q, 1)] * d[1] + (double)B[hpl_at(q, 2)] * d[2];
  }
  __shared__ double red[THREADS / 32][6];
  block_sum_array<double, 6, THREADS>(acc, &red[0][0]);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 6; ++q) bs[(size_t)h * 6 + q] = r_p[(size_t)h * 6 + q] - acc[q];
  }
}

// Landmark back-substitution (block_solver.hpp:449-474):
// x_l = Dinv (r_l - sum_a B_a^T x_p(row a))
template <typename Real>
__global__ void ba_backsub(const int* hb_ptr, const int* hpl_row, int Pf, const Real* hpl, const Real* dinv,
                           const double* r_l, const double* x_p, double* x_l) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= Pf) return;
  double cl[3] = {r_l[(size_t)l * 3], r_l[(size_t)l * 3 + 1], r_l[(size_t)l * 3 + 2]};
  const int b1 = hb_ptr[l + 1];
  for (int a = hb_ptr[l]; a < b1; ++a) {
    const Real* B = hpl + (size_t)a * 18;
    const double* xp = x_p + (size_t)hpl_row[a] * 6;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double s = 0.0;
#pragma unroll
      for (int r = 0; r < 6; ++r) s += (double)B[hpl_at(r, c)] * xp[r];
      cl[c] -= s;
    }
  }
  const Real* D = dinv + (size_t)l * 9;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    x_l[(size_t)l * 3 + i] = (double)D[i * 3] * cl[0] + (double)D[i * 3 + 1] * cl[1] + (double)D[i * 3 + 2] * cl[2];
}

// Back-substitution, one warp per chunk of whole landmarks (lane per edge,
// each edge of a free camera owns one Hpl block when the chunks exist),
// segmented warp scan by landmark.
template <typename Real>
__global__ void ba_backsub_warp(const int* e_hpl, const int* hpl_row, const int* chunk_ptr, int nchunks,
                                const int* e_lm, const Real* hpl, const Real* dinv, const double* r_l,
                                const double* x_p, double* x_l) {
  const int lane = threadIdx.x & 31;
  const int ch = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (ch >= nchunks) return;
  const int e0 = chunk_ptr[ch], e1 = chunk_ptr[ch + 1];
  const int k = e0 + lane;
  const bool act = k < e1;
  double acc[3] = {0, 0, 0};
  int key = -1 - lane;
  if (act) {
    key = e_lm[k];
    const int blk = e_hpl[k];
    if (blk >= 0) {
      const Real* B = hpl + (size_t)blk * 18;
      const double* xp = x_p + (size_t)hpl_row[blk] * 6;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double t = 0.0;
#pragma unroll
        for (int r = 0; r < 6; ++r) t += (double)B[hpl_at(r, c)] * xp[r];
        acc[c] = t;
      }
    }
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int ko = __shfl_up_sync(0xffffffffu, key, off);
    double ao[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) ao[i] = __shfl_up_sync(0xffffffffu, acc[i], off);
    if (lane >= off && ko == key) {
#pragma unroll
      for (int i = 0; i < 3; ++i) acc[i] += ao[i];
    }
  }
  const int knext = __shfl_down_sync(0xffffffffu, key, 1);
  if (act && (lane == 31 || knext != key)) {
    const double cl[3] = {r_l[(size_t)key * 3] - acc[0], r_l[(size_t)key * 3 + 1] - acc[1],
                          r_l[(size_t)key * 3 + 2] - acc[2]};
    const Real* D = dinv + (size_t)key * 9;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      x_l[(size_t)key * 3 + i] = (double)D[i * 3] * cl[0] + (double)D[i * 3 + 1] * cl[1] + (double)D[i * 3 + 2] * cl[2];
  }
}

// Matrix-free FP64 residual of the damped normal equations for the
// mixed-precision refinement, r = b - (J^T Om' J + lambda I) x, with the
// Jacobians recomputed in FP64 from the edges (no FP32 Hessian involved).
// Landmark side: one thread per free landmark over its edges.
static __global__ void ba_resid64_landmark(BAEdges E, BAVertices V, const int* l_ptr, int Pf, const int* pose_h,
                                    double lambda, const double* b_l, const double* x_p, const double* x_l,
                                    double* r_l) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= Pf) return;
  const double* xl = x_l + (size_t)l * 3;
  double acc[3] = {lambda * xl[0], lambda * xl[1], lambda * xl[2]};
  const int k1 = l_ptr[l + 1];
  for (int k = l_ptr[l]; k < k1; ++k) {
    const int2 v = E.v[k];
    const double4 om = ba_om(E, k);
    double e[2], Xc[3], chi2, w;
    ba_edge_error(V, v, E.z[k], om, e, Xc, chi2, w);
    double Jp[6], Jc[12];
    ba_jacobians_from_xc(V.cam + (size_t)v.y * 8, Xc, V.fx, V.fy, Jp, Jc);
    double u0 = Jp[0] * xl[0] + Jp[1] * xl[1] + Jp[2] * xl[2];
    double u1 = Jp[3] * xl[0] + Jp[4] * xl[1] + Jp[5] * xl[2];
    const int h = pose_h[v.y];
    if (h >= 0) {
      const double* xp = x_p + (size_t)h * 6;
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        u0 += Jc[q] * xp[q];
        u1 += Jc[6 + q] * xp[q];
      }
    }
    const double o0 = w * (om.x * u0 + om.y * u1), o1 = w * (om.y * u0 + om.z * u1);
#pragma unroll
    for (int i = 0; i < 3; ++i) acc[i] += Jp[i] * o0 + Jp[3 + i] * o1;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) r_l[(size_t)l * 3 + i] = b_l[(size_t)l * 3 + i] - acc[i];
}

// Landmark side, one warp per chunk of whole landmarks (<= 32 edges, lane
// per edge) with a segmented warp scan, as ba_landmark_warp.
static __global__ void ba_resid64_landmark_warp(BAEdges E, BAVertices V, const int* chunk_ptr, int nchunks,
                                                const int* e_lm, const int* pose_h, double lambda, const double* b_l,
                                                const double* x_p, const double* x_l, double* r_l) {
  const int lane = threadIdx.x & 31;
  const int ch = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (ch >= nchunks) return;
  const int e0 = chunk_ptr[ch], e1 = chunk_ptr[ch + 1];
  const int k = e0 + lane;
  const bool act = k < e1;
  double acc[3] = {0, 0, 0};
  int key = -1 - lane;  // distinct for idle lanes
  if (act) {
    key = e_lm[k];
    const double* xl = x_l + (size_t)key * 3;
    const int2 v = E.v[k];
    const double4 om = ba_om(E, k);
    double e[2], Xc[3], chi2, w;
    ba_edge_error(V, v, E.z[k], om, e, Xc, chi2, w);
    double Jp[6], Jc[12];
    ba_jacobians_from_xc(V.cam + (size_t)v.y * 8, Xc, V.fx, V.fy, Jp, Jc);
    double u0 = Jp[0] * xl[0] + Jp[1] * xl[1] + Jp[2] * xl[2];
    double u1 = Jp[3] * xl[0] + Jp[4] * xl[1] + Jp[5] * xl[2];
    const int h = pose_h[v.y];
    if (h >= 0) {
      const double* xp = x_p + (size_t)h * 6;
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        u0 += Jc[q] * xp[q];
        u1 += Jc[6 + q] * xp[q];
      }
    }
    const double o0 = w * (om.x * u0 + om.y * u1), o1 = w * (om.y * u0 + om.z * u1);
#pragma unroll
    for (int i = 0; i < 3; ++i) acc[i] = Jp[i] * o0 + Jp[3 + i] * o1;
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int ko = __shfl_up_sync(0xffffffffu, key, off);
    double ao[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) ao[i] = __shfl_up_sync(0xffffffffu, acc[i], off);
    if (lane >= off && ko == key) {
#pragma unroll
      for (int i = 0; i < 3; ++i) acc[i] += ao[i];
    }
  }
  const int knext = __shfl_down_sync(0xffffffffu, key, 1);
  if (act && (lane == 31 || knext != key)) {
    const double* xl = x_l + (size_t)key * 3;
#pragma unroll
    for (int i = 0; i < 3; ++i) r_l[(size_t)key * 3 + i] = b_l[(size_t)key * 3 + i] - lambda * xl[i] - acc[i];
  }
}

// Camera side: one CTA per free camera over its edges, fixed-order reduction.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) ba_resid64_camera(BACamEdges CE, BAVertices V, const int* point_l,
                                                             double lambda, const double* b_p, const double* x_p,
                                                             const double* x_l, double* r_p) {
  const int h = blockIdx.x;
  const double* xp = x_p + (size_t)h * 6;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  const int j1 = CE.ptr[h + 1];
  for (int j = CE.ptr[h] + threadIdx.x; j < j1; j += THREADS) {
    const int2 v = CE.v[j];
    const double4 om = ba_om(CE, j);
    double e[2], Xc[3], chi2, w;
    ba_edge_error(V, v, CE.z[j], om, e, Xc, chi2, w);
    double Jp[6], Jc[12];
    ba_jacobians_from_xc(V.cam + (size_t)v.y * 8, Xc, V.fx, V.fy, Jp, Jc);
    double u0 = 0.0, u1 = 0.0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      u0 += Jc[q] * xp[q];
      u1 += Jc[6 + q] * xp[q];
    }
    const int l = point_l[v.x];
    if (l >= 0) {
      const double* xl = x_l + (size_t)l * 3;
      u0 += Jp[0] * xl[0] + Jp[1] * xl[1] + Jp[2] * xl[2];
      u1 += Jp[3] * xl[0] + Jp[4] * xl[1] + Jp[5] * xl[2];
    }
    const double o0 = w * (om.x * u0 + om.y * u1), o1 = w * (om.y * u0 + om.z * u1);
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] += Jc[q] * o0 + Jc[6 + q] * o1;
  }
  __shared__ double red[THREADS / 32][6];
  block_sum_array<double, 6, THREADS>(acc, &red[0][0]);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 6; ++q) r_p[(size_t)h * 6 + q] = b_p[(size_t)h * 6 + q] - lambda * xp[q] - acc[q];
  }
}

// SparseOptimizer::update (sparse_optimizer.cpp:457-468) with
// VertexSE3Expmap::oplusImpl (g2o/types/sba/vertex_se3_expmap.cpp:48-51):
// T <- exp(dx) * T; VertexPointXYZ: p <- p + dx (vertex_pointxyz.h:47-50)
// cam_bak / pt_bak (nullptr: none): the estimates before the update. still: a
// camera whose step is zero keeps its bits (exp(0) T normalizes the quaternion):
// a finished window of a batch, in the rounds that others need
static __global__ void ba_oplus(BAVertices V, int Cf, int Pf, const double* x, int* nonfinite, double* cam_bak,
                                double* pt_bak, bool still) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < Cf) {
    double u[6];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      u[i] = x[(size_t)t * 6 + i];
      bad |= !isfinite(u[i]);
    }
    if (bad) *nonfinite = 1;
    double* cam = V.cam + (size_t)V.free_pose[t] * 8;
    if (cam_bak) {
      double* s = cam_bak + (size_t)V.free_pose[t] * 8;
#pragma unroll
      for (int i = 0; i < 7; ++i) s[i] = cam[i];
    }
    if (still && u[0] == 0.0 && u[1] == 0.0 && u[2] == 0.0 && u[3] == 0.0 && u[4] == 0.0 && u[5] == 0.0) return;
    SE3Q<double> T;
    T.q = Q4<double>{cam[0], cam[1], cam[2], cam[3]};
    T.t[0] = cam[4]; T.t[1] = cam[5]; T.t[2] = cam[6];
    SE3Q<double> R = se3q_mul(se3q_exp(u), T);
    cam[0] = R.q.x; cam[1] = R.q.y; cam[2] = R.q.z; cam[3] = R.q.w;
    cam[4] = R.t[0]; cam[5] = R.t[1]; cam[6] = R.t[2];
  } else if (t < Cf + Pf) {
    const int l = t - Cf;
    double* p = V.pt + (size_t)V.free_point[l] * 4;
    const double* u = x + (size_t)Cf * 6 + (size_t)l * 3;
    if (!isfinite(u[0]) || !isfinite(u[1]) || !isfinite(u[2])) *nonfinite = 1;
    if (pt_bak) {
      double* s = pt_bak + (size_t)V.free_point[l] * 4;
      s[0] = p[0];
      s[1] = p[1];
      s[2] = p[2];
    }
    p[0] += u[0];
    p[1] += u[1];
    p[2] += u[2];
  }
}

// max |diag| over Hpp and H_ll (computeLambdaInit,
// optimization_algorithm_levenberg.cpp:155-167): partial maxima per block
// sharded bundle adjustment: the diagonal of this rank's part of Hpp
template <typename Real>
__global__ void ba_hpp_diag(const Real* hpp, int Cf, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < Cf * 6) out[t] = (double)hpp[(size_t)(t / 6) * 36 + (t % 6) * 7];
}

// max |diag H| from the summed Hpp diagonal (all ranks) and this rank's Hll
template <typename Real>
__global__ void ba_max_diag_summed(const double* pdiag, int Cf, const Real* hll, int Pf, double* partials) {
  double m = 0.0;
  const int n = Cf * 6 + Pf * 3;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    double v;
    if (t < Cf * 6) {
      v = fabs(pdiag[t]);
    } else {
      const int l = (t - Cf * 6) / 3, d = (t - Cf * 6) % 3;
      const int idx = d == 0 ? 0 : d == 1 ? 3 : 5;
      v = fabs((double)hll[(size_t)l * 6 + idx]);
    }
    m = fmax(m, v);
  }
  block_max(m, partials + blockIdx.x);
}

template <typename Real>
__global__ void ba_max_diag(const Real* hpp, int Cf, const Real* hll, int Pf, double* partials) {
  double m = 0.0;
  const int n = Cf * 6 + Pf * 3;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    double v;
    if (t < Cf * 6) {
      const int h = t / 6, d = t % 6;
      v = fabs((double)hpp[(size_t)h * 36 + d * 7]);
    } else {
      const int l = (t - Cf * 6) / 3, d = (t - Cf * 6) % 3;
      const int idx = d == 0 ? 0 : d == 1 ? 3 : 5;
      v = fabs((double)hll[(size_t)l * 6 + idx]);
    }
    m = fmax(m, v);
  }
  block_max(m, partials + blockIdx.x);
}

}  // namespace g2oc
