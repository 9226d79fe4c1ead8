// fm_mgpcg.cu -- MGPCG pressure projection for sm_100a.
//
// Restates the reference solver (3D/mgpcg.py:12-439; 2D/vortex/mgpcg_solid.py
// with an empty obstacle mask): all-Neumann 5/7-point Laplacian, red-black
// Gauss-Seidel V-cycle (2 pre + 2 post sweeps, piecewise-constant prolongation,
// restriction summing fine residuals into I//2 scaled 1/(dim-1), bottom RBGS),
// recentring of r, PCG with absolute (and optional relative) rTr tolerance.
//
// B200 design:
//  * alpha/beta/convergence live on the device (FP64), so an iteration issues
//    no host read; the host only polls the `done` word every check_every
//    iterations (the reference syncs three times per iteration).
//  * inner products use fixed-grid block partials reduced in a fixed order
//    (deterministic, FP64 accumulation).
//  * restriction is a gather over the 2^dim children (no atomics, no zero-fill);
//    the first red sweep of every level fuses the zero-fill of z (and, on the
//    fine level, the recentring of r); the last fine sweep fuses z.r.
//  * the coarsest level is smoothed by one CTA in shared memory (the reference
//    issues 2*bottom launches there).
//  * one PCG iteration (~40 launches) is captured once into a CUDA graph.
#include <cuda_bf16.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>

#include "fm_common.cuh"
#include "fm_internal.h"
#include "fm_mg_cluster.cuh"

namespace fm {

std::atomic<long long> g_launch_count{0};
std::atomic<int> g_last_cuda_error{0};
std::atomic<int> g_pdl{1};

constexpr int kRedBlocks = 148 * 4;  // fixed reduction grid: 4 CTAs per SM
constexpr int kRedThreads = 256;
constexpr int kMaxLevels = 16;
// single-CTA bottom solve: 512 threads x up to 8 cells each
constexpr int kBottomThreads = 512;
constexpr int kBottomCellsPerThread = 8;
constexpr int kBottomMaxCells = kBottomThreads * kBottomCellsPerThread;

struct DevState {
  double zTr_old, tol, rTr, alpha, beta, mean, pAp;
  int it;        // completed PCG iterations (reference `it`)
  int done;      // converged, max_iters reached or non-finite
  int conv;
  int nonfinite;
  int result_it;
  int max_it_seen;
  // cumulative over all solves since create / the last stats reset
  long long solves, iters_total, not_converged, nonfinite_count;
  long long bodies;  // while-loop bodies executed (device mode), for the launch count
  // outer defect correction (fm_mgpcg_solve_dc): mean of b, |b - mean|^2, |r|^2,
  // and an rTr floor for the inner solves (0 outside a defect correction)
  double dc_mean, dc_b2, dc_r2, dc_tol;
  // device-side defect correction (fm_project_dc): set once |r| <= rel_tol |b|;
  // every later correction, and the inner solves inside them, skip their work
  int dc_done;
};

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

template <int D>
__device__ __forceinline__ int parity(int i, int j, int k) {
  return (i + j + (D == 3 ? k : 0)) & 1;
}

// neighbor_sum / num_fluid_neighbors (3D/mgpcg.py:97-120), all-Neumann walls.
template <typename T, int D>
__device__ __forceinline__ T nb_sum(const T* __restrict__ x, const Shape& s, int i, int j, int k, T& diag) {
  T acc = 0;
  int nd = 2 * D;
  const long q = s.idx(i, j, k);
  if (i < s.s0 - 1) acc += x[q + (long)s.s1 * s.s2]; else --nd;
  if (i > 0) acc += x[q - (long)s.s1 * s.s2]; else --nd;
  if (j < s.s1 - 1) acc += x[q + s.s2]; else --nd;
  if (j > 0) acc += x[q - s.s2]; else --nd;
  if (D == 3) {
    if (k < s.s2 - 1) acc += x[q + 1]; else --nd;
    if (k > 0) acc += x[q - 1]; else --nd;
  }
  diag = (T)nd;
  return acc;
}

// Storage of MG levels: the compute type T, or BF16 for the levels between the
// finest and the cluster-resident ones when coarse_bf16 is set (FP32 solvers).
__device__ __forceinline__ float to_c(float v) { return v; }
__device__ __forceinline__ double to_c(double v) { return v; }
__device__ __forceinline__ float to_c(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename S, typename T>
__device__ __forceinline__ S to_s(T v) {
  if constexpr (std::is_same<S, __nv_bfloat16>::value) return __float2bfloat16_rn((float)v);
  else return (S)v;
}

// nb_sum over a stored level (values converted to the compute type T)
template <typename T, int D, typename S>
__device__ __forceinline__ T nb_sum_s(const S* __restrict__ x, const Shape& s, int i, int j, int k, T& diag) {
  T acc = 0;
  int nd = 2 * D;
  const long q = s.idx(i, j, k);
  if (i < s.s0 - 1) acc += (T)to_c(x[q + (long)s.s1 * s.s2]); else --nd;
  if (i > 0) acc += (T)to_c(x[q - (long)s.s1 * s.s2]); else --nd;
  if (j < s.s1 - 1) acc += (T)to_c(x[q + s.s2]); else --nd;
  if (j > 0) acc += (T)to_c(x[q - s.s2]); else --nd;
  if (D == 3) {
    if (k < s.s2 - 1) acc += (T)to_c(x[q + 1]); else --nd;
    if (k > 0) acc += (T)to_c(x[q - 1]); else --nd;
  }
  diag = (T)nd;
  return acc;
}

template <int D>
__device__ __forceinline__ int diag_of(const Shape& s, int i, int j, int k) {
  int nd = 2 * D;
  nd -= (i == 0) + (i == s.s0 - 1) + (j == 0) + (j == s.s1 - 1);
  if (D == 3) nd -= (k == 0) + (k == s.s2 - 1);
  return nd;
}

__device__ __forceinline__ void block_reduce2(double a, double b, double* out2) {
  __shared__ double sa[32], sb[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) { sa[w] = a; sb[w] = b; }
  __syncthreads();
  if (w == 0) {
    a = lane < nw ? sa[lane] : 0.0;
    b = lane < nw ? sb[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if (lane == 0) { out2[0] = a; out2[1] = b; }
  }
}

// the same for a block of 32 x n threads (its partial sums in the same place)
__device__ __forceinline__ void block_reduce2_2d(double a, double b, double* out2) {
  __shared__ double sa[32], sb[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  if (threadIdx.x == 0) { sa[threadIdx.y] = a; sb[threadIdx.y] = b; }
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    a = b = 0.0;
    for (unsigned k = 0; k < blockDim.y; ++k) a += sa[k], b += sb[k];
    out2[0] = a;
    out2[1] = b;
  }
}
// a grid of fewer blocks than partial sums: the rest is zero
__device__ __forceinline__ void walk_clear(double* part) {
  if (blockIdx.x == 0)
    for (unsigned q = gridDim.x + threadIdx.y * blockDim.x + threadIdx.x; q < kRedBlocks; q += blockDim.x * blockDim.y)
      part[2 * q] = part[2 * q + 1] = 0.0;
}

// Sum the fixed-grid partials in a fixed order (one CTA of 256 threads).
__device__ __forceinline__ void sum_partials(const double* __restrict__ part, double& a, double& b) {
  double x = 0, y = 0;
  for (int i = threadIdx.x; i < kRedBlocks; i += blockDim.x) { x += part[2 * i]; y += part[2 * i + 1]; }
  __shared__ double res[2];
  block_reduce2(x, y, res);
  __syncthreads();
  a = res[0];
  b = res[1];
}

#define FM_GRID_STRIDE(q, n) for (long q = (long)blockIdx.x * blockDim.x + threadIdx.x; q < (n); q += (long)gridDim.x * blockDim.x)

// ---------------------------------------------------------------------------
// projection front/back end
// ---------------------------------------------------------------------------
// apply_bc + divergence + init(r = -div) + x = 0, with partial sums of r for
// the recentring (3D/mgpcg.py:368-399, :76-84, :179-185).
// Each thread takes kDivUnroll cells of its grid-stride sequence at a time and
// issues all their face loads before any store, so 6 x kDivUnroll loads are in
// flight (a plain grid-stride loop waits one memory latency per cell).  The
// hoisting is safe: the only faces written are domain-wall faces, and every
// cell that reads one replaces the loaded value by 0.  The per-thread sum runs
// over the same cells in the same order as the plain loop.
constexpr int kDivUnroll = 2;

template <typename T, int D>
__global__ void __launch_bounds__(kRedThreads, 4) k_div_bc(fm_grid g, MacW<T> u, T* __restrict__ r,
                                                           T* __restrict__ x, double* __restrict__ part) {
  pdl_begin();
  const Shape cs = cell_shape(g);
  const unsigned n = (unsigned)cs.size();  // every field has fewer than 2^32 entries
  const unsigned stride = gridDim.x * blockDim.x;
  unsigned fstep[3];  // face offset of the high face of a cell, per component
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const Shape fs = face_shape(g, c);
    fstep[c] = c == 0 ? (unsigned)fs.s1 * fs.s2 : (c == 1 ? (unsigned)fs.s2 : 1u);
  }
  double sum = 0;
  for (unsigned base = blockIdx.x * blockDim.x + threadIdx.x; base < n; base += kDivUnroll * stride) {
    T vl[kDivUnroll][3], vr[kDivUnroll][3];
    unsigned qf[kDivUnroll][3];
    int I[kDivUnroll][3];
#pragma unroll
    for (int m = 0; m < kDivUnroll; ++m) {
      const unsigned q = base + m * stride;
      if (q >= n) break;
      unflatten(cs, q, I[m][0], I[m][1], I[m][2]);
#pragma unroll
      for (int c = 0; c < D; ++c) {
        const Shape fs = face_shape(g, c);
        const unsigned ql = ((unsigned)I[m][0] * fs.s1 + I[m][1]) * fs.s2 + I[m][2];
        qf[m][c] = ql;
        vl[m][c] = u.c[c][ql];
        vr[m][c] = u.c[c][ql + fstep[c]];
      }
    }
#pragma unroll
    for (int m = 0; m < kDivUnroll; ++m) {
      const unsigned q = base + m * stride;
      if (q >= n) break;
      T acc = 0;
#pragma unroll
      for (int c = 0; c < D; ++c) {
        T a = vl[m][c], b = vr[m][c];
        if (I[m][c] == 0) { a = 0; u.c[c][qf[m][c]] = 0; }
        if (I[m][c] == axis_len(cs, c) - 1) { b = 0; u.c[c][qf[m][c] + fstep[c]] = 0; }
        if (c == 0) acc = b - a;
        else { acc = acc + b; acc = acc - a; }
      }
      const T bq = acc * (T)-1;
      r[q] = bq;
      x[q] = 0;
      sum += (double)bq;
    }
  }
  block_reduce2(sum, 0.0, part + 2 * blockIdx.x);
}

// rhs given directly (fm_mgpcg_solve)
template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_load_rhs(long n, const T* __restrict__ b, T* __restrict__ r,
                                                          T* __restrict__ x, double* __restrict__ part) {
  pdl_begin();
  double sum = 0;
  FM_GRID_STRIDE(q, n) {
    const T v = b[q];
    r[q] = v;
    x[q] = 0;
    sum += (double)v;
  }
  block_reduce2(sum, 0.0, part + 2 * blockIdx.x);
}

// ---------------------------------------------------------------------------
// outer defect correction in FP64 around FP32 MGPCG solves (fm_mgpcg_solve_dc)
// ---------------------------------------------------------------------------
template <typename TB>
__global__ void __launch_bounds__(kRedThreads) k_dc_sum(long n, const TB* __restrict__ b, double* __restrict__ part) {
  pdl_begin();
  double sum = 0;
  FM_GRID_STRIDE(q, n) sum += (double)b[q];
  block_reduce2(sum, 0.0, part + 2 * blockIdx.x);
}

// which = 0: dc_mean = sum / n;  1: dc_b2 = dc_r2 = sum of squares;  2: dc_r2 = sum of squares
__global__ void k_dc_fin(DevState* st, const double* part, double n, int which) {
  pdl_begin();
  double a, b;
  sum_partials(part, a, b);
  if (threadIdx.x == 0) {
    if (which == 0) st->dc_mean = a / n;
    else {
      st->dc_r2 = b;
      if (which == 1) st->dc_b2 = b;
    }
  }
}

// work = (b - mean) - A x in FP64, partial sums of work^2 (second slot).
template <typename TB, int D>
__global__ void __launch_bounds__(kRedThreads) k_dc_residual(Shape s, const TB* __restrict__ b,
                                                             const double* __restrict__ x, double* __restrict__ work,
                                                             double* __restrict__ part, const DevState* st) {
  pdl_begin();
  const double mean = st->dc_mean;
  double acc = 0;
  FM_GRID_STRIDE(q, s.size()) {
    int i, j, k;
    unflatten(s, q, i, j, k);
    double diag;
    const double nb = nb_sum<double, D>(x, s, i, j, k, diag);
    const double r = ((double)b[q] - mean) - (diag * x[q] - nb);
    work[q] = r;
    acc += r * r;
  }
  block_reduce2(0.0, acc, part + 2 * blockIdx.x);
}

// Inner right-hand side r32 = work / |work| (unit norm keeps FP32 away from
// underflow as the residual shrinks), x32 = 0, partial sums of r32 for the
// recentring of the inner solve.
__global__ void __launch_bounds__(kRedThreads) k_dc_load(long n, const double* __restrict__ work,
                                                         float* __restrict__ r, float* __restrict__ x,
                                                         double* __restrict__ part, const DevState* st) {
  pdl_begin();
  const double inv = 1.0 / sqrt(st->dc_r2);
  double sum = 0;
  FM_GRID_STRIDE(q, n) {
    const float v = (float)(work[q] * inv);
    r[q] = v;
    x[q] = 0.f;
    sum += (double)v;
  }
  block_reduce2(sum, 0.0, part + 2 * blockIdx.x);
}

// rTr floor of the next inner solve (unit-norm right-hand side): a correction
// only has to bring |r| down to rel_tol |b|, with a factor 2 margin; 0 clears it.
__global__ void k_dc_set_tol(DevState* st, double rel_tol, int clear) {
  pdl_begin();
  const double t = clear ? 0.0 : 0.5 * rel_tol * sqrt(st->dc_b2 / st->dc_r2);
  st->dc_tol = t * t;
}

// x += |r| * e
__global__ void k_dc_update(long n, double* __restrict__ x, const float* __restrict__ e, const DevState* st) {
  pdl_begin();
  const double s = sqrt(st->dc_r2);
  FM_GRID_STRIDE(q, n) x[q] += s * (double)e[q];
}

// fm_project_dc: b = -div(u) of the FP32 velocity formed in FP64 (apply_bc
// zeroes the wall faces, as k_div_bc does), x = 0, partial sums of b.
template <int D>
__global__ void __launch_bounds__(kRedThreads) k_dc_div(fm_grid g, MacW<float> u, double* __restrict__ b,
                                                        double* __restrict__ x, double* __restrict__ part) {
  pdl_begin();
  const Shape cs = cell_shape(g);
  double sum = 0;
  FM_GRID_STRIDE(q, cs.size()) {
    int I[3];
    unflatten(cs, q, I[0], I[1], I[2]);
    double acc = 0;
#pragma unroll
    for (int c = 0; c < D; ++c) {
      const Shape fs = face_shape(g, c);
      const long step = c == 0 ? (long)fs.s1 * fs.s2 : (c == 1 ? (long)fs.s2 : 1);
      const long ql = fs.idx(I[0], I[1], I[2]);
      double a = (double)u.c[c][ql], bb = (double)u.c[c][ql + step];
      if (I[c] == 0) { a = 0; u.c[c][ql] = 0.f; }
      if (I[c] == axis_len(cs, c) - 1) { bb = 0; u.c[c][ql + step] = 0.f; }
      acc += bb - a;
    }
    b[q] = -acc;
    x[q] = 0;
    sum += -acc;
  }
  block_reduce2(sum, 0.0, part + 2 * blockIdx.x);
}

// fm_project_dc: after a residual, |r|^2 (which = 1 also |b|^2) and the stop
// test |r| <= rel_tol |b|; nothing once the correction loop is done.
__global__ void k_dc_check(DevState* st, const double* part, double rel_tol, int which) {
  pdl_begin();
  if (st->dc_done) return;
  double a, b;
  sum_partials(part, a, b);
  if (threadIdx.x == 0) {
    st->dc_r2 = b;
    if (which == 1) st->dc_b2 = b;
    if (!isfinite(b)) { st->dc_done = 1; st->nonfinite_count += 1; }
    else if (st->dc_b2 == 0.0 || b <= rel_tol * rel_tol * st->dc_b2) st->dc_done = 1;
  }
}

// The correction-loop versions of k_dc_residual / k_dc_load / k_dc_set_tol /
// k_dc_update: each returns at once when the loop is done.
template <int D>
__global__ void __launch_bounds__(kRedThreads) k_dc_residual_g(Shape s, const double* __restrict__ b,
                                                               const double* __restrict__ x, double* __restrict__ w,
                                                               double* __restrict__ part, const DevState* st) {
  pdl_begin();
  if (st->dc_done) return;
  const double mean = st->dc_mean;
  double acc = 0;
  FM_GRID_STRIDE(q, s.size()) {
    int i, j, k;
    unflatten(s, q, i, j, k);
    double diag;
    const double nb = nb_sum<double, D>(x, s, i, j, k, diag);
    const double r = (b[q] - mean) - (diag * x[q] - nb);
    w[q] = r;
    acc += r * r;
  }
  block_reduce2(0.0, acc, part + 2 * blockIdx.x);
}

__global__ void __launch_bounds__(kRedThreads) k_dc_load_g(long n, const double* __restrict__ w,
                                                           float* __restrict__ r, float* __restrict__ x,
                                                           double* __restrict__ part, const DevState* st) {
  pdl_begin();
  if (st->dc_done) return;
  const double inv = 1.0 / sqrt(st->dc_r2);
  double sum = 0;
  FM_GRID_STRIDE(q, n) {
    const float v = (float)(w[q] * inv);
    r[q] = v;
    x[q] = 0.f;
    sum += (double)v;
  }
  block_reduce2(sum, 0.0, part + 2 * blockIdx.x);
}

__global__ void k_dc_set_tol_g(DevState* st, double rel_tol) {
  pdl_begin();
  if (st->dc_done) return;
  const double t = 0.5 * rel_tol * sqrt(st->dc_b2 / st->dc_r2);
  st->dc_tol = t * t;
}

__global__ void k_dc_update_g(long n, double* __restrict__ x, const float* __restrict__ e, const DevState* st) {
  pdl_begin();
  if (st->dc_done) return;
  const double sc = sqrt(st->dc_r2);
  FM_GRID_STRIDE(q, n) x[q] += sc * (double)e[q];
}

// End of fm_project_dc: an unconverged loop counts as a not-converged solve;
// the state returns to plain solves (no floor, not done).
__global__ void k_dc_finish(DevState* st) {
  pdl_begin();
  if (!st->dc_done) st->not_converged += 1;
  st->dc_done = 0;
  st->dc_tol = 0.0;
}

// subtract_grad_p + apply_bc (3D/mgpcg.py:401-427), 2D.  T: the pressure's type (FP64 for
// a defect-corrected FP32 velocity).
template <typename T, typename U>
__global__ void k_subgrad_bc2(fm_grid g, const T* __restrict__ p, MacW<U> u) {
  pdl_begin();
  const int c = blockIdx.y;
  const Shape fs = face_shape(g, c);
  const Shape cs = cell_shape(g);
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= fs.size()) return;
  int I[3];
  unflatten(fs, q, I[0], I[1], I[2]);
  if (I[c] == 0 || I[c] == axis_len(cs, c)) { u.c[c][q] = 0; return; }
  const long pc = cs.idx(I[0], I[1], I[2]);
  const long step = c == 0 ? cs.s1 : 1;
  u.c[c][q] = (U)((T)u.c[c][q] - (p[pc] - p[pc - step]));
}

// ---------------------------------------------------------------------------
// scalar finalizers (one CTA)
// ---------------------------------------------------------------------------
__global__ void k_fin_mean(DevState* st, const double* part, double n) {
  pdl_begin();
  double a, b;
  sum_partials(part, a, b);
  if (threadIdx.x == 0) {
    st->mean = a / n;
    st->done = st->dc_done;  // 0 outside fm_project_dc
    st->conv = 0; st->nonfinite = 0; st->it = 0; st->result_it = 0;
    st->beta = 0; st->alpha = 0;
  }
}

__global__ void k_fin_alpha(DevState* st, const double* part, double eps) {
  pdl_begin();
  if (st->done) return;
  double a, b;
  sum_partials(part, a, b);
  if (threadIdx.x == 0) {
    st->pAp = a;
    st->alpha = st->zTr_old / (a + eps);
  }
}

// Called by thread 0 when a solve ends: fold it into the cumulative counters.
__device__ __forceinline__ void finish_solve(DevState* st) {
  st->done = 1;
  st->result_it = st->it;
  st->solves += 1;
  st->iters_total += st->it;
  if (st->it > st->max_it_seen) st->max_it_seen = st->it;
  if (st->nonfinite) st->nonfinite_count += 1;
  else if (!st->conv) st->not_converged += 1;
}

__global__ void k_fin_conv(DevState* st, const double* part, double n) {
  pdl_begin();
  if (st->done) return;
  double a, b;
  sum_partials(part, a, b);
  if (threadIdx.x == 0) {
    st->rTr = a;
    st->mean = b / n;
    if (!isfinite(a)) { st->nonfinite = 1; finish_solve(st); }
    else if (a < st->tol) { st->conv = 1; finish_solve(st); }
  }
}

// Node before a while loop: skip the loop when the solve is already done at
// its start (an inner solve of a finished defect correction, a non-finite
// start), instead of running one body of early-returning kernels.
__global__ void k_loop_init(cudaGraphConditionalHandle h, const DevState* st) {
  cudaGraphSetConditional(h, st->done ? 0u : 1u);
}

// Last node of the while-loop body: keep iterating until the solve is done.
__global__ void k_loop_cond(cudaGraphConditionalHandle h, DevState* st) {
  pdl_begin();
  st->bodies += 1;
  cudaGraphSetConditional(h, st->done ? 0u : 1u);
}

__global__ void k_fin_beta(DevState* st, const double* part, double eps, double abs_tol, double rel_tol,
                           int max_iters, int first) {
  pdl_begin();
  if (st->done) return;
  double a, b;
  sum_partials(part, a, b);
  if (threadIdx.x == 0) {
    if (first) {
      st->zTr_old = a;
      double tol = abs_tol;
      if (rel_tol > 0 && a * rel_tol > tol) tol = a * rel_tol;
      if (st->dc_tol > tol) tol = st->dc_tol;
      st->tol = tol;
      st->beta = 0;
      if (!isfinite(a)) { st->nonfinite = 1; finish_solve(st); }
      // z.r = 0 means r = 0 (the preconditioner is SPD on mean-zero fields): the
      // zero start is the solution.  Stopping here keeps alpha = 0 / (0 + eps)
      // from becoming NaN when eps = 0.
      else if (a == 0.0) { st->conv = 1; finish_solve(st); }
    } else {
      st->beta = a / (st->zTr_old + eps);
      st->zTr_old = a;
      st->it += 1;
      if (st->it >= max_iters) finish_solve(st);
    }
  }
}

// ---------------------------------------------------------------------------
// PCG vector kernels
// ---------------------------------------------------------------------------
// Neighbour values of cell (i, j, k) at 32-bit index q in the reference's
// summation order (+i, -i, +j, -j, +k, -k), 0 where the neighbour is outside.
// Summing all six (or four) from +0.0 gives the skipping sum bit for bit: a
// round-to-nearest sum that starts at +0.0 is never -0.0, so adding +0.0
// changes nothing.
template <typename T, int D>
__device__ __forceinline__ void nb_load(const T* x, const Shape& s, unsigned q, int i, int j, int k, T* v) {
  const unsigned si = (unsigned)s.s1 * s.s2, sj = s.s2;
  v[0] = i < s.s0 - 1 ? x[q + si] : (T)0;
  v[1] = i > 0 ? x[q - si] : (T)0;
  v[2] = j < s.s1 - 1 ? x[q + sj] : (T)0;
  v[3] = j > 0 ? x[q - sj] : (T)0;
  if (D == 3) {
    v[4] = k < s.s2 - 1 ? x[q + 1] : (T)0;
    v[5] = k > 0 ? x[q - 1] : (T)0;
  }
}
template <typename T, int D>
__device__ __forceinline__ T nb_add(const T* v) {
  T acc = 0;
#pragma unroll
  for (int m = 0; m < 2 * D; ++m) acc += v[m];
  return acc;
}

// The grid-stride vector kernels below take kVecUnroll cells of a thread's
// sequence at a time and issue all their loads before any store (memory-level
// parallelism); the per-thread partial sums keep the cell order of a plain
// grid-stride loop.
constexpr int kVecUnroll = 2;

template <typename T, int D>
__global__ void __launch_bounds__(kRedThreads) k_Ap_dot(Shape s, const T* __restrict__ p, T* __restrict__ Ap,
                                                        double* __restrict__ part, const DevState* st) {
  pdl_begin();
  if (st->done) return;
  const unsigned n = (unsigned)s.size(), stride = gridDim.x * blockDim.x;
  double acc = 0;
  for (unsigned base = blockIdx.x * blockDim.x + threadIdx.x; base < n; base += kVecUnroll * stride) {
    T v[kVecUnroll][6], pv[kVecUnroll];
    int nd[kVecUnroll];
#pragma unroll
    for (int m = 0; m < kVecUnroll; ++m) {
      const unsigned q = base + m * stride;
      if (q >= n) break;
      int i, j, k;
      unflatten(s, q, i, j, k);
      nb_load<T, D>(p, s, q, i, j, k, v[m]);
      pv[m] = p[q];
      nd[m] = diag_of<D>(s, i, j, k);
    }
#pragma unroll
    for (int m = 0; m < kVecUnroll; ++m) {
      const unsigned q = base + m * stride;
      if (q >= n) break;
      const T a = rn_sub(rn_mul((T)nd[m], pv[m]), nb_add<T, D>(v[m]));
      Ap[q] = a;
      acc += (double)pv[m] * (double)a;
    }
  }
  block_reduce2(acc, 0.0, part + 2 * blockIdx.x);
}

template <typename T>
__global__ void __launch_bounds__(kRedThreads) k_update_xr(long n, T* __restrict__ x, T* __restrict__ r,
                                                           const T* __restrict__ p, const T* __restrict__ Ap,
                                                           double* __restrict__ part, const DevState* st) {
  pdl_begin();
  if (st->done) return;
  const T alpha = (T)st->alpha;
  double rr = 0, rs = 0;
  FM_GRID_STRIDE(q, n) {
    x[q] = rn_add(x[q], rn_mul(alpha, p[q]));
    const T rv = rn_sub(r[q], rn_mul(alpha, Ap[q]));
    r[q] = rv;
    rr += (double)rv * (double)rv;
    rs += (double)rv;
  }
  block_reduce2(rr, rs, part + 2 * blockIdx.x);
}

template <typename T>
__global__ void k_update_p(long n, T* __restrict__ p, const T* __restrict__ z, const DevState* st, int first) {
  pdl_begin();
  if (st->done) return;
  const T beta = (T)st->beta;
  FM_GRID_STRIDE(q, n) p[q] = first ? z[q] : rn_add(z[q], rn_mul(beta, p[q]));
}

// ---------------------------------------------------------------------------
// V-cycle kernels
// ---------------------------------------------------------------------------
// First red sweep from z == 0 (fuses z.fill(0)); optionally recentres r.
template <typename T, int D>
__global__ void k_smooth_first(Shape s, T* __restrict__ r, T* __restrict__ z, const DevState* st, int recenter) {
  pdl_begin();
  if (st->done) return;
  const T mean = recenter ? (T)st->mean : (T)0;
  FM_GRID_STRIDE(q, s.size()) {
    int i, j, k;
    unflatten(s, q, i, j, k);
    T rv = r[q];
    if (recenter) { rv = rv - mean; r[q] = rv; }
    z[q] = parity<D>(i, j, k) == 0 ? div_nd(rv, diag_of<D>(s, i, j, k)) : (T)0;
  }
}

// Pair-per-thread RBGS sweeps for the levels above the cluster kernel.  A
// thread owns cells (.., 2m) and (.., 2m+1) along the innermost axis (k in 3D,
// j in 2D), one red and one black, so every lane updates a cell in every
// half-sweep.  Launch: block (32, 8); 3D grid (pairs/32, n1/8, n0) over
// (pair, j, i), 2D grid (pairs/32, n0/8) over (pair, i).
constexpr int kPairBX = 32, kPairBY = 8;

template <int D>
__device__ __forceinline__ bool pair_coords(const Shape& s, int& i, int& j, int& k0) {
  const int m = blockIdx.x * kPairBX + threadIdx.x;
  if (D == 3) {
    i = blockIdx.z;
    j = blockIdx.y * kPairBY + threadIdx.y;
    k0 = 2 * m;
    return j < s.s1 && k0 < s.s2;
  }
  i = blockIdx.y * kPairBY + threadIdx.y;
  j = 2 * m;
  k0 = 0;
  return i < s.s0 && j < s.s1;
}

// Neighbour sum (reference order +i, -i, +j, -j, +k, -k) and neighbour count
// of cell (i, j, k) at 32-bit index q.
template <typename T, int D, typename S>
__device__ __forceinline__ T nb_sum32(const S* __restrict__ x, const Shape& s, unsigned q, int i, int j, int k,
                                      int& nd) {
  const unsigned si = (unsigned)s.s1 * s.s2, sj = s.s2;
  T acc = 0;
  nd = 0;
  if (i < s.s0 - 1) { acc += (T)to_c(x[q + si]); ++nd; }
  if (i > 0) { acc += (T)to_c(x[q - si]); ++nd; }
  if (j < s.s1 - 1) { acc += (T)to_c(x[q + sj]); ++nd; }
  if (j > 0) { acc += (T)to_c(x[q - sj]); ++nd; }
  if (D == 3) {
    if (k < s.s2 - 1) { acc += (T)to_c(x[q + 1]); ++nd; }
    if (k > 0) { acc += (T)to_c(x[q - 1]); ++nd; }
  }
  return acc;
}

// smooth(l, phase) over pairs: only the cell of colour `phase` is updated.
// S: storage type of the level (T, or BF16 with coarse_bf16).
template <typename T, int D, typename S = T>
__global__ void __launch_bounds__(kPairBX* kPairBY) k_smooth_pair(Shape s, const S* __restrict__ r, S* z, int phase,
                                                                 const DevState* st) {
  pdl_begin();
  if (st->done) return;
  int i, j, k;
  if (!pair_coords<D>(s, i, j, k)) return;
  // the colour-`phase` cell of the pair: parity(i, j, k0) is (i + j) & 1 in 3D, i & 1 in 2D
  const int shift = ((D == 3 ? i + j : i) + phase) & 1;
  if (D == 3) k += shift; else j += shift;
  if ((D == 3 ? k : j) >= (D == 3 ? s.s2 : s.s1)) return;
  const unsigned q = ((unsigned)i * s.s1 + j) * s.s2 + k;
  int nd;
  const T nb = nb_sum32<T, D, S>(z, s, q, i, j, k, nd);
  z[q] = to_s<S>(div_nd((T)to_c(r[q]) + nb, nd));
}

// First red sweep from z == 0 over pairs (fuses z.fill(0)); optionally recentres r.
template <typename T, int D, typename S = T>
__global__ void __launch_bounds__(kPairBX* kPairBY) k_smooth_first_pair(Shape s, S* __restrict__ r, S* __restrict__ z,
                                                                       const DevState* st, int recenter) {
  pdl_begin();
  if (st->done) return;
  int i, j, k;
  if (!pair_coords<D>(s, i, j, k)) return;
  const T mean = recenter ? (T)st->mean : (T)0;
  const int red_second = (D == 3 ? i + j : i) & 1;  // the pair's second cell is red
  const unsigned q0 = ((unsigned)i * s.s1 + j) * s.s2 + k;
  const bool has2 = (D == 3 ? k : j) + 1 < (D == 3 ? s.s2 : s.s1);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (c == 1 && !has2) break;
    const unsigned q = q0 + c;
    T rv = (T)to_c(r[q]);
    if (recenter) { rv = rv - mean; r[q] = to_s<S>(rv); }
    if (c == red_second) {
      const int ci = i, cj = D == 3 ? j : j + c, ck = D == 3 ? k + c : 0;
      z[q] = to_s<S>(div_nd(rv, diag_of<D>(s, ci, cj, ck)));
    } else {
      z[q] = to_s<S>((T)0);
    }
  }
}

// smooth(l, phase) (3D/mgpcg.py:170-177); with part != nullptr also z.r over all cells.
// A half-sweep reads only cells of the other colour and writes only cells of
// colour `phase`, so the hoisted loads never see a value written in this launch.
template <typename T, int D, bool DOT>
__global__ void __launch_bounds__(kRedThreads) k_smooth(Shape s, const T* __restrict__ r, T* z, int phase,
                                                        double* __restrict__ part, const DevState* st) {
  pdl_begin();
  if (st->done) return;
  const unsigned n = (unsigned)s.size(), stride = gridDim.x * blockDim.x;
  double acc = 0;
  for (unsigned base = blockIdx.x * blockDim.x + threadIdx.x; base < n; base += kVecUnroll * stride) {
    T v[kVecUnroll][6], rv[kVecUnroll], zo[kVecUnroll];
    int nd[kVecUnroll];
    bool upd[kVecUnroll];
#pragma unroll
    for (int m = 0; m < kVecUnroll; ++m) {
      const unsigned q = base + m * stride;
      if (q >= n) break;
      int i, j, k;
      unflatten(s, q, i, j, k);
      upd[m] = parity<D>(i, j, k) == phase;
      rv[m] = r[q];
      if (upd[m]) {
        nb_load<T, D>(z, s, q, i, j, k, v[m]);
        nd[m] = diag_of<D>(s, i, j, k);
      } else {
        zo[m] = z[q];
      }
    }
#pragma unroll
    for (int m = 0; m < kVecUnroll; ++m) {
      const unsigned q = base + m * stride;
      if (q >= n) break;
      T zv;
      if (upd[m]) {
        zv = div_nd(rv[m] + nb_add<T, D>(v[m]), nd[m]);
        z[q] = zv;
      } else {
        zv = zo[m];
      }
      if (DOT) acc += (double)zv * (double)rv[m];
    }
  }
  if (DOT) block_reduce2(acc, 0.0, part + 2 * blockIdx.x);
}

// restrict(l) (3D/mgpcg.py:157-163) as a gather over the 4 children, 2D (3D: k_restrict_walk).
// SF / SC: storage types of the fine and the coarse level.
template <typename T, typename SF = T, typename SC = T>
__global__ void k_restrict(Shape sf, Shape sc, const SF* __restrict__ rf, const SF* __restrict__ zf,
                           SC* __restrict__ rc, const DevState* st) {
  pdl_begin();
  if (st->done) return;
  FM_GRID_STRIDE(q, sc.size()) {
    int I, J, K;
    unflatten(sc, q, I, J, K);
    T acc = 0;
#pragma unroll
    for (int di = 0; di < 2; ++di)
#pragma unroll
      for (int dj = 0; dj < 2; ++dj) {
        const int i = 2 * I + di, j = 2 * J + dj;
        const long f = sf.idx(i, j, 0);
        T diag;
        const T nb = nb_sum_s<T, 2, SF>(zf, sf, i, j, 0, diag);
        acc = rn_add(acc, rn_sub((T)to_c(rf[f]), rn_sub(rn_mul(diag, (T)to_c(zf[f])), nb)));  // scale 1 / (D - 1)
      }
    rc[q] = to_s<SC>(acc);
  }
}

// prolongate(l) (3D/mgpcg.py:165-168), 2D (3D: k_prolong_walk)
template <typename T, typename SF = T, typename SC = T>
__global__ void k_prolong(Shape sf, Shape sc, SF* __restrict__ zf, const SC* __restrict__ zc, const DevState* st) {
  pdl_begin();
  if (st->done) return;
  FM_GRID_STRIDE(q, sf.size()) {
    int i, j, k;
    unflatten(sf, q, i, j, k);
    zf[q] = to_s<SF>((T)to_c(zf[q]) + (T)to_c(zc[sc.idx(i >> 1, j >> 1, 0)]));
  }
}

// ---------------------------------------------------------------------------
// 3D: columns of planes
// ---------------------------------------------------------------------------
// The fine levels of a 3D solve live in the L2, and a kernel that reads the 7-point
// neighbourhood of each cell by itself fetches every cell about four times and spends
// most of its issue slots on indices.  The kernels below walk along axis 0 instead: a
// thread owns a pair of cells (.., 2m), (.., 2m+1) and keeps the planes before and
// after in registers, the neighbours along k come from the next lanes by shuffles,
// those along j from the L1, and the loads of the next plane are issued before the
// current one is used.  A block is 32 pairs x 8 rows, an item of work a stretch of
// planes of such a tile, blocks take items in a stride (so that the reductions have at
// most kRedBlocks partial sums).  Seven blocks fit an SM: the stretch is as long as
// leaves about that many.  128^3 FP32, us, warm: last half-sweep with its inner product
// 16.6 -> 9.2, A p and its inner product 12.9 -> 8.5, restriction 9.0 -> 7.5, prolongation
// 9.0 -> 5.2, gradient subtraction 37.8 -> 14.4.  (A plain half-sweep gains nothing: 7.2 by
// pairs of one plane, 9.3 walking with the walls worked out per plane.)
struct Walk {
  int tk, tj, planes, items;
};
constexpr int kWalkBX = 32, kWalkBY = 8, kWalkBlocks = 148 * 7;
// The two kernels with an inner product walk in FP32 only: in FP64 the grid-stride ones are faster
// (144^3, us, walking / not: last half-sweep 30.1 / 23.7, A p 28.0 / 19.0; 128^3 18.4 / 17.7 and 12.6 / 10.6;
// 40^3 4.9 / 4.3 and 3.8 / 3.4).
template <typename T, int D>
constexpr bool kWalkDots = D == 3 && std::is_same<T, float>::value;
// over n0 planes, n1 rows, nk columns of the threads, in at most `most` items where
// stretches of whole columns allow
inline Walk walk_of(int n0, int n1, int nk, int most) {
  Walk w;
  w.tk = (nk + kWalkBX - 1) / kWalkBX;
  w.tj = (n1 + kWalkBY - 1) / kWalkBY;
  const long tiles = (long)w.tk * w.tj;
  const int segs = tiles < most ? (int)(most / tiles) : 1;
  w.planes = (n0 + segs - 1) / segs;
  w.items = (int)(tiles * ((n0 + w.planes - 1) / w.planes));
  return w;
}
inline Walk walk_pairs(const Shape& s, int most) { return walk_of(s.s0, s.s1, (s.s2 + 1) / 2, most); }
constexpr dim3 kWalkBlock(kWalkBX, kWalkBY);
__device__ __forceinline__ void walk_item(const Walk& w, int it, int n0, int& i0, int& i1, int& j, int& m) {
  const int t = it / w.tk;
  m = (it - t * w.tk) * kWalkBX + threadIdx.x;
  const int seg = t / w.tj;
  j = (t - seg * w.tj) * kWalkBY + threadIdx.y;
  i0 = seg * w.planes;
  i1 = min(i0 + w.planes, n0);
}

// How a pair of cells of a row is stored: side by side, read by one aligned load (rows of
// every level but the coarsest have an even length: creation asks for cell counts that are
// multiples of 2^(levels - 1)), or by colour (below).
enum { kVec = 0, kSplit = 1 };
// The pair at p, zeros where `on` is false; oa: kSplit, the offset of the first one's
// colour (0 or h), p then points at the pair in the first colour.
template <int MODE, typename T, typename S>
__device__ __forceinline__ void load_two(const S* p, bool on, T& a, T& b, int oa = 0, int h = 0) {
  if constexpr (MODE == kSplit) {
    a = on ? (T)to_c(p[oa]) : (T)0;
    b = on ? (T)to_c(p[h - oa]) : (T)0;
  } else {
    a = b = (T)0;
    if (on) {
      if constexpr (std::is_same<S, __nv_bfloat16>::value) {
        const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(p);
        a = (T)__low2float(v), b = (T)__high2float(v);
      } else {
        using V = std::conditional_t<std::is_same<S, float>::value, float2, double2>;
        const V v = *reinterpret_cast<const V*>(p);
        a = (T)v.x, b = (T)v.y;
      }
    }
  }
}
// neighbours of a cell within its plane
__device__ __forceinline__ int plane_nd(const Shape& s, int j, int k) {
  return 6 - (j == 0) - (j == s.s1 - 1) - (k == 0) - (k == s.s2 - 1);
}
// smooth(l, phase) (3D/mgpcg.py:170-177), only the cells of colour `phase`, and
// the partial sums of z.r over all cells.  The other colour's cell of a
// pair is the +-i neighbour of the updated cells in the planes beside, and a +-k
// neighbour of this plane's and of the next pair's updated cell; none of them is
// written here, so loads may run ahead of the stores.  Which cell of the pair is
// updated alternates with the planes and is the same for the whole warp (a row):
// planes are taken by twos with it known at compile time, and what a column needs
// of the walls is worked out once (with both done per plane the kernel is bound by
// issue slots, 174 instructions a plane).
template <typename T>
__global__ void __launch_bounds__(kWalkBX* kWalkBY) k_smooth_dot_walk(Shape s, Walk w, const T* __restrict__ r, T* z,
                                                                 int phase, double* __restrict__ part,
                                                                 const DevState* st) {
  pdl_begin();
  if (st->done) return;
  constexpr unsigned all = 0xffffffffu;
  const int lane = threadIdx.x;
  const long sj = s.s2, si = (long)s.s1 * s.s2;
  double acc = 0;
  for (int it = blockIdx.x; it < w.items; it += gridDim.x) {
    int i0, i1, j, m;
    walk_item(w, it, s.s0, i0, i1, j, m);
    if (j >= s.s1) continue;  // the whole warp: a warp is one row
    const int k0 = 2 * m;
    // per cell of the pair: it exists, its +-j neighbours do, its k neighbour of another warp does
    const bool kv[2] = {k0 < s.s2, k0 + 1 < s.s2};
    const bool kp[2] = {kv[0] && j < s.s1 - 1, kv[1] && j < s.s1 - 1}, km[2] = {kv[0] && j > 0, kv[1] && j > 0};
    const bool kf[2] = {kv[0] && lane == 0 && k0 > 0, lane == 31 && k0 + 2 < s.s2};
    const int nd[2] = {plane_nd(s, j, k0), plane_nd(s, j, k0 + 1)};
    const ClQuot<T> quot[2] = {ClQuot<T>(nd[0]), ClQuot<T>(nd[1])};
    const long q = ((long)i0 * s.s1 + j) * s.s2 + k0;
    T* zp = z + q;  // the pair in plane i
    const T* rp = r + q;
    struct Plane {
      T o, jp, jm, r, ro, far;
    };
    // what the plane at zp needs, SH the updated cell: the other colour's cell (`in`:
    // the plane exists), the +-j neighbours, the residual(s), the outer k neighbour
    const auto fetch = [&](auto sh_, const T* zq, const T* rq, bool in, bool whole) {
      constexpr int SH = decltype(sh_)::value;
      Plane p;
      p.o = in && kv[1 - SH] ? (zq[1 - SH]) : (T)0;
      p.jp = whole && kp[SH] ? (zq[SH + sj]) : (T)0;
      p.jm = whole && km[SH] ? (zq[SH - sj]) : (T)0;
      p.r = whole && kv[SH] ? (rq[SH]) : (T)0;
      p.ro = whole && kv[1 - SH] ? (rq[1 - SH]) : (T)0;
      p.far = whole && kf[SH] ? (zq[SH ? 2 : -1]) : (T)0;
      return p;
    };
    const auto walk = [&](auto first) {
      constexpr int S0 = decltype(first)::value;
      using A = std::integral_constant<int, S0>;
      using B = std::integral_constant<int, 1 - S0>;
      T om = i0 > 0 && kv[S0] ? (zp[S0 - si]) : (T)0;
      Plane c = fetch(A(), zp, rp, true, true);
      const auto step = [&](auto sh_, auto next_, int i) {
        constexpr int SH = decltype(sh_)::value;
        const Plane n = fetch(next_, zp + si, rp + si, i + 1 < s.s0, i + 1 < i1);
        const T side = SH ? __shfl_down_sync(all, c.o, 1) : __shfl_up_sync(all, c.o, 1);
        const T far = lane == (SH ? 31 : 0) ? c.far : side;
        T nb = (T)0;
        nb += n.o;
        nb += om;
        nb += c.jp;
        nb += c.jm;
        nb += SH ? far : c.o;
        nb += SH ? c.o : far;
        const T x = c.r + nb;
        T v;
        if (i > 0 && i < s.s0 - 1) {
          v = quot[SH].fast(x);
          if (quot[SH].template bad<true>(x)) v = quot[SH].slow(x);
        } else {
          v = div_nd(x, nd[SH] - (i == 0) - (i == s.s0 - 1));
        }
        if (kv[SH]) zp[SH] = v;
        acc += kv[SH] ? (double)v * (double)c.r : 0.0;
        acc += (double)c.o * (double)c.ro;
        om = c.o;
        c = n;
        zp += si;
        rp += si;
      };
      int i = i0;
      for (; i + 1 < i1; i += 2) {
        step(A(), B(), i);
        step(B(), A(), i + 1);
      }
      if (i < i1) step(A(), B(), i);
    };
    if ((i0 + j + phase) & 1) walk(std::integral_constant<int, 1>());
    else walk(std::integral_constant<int, 0>());
  }
  block_reduce2_2d(acc, 0.0, part + 2 * blockIdx.x);
  walk_clear(part);
}

// Ap = A p and the partial sums of p.Ap
template <typename T>
__global__ void __launch_bounds__(kWalkBX* kWalkBY) k_Ap_walk(Shape s, Walk w, const T* __restrict__ p,
                                                             T* __restrict__ Ap, double* __restrict__ part,
                                                             const DevState* st) {
  pdl_begin();
  if (st->done) return;
  constexpr unsigned all = 0xffffffffu;
  const int lane = threadIdx.x;
  const long sj = s.s2, si = (long)s.s1 * s.s2;
  double acc = 0;
  for (int it = blockIdx.x; it < w.items; it += gridDim.x) {
    int i0, i1, j, m;
    walk_item(w, it, s.s0, i0, i1, j, m);
    if (j >= s.s1) continue;  // the whole warp
    const int k0 = 2 * m;
    const bool on = k0 < s.s2, jp = on && j < s.s1 - 1, jm = on && j > 0;
    const bool edge = (lane == 0 && on && k0 > 0) || (lane == 31 && k0 + 2 < s.s2);
    const int eo = lane == 0 ? -1 : 2;
    const T nda = (T)plane_nd(s, j, k0), ndb = (T)plane_nd(s, j, k0 + 1);
    const long q = ((long)i0 * s.s1 + j) * s.s2 + k0;
    const T* pp = p + q;
    T* ap = Ap + q;
    struct Plane {
      T a, b, pa, pb, ma, mb, far;  // the pair, its +j and -j pairs, the k neighbour outside the warp
    };
    const auto fetch = [&](const T* x, bool in, bool whole) {
      Plane v;
      load_two<kVec>(x, in && on, v.a, v.b);
      load_two<kVec>(x + sj, whole && jp, v.pa, v.pb);
      load_two<kVec>(x - sj, whole && jm, v.ma, v.mb);
      v.far = whole && edge ? x[eo] : (T)0;
      return v;
    };
    T ma, mb;
    load_two<kVec>(pp - si, i0 > 0 && on, ma, mb);
    Plane c = fetch(pp, true, true);
#pragma unroll 2
    for (int i = i0; i < i1; ++i) {
      const Plane n = fetch(pp + si, i + 1 < s.s0, i + 1 < i1);
      const T up = __shfl_down_sync(all, c.a, 1), dn = __shfl_up_sync(all, c.b, 1);
      const T left = lane == 0 ? c.far : dn, right = lane == 31 ? c.far : up;
      T na = (T)0, nb = (T)0;
      na += n.a, na += ma, na += c.pa, na += c.ma, na += c.b, na += left;
      nb += n.b, nb += mb, nb += c.pb, nb += c.mb, nb += right, nb += c.a;
      const T wall = (T)((i == 0) + (i == s.s0 - 1));
      const T ra = rn_sub(rn_mul(nda - wall, c.a), na), rb = rn_sub(rn_mul(ndb - wall, c.b), nb);
      using V = std::conditional_t<std::is_same<T, float>::value, float2, double2>;
      if (on) *reinterpret_cast<V*>(ap) = V{ra, rb};
      acc += (double)c.a * (double)ra;  // a missing cell is 0
      acc += (double)c.b * (double)rb;
      ma = c.a, mb = c.b;
      c = n;
      pp += si;
      ap += si;
    }
  }
  block_reduce2_2d(acc, 0.0, part + 2 * blockIdx.x);
  walk_clear(part);
}

// restrict(l) (3D/mgpcg.py:157-163): a thread owns the coarse cell of a pair column and
// two rows, and walks the fine planes; children in the order of the gather.
// out_split: the coarse level is stored by colour.
template <typename T, typename SF, typename SC, int MODE>
__global__ void __launch_bounds__(kWalkBX* kWalkBY) k_restrict_walk(Shape sf, Shape sc, Walk w,
                                                                   const SF* __restrict__ rf,
                                                                   const SF* __restrict__ zf, SC* __restrict__ rc,
                                                                   int out_split, const DevState* st) {
  pdl_begin();
  if (st->done) return;
  constexpr unsigned all = 0xffffffffu;
  const T scale = (T)1.0 / (T)2.0;
  const int lane = threadIdx.x;
  const long sj = sf.s2, si = (long)sf.s1 * sf.s2;
  const int h = sf.s2 / 2;
  for (int it = blockIdx.x; it < w.items; it += gridDim.x) {
    int I0, I1, J, K;
    walk_item(w, it, sc.s0, I0, I1, J, K);
    if (J >= sc.s1) continue;  // the whole warp
    const bool on = K < sc.s2;  // then the fine pairs exist
    const int k0 = 2 * K, j0 = 2 * J;
    const bool jl = on && j0 > 0, jh = on && j0 + 2 < sf.s1;
    const bool el = on && lane == 0 && k0 > 0;
    const bool er = on && lane == 31 && k0 + 2 < sf.s2;
    T nd[2][2];
#pragma unroll
    for (int d = 0; d < 2; ++d) nd[d][0] = (T)plane_nd(sf, j0 + d, k0), nd[d][1] = (T)plane_nd(sf, j0 + d, k0 + 1);
    // by colour: the first cell of a pair in row j0 + d of plane i has colour (d + i) & 1 (j0 and k0 are even)
    const long q = ((long)(2 * I0) * sf.s1 + j0) * sf.s2 + (MODE == kSplit ? K : k0);
    const SF* zp = zf + q;
    const SF* rp = rf + q;
    SC* out = rc + ((long)I0 * sc.s1 + J) * sc.s2;
    T ma[2], mb[2], ca[2], cb[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      load_two<MODE>(zp - si + d * sj, on && I0 > 0, ma[d], mb[d], d ? 0 : h, h);
      load_two<MODE>(zp + d * sj, on, ca[d], cb[d], d ? h : 0, h);
    }
    for (int I = I0; I < I1; ++I) {
      T acc = (T)0;
#pragma unroll
      for (int di = 0; di < 2; ++di) {
        const int i = 2 * I + di;
        T na[2], nb[2], xa[2], xb[2], ra[2], rb[2], eL[2], eR[2];
        const bool up = on && i + 1 < sf.s0;
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int oa = ((d + di) & 1) ? h : 0;  // the first cell's colour
          load_two<MODE>(zp + si + d * sj, up, na[d], nb[d], h - oa, h);
          load_two<MODE>(rp + d * sj, on, ra[d], rb[d], oa, h);
          eL[d] = el ? (T)to_c(zp[d * sj + (MODE == kSplit ? h - oa - 1 : -1)]) : (T)0;
          eR[d] = er ? (T)to_c(zp[d * sj + (MODE == kSplit ? oa + 1 : 2)]) : (T)0;
        }
        load_two<MODE>(zp - sj, jl, xa[0], xb[0], di ? 0 : h, h);
        load_two<MODE>(zp + 2 * sj, jh, xa[1], xb[1], di ? h : 0, h);
        const T wall = (T)((i == 0) + (i == sf.s0 - 1));
#pragma unroll
        for (int d = 0; d < 2; ++d) {  // row j0 + d
          T left = __shfl_up_sync(all, cb[d], 1), right = __shfl_down_sync(all, ca[d], 1);
          if (lane == 0) left = eL[d];
          if (lane == 31) right = eR[d];
          const T pa = d == 0 ? ca[1] : xa[1], pb = d == 0 ? cb[1] : xb[1];  // +j
          const T la = d == 0 ? xa[0] : ca[0], lb = d == 0 ? xb[0] : cb[0];  // -j
          T sa = (T)0, sb = (T)0;
          sa += na[d], sa += ma[d], sa += pa, sa += la, sa += cb[d], sa += left;
          sb += nb[d], sb += mb[d], sb += pb, sb += lb, sb += right, sb += ca[d];
          const T ga = rn_sub(ra[d], rn_sub(rn_mul(nd[d][0] - wall, ca[d]), sa));
          const T gb = rn_sub(rb[d], rn_sub(rn_mul(nd[d][1] - wall, cb[d]), sb));
          acc = rn_add(acc, rn_mul(ga, scale));
          acc = rn_add(acc, rn_mul(gb, scale));
        }
#pragma unroll
        for (int d = 0; d < 2; ++d) ma[d] = ca[d], mb[d] = cb[d], ca[d] = na[d], cb[d] = nb[d];
        zp += si;
        rp += si;
      }
      if (on) out[out_split ? ((I + J + K) & 1) * (sc.s2 / 2) + (K >> 1) : K] = to_s<SC>(acc);
      out += (long)sc.s1 * sc.s2;
    }
  }
}

// prolongate(l) (3D/mgpcg.py:165-168), a coarse cell's column of fine pairs per thread;
// in_split: the coarse level is stored by colour
template <typename T, typename SF, typename SC, int MODE>
__global__ void __launch_bounds__(kWalkBX* kWalkBY) k_prolong_walk(Shape sf, Shape sc, Walk w, SF* __restrict__ zf,
                                                                  const SC* __restrict__ zc, int in_split,
                                                                  const DevState* st) {
  pdl_begin();
  if (st->done) return;
  const unsigned si = (unsigned)sf.s1 * sf.s2;
  for (int it = blockIdx.x; it < w.items; it += gridDim.x) {
    int i0, i1, j, m;
    walk_item(w, it, sf.s0, i0, i1, j, m);
    const int k0 = 2 * m;
    if (j >= sf.s1 || k0 >= sf.s2) continue;
    unsigned q = ((unsigned)i0 * sf.s1 + j) * sf.s2 + (MODE == kSplit ? m : k0);
    const SC* const zcol = zc + (j >> 1) * (unsigned)sc.s2;
    const int h = sf.s2 / 2;
    const unsigned sci = (unsigned)sc.s1 * sc.s2;
#pragma unroll 4
    for (int i = i0; i < i1; ++i, q += si) {
      const int I = i >> 1, at = in_split ? ((I + (j >> 1) + m) & 1) * (sc.s2 / 2) + (m >> 1) : m;
      const T c = (T)to_c(zcol[I * sci + at]);
      const int oa = MODE == kSplit && ((i + j) & 1) ? h : 0, ob = MODE == kSplit ? h - oa : 1;
      T a, b;
      load_two<MODE>(zf + q, true, a, b, oa, h);
      zf[q + oa] = to_s<SF>(a + c);
      zf[q + ob] = to_s<SF>(b + c);
    }
  }
}

// subtract_grad_p + apply_bc (3D/mgpcg.py:401-427): a column of cells per thread, each with
// its three low faces (and the high ones at the walls)
template <typename T, typename U>
__global__ void __launch_bounds__(kWalkBX* kWalkBY) k_subgrad_walk(Shape s, Walk w, const T* __restrict__ p,
                                                                  U* __restrict__ ux, U* __restrict__ uy,
                                                                  U* __restrict__ uz) {
  pdl_begin();
  const unsigned si = (unsigned)s.s1 * s.s2;
  for (int it = blockIdx.x; it < w.items; it += gridDim.x) {
    int i0, i1, j, k;
    walk_item(w, it, s.s0, i0, i1, j, k);
    if (j >= s.s1 || k >= s.s2) continue;
    unsigned q = ((unsigned)i0 * s.s1 + j) * s.s2 + k;
    unsigned qy = ((unsigned)i0 * (s.s1 + 1) + j) * s.s2 + k;
    unsigned qz = ((unsigned)i0 * s.s1 + j) * (s.s2 + 1) + k;
    T below = i0 > 0 ? p[q - si] : (T)0;
#pragma unroll 4
    for (int i = i0; i < i1; ++i) {
      const T c = p[q];
      const U vy = j > 0 ? (U)((T)uy[qy] - (c - p[q - s.s2])) : (U)0;
      const U vz = k > 0 ? (U)((T)uz[qz] - (c - p[q - 1])) : (U)0;
      ux[q] = i > 0 ? (U)((T)ux[q] - (c - below)) : (U)0;
      uy[qy] = vy;
      uz[qz] = vz;
      if (i == s.s0 - 1) ux[q + si] = (U)0;
      if (j == s.s1 - 1) uy[qy + s.s2] = (U)0;
      if (k == s.s2 - 1) uz[qz + 1] = (U)0;
      below = c;
      q += si;
      qy += (unsigned)(s.s1 + 1) * s.s2;
      qz += (unsigned)s.s1 * (s.s2 + 1);
    }
  }
}
template <typename T, typename U>
static void launch_subgrad(const fm_grid& g, const T* p, const MacW<U>& u, cudaStream_t s) {
  if (g.dim == 3) {
    const Shape cs = cell_shape(g);
    const Walk w = walk_of(cs.s0, cs.s1, cs.s2, kWalkBlocks);
    launch_pdl(k_subgrad_walk<T, U>, (unsigned)w.items, kWalkBlock, 0, s, cs, w, p, u.c[0], u.c[1], u.c[2]);
  } else {
    const long f0 = face_shape(g, 0).size(), f1 = face_shape(g, 1).size(), n = f0 > f1 ? f0 : f1;
    launch_pdl(k_subgrad_bc2<T, U>, dim3((unsigned)((n + 255) / 256), 2), 256, 0, s, g, p, u);
  }
}

// ---------------------------------------------------------------------------
// 3D, levels stored by colour
// ---------------------------------------------------------------------------
// Whatever the kernel, an interleaved half-sweep at 128^3 takes 7.2 us: it moves 25 MB
// (z and r whole, z back) through the L2, of which it uses half.  Where every per-level
// row has 16 n cells the V-cycle of a large FP32 solver therefore stores z and r of those
// levels by colour within the row: cell k of colour c = (i + j + k) & 1 at c s2 / 2 +
// (k >> 1).  The first sweep splits the residual (into rs), the last one writes z in natural
// order (into A p's array, which is free then), so that the rest of the solver does not see
// it; a half-sweep moves 12.6 MB.  A thread updates 8 cells of a row: 16-byte loads of the
// other colour in the row and its four neighbours and of the residual.  Within a
// row the neighbours of the cell at m with sigma = (i + j + c) & 1 are the other colour's
// m + sigma (k + 1) and m + sigma - 1.  Lanes of a warp have rows of the same parity,
// so that sigma is the same for all.  128^3 FP32, us, warm: half-sweep 7.2 -> 5.2, first
// 7.8 -> 8.6 (it writes the split residual too), last with its inner product 16.6 -> 8.8,
// restriction 7.5 -> 9.2 and prolongation 5.2 -> 6.1 (walking); 64^3 in BF16 all as before (3.2 a
// half-sweep: a launch).  A V-cycle with three smoothing steps: 220 -> 180.
constexpr int kRow = 8;
// FP32 solvers of at least this many cells.  Projections of five iterations by colour and in
// natural order, us: 48^3 439 and 418, 64^3 508 and 499, 64x96x128 625 and 611, 96^3 699 and
// 702, 128^3 897 and 926 (on less, eight cells a thread leave too few threads); FP64 64^3
// 682 and 604, 128^3 1555 and 1253 (a half-sweep is then bound by its divisions).
constexpr long kSplitCells = 850000;
inline bool split_fits(const Shape& s) { return s.s2 % (2 * kRow) == 0; }
struct Rows {
  int lx, by, gx, gy, items;  // threads per row (log2), rows per block, blocks along the row and along j, blocks
};
inline Rows rows_of(const Shape& s, int threads) {
  Rows w;
  const int chunks = s.s2 / (2 * kRow);
  w.lx = 0;
  while (w.lx < 5 && (1 << w.lx) < chunks) ++w.lx;
  w.by = threads >> w.lx;
  w.gx = (chunks + (1 << w.lx) - 1) >> w.lx;
  w.gy = (s.s1 + w.by - 1) / w.by;
  w.items = w.gx * w.gy * s.s0;
  return w;
}
// block b's row group: plane i, row j, first m of a colour; false past the end.  A
// warp holds rows a multiple of the number of warps (even) apart.
__device__ __forceinline__ bool rows_at(const Rows& w, const Shape& s, int b, int& i, int& j, int& m) {
  const int tx = threadIdx.x & ((1 << w.lx) - 1), ty = threadIdx.x >> w.lx;
  const int rpw = 32 >> w.lx, nw = blockDim.x >> 5;  // rows per warp, warps
  const int bx = w.gx == 1 ? 0 : b % w.gx, t = w.gx == 1 ? b : b / w.gx;
  i = t / w.gy;
  j = (t - i * w.gy) * w.by + (ty >> (5 - w.lx)) + (ty & (rpw - 1)) * nw;
  m = ((bx << w.lx) + tx) * kRow;
  return j < s.s1 && 2 * m < s.s2;
}
// 8 cells, 16-byte aligned (zeros when `on` is false)
template <typename T>
__device__ __forceinline__ void load_row(const float* p, bool on, T* v) {
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  if (on) a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
template <typename T>
__device__ __forceinline__ void load_row(const __nv_bfloat16* p, bool on, T* v) {
  uint4 a = make_uint4(0, 0, 0, 0);
  if (on) a = *reinterpret_cast<const uint4*>(p);
  const unsigned x[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int m = 0; m < 4; ++m) v[2 * m] = (T)__uint_as_float(x[m] << 16), v[2 * m + 1] = (T)__uint_as_float(x[m] & 0xffff0000u);
}
template <typename T>
__device__ __forceinline__ void store_row(float* p, const T* v) {
  reinterpret_cast<float4*>(p)[0] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4((float)v[4], (float)v[5], (float)v[6], (float)v[7]);
}
template <typename T>
__device__ __forceinline__ void store_row(__nv_bfloat16* p, const T* v) {
  unsigned x[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const __nv_bfloat162 h = __halves2bfloat162(to_s<__nv_bfloat16>(v[2 * m]), to_s<__nv_bfloat16>(v[2 * m + 1]));
    x[m] = *reinterpret_cast<const unsigned*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(x[0], x[1], x[2], x[3]);
}

// smooth(l, phase) (3D/mgpcg.py:170-177) of a level stored by colour.  OUT: instead of into
// z the updated cells go, with the other colour's, to `out` in natural order, and
// the partial sums of z.r over all cells to part (blocks take several items then).
template <typename T, typename S, bool OUT>
__global__ void __launch_bounds__(OUT ? 256 : 128) k_smooth_split(Shape s, Rows w, const S* __restrict__ r, S* z,
                                                                int phase, S* __restrict__ out,
                                                                double* __restrict__ part, const DevState* st) {
  pdl_begin();
  if (st->done) return;
  const long sj = s.s2, si = (long)s.s1 * s.s2;
  const int h = s.s2 / 2;
  double acc = 0;
  for (int it = blockIdx.x; it < w.items; it += gridDim.x) {
    int i, j, m;
    if (!rows_at(w, s, it, i, j, m)) continue;
    const long row = (long)i * si + (long)j * sj;
    const S* const o = z + row + (1 - phase) * h + m;  // the other colour
    const int nd = 6 - (i == 0) - (i == s.s0 - 1) - (j == 0) - (j == s.s1 - 1);
    T x[kRow], ip[kRow], im[kRow], jp[kRow], jm[kRow], rv[kRow], ro[kRow], v[kRow];
    // the neighbour rows' other colour has the same place in the row
    load_row(o, true, x);
    load_row(o + si, i < s.s0 - 1, ip);
    load_row(o - si, i > 0, im);
    load_row(o + sj, j < s.s1 - 1, jp);
    load_row(o - sj, j > 0, jm);
    load_row(r + row + phase * h + m, true, rv);
    if (OUT) load_row(r + row + (1 - phase) * h + m, true, ro);
    const auto body = [&](auto sg_) {
      constexpr int SG = decltype(sg_)::value, E = SG ? kRow - 1 : 0;  // E: the cell whose outer k neighbour is another thread's
      const bool wall = SG ? m + kRow >= h : m == 0;
      const T far = wall ? (T)0 : (T)to_c(o[SG ? kRow : -1]);
      const ClQuot<T> quot(nd), quot_e(nd - wall);
      T y[kRow];
      bool bad = false;
#pragma unroll
      for (int a = 0; a < kRow; ++a) {
        T nb = (T)0;
        nb += ip[a];
        nb += im[a];
        nb += jp[a];
        nb += jm[a];
        nb += SG ? (a == kRow - 1 ? far : x[a == kRow - 1 ? a : a + 1]) : x[a];
        nb += SG ? x[a] : (a == 0 ? far : x[a == 0 ? a : a - 1]);
        y[a] = rv[a] + nb;
        v[a] = a == E ? quot_e.fast(y[a]) : quot.fast(y[a]);
        bad |= a == E ? quot_e.template bad<true>(y[a]) : quot.template bad<true>(y[a]);
      }
      if (bad) {
#pragma unroll
        for (int a = 0; a < kRow; ++a) v[a] = div_nd(y[a], a == E ? nd - wall : nd);
      }
      if constexpr (OUT) {
        T nat[2 * kRow];  // cell 2 a + SG is the updated one
#pragma unroll
        for (int a = 0; a < kRow; ++a) {
          nat[2 * a + SG] = v[a];
          nat[2 * a + 1 - SG] = x[a];
          acc += (double)v[a] * (double)rv[a];
          acc += (double)x[a] * (double)ro[a];
        }
        store_row(out + row + 2 * m, nat);
        store_row(out + row + 2 * m + kRow, nat + kRow);
      } else {
        store_row(z + row + phase * h + m, v);
      }
    };
    if ((i + j + phase) & 1) body(std::integral_constant<int, 1>());
    else body(std::integral_constant<int, 0>());
  }
  if constexpr (OUT) {
    block_reduce2(acc, 0.0, part + 2 * blockIdx.x);
    walk_clear(part);
  }
}

// First red sweep from z == 0 (the black cells need no zeros: the next half-sweep
// writes them from the red ones).  rn: the residual in natural order (the finest
// level), stored by colour into r; recentre: less its mean, also in rn.
template <typename T, typename S>
__global__ void __launch_bounds__(128) k_first_split(Shape s, Rows w, S* __restrict__ rn, S* __restrict__ r,
                                                     S* __restrict__ z, const DevState* st, int recenter) {
  pdl_begin();
  if (st->done) return;
  int i, j, m;
  if (!rows_at(w, s, blockIdx.x, i, j, m)) return;
  const int h = s.s2 / 2;
  const long row = ((long)i * s.s1 + j) * s.s2;
  const int sg = (i + j) & 1;  // the red cell of a pair
  T red[kRow];
  if (rn) {
    T nat[2 * kRow], black[kRow];
    load_row(rn + row + 2 * m, true, nat);
    load_row(rn + row + 2 * m + kRow, true, nat + kRow);
    if (recenter) {
      const T mean = (T)st->mean;
#pragma unroll
      for (int a = 0; a < 2 * kRow; ++a) nat[a] = nat[a] - mean;
      store_row(rn + row + 2 * m, nat);
      store_row(rn + row + 2 * m + kRow, nat + kRow);
    }
#pragma unroll
    for (int a = 0; a < kRow; ++a) {
      red[a] = sg ? nat[2 * a + 1] : nat[2 * a];
      black[a] = sg ? nat[2 * a] : nat[2 * a + 1];
    }
    store_row(r + row + m, red);
    store_row(r + row + h + m, black);
  } else {
    load_row(r + row + m, true, red);
  }
  const int nd = 6 - (i == 0) - (i == s.s0 - 1) - (j == 0) - (j == s.s1 - 1);
#pragma unroll
  for (int a = 0; a < kRow; ++a)
    red[a] = div_nd(red[a], nd - (a == 0 && m == 0 && !sg) - (a == kRow - 1 && m + kRow >= h && sg));
  store_row(z + row + m, red);
}

// Bottom smoothing on the coarsest level by one CTA in shared memory.
// z starts at zero (the reference zero-fills before restricting).
template <typename T, int D>
__global__ void k_bottom(Shape s, const T* __restrict__ r, T* __restrict__ z, int bottom, int mode,
                         const DevState* st) {
  pdl_begin();
  if (st->done) return;
  extern __shared__ unsigned char smem_raw[];
  T* zs = reinterpret_cast<T*>(smem_raw);
  T* rs = zs + s.size();
  const int n = (int)s.size();
  for (int q = threadIdx.x; q < n; q += blockDim.x) { zs[q] = 0; rs[q] = r[q]; }
  // per-thread cells (n <= kBottomMaxCells = 8 * blockDim): index, parity,
  // in-domain neighbour mask and diagonal computed once, outside the sweeps
  int cq[kBottomCellsPerThread], cinfo[kBottomCellsPerThread];
  const int si = s.s1 * s.s2, sj = s.s2;
#pragma unroll
  for (int m = 0; m < kBottomCellsPerThread; ++m) {
    const int q = threadIdx.x + m * blockDim.x;
    cq[m] = q;
    cinfo[m] = -1;
    if (q < n) {
      int i, j, k;
      unflatten(s, q, i, j, k);
      int mask = 0;
      mask |= (i < s.s0 - 1) << 0;
      mask |= (i > 0) << 1;
      mask |= (j < s.s1 - 1) << 2;
      mask |= (j > 0) << 3;
      if (D == 3) { mask |= (k < s.s2 - 1) << 4; mask |= (k > 0) << 5; }
      cinfo[m] = mask | (parity<D>(i, j, k) << 6);
    }
  }
  __syncthreads();
  auto sweep = [&](int phase) {
#pragma unroll
    for (int m = 0; m < kBottomCellsPerThread; ++m) {
      const int info = cinfo[m];
      if (info >= 0 && (info >> 6) == phase) {
        const int q = cq[m];
        T nb = 0;
        if (info & 1) nb += zs[q + si];
        if (info & 2) nb += zs[q - si];
        if (info & 4) nb += zs[q + sj];
        if (info & 8) nb += zs[q - sj];
        if (D == 3) {
          if (info & 16) nb += zs[q + 1];
          if (info & 32) nb += zs[q - 1];
        }
        zs[q] = div_nd(rs[q] + nb, __popc(info & 63));
      }
    }
    __syncthreads();
  };
  if (mode == 0) {
    for (int it = 0; it < bottom; ++it) { sweep(0); sweep(1); }
  } else {
    for (int it = 0; it < bottom / 2; ++it) { sweep(0); sweep(1); }
    for (int it = 0; it < bottom / 2; ++it) { sweep(1); sweep(0); }
  }
  for (long q = threadIdx.x; q < n; q += blockDim.x) z[q] = zs[q];
}

template <typename T, int D>
__global__ void k_laplacian(Shape s, const T* __restrict__ p, T* __restrict__ Ap) {
  pdl_begin();
  FM_GRID_STRIDE(q, s.size()) {
    int i, j, k;
    unflatten(s, q, i, j, k);
    T diag;
    const T nb = nb_sum<T, D>(p, s, i, j, k, diag);
    Ap[q] = rn_sub(rn_mul(diag, p[q]), nb);
  }
}

// k_pcg_cluster's connection to the solver state
__device__ __forceinline__ bool pcg_skip(const DevState* st) { return st->dc_done != 0; }  // 0 outside fm_project_dc
__device__ __forceinline__ double pcg_floor(const DevState* st) { return st->dc_tol; }
__device__ __forceinline__ void pcg_finish(DevState* st, const PcgOutcome& R) {
  st->zTr_old = R.zTr;
  st->tol = R.tol;
  st->alpha = R.alpha;
  st->beta = R.beta;
  st->mean = R.mean;
  st->pAp = R.pAp;
  if (R.stepped) st->rTr = R.rTr;
  st->it = R.it;
  st->conv = R.conv;
  st->nonfinite = R.nonfinite;
  finish_solve(st);
}

}  // namespace fm

#include "fm_mg_ring.cuh"

using namespace fm;

struct fm_mgpcg {
  fm_grid g;
  int dtype;
  fm_mg_params P;
  int L;
  Shape lv[kMaxLevels];
  void* r[kMaxLevels];
  void* z[kMaxLevels];
  void* x;
  void* p;
  void* Ap;
  void* rs;        // the finest residual by colour, for V-cycles on levels stored so (null: natural order)
  double* part;
  DevState* st;
  DevState* h_st;  // pinned
  cudaStream_t cap;
  cudaGraphExec_t prologue;    // recentring, first V-cycle, p = z, zTr
  long long prologue_kernels;
  cudaGraphExec_t chunk;       // host-checked mode: check_every iterations
  long long chunk_kernels;
  cudaGraphExec_t loop;        // device mode: conditional WHILE node around one iteration
  long long loop_kernels;      // kernels per loop iteration
  size_t bottom_smem;
  int lc;                      // levels lc .. L-1 run as one cluster launch (<= 0: per-level launches)
  int nc;                      // CTAs in that cluster
  size_t coarse_smem;
  bool push;                   // which kernel: k_mg_coarse ...
  ClArgs coarse;
  RingArgs ring;               // ... or k_mg_ring
  ClArgs* d_coarse;
  int pcg_nc;                  // CTAs of the cluster that runs a whole solve (0: the solve is a sequence of launches)
  size_t pcg_smem;
  ClArgs pcg;
  ClArgs* d_pcg;
  int bf16_hi;                 // levels 1 .. bf16_hi-1 stored in BF16 (0: none)
};

namespace fm {

// Picks the finest level lc >= 1 from which the rest of the V-cycle runs as one
// cluster launch: level lc split into nc <= 8 slabs (enable_coarse: 16) of an even number of
// planes, every slab and every deeper level at most 4096 cells (two pairs per thread:
// beyond that a per-level launch spread over the chip is faster).  lc = -1 when
// no level qualifies (the V-cycle launches per level).
constexpr int kCoarseMaxNC = 8;
constexpr long kCoarseMaxPairs = 2 * kClThreads;
static_assert(kRingThreads == kClThreads && kRingPPT == 2, "one rule for both kernels");

// Which kernel that is: k_mg_coarse in 3D FP32, k_mg_ring in 3D FP64 (fm_mg_ring.cuh has the figures).  In 2D the ring,
// unless the coarsest level is so large that its sweeps decide and its rows are multiples of 32 cells, whose
// natural order meets bank conflicts (V-cycles on four levels, us, ring / push: FP32 512^2 and 448x512 84.3 / 78.1, 83.0 /
// 78.4, without such rows 384^2 74.4 / 74.9, 416^2 81.1 / 81.5; FP64 256^2 68.5 / 65.1,
// 512x256 79.5 / 74.7, without 304^2 79.9 / 81.9).  In FP64 the push kernel takes only one pair a thread in
// registers (384^2 83.0 / 104.9).
template <typename T, int D>
constexpr bool kCanPush = D == 2 || sizeof(T) == 4;
template <typename T, int D>
constexpr bool kCanRing = D == 2 || sizeof(T) == 8;

static long coarse_pairs(const Shape& s, int dim, int planes) {
  const long nin = dim == 3 ? s.s2 : s.s1;
  return (long)planes * (dim == 3 ? s.s1 : 1) * ((nin + 1) / 2);
}
static long coarse_ring(const Shape& s, int dim, int planes) {
  return (long)planes * (s.s1 + 2) * (dim == 3 ? s.s2 + 2 : 1);
}

// k_mg_ring's shared memory for level lc on nc CTAs: slab, then CTA 0's deep levels (compact r, zero-ringed z).
static size_t ring_layout(RingArgs& a, const fm_mgpcg* S, int lc, int nc, size_t es) {
  const int dim = S->g.dim;
  long off = 0;
  for (int l = 0; l < S->L; ++l) {
    const Shape& t = S->lv[l];
    a.lv[l] = t;
    a.roff[l] = a.zoff[l] = 0;
    if (l <= lc) continue;
    a.roff[l] = (int)off;
    a.zoff[l] = (int)(off + t.size());
    off += t.size() + coarse_ring(t, dim, t.s0 + 2);
  }
  a.lc = lc;
  a.L = S->L;
  a.pre_post = S->P.pre_post;
  a.bottom = S->P.bottom;
  a.bottom_mode = S->P.bottom_mode;
  const Shape& t = S->lv[lc];
  const int planes = t.s0 / nc;
  return es * (size_t)(off + coarse_ring(t, dim, planes + 2) + (long)planes * t.s1 * t.s2);
}

template <typename T, int D>
static bool push_coarse(const fm_mgpcg* S) {
  if (D == 3) return kCanPush<T, D>;
  const Shape& b = S->lv[S->L - 1];
  const long pairs = coarse_pairs(b, D, b.s0);
  return b.s1 % 32 == 0 && pairs >= 512 && pairs <= (sizeof(T) == 4 ? kCoarseMaxPairs : (long)kClThreads);
}

template <typename T, int D>
static void plan_coarse(fm_mgpcg* S) {
  S->push = push_coarse<T, D>(S);
  S->lc = -1;
  S->nc = 0;
  S->coarse_smem = 0;
  for (int l = 1; l < S->L - 1; ++l) {
    const Shape t = S->lv[l];
    int nc = kCoarseMaxNC;
    while (nc > 1 && t.s0 % (2 * nc) != 0) nc >>= 1;
    if (t.s0 % (2 * nc) != 0 || coarse_pairs(t, D, t.s0 / nc) > kCoarseMaxPairs) continue;
    bool fits = true;
    for (int m = l + 1; m < S->L; ++m) fits = fits && coarse_pairs(S->lv[m], D, S->lv[m].s0) <= kCoarseMaxPairs;
    const size_t smem = S->push ? cl_layout(S->coarse, S->lv, l, l + 1, S->L, D, sizeof(T), nc, false, false)
                                : ring_layout(S->ring, S, l, nc, sizeof(T));
    if (!fits || smem == 0 || smem > (S->push ? kClMaxSmem : 200 * 1024)) continue;
    S->lc = l;
    S->nc = nc;
    S->coarse_smem = smem;
    S->coarse.pre_post = S->P.pre_post;
    S->coarse.bottom = S->P.bottom;
    S->coarse.bottom_mode = S->P.bottom_mode;
    return;
  }
}

// Makes the plan launchable.  Slabs of more than one pair a thread are halved over 16 CTAs
// (beyond the portable cluster size) where the device takes such a cluster: 32^3 on
// 16 CTAs instead of 8, FP32, a 128^3 projection: 443 -> 434 us.
template <typename T, int D>
static bool enable_coarse(fm_mgpcg* S) {
  if constexpr (kCanPush<T, D>)
    if (S->push) {
      const Shape t = S->lv[S->lc];
      const int nc = 2 * kCoarseMaxNC;
      if (S->nc == kCoarseMaxNC && t.s0 % (2 * nc) == 0 && coarse_pairs(t, D, t.s0 / S->nc) > kClThreads) {
        ClArgs a = S->coarse;
        const size_t smem = cl_layout(a, S->lv, S->lc, S->lc + 1, S->L, D, sizeof(T), nc, false, false);
        if (smem > 0 && smem <= kClMaxSmem && cl_enable(k_mg_coarse<T, D, DevState>, nc, smem)) {
          S->coarse = a;
          S->nc = nc;
          S->coarse_smem = smem;
          return true;
        }
        cudaGetLastError();
      }
      return raise_smem_limit(k_mg_coarse<T, D, DevState>, S->coarse_smem);
    }
  if constexpr (kCanRing<T, D>) return raise_smem_limit(k_mg_ring<T, D>, S->coarse_smem);
  return false;
}

// The coarse levels in one cluster launch where they fit.
template <typename T, int D>
static void plan_coarse_t(fm_mgpcg* S) {
  plan_coarse<T, D>(S);
  if (S->lc > 0 && !enable_coarse<T, D>(S)) {
    cudaGetLastError();
    S->lc = -1;
  }
}

template <typename T, int D>
static void plan_pcg_t(fm_mgpcg* S) {
  S->pcg_nc = cl_plan_pcg(S->pcg, k_pcg_cluster<T, D, false, DevState*>, S->lv, S->L, S->P, D, sizeof(T), false,
                          &S->pcg_smem);
  // Near the top of the range the largest slab decides: where it is a fifth above the mean and over 10 500 cells the
  // launches are as fast, if they have a coarse-level kernel (projections of five levels, us, launches / one cluster:
  // 288x448 798 / 807, 320x448 768 / 781; smaller slabs, 400x320 868 / 821, 272x432 815 / 799, 304x384 816 / 726;
  // without a coarse-level kernel, 400x352 on four levels, 2039 / 1618).
  const long slab = S->pcg_nc ? (long)S->pcg.lv[0].pmax * S->lv[0].s1 : 0;
  if (D == 2 && sizeof(T) == 4 && S->lc > 0 && slab > 10500 && 5 * slab * S->pcg_nc >= 6 * S->lv[0].size()) S->pcg_nc = 0;
}

static inline unsigned blocks_for(long n, int threads, long cap) {
  long b = (n + threads - 1) / threads;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

// Levels lc .. L-1 of the V-cycle as one cluster launch.
template <typename T, int D>
static void launch_coarse(fm_mgpcg* S, cudaStream_t s) {
  if constexpr (kCanPush<T, D>)
    if (S->push) {
      cl_launch(k_mg_coarse<T, D, DevState>, S->nc, S->coarse_smem, s, (const ClArgs*)S->d_coarse, (const T*)S->r[S->lc],
                (T*)S->z[S->lc], (const DevState*)S->st);
      return;
    }
  if constexpr (kCanRing<T, D>) {
    RingArgs a = S->ring;
    a.r_top = S->r[S->lc];
    a.z_top = S->z[S->lc];
    cl_launch(k_mg_ring<T, D>, S->nc, S->coarse_smem, s, a, (const DevState*)S->st);
  }
}

// Where a V-cycle leaves its result, in natural order.
static void* zout(const fm_mgpcg* S) { return S->rs ? S->Ap : S->z[0]; }

// One V-cycle (apply_preconditioner, 3D/mgpcg.py:187-205) on r[0] -> zout.
// recenter: subtract st->mean from r[0] first (fused into the first sweep);
// dot_last: the last fine sweep also writes z.r block partials.
template <typename T, int D>
static void launch_vcycle(fm_mgpcg* S, cudaStream_t s, bool dot_last, bool recenter = true) {
  const int L = S->L;
  const fm_mg_params& P = S->P;
  T** r = (T**)S->r;
  T** z = (T**)S->z;
  const long cap = 148L * 16;
  const int lc = S->lc > 0 ? S->lc : L - 1;  // first level not smoothed by per-level launches
  const dim3 pblk(kPairBX, kPairBY, 1);
  auto pair_grid = [](const Shape& sh) {
    if (D == 3)
      return dim3((unsigned)((sh.s2 + 1) / 2 + kPairBX - 1) / kPairBX, (unsigned)(sh.s1 + kPairBY - 1) / kPairBY,
                  (unsigned)sh.s0);
    return dim3((unsigned)((sh.s1 + 1) / 2 + kPairBX - 1) / kPairBX, (unsigned)(sh.s0 + kPairBY - 1) / kPairBY, 1);
  };
  // level storage: T, or BF16 for levels 1 .. bf16_hi-1 (FP32 solvers with coarse_bf16)
  using BF = __nv_bfloat16;
  auto bf = [&](int l) { return std::is_same<T, float>::value && l >= 1 && l < S->bf16_hi; };
  constexpr bool kCanSplit = D == 3 && std::is_same<T, float>::value;
  const bool split = kCanSplit && S->rs;  // the per-level levels are stored by colour
  auto rl = [&](int l) { return l == 0 && split ? (T*)S->rs : r[l]; };
  auto sweep = [&](int l, int phase) {
    const Shape sh = S->lv[l];
    if constexpr (kCanSplit) {
      if (split) {
        const Rows w = rows_of(sh, 128);
        if (bf(l)) launch_pdl(k_smooth_split<T, BF, false>, (unsigned)w.items, 128, 0, s, sh, w, (const BF*)S->r[l], (BF*)S->z[l], phase, (BF*)nullptr, nullptr, S->st);
        else launch_pdl(k_smooth_split<T, T, false>, (unsigned)w.items, 128, 0, s, sh, w, (const T*)rl(l), z[l], phase, (T*)nullptr, nullptr, S->st);
        return;
      }
    }
    if (bf(l)) launch_pdl(k_smooth_pair<T, D, BF>, pair_grid(sh), pblk, 0, s, sh, (const BF*)S->r[l], (BF*)S->z[l], phase, S->st);
    else launch_pdl(k_smooth_pair<T, D>, pair_grid(sh), pblk, 0, s, sh, (const T*)r[l], z[l], phase, S->st);
  };
  auto first_sweep = [&](int l) {
    const Shape sh = S->lv[l];
    const int rec = l == 0 && recenter ? 1 : 0;
    if constexpr (kCanSplit) {
      if (split) {
        const Rows w = rows_of(sh, 128);
        if (bf(l)) launch_pdl(k_first_split<T, BF>, (unsigned)w.items, 128, 0, s, sh, w, (BF*)nullptr, (BF*)S->r[l], (BF*)S->z[l], S->st, 0);
        else launch_pdl(k_first_split<T, T>, (unsigned)w.items, 128, 0, s, sh, w, l == 0 ? r[0] : (T*)nullptr, rl(l), z[l], S->st, rec);
        return;
      }
    }
    if (bf(l)) launch_pdl(k_smooth_first_pair<T, D, BF>, pair_grid(sh), pblk, 0, s, sh, (BF*)S->r[l], (BF*)S->z[l], S->st, 0);
    else launch_pdl(k_smooth_first_pair<T, D>, pair_grid(sh), pblk, 0, s, sh, r[l], z[l], S->st, rec);
  };
  for (int l = 0; l < lc; ++l) {
    const Shape sh = S->lv[l];
    for (int it = 0; it < P.pre_post; ++it) {
      if (it == 0) first_sweep(l);
      else sweep(l, 0);
      sweep(l, 1);
    }
    const Shape sc = S->lv[l + 1];
    if constexpr (D == 3) {
      const Walk w = walk_of(sc.s0, sc.s1, sc.s2, kWalkBlocks);
      auto go = [&](auto* rf, auto* zf, auto* rc) {
        using SF = std::remove_pointer_t<decltype(rf)>;
        const int out_split = split && l + 1 < lc;
        using SC = std::remove_pointer_t<decltype(rc)>;
        auto k = k_restrict_walk<T, SF, SC, kVec>;
        if constexpr (kCanSplit) k = split ? k_restrict_walk<T, SF, SC, kSplit> : k;
        launch_pdl(k, (unsigned)w.items, kWalkBlock, 0, s, sh, sc, w, (const SF*)rf, (const SF*)zf, rc, out_split, (const DevState*)S->st);
      };
      if (bf(l) && bf(l + 1)) go((BF*)S->r[l], (BF*)S->z[l], (BF*)S->r[l + 1]);
      else if (bf(l)) go((BF*)S->r[l], (BF*)S->z[l], r[l + 1]);
      else if (bf(l + 1)) go(rl(l), z[l], (BF*)S->r[l + 1]);
      else go(rl(l), z[l], r[l + 1]);
    } else {
      const unsigned rb = blocks_for(sc.size(), 256, cap);
      if (bf(l) && bf(l + 1))
        launch_pdl(k_restrict<T, BF, BF>, rb, 256, 0, s, sh, sc, (const BF*)S->r[l], (const BF*)S->z[l], (BF*)S->r[l + 1], S->st);
      else if (bf(l))
        launch_pdl(k_restrict<T, BF, T>, rb, 256, 0, s, sh, sc, (const BF*)S->r[l], (const BF*)S->z[l], r[l + 1], S->st);
      else if (bf(l + 1))
        launch_pdl(k_restrict<T, T, BF>, rb, 256, 0, s, sh, sc, (const T*)r[l], (const T*)z[l], (BF*)S->r[l + 1], S->st);
      else
        launch_pdl(k_restrict<T>, rb, 256, 0, s, sh, sc, (const T*)r[l], (const T*)z[l], r[l + 1], S->st);
    }
  }
  const Shape sb = S->lv[L - 1];
  if (S->lc > 0) {
    launch_coarse<T, D>(S, s);
  } else if (S->bottom_smem) {
    launch_pdl(k_bottom<T, D>, 1, kBottomThreads, S->bottom_smem, s, sb, r[L - 1], z[L - 1], P.bottom, P.bottom_mode,
           S->st);
  } else {
    // large coarsest level: per-sweep launches (z zero-filled by the first sweep)
    const unsigned nb = blocks_for(sb.size(), 256, cap);
    int first = 1;
    auto pair = [&](int a, int b) {
      if (first && a == 0) launch_pdl(k_smooth_first<T, D>, nb, 256, 0, s, sb, r[L - 1], z[L - 1], S->st, 0);
      else {
        if (first) cudaMemsetAsync(z[L - 1], 0, sizeof(T) * sb.size(), s);
        launch_pdl(k_smooth<T, D, false>, nb, 256, 0, s, sb, r[L - 1], z[L - 1], a, nullptr, S->st);
      }
      first = 0;
      launch_pdl(k_smooth<T, D, false>, nb, 256, 0, s, sb, r[L - 1], z[L - 1], b, nullptr, S->st);
    };
    if (P.bottom_mode == 0) for (int i = 0; i < P.bottom; ++i) pair(0, 1);
    else {
      for (int i = 0; i < P.bottom / 2; ++i) pair(0, 1);
      for (int i = 0; i < P.bottom / 2; ++i) pair(1, 0);
    }
    if (first) cudaMemsetAsync(z[L - 1], 0, sizeof(T) * sb.size(), s);  // no bottom sweeps
  }
  for (int l = lc - 1; l >= 0; --l) {
    const Shape sh = S->lv[l];
    const Shape sc = S->lv[l + 1];
    if constexpr (D == 3) {
      const Walk w = walk_pairs(sh, kWalkBlocks);
      auto go = [&](auto* zf, auto* zc) {
        using SF = std::remove_pointer_t<decltype(zf)>;
        using SC = std::remove_pointer_t<decltype(zc)>;
        auto k = k_prolong_walk<T, SF, SC, kVec>;
        if constexpr (kCanSplit) k = split ? k_prolong_walk<T, SF, SC, kSplit> : k;
        launch_pdl(k, (unsigned)w.items, kWalkBlock, 0, s, sh, sc, w, zf, (const SC*)zc, (int)(split && l + 1 < lc),
                   (const DevState*)S->st);
      };
      if (bf(l) && bf(l + 1)) go((BF*)S->z[l], (BF*)S->z[l + 1]);
      else if (bf(l)) go((BF*)S->z[l], z[l + 1]);
      else if (bf(l + 1)) go(z[l], (BF*)S->z[l + 1]);
      else go(z[l], z[l + 1]);
    } else {
      const unsigned nb = blocks_for(sh.size(), 256, cap);
      if (bf(l) && bf(l + 1))
        launch_pdl(k_prolong<T, BF, BF>, nb, 256, 0, s, sh, sc, (BF*)S->z[l], (const BF*)S->z[l + 1], S->st);
      else if (bf(l))
        launch_pdl(k_prolong<T, BF, T>, nb, 256, 0, s, sh, sc, (BF*)S->z[l], (const T*)z[l + 1], S->st);
      else if (bf(l + 1))
        launch_pdl(k_prolong<T, T, BF>, nb, 256, 0, s, sh, sc, z[l], (const BF*)S->z[l + 1], S->st);
      else
        launch_pdl(k_prolong<T>, nb, 256, 0, s, sh, sc, z[l], (const T*)z[l + 1], S->st);
    }
    for (int it = 0; it < P.pre_post; ++it) {
      sweep(l, 1);
      const bool end = l == 0 && it == P.pre_post - 1, last = dot_last && end;
      if constexpr (kCanSplit) {
        if (end && split) {
          const Rows w = rows_of(sh, 256);
          launch_pdl(k_smooth_split<T, T, true>, (unsigned)(w.items < kRedBlocks ? w.items : kRedBlocks), 256, 0, s, sh, w,
                     (const T*)S->rs, z[0], 0, (T*)S->Ap, S->part, S->st);
          continue;
        }
      }
      if (!last) {
        sweep(l, 0);
      } else if constexpr (kWalkDots<T, D>) {
        const Walk w = walk_pairs(sh, kRedBlocks);
        launch_pdl(k_smooth_dot_walk<T>, (unsigned)(w.items < kRedBlocks ? w.items : kRedBlocks), kWalkBlock, 0, s, sh, w,
                   (const T*)r[l], z[l], 0, S->part, S->st);
      } else {
        launch_pdl(k_smooth<T, D, true>, kRedBlocks, kRedThreads, 0, s, sh, r[l], z[l], 0, S->part, S->st);
      }
    }
  }
}

// x += alpha p, r -= alpha A p and the convergence test: the second half of a
// PCG iteration (3D/mgpcg.py:240-260).
template <typename T, int D>
static void launch_step(fm_mgpcg* S, cudaStream_t s) {
  const Shape s0 = S->lv[0];
  const long n = s0.size();
  if constexpr (kWalkDots<T, D>) {
    const Walk w = walk_pairs(s0, kRedBlocks);
    launch_pdl(k_Ap_walk<T>, (unsigned)(w.items < kRedBlocks ? w.items : kRedBlocks), kWalkBlock, 0, s, s0, w, (const T*)S->p,
               (T*)S->Ap, S->part, S->st);
  } else {
    launch_pdl(k_Ap_dot<T, D>, kRedBlocks, kRedThreads, 0, s, s0, (T*)S->p, (T*)S->Ap, S->part, S->st);
  }
  launch_pdl(k_fin_alpha, 1, 256, 0, s, S->st, S->part, S->P.eps);
  launch_pdl(k_update_xr<T>, kRedBlocks, kRedThreads, 0, s, n, (T*)S->x, (T*)S->r[0], (T*)S->p, (T*)S->Ap,
             S->part, S->st);
  launch_pdl(k_fin_conv, 1, 256, 0, s, S->st, S->part, (double)n);
}

// One PCG iteration (3D/mgpcg.py:240-284) as a fixed launch sequence, rotated
// so that the convergence test ends it: z = M r, beta, p = z + beta p, then the
// next x / r update and its test.  A solve that converges stops right after
// its test, with no V-cycle of early-returning kernels behind it; the kernels
// run in the same order as the unrotated loop, so results are unchanged.
template <typename T, int D>
static void launch_iteration(fm_mgpcg* S, cudaStream_t s) {
  const long n = S->lv[0].size();
  launch_vcycle<T, D>(S, s, true);
  launch_pdl(k_fin_beta, 1, 256, 0, s, S->st, S->part, S->P.eps, S->P.abs_tol, S->P.rel_tol, S->P.max_iters, 0);
  launch_pdl(k_update_p<T>, blocks_for(n, 256, 148L * 16), 256, 0, s, n, (T*)S->p, (const T*)zout(S), S->st, 0);
  launch_step<T, D>(S, s);
}

// Prologue after r0 = b and partial sums of b: recentre, V-cycle, p = z, zTr,
// and the first x / r update with its convergence test.
template <typename T, int D>
static void launch_prologue(fm_mgpcg* S, cudaStream_t s) {
  const long n = S->lv[0].size();
  launch_pdl(k_fin_mean, 1, 256, 0, s, S->st, S->part, (double)n);
  launch_vcycle<T, D>(S, s, true);
  launch_pdl(k_fin_beta, 1, 256, 0, s, S->st, S->part, S->P.eps, S->P.abs_tol, S->P.rel_tol, S->P.max_iters, 1);
  launch_pdl(k_update_p<T>, blocks_for(n, 256, 148L * 16), 256, 0, s, n, (T*)S->p, (const T*)zout(S), S->st, 1);
  launch_step<T, D>(S, s);
}

// Device mode: one graph holding a conditional WHILE node whose body is one PCG
// iteration followed by k_loop_cond.  The solve then needs no host round trip.
template <typename T>
static int build_loop_graph(fm_mgpcg* S) {
  const int D = S->g.dim;
  cudaGraph_t graph = nullptr;
  if (cudaGraphCreate(&graph, 0) != cudaSuccess) return FM_ERR_CUDA;
  int status = FM_ERR_CUDA;
  do {
    cudaGraphConditionalHandle h;
    if (cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault) != cudaSuccess) break;
    cudaKernelNodeParams kp = {};
    DevState* st_arg = S->st;
    void* kargs[2] = {&h, &st_arg};
    kp.func = (void*)k_loop_init;
    kp.gridDim = dim3(1, 1, 1);
    kp.blockDim = dim3(1, 1, 1);
    kp.kernelParams = kargs;
    cudaGraphNode_t init;
    if (cudaGraphAddKernelNode(&init, graph, nullptr, 0, &kp) != cudaSuccess) break;
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    if (cudaGraphAddNode(&node, graph, &init, 1, &cp) != cudaSuccess) break;
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    if (cudaStreamBeginCaptureToGraph(S->cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) !=
        cudaSuccess)
      break;
    const long long before = g_launch_count.load();
    if (D == 3) launch_iteration<T, 3>(S, S->cap); else launch_iteration<T, 2>(S, S->cap);
    launch_pdl(k_loop_cond, 1, 1, 0, S->cap, h, S->st);
    S->loop_kernels = g_launch_count.load() - before;
    g_launch_count.fetch_sub(S->loop_kernels);
    cudaGraph_t captured = nullptr;
    if (cudaStreamEndCapture(S->cap, &captured) != cudaSuccess) break;
    if (cudaGraphInstantiate(&S->loop, graph, 0) != cudaSuccess) { S->loop = nullptr; break; }
    status = FM_OK;
  } while (0);
  cudaGraphDestroy(graph);
  cudaGetLastError();
  return status;
}

// The prologue (~45 kernels, internal buffers only) captured once into a graph.
template <typename T>
static int build_prologue_graph(fm_mgpcg* S) {
  cudaGraph_t graph;
  if (cudaStreamBeginCapture(S->cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return FM_ERR_CUDA;
  const long long before = g_launch_count.load();
  if (S->g.dim == 3) launch_prologue<T, 3>(S, S->cap); else launch_prologue<T, 2>(S, S->cap);
  S->prologue_kernels = g_launch_count.load() - before;
  g_launch_count.fetch_sub(S->prologue_kernels);  // captured, not executed
  if (cudaStreamEndCapture(S->cap, &graph) != cudaSuccess) return FM_ERR_CUDA;
  const cudaError_t e = cudaGraphInstantiate(&S->prologue, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) { S->prologue = nullptr; return FM_ERR_CUDA; }
  return FM_OK;
}

// True while `s` records into a CUDA graph (a caller capturing a whole
// gradient); the solver then adds its work to that graph instead of launching
// its own executable graphs.
static bool stream_capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) return false;
  return cs == cudaStreamCaptureStatusActive;
}

// A device-mode solve recorded into the graph being captured on `s`: the
// prologue's kernels go onto `s`, and the PCG loop becomes a conditional WHILE
// node appended to the captured graph (after the prologue), its body one PCG
// iteration and k_loop_cond recorded from S->cap.  Every solve recorded this
// way owns its own node and condition handle.
template <typename T>
static int capture_solve(fm_mgpcg* S, cudaStream_t s) {
  const int D = S->g.dim;
  if (D == 3) launch_prologue<T, 3>(S, s); else launch_prologue<T, 2>(S, s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e);
  cudaStreamCaptureStatus cs;
  cudaGraph_t graph = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t ndeps = 0;
  if ((e = cudaStreamGetCaptureInfo(s, &cs, nullptr, &graph, &deps, &ndeps)) != cudaSuccess) return cuda_fail(e);
  if (cs != cudaStreamCaptureStatusActive) return cuda_fail(cudaErrorStreamCaptureInvalidated);
  cudaGraphConditionalHandle h;
  if ((e = cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault)) != cudaSuccess)
    return cuda_fail(e);
  k_loop_init<<<1, 1, 0, s>>>(h, S->st);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e);
  if ((e = cudaStreamGetCaptureInfo(s, &cs, nullptr, &graph, &deps, &ndeps)) != cudaSuccess) return cuda_fail(e);
  cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  if ((e = cudaGraphAddNode(&node, graph, deps, ndeps, &cp)) != cudaSuccess) return cuda_fail(e);
  if ((e = cudaStreamUpdateCaptureDependencies(s, &node, 1, cudaStreamSetCaptureDependencies)) != cudaSuccess)
    return cuda_fail(e);
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  if ((e = cudaStreamBeginCaptureToGraph(S->cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
      cudaSuccess)
    return cuda_fail(e);
  const long long before = g_launch_count.load();
  if (D == 3) launch_iteration<T, 3>(S, S->cap); else launch_iteration<T, 2>(S, S->cap);
  launch_pdl(k_loop_cond, 1, 1, 0, S->cap, h, S->st);
  g_launch_count.fetch_sub(g_launch_count.load() - before);  // the loop body runs a data-dependent number of times
  cudaGraph_t captured = nullptr;
  if ((e = cudaStreamEndCapture(S->cap, &captured)) != cudaSuccess) return cuda_fail(e);
  return FM_OK;
}

// The outcome of the solve just enqueued on s (a host synchronisation).
static int read_outcome(fm_mgpcg* S, cudaStream_t s, int* iters, double* rtr) {
  if (cudaMemcpyAsync(S->h_st, S->st, sizeof(DevState), cudaMemcpyDeviceToHost, s) != cudaSuccess) return FM_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return FM_ERR_CUDA;
  if (iters) *iters = S->h_st->result_it;
  if (rtr) *rtr = S->h_st->rTr;
  if (S->h_st->nonfinite) return FM_ERR_NONFINITE;
  if (!S->h_st->conv) return FM_ERR_NOT_CONVERGED;
  return FM_OK;
}

template <typename T>
static int run_solve(fm_mgpcg* S, cudaStream_t s, int* iters, double* rtr) {
  const int D = S->g.dim;
  if (stream_capturing(s)) {
    // recorded, not run: no host read of the outcome, no host-checked loop
    if (iters || rtr || S->P.check_every != 0) return FM_ERR_ARG;
    if (!S->pcg_nc) return capture_solve<T>(S, s);
  }
  if (S->pcg_nc) {
    const PcgParams pp{S->P.max_iters, S->P.abs_tol, S->P.rel_tol, S->P.eps};
    auto go = [&](auto k) { cl_launch(k, S->pcg_nc, S->pcg_smem, s, (const ClArgs*)S->d_pcg, pp, (const T*)S->r[0], (T*)S->x, S->st); };
    if (D == 3) go(k_pcg_cluster<T, 3, false, DevState*>);
    else go(k_pcg_cluster<T, 2, false, DevState*>);
    const int e = check_cuda();
    if (e) return e;
    if (S->P.check_every == 0 && !iters && !rtr) return FM_OK;  // asynchronous: outcome via fm_mgpcg_stats
    return read_outcome(S, s, iters, rtr);
  }
  if (!S->prologue) {
    const int e = build_prologue_graph<T>(S);
    if (e) return e;
  }
  if (cudaGraphLaunch(S->prologue, s) != cudaSuccess) return FM_ERR_CUDA;
  count_launch(S->prologue_kernels);
  if (S->P.check_every == 0) {
    if (!S->loop) {
      int e = build_loop_graph<T>(S);
      if (e) return e;
    }
    if (cudaGraphLaunch(S->loop, s) != cudaSuccess) return FM_ERR_CUDA;
    if (!iters && !rtr) return FM_OK;  // asynchronous: outcome via fm_mgpcg_stats
    return read_outcome(S, s, iters, rtr);
  }
  if (!S->chunk) {
    cudaGraph_t graph;
    if (cudaStreamBeginCapture(S->cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return FM_ERR_CUDA;
    const long long before = g_launch_count.load();
    for (int i = 0; i < S->P.check_every; ++i) {
      if (D == 3) launch_iteration<T, 3>(S, S->cap); else launch_iteration<T, 2>(S, S->cap);
    }
    // captured, not executed: count them per graph launch instead
    S->chunk_kernels = g_launch_count.load() - before;
    g_launch_count.fetch_sub(S->chunk_kernels);
    if (cudaStreamEndCapture(S->cap, &graph) != cudaSuccess) return FM_ERR_CUDA;
    cudaError_t e = cudaGraphInstantiate(&S->chunk, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) { S->chunk = nullptr; return FM_ERR_CUDA; }
  }
  long launched = 0;
  const long limit = (long)S->P.max_iters + S->P.check_every;
  for (;;) {
    if (cudaGraphLaunch(S->chunk, s) != cudaSuccess) return FM_ERR_CUDA;
    count_launch(S->chunk_kernels);
    launched += S->P.check_every;
    if (cudaMemcpyAsync(S->h_st, S->st, sizeof(DevState), cudaMemcpyDeviceToHost, s) != cudaSuccess) return FM_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return FM_ERR_CUDA;
    if (S->h_st->done || launched >= limit) break;
  }
  if (iters) *iters = S->h_st->result_it;
  if (rtr) *rtr = S->h_st->rTr;
  if (S->h_st->nonfinite) return FM_ERR_NONFINITE;
  if (!S->h_st->conv) return FM_ERR_NOT_CONVERGED;
  return FM_OK;
}

}  // namespace fm

extern "C" {

int fm_mgpcg_create(const fm_grid* g, int dtype, const fm_mg_params* params, fm_mgpcg** out) {
  if (!out || !params) return FM_ERR_ARG;
  *out = nullptr;
  int st = validate_grid(g, dtype);
  if (st) return st;
  const fm_mg_params& P = *params;
  if (P.levels < 2 || P.levels > kMaxLevels || P.pre_post < 1 || P.bottom < 0 || P.max_iters < 1 ||
      P.check_every < 0 || (P.bottom_mode != 0 && P.bottom_mode != 1))
    return FM_ERR_ARG;
  if (P.coarse_bf16 && dtype != FM_F32) return FM_ERR_ARG;
  for (int a = 0; a < g->dim; ++a)
    if (g->n[a] % (1 << (P.levels - 1)) != 0 || (g->n[a] >> (P.levels - 1)) < 1) return FM_ERR_SHAPE;
  fm_mgpcg* S = (fm_mgpcg*)calloc(1, sizeof(fm_mgpcg));
  if (!S) return FM_ERR_ARG;
  S->g = *g;
  S->dtype = dtype;
  S->P = P;
  S->L = P.levels;
  const size_t es = dtype == FM_F32 ? sizeof(float) : sizeof(double);
  bool ok = true;
  for (int l = 0; l < S->L; ++l) {
    Shape sh{1, 1, 1};
    sh.s0 = g->n[0] >> l;
    sh.s1 = g->n[1] >> l;
    sh.s2 = g->dim == 3 ? (g->n[2] >> l) : 1;
    S->lv[l] = sh;
  }
  if (dtype == FM_F32) g->dim == 3 ? plan_coarse_t<float, 3>(S) : plan_coarse_t<float, 2>(S);
  else g->dim == 3 ? plan_coarse_t<double, 3>(S) : plan_coarse_t<double, 2>(S);
  // BF16 storage for the per-level coarse levels 1 .. lc-1 (needs the cluster path)
  S->bf16_hi = (P.coarse_bf16 && S->lc > 1) ? S->lc : 0;
  // a grid that fits one cluster is solved in one launch (with BF16 levels it keeps those)
  if (S->bf16_hi == 0) {
    if (dtype == FM_F32) g->dim == 3 ? plan_pcg_t<float, 3>(S) : plan_pcg_t<float, 2>(S);
    else g->dim == 3 ? plan_pcg_t<double, 3>(S) : plan_pcg_t<double, 2>(S);
  }
  for (int l = 0; l < S->L; ++l) {
    const size_t e = (l >= 1 && l < S->bf16_hi) ? sizeof(__nv_bfloat16) : es;
    ok = ok && cudaMalloc(&S->r[l], e * S->lv[l].size()) == cudaSuccess;
    ok = ok && cudaMalloc(&S->z[l], e * S->lv[l].size()) == cudaSuccess;
  }
  const long n0 = S->lv[0].size();
  // levels of 16 n cells a row of a large 3D FP32 solver are stored by colour: a second residual, in x's
  // allocation; without the memory for it the levels stay in natural order
  const int fine = S->lc > 0 ? S->lc : S->L - 1;
  bool split = g->dim == 3 && dtype == FM_F32 && n0 >= kSplitCells && !S->pcg_nc && fine > 0;
  for (int l = 0; l < fine; ++l) split = split && split_fits(S->lv[l]);
  if (split && ok) {
    const size_t xb = (es * n0 + 255) / 256 * 256;
    if (cudaMalloc(&S->x, xb + es * n0) == cudaSuccess) S->rs = (char*)S->x + xb;
    else cudaGetLastError(), S->x = nullptr;
  }
  if (!S->x) ok = ok && cudaMalloc(&S->x, es * n0) == cudaSuccess;
  if (!S->pcg_nc) {  // a cluster solve keeps p and A p in shared memory
    ok = ok && cudaMalloc(&S->p, es * n0) == cudaSuccess;
    ok = ok && cudaMalloc(&S->Ap, es * n0) == cudaSuccess;
  }
  // partials, state and the cluster geometries in one allocation
  struct Small {
    double part[2 * kRedBlocks];
    ClArgs coarse, pcg;
    DevState st;
  };
  Small* small = nullptr;
  ok = ok && cudaMalloc((void**)&small, sizeof(Small)) == cudaSuccess;
  if (ok) {
    S->part = small->part;
    S->st = &small->st;
    S->d_coarse = &small->coarse;
    S->d_pcg = &small->pcg;
    ClArgs both[2] = {S->coarse, S->pcg};
    ok = cudaMemcpy(S->d_coarse, both, sizeof(both), cudaMemcpyHostToDevice) == cudaSuccess;
  }
  ok = ok && cudaMallocHost(&S->h_st, sizeof(DevState)) == cudaSuccess;
  ok = ok && cudaStreamCreateWithFlags(&S->cap, cudaStreamNonBlocking) == cudaSuccess;
  if (ok) ok = cudaMemset(S->st, 0, sizeof(DevState)) == cudaSuccess;
  // both may still be under way; the first solve may come on a stream that the default one does not order
  if (ok) ok = cudaStreamSynchronize(nullptr) == cudaSuccess;
  const long nb = S->lv[S->L - 1].size();
  const size_t smem = 2 * es * nb;
  if (ok && smem <= 200 * 1024 && nb <= kBottomMaxCells) {
    S->bottom_smem = smem;
    if (smem > 48 * 1024) {
      bool e;
      if (dtype == FM_F32)
        e = g->dim == 3 ? raise_smem_limit(k_bottom<float, 3>, smem) : raise_smem_limit(k_bottom<float, 2>, smem);
      else
        e = g->dim == 3 ? raise_smem_limit(k_bottom<double, 3>, smem) : raise_smem_limit(k_bottom<double, 2>, smem);
      if (!e) {
        cudaGetLastError();
        S->bottom_smem = 0;
      }
    }
  }
  if (!ok) {
    fm_mgpcg_destroy(S);
    return FM_ERR_CUDA;
  }
  *out = S;
  return FM_OK;
}

int fm_mgpcg_destroy(fm_mgpcg* S) {
  if (!S) return FM_OK;
  for (int l = 0; l < kMaxLevels; ++l) {
    if (S->r[l]) cudaFree(S->r[l]);
    if (S->z[l]) cudaFree(S->z[l]);
  }
  if (S->x) cudaFree(S->x);
  if (S->p) cudaFree(S->p);
  if (S->Ap) cudaFree(S->Ap);
  if (S->part) cudaFree(S->part);  // and the state and the cluster geometries with it
  if (S->h_st) cudaFreeHost(S->h_st);
  if (S->chunk) cudaGraphExecDestroy(S->chunk);
  if (S->prologue) cudaGraphExecDestroy(S->prologue);
  if (S->loop) cudaGraphExecDestroy(S->loop);
  if (S->cap) cudaStreamDestroy(S->cap);
  free(S);
  return FM_OK;
}

int fm_project(fm_mgpcg* S, void* ux, void* uy, void* uz, void* p_out, void* stream, int* iters, double* rtr) {
  if (!S || !ux || !uy || (S->g.dim == 3 && !uz)) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const fm_grid g = S->g;
  const long n = S->lv[0].size();
  int status;
  if (S->dtype == FM_F32) {
    MacW<float> u{{(float*)ux, (float*)uy, (float*)uz}};
    if (g.dim == 3) launch_pdl(k_div_bc<float, 3>, kRedBlocks, kRedThreads, 0, s, g, u, (float*)S->r[0], (float*)S->x, S->part);
    else launch_pdl(k_div_bc<float, 2>, kRedBlocks, kRedThreads, 0, s, g, u, (float*)S->r[0], (float*)S->x, S->part);
    status = run_solve<float>(S, s, iters, rtr);
    if (status == FM_ERR_CUDA) return status;
    launch_subgrad(g, (const float*)S->x, u, s);
  } else {
    MacW<double> u{{(double*)ux, (double*)uy, (double*)uz}};
    if (g.dim == 3) launch_pdl(k_div_bc<double, 3>, kRedBlocks, kRedThreads, 0, s, g, u, (double*)S->r[0], (double*)S->x, S->part);
    else launch_pdl(k_div_bc<double, 2>, kRedBlocks, kRedThreads, 0, s, g, u, (double*)S->r[0], (double*)S->x, S->part);
    status = run_solve<double>(S, s, iters, rtr);
    if (status == FM_ERR_CUDA) return status;
    launch_subgrad(g, (const double*)S->x, u, s);
  }
  if (p_out) cudaMemcpyAsync(p_out, S->x, (S->dtype == FM_F32 ? 4 : 8) * n, cudaMemcpyDeviceToDevice, s);
  if (check_cuda()) return FM_ERR_CUDA;
  return status;
}

int fm_mgpcg_solve(fm_mgpcg* S, const void* b, void* x, void* stream, int* iters, double* rtr) {
  if (!S || !b || !x) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const long n = S->lv[0].size();
  int status;
  if (S->dtype == FM_F32) {
    launch_pdl(k_load_rhs<float>, kRedBlocks, kRedThreads, 0, s, n, (const float*)b, (float*)S->r[0], (float*)S->x, S->part);
    status = run_solve<float>(S, s, iters, rtr);
  } else {
    launch_pdl(k_load_rhs<double>, kRedBlocks, kRedThreads, 0, s, n, (const double*)b, (double*)S->r[0], (double*)S->x, S->part);
    status = run_solve<double>(S, s, iters, rtr);
  }
  if (status == FM_ERR_CUDA) return status;
  cudaMemcpyAsync(x, S->x, (S->dtype == FM_F32 ? 4 : 8) * n, cudaMemcpyDeviceToDevice, s);
  if (check_cuda()) return FM_ERR_CUDA;
  return status;
}

int fm_mg_vcycle(fm_mgpcg* S, const void* r, void* z, void* stream) {
  if (!S || !r || !z) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t bytes = (S->dtype == FM_F32 ? 4 : 8) * (size_t)S->lv[0].size();
  if (cudaMemcpyAsync(S->r[0], r, bytes, cudaMemcpyDeviceToDevice, s) != cudaSuccess) return FM_ERR_CUDA;
  // every V-cycle kernel is gated on the solver's `done` word
  if (cudaMemsetAsync(&S->st->done, 0, sizeof(int), s) != cudaSuccess) return FM_ERR_CUDA;
  if (S->dtype == FM_F32) {
    if (S->g.dim == 3) launch_vcycle<float, 3>(S, s, false, false);
    else launch_vcycle<float, 2>(S, s, false, false);
  } else {
    if (S->g.dim == 3) launch_vcycle<double, 3>(S, s, false, false);
    else launch_vcycle<double, 2>(S, s, false, false);
  }
  if (cudaMemcpyAsync(z, zout(S), bytes, cudaMemcpyDeviceToDevice, s) != cudaSuccess) return FM_ERR_CUDA;
  return check_cuda();
}

int fm_mgpcg_solve_dc(fm_mgpcg* S, int b_dtype, const void* b, double* x, double* work, double rel_tol,
                      int max_outer, void* stream, int* outer_iters, int* inner_iters, double* rel_res) {
  if (!S || !b || !x || !work || max_outer < 0 || !(rel_tol >= 0.0)) return FM_ERR_ARG;
  if (S->dtype != FM_F32 || (b_dtype != FM_F32 && b_dtype != FM_F64)) return FM_ERR_DTYPE;
  cudaStream_t s = (cudaStream_t)stream;
  const Shape s0 = S->lv[0];
  const long n = s0.size();
  const int D = S->g.dim;
  const unsigned nb = blocks_for(n, 256, 148L * 16);
  if (b_dtype == FM_F32) launch_pdl(k_dc_sum<float>, kRedBlocks, kRedThreads, 0, s, n, (const float*)b, S->part);
  else launch_pdl(k_dc_sum<double>, kRedBlocks, kRedThreads, 0, s, n, (const double*)b, S->part);
  launch_pdl(k_dc_fin, 1, 256, 0, s, S->st, S->part, (double)n, 0);
  if (cudaMemsetAsync(x, 0, sizeof(double) * n, s) != cudaSuccess) return FM_ERR_CUDA;
  auto residual = [&](int which) {
    if (b_dtype == FM_F32) {
      if (D == 3) launch_pdl(k_dc_residual<float, 3>, kRedBlocks, kRedThreads, 0, s, s0, (const float*)b, x, work, S->part, S->st);
      else launch_pdl(k_dc_residual<float, 2>, kRedBlocks, kRedThreads, 0, s, s0, (const float*)b, x, work, S->part, S->st);
    } else {
      if (D == 3) launch_pdl(k_dc_residual<double, 3>, kRedBlocks, kRedThreads, 0, s, s0, (const double*)b, x, work, S->part, S->st);
      else launch_pdl(k_dc_residual<double, 2>, kRedBlocks, kRedThreads, 0, s, s0, (const double*)b, x, work, S->part, S->st);
    }
    launch_pdl(k_dc_fin, 1, 256, 0, s, S->st, S->part, (double)n, which);
  };
  residual(1);
  int outer = 0, inner = 0, status = FM_OK;
  double rel = 0;
  for (;;) {
    if (cudaMemcpyAsync(S->h_st, S->st, sizeof(DevState), cudaMemcpyDeviceToHost, s) != cudaSuccess) return FM_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return FM_ERR_CUDA;
    const double b2 = S->h_st->dc_b2, r2 = S->h_st->dc_r2;
    rel = b2 > 0 ? sqrt(r2 / b2) : 0.0;
    if (!isfinite(rel)) { status = FM_ERR_NONFINITE; break; }
    if (rel <= rel_tol || r2 == 0.0) break;
    if (outer >= max_outer) { status = FM_ERR_NOT_CONVERGED; break; }
    launch_pdl(k_dc_load, kRedBlocks, kRedThreads, 0, s, n, (const double*)work, (float*)S->r[0], (float*)S->x, S->part,
           (const DevState*)S->st);
    launch_pdl(k_dc_set_tol, 1, 1, 0, s, S->st, rel_tol, 0);
    int it = 0;
    double rtr = 0;
    const int st = run_solve<float>(S, s, &it, &rtr);  // reaching max_iters is fine: the outer loop corrects
    inner += it;
    if (st == FM_ERR_CUDA || st == FM_ERR_NONFINITE) { status = st; break; }
    launch_pdl(k_dc_update, nb, 256, 0, s, n, x, (const float*)S->x, (const DevState*)S->st);
    ++outer;
    residual(2);
  }
  launch_pdl(k_dc_set_tol, 1, 1, 0, s, S->st, 0.0, 1);
  if (outer_iters) *outer_iters = outer;
  if (inner_iters) *inner_iters = inner;
  if (rel_res) *rel_res = rel;
  if (check_cuda()) return FM_ERR_CUDA;
  return status;
}

int fm_project_dc(fm_mgpcg* S, void* ux, void* uy, void* uz, double* work, double rel_tol, int max_outer,
                  double* p_out, void* stream) {
  if (!S || !ux || !uy || (S->g.dim == 3 && !uz) || !work || max_outer < 1 || max_outer > 16 ||
      !(rel_tol > 0.0))
    return FM_ERR_ARG;
  if (S->dtype != FM_F32) return FM_ERR_DTYPE;
  if (S->P.check_every != 0) return FM_ERR_ARG;  // device-side loops only
  cudaStream_t s = (cudaStream_t)stream;
  const fm_grid g = S->g;
  const Shape s0 = S->lv[0];
  const long n = s0.size();
  const int D = g.dim;
  double* b = work;
  double* x = work + n;
  double* w = work + 2 * n;
  MacW<float> u{{(float*)ux, (float*)uy, (float*)uz}};
  const unsigned nb = blocks_for(n, 256, 148L * 16);
  if (D == 3) launch_pdl(k_dc_div<3>, kRedBlocks, kRedThreads, 0, s, g, u, b, x, S->part);
  else launch_pdl(k_dc_div<2>, kRedBlocks, kRedThreads, 0, s, g, u, b, x, S->part);
  launch_pdl(k_dc_fin, 1, 256, 0, s, S->st, S->part, (double)n, 0);  // dc_mean
  auto residual = [&](int which) {
    if (D == 3) launch_pdl(k_dc_residual_g<3>, kRedBlocks, kRedThreads, 0, s, s0, (const double*)b, (const double*)x, w, S->part, (const DevState*)S->st);
    else launch_pdl(k_dc_residual_g<2>, kRedBlocks, kRedThreads, 0, s, s0, (const double*)b, (const double*)x, w, S->part, (const DevState*)S->st);
    launch_pdl(k_dc_check, 1, 256, 0, s, S->st, S->part, rel_tol, which);
  };
  residual(1);
  for (int o = 0; o < max_outer; ++o) {
    launch_pdl(k_dc_load_g, kRedBlocks, kRedThreads, 0, s, n, (const double*)w, (float*)S->r[0], (float*)S->x,
               S->part, (const DevState*)S->st);
    launch_pdl(k_dc_set_tol_g, 1, 1, 0, s, S->st, rel_tol);
    const int st = run_solve<float>(S, s, nullptr, nullptr);
    if (st) return st;
    launch_pdl(k_dc_update_g, nb, 256, 0, s, n, x, (const float*)S->x, (const DevState*)S->st);
    residual(2);
  }
  launch_subgrad(g, (const double*)x, u, s);
  launch_pdl(k_dc_finish, 1, 1, 0, s, S->st);
  if (p_out) cudaMemcpyAsync(p_out, x, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
  if (check_cuda()) return FM_ERR_CUDA;
  return FM_OK;
}

int fm_mgpcg_stats(fm_mgpcg* S, void* stream, int reset, fm_mg_stats* out) {
  if (!S || !out) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(S->h_st, S->st, sizeof(DevState), cudaMemcpyDeviceToHost, s) != cudaSuccess) return FM_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return FM_ERR_CUDA;
  const DevState& h = *S->h_st;
  out->solves = h.solves;
  out->iterations = h.iters_total;
  out->not_converged = h.not_converged;
  out->nonfinite = h.nonfinite_count;
  out->last_iters = h.result_it;
  out->max_iters_seen = h.max_it_seen;
  out->last_rtr = h.rTr;
  // kernels run inside device-mode while loops since the last call
  count_launch(h.bodies * S->loop_kernels);
  long long zero_bodies = 0;
  if (cudaMemcpyAsync(&S->st->bodies, &zero_bodies, sizeof(long long), cudaMemcpyHostToDevice, s) != cudaSuccess)
    return FM_ERR_CUDA;
  if (reset) {
    DevState z = h;
    z.solves = z.iters_total = z.not_converged = z.nonfinite_count = 0;
    z.max_it_seen = 0;
    z.bodies = 0;
    if (cudaMemcpyAsync(S->st, &z, sizeof(DevState), cudaMemcpyHostToDevice, s) != cudaSuccess) return FM_ERR_CUDA;
  }
  if (cudaStreamSynchronize(s) != cudaSuccess) return FM_ERR_CUDA;
  return FM_OK;
}

int fm_laplacian(const fm_grid* g, int dtype, const void* p, void* Ap, void* stream) {
  int st = validate_grid(g, dtype);
  if (st) return st;
  if (!p || !Ap) return FM_ERR_ARG;
  Shape s = cell_shape(*g);
  cudaStream_t cs = (cudaStream_t)stream;
  unsigned nb = blocks_for(s.size(), 256, 148L * 16);
  if (dtype == FM_F32) {
    if (g->dim == 3) launch_pdl(k_laplacian<float, 3>, nb, 256, 0, cs, s, (const float*)p, (float*)Ap);
    else launch_pdl(k_laplacian<float, 2>, nb, 256, 0, cs, s, (const float*)p, (float*)Ap);
  } else {
    if (g->dim == 3) launch_pdl(k_laplacian<double, 3>, nb, 256, 0, cs, s, (const double*)p, (double*)Ap);
    else launch_pdl(k_laplacian<double, 2>, nb, 256, 0, cs, s, (const double*)p, (double*)Ap);
  }
  return check_cuda();
}

int fm_abi_version(void) { return 1; }

long long fm_launch_count(int reset) {
  if (reset) return g_launch_count.exchange(0);
  return g_launch_count.load();
}

int fm_set_pdl(int enable) {
  return g_pdl.exchange(enable ? 1 : 0);
}

int fm_last_cuda_error(char* buf, int len) {
  const int e = g_last_cuda_error.load();
  if (buf && len > 0) {
    const char* name = e ? cudaGetErrorName((cudaError_t)e) : "cudaSuccess";
    int i = 0;
    for (; name && name[i] && i < len - 1; ++i) buf[i] = name[i];
    buf[i] = 0;
  }
  return e;
}

const char* fm_status_string(int status) {
  switch (status) {
    case FM_OK: return "ok";
    case FM_ERR_SHAPE: return "unsupported grid shape";
    case FM_ERR_ARG: return "invalid argument";
    case FM_ERR_NOT_CONVERGED: return "MGPCG did not converge within max_iters";
    case FM_ERR_NONFINITE: return "non-finite residual in MGPCG";
    case FM_ERR_TIMEOUT: return "bounded device wait timed out";
    case FM_ERR_CUDA: return "CUDA runtime error";
    case FM_ERR_DTYPE: return "unsupported dtype";
    case FM_ERR_CAPACITY: return "grid too large for the static scratch of fm_project_noalloc";
    default: return "unknown status";
  }
}

}  // extern "C"

// ---------------------------------------------------------------------------
// fm_project_noalloc: the projection without any allocation.
//
// Its MG hierarchy, PCG vectors, reduction partials and solver state are carved
// out of one file-scope __device__ array (kNoAllocScratchBytes), which every
// GPU that loads this library holds until the process exits.  Host code cannot
// use the array's name as a device address (it names a host-side shadow), so
// the address is fetched with cudaGetSymbolAddress once per device, with that
// device current, on the first call made on it; that first call should
// therefore come before any stream capture.  Under CUDA's lazy module loading
// (the default) that first call is also when the array and this library's
// kernels receive their device memory, so it must come before another runtime
// claims the device's memory (or the process sets CUDA_MODULE_LOADING=EAGER,
// which places them when the library loads).  Kernels are launched directly (no
// CUDA graph, whose instantiation may allocate) and convergence is polled
// through a host stack variable (no pinned buffer).
// ---------------------------------------------------------------------------
namespace fm {

constexpr size_t kNoAllocScratchBytes = size_t(48) << 20;  // 48 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
static void* g_noalloc_base[kMaxDevices];
static std::mutex g_noalloc_mu;

static int noalloc_scratch(void** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return FM_ERR_CUDA;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_base[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
      cudaGetLastError();  // leave no pending error for an unrelated later check
      return FM_ERR_CUDA;
    }
    g_noalloc_base[dev] = p;
  }
  *out = g_noalloc_base[dev];
  return FM_OK;
}

// Lays the solver's buffers out from `base` (nullptr: size only); returns bytes.
static size_t noalloc_layout(const fm_grid& g, int dtype, int levels, fm_mgpcg* S, unsigned char* base) {
  size_t off = 0;
  auto take = [&](size_t bytes) -> void* {
    off = (off + 255) & ~size_t(255);
    void* p = base ? (void*)(base + off) : nullptr;
    off += bytes;
    return p;
  };
  const size_t es = dtype == FM_F32 ? sizeof(float) : sizeof(double);
  for (int l = 0; l < levels; ++l) {
    Shape sh{g.n[0] >> l, g.n[1] >> l, g.dim == 3 ? (g.n[2] >> l) : 1};
    S->lv[l] = sh;
    S->r[l] = take(es * sh.size());
    S->z[l] = take(es * sh.size());
  }
  const long n0 = S->lv[0].size();
  S->x = take(es * n0);
  S->p = take(es * n0);
  S->Ap = take(es * n0);
  S->part = (double*)take(sizeof(double) * 2 * kRedBlocks);
  S->st = (DevState*)take(sizeof(DevState));
  return off;
}

// Host-checked solve with direct launches (no graph).
template <typename T>
static int run_solve_direct(fm_mgpcg* S, cudaStream_t s, int* iters, double* rtr) {
  const int D = S->g.dim;
  const int every = S->P.check_every > 0 ? S->P.check_every : 4;
  if (D == 3) launch_prologue<T, 3>(S, s); else launch_prologue<T, 2>(S, s);
  DevState h;
  long launched = 0;
  const long limit = (long)S->P.max_iters + every;
  for (;;) {
    for (int i = 0; i < every; ++i) {
      if (D == 3) launch_iteration<T, 3>(S, s); else launch_iteration<T, 2>(S, s);
    }
    launched += every;
    if (cudaMemcpyAsync(&h, S->st, sizeof(DevState), cudaMemcpyDeviceToHost, s) != cudaSuccess) return FM_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return FM_ERR_CUDA;
    if (h.done || launched >= limit) break;
  }
  if (iters) *iters = h.result_it;
  if (rtr) *rtr = h.rTr;
  if (h.nonfinite) return FM_ERR_NONFINITE;
  if (!h.conv) return FM_ERR_NOT_CONVERGED;
  return FM_OK;
}

}  // namespace fm

extern "C" int fm_project_noalloc(const fm_grid* g, int dtype, const fm_mg_params* params, void* ux, void* uy,
                                  void* uz, void* stream, int* iters, double* rtr) {
  int st = validate_grid(g, dtype);
  if (st) return st;
  if (!params) return FM_ERR_ARG;
  const fm_mg_params& P = *params;
  if (P.levels < 2 || P.levels > kMaxLevels || P.pre_post < 1 || P.bottom < 0 || P.max_iters < 1 ||
      P.check_every < 0 || (P.bottom_mode != 0 && P.bottom_mode != 1) || P.coarse_bf16)
    return FM_ERR_ARG;
  for (int a = 0; a < g->dim; ++a)
    if (g->n[a] % (1 << (P.levels - 1)) != 0) return FM_ERR_SHAPE;
  fm_mgpcg S;
  memset(&S, 0, sizeof(S));
  S.g = *g;
  S.dtype = dtype;
  S.P = P;
  S.L = P.levels;
  // capacity before the field pointers: a caller can ask whether a grid fits without passing any
  if (noalloc_layout(*g, dtype, P.levels, &S, nullptr) > kNoAllocScratchBytes) return FM_ERR_CAPACITY;
  if (!ux || !uy || (g->dim == 3 && !uz)) return FM_ERR_ARG;
  void* base = nullptr;
  if ((st = noalloc_scratch(&base))) return st;
  noalloc_layout(*g, dtype, P.levels, &S, (unsigned char*)base);
  const size_t es = dtype == FM_F32 ? sizeof(float) : sizeof(double);
  const size_t smem = 2 * es * S.lv[S.L - 1].size();
  // larger coarsest levels: per-sweep launches
  S.bottom_smem = (smem <= 48 * 1024 && S.lv[S.L - 1].size() <= kBottomMaxCells) ? smem : 0;
  cudaStream_t s = (cudaStream_t)stream;
  // the scratch keeps the previous call's contents: the solver state must start at zero
  if (cudaMemsetAsync(S.st, 0, sizeof(DevState), s) != cudaSuccess) return FM_ERR_CUDA;
  const fm_grid gg = *g;
  int status;
  if (dtype == FM_F32) {
    MacW<float> u{{(float*)ux, (float*)uy, (float*)uz}};
    if (gg.dim == 3) launch_pdl(k_div_bc<float, 3>, kRedBlocks, kRedThreads, 0, s, gg, u, (float*)S.r[0], (float*)S.x, S.part);
    else launch_pdl(k_div_bc<float, 2>, kRedBlocks, kRedThreads, 0, s, gg, u, (float*)S.r[0], (float*)S.x, S.part);
    status = run_solve_direct<float>(&S, s, iters, rtr);
    if (status == FM_ERR_CUDA) return status;
    launch_subgrad(gg, (const float*)S.x, u, s);
  } else {
    MacW<double> u{{(double*)ux, (double*)uy, (double*)uz}};
    if (gg.dim == 3) launch_pdl(k_div_bc<double, 3>, kRedBlocks, kRedThreads, 0, s, gg, u, (double*)S.r[0], (double*)S.x, S.part);
    else launch_pdl(k_div_bc<double, 2>, kRedBlocks, kRedThreads, 0, s, gg, u, (double*)S.r[0], (double*)S.x, S.part);
    status = run_solve_direct<double>(&S, s, iters, rtr);
    if (status == FM_ERR_CUDA) return status;
    launch_subgrad(gg, (const double*)S.x, u, s);
  }
  if (check_cuda()) return FM_ERR_CUDA;
  return status;
}
