// fm_force.cu -- Gaussian control forces and their parameter adjoint.
//
// Force (apply_gausion_force_kernel, 3D/lfm_midpoint_simulator.py:309-344,
// 2D/shape/lfm_midpoint_simulator.py:283-299): on every MAC face X of
// component c,
//     f_c(X) = sum over I < n with q_I(X) < 5 of exp(-q_I(X)) s_I[c],
//     q_I(X) = |X - c_I|^2 r_I   (|.| = sqrt of the sum of squares, squared),
// summed in ascending I as the reference's per-face loop does; r_I is the
// inverse squared radius.
//
// Adjoint (calculate_adj_gausion_force_kernel,
// 3D/lfm_midpoint_diff_simulator.py:63-110): for every Gaussian the sums over
// the faces of its support of
//     adj_strength[c] += e a_c            adj_center += s_c e 2 (X - c) r a_c
//     pen_strength[c] += 2 f e            pen_center += 2 f s_c e 2 (X - c) r
// with e = exp(-q), f = e s_c and a the adjoint velocity.
//
// Inclusion is decided exactly as the reference rounds it: s2 = sum (X - c)^2
// (left to right, no FMA contraction), d = sqrt(s2), q = (d d) r, q < 5.
// Off the boundary (s2 r outside 5 (1 -+ 1e-4)) the decision cannot depend on
// the rounding of d d and is taken without the square root (against
// 5 (1 -+ 1e-4) / r - s2_other, for the faces of a column).  The weight uses
// the Gaussian's separability, exp(-r s2) = exp(-r s2_other) exp(-r dz^2),
// which differs from exp(-q) by a few ulps.
//
// B200 mapping.  3000 Gaussians against every face is compute work, bound by
// issue slots.  Both kernels tabulate per Gaussian and axis the squared offsets and
// the factors exp(-r dx_a^2) in shared memory, so that a face costs a few
// additions, a compare and a multiply-add.
//  * k_gauss_force: one CTA per tile of cells (16x16 in 2D, 8x8x8 in 3D), a
//    column of faces along the fastest axis (k in 3D, j in 2D) per thread.  The
//    CTA walks the Gaussians in chunks of 256, read one chunk ahead, and appends
//    those whose support ball (radius sqrt(5/r), widened) reaches the tile's box
//    to a list in shared memory, in ascending order (ballot + popc prefix); once
//    the list could not take another chunk, or at the end, it tabulates the
//    listed Gaussians a sub-chunk at a time (each thread its own table entry) and
//    every thread accumulates its column segment over them in list order, the
//    other axes combined once per (column, Gaussian), four faces per shared load.
//    The cull is a superset of the exact test.  3000 Gaussians of radius 1..9 cells
//    on 128^3 in FP32: 289 us with the cull in FP64 and scalar table loads, 210 us now.
//  * k_gauss_grad: one CTA per Gaussian over its support; what a lane sums of one
//    short stretch of faces is of the run's type, everything beyond it FP64;
//    fixed-order warp-shuffle + shared-memory reduction, so the result is
//    deterministic (the reference's atomics are not).  Gaussians with r <= 0 or a
//    support longer than the table along the columns take a per-face path in the
//    reference's operation order.
#include <math.h>

#include "fm_common.cuh"
#include "fm_internal.h"

namespace fm {

constexpr int kGfThreads = 256;
constexpr int kGfWarps = kGfThreads / 32;
constexpr int kGfMaxN = 1 << 24;
constexpr int kGfTab = 256;   // table capacity of the adjoint kernel (faces of an axis)

// Tiles of the force kernel; the column axis is D-1.  SEG: faces per thread
// along it (one segment per thread: 3D 9*8 + 8*9 + 8*8 = 208, 2D 17*4 + 16*5 = 148).
template <int D> struct GfTile;
template <> struct GfTile<2> { static constexpr int B0 = 16, B1 = 16, B2 = 1, BC = 16, SEG = 4; };
template <> struct GfTile<3> { static constexpr int B0 = 8, B1 = 8, B2 = 8, BC = 8, SEG = 9; };

// Relative widening of the support radius used by the culls and by the
// square-root-free decisions; far above the few ulps by which the rounding of
// the exact test can move the boundary.
constexpr double kGfMargin = 1e-4;

// Position of index i along an axis: face grids at i dx on their own axis,
// (i + 1/2) dx elsewhere (node_pos, 3D/taichi_utils.py:95-128).
template <typename T>
__device__ __forceinline__ T gf_pos(int i, bool face, T dx) {
  T f = (T)i;
  if (!face) f = f + (T)0.5;
  return f * dx;
}

// Inclusion of a face with squared distance s2 (rounded as the reference
// rounds it) for inverse radius r.
template <typename T>
__device__ __forceinline__ bool gf_inside(T s2, T r) {
  const T t = rn_mul(s2, r);
  if (t < (T)(5.0 * (1.0 - kGfMargin))) return true;   // r <= 0 lands here too
  if (t > (T)(5.0 * (1.0 + kGfMargin))) return false;
  const T d = sqrt(s2);                                   // near the boundary: the exact test
  return rn_mul(rn_mul(d, d), r) < (T)5;                  // NaN excluded
}

// The per-face path: exact test and weight at one face.
template <typename T, int D>
__device__ __forceinline__ bool gf_weight(const T* p, const T* c, T r, T* dp, T& e) {
#pragma unroll
  for (int a = 0; a < D; ++a) dp[a] = rn_sub(p[a], c[a]);
  T s2 = rn_mul(dp[0], dp[0]);
#pragma unroll
  for (int a = 1; a < D; ++a) s2 = rn_add(s2, rn_mul(dp[a], dp[a]));
  if (!gf_inside(s2, r)) return false;
  e = exp(-rn_mul(s2, r));
  return true;
}

// Tile cull: does Gaussian (c, r) possibly reach a face inside [lo, hi]?  In the
// run's type (every Gaussian is tested against every tile): the box is wider
// than the faces by a hundredth of a cell and the bound by kGfMargin, far above the
// rounding here, and s2 r is compared so that no division is needed.
template <typename T, int D>
__device__ __forceinline__ bool gf_touches(const T* c, T r, const T* lo, const T* hi) {
  if (r != r) return false;          // NaN radius: the exact test excludes every face
  if (!(r > (T)0)) return true;      // r <= 0: q <= 0 everywhere (left to the exact test)
  T d2 = (T)0;
#pragma unroll
  for (int a = 0; a < D; ++a) {
    const T t = c[a] < lo[a] ? lo[a] - c[a] : (c[a] > hi[a] ? c[a] - hi[a] : (T)0);
    d2 += t * t;
  }
  return !(d2 * r > (T)(5.0 * (1.0 + kGfMargin)));  // NaN (0 times infinity, a NaN centre): left to the exact test
}

// four consecutive table entries, 16-byte aligned
__device__ __forceinline__ void load4(const float* p, float* v) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
__device__ __forceinline__ void load4(const double* p, double* v) {
  const double2 x = *reinterpret_cast<const double2*>(p), y = *reinterpret_cast<const double2*>(p + 2);
  v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
}

template <typename T, int D>
__global__ void __launch_bounds__(kGfThreads) k_gauss_force(fm_grid g, T dx, int n, const T* __restrict__ cen,
                                                            const T* __restrict__ ir, const T* __restrict__ str,
                                                            T* __restrict__ f0, T* __restrict__ f1,
                                                            T* __restrict__ f2) {
  using Tl = GfTile<D>;
  constexpr int CA = D - 1, SEG = Tl::SEG;
  // table entries per axis and variant, rounded up for 16-byte loads
  constexpr int BM = ((Tl::B0 > Tl::BC ? Tl::B0 : Tl::BC) + 1 + 3) / 4 * 4;
  constexpr int SUB = sizeof(T) == 4 ? 48 : 24;                       // Gaussians tabulated at a time
  constexpr int TS = D * 2 * BM;                                      // table entries per Gaussian
  constexpr int CAP = sizeof(T) == 4 ? 2 * kGfThreads : kGfThreads;  // culled-list capacity
  __shared__ T s_c[D][CAP], s_s[D][CAP], s_r[CAP];
  // per tabulated Gaussian l, axis a, variant v (0 cell, 1 face), index q - lo[a]:
  // squared offset and exp(-r offset^2)
  __shared__ alignas(16) T t_sq[SUB][D][2][BM], t_ex[SUB][D][2][BM];
  __shared__ T t_lo[SUB], t_hi[SUB];  // 5 (1 -+ m) / r, or +inf for r <= 0
  __shared__ int s_cnt[kGfWarps];

  const int nt1 = (g.n[1] + Tl::B1 - 1) / Tl::B1, nt2 = (g.n[2] + Tl::B2 - 1) / Tl::B2;
  int t = blockIdx.x;
  const int t2 = t % nt2;
  t /= nt2;
  const int t1 = t % nt1, t0 = t / nt1;
  const int lo[3] = {t0 * Tl::B0, t1 * Tl::B1, t2 * Tl::B2};
  const int hc[3] = {min(lo[0] + Tl::B0, g.n[0]), min(lo[1] + Tl::B1, g.n[1]), min(lo[2] + Tl::B2, g.n[2])};
  // the tile's box: faces at i dx (the last tile along an axis also owns the
  // face at n dx), centres at (i + 1/2) dx, widened by a hundredth of a cell
  T blo[3], bhi[3];
#pragma unroll
  for (int a = 0; a < D; ++a) {
    blo[a] = (T)(((double)lo[a] - 0.01) * (double)dx);
    bhi[a] = (T)(((double)hc[a] + 1.01) * (double)dx);
  }

  // this thread's segment: component cc, tile-local other-axis indices io[],
  // tile-local column indices [k0, k0 + len)
  int cc = -1, io[2] = {0, 0}, k0 = 0, len = 0;
  {
    int q = threadIdx.x;
#pragma unroll
    for (int comp = 0; comp < D; ++comp) {
      if (cc < 0) {
        int e[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) e[a] = hc[a] + (comp == a && hc[a] == g.n[a]) - lo[a];
        const int nseg = (e[CA] + SEG - 1) / SEG;
        const int cnt = (D == 3 ? e[0] * e[1] : e[0]) * nseg;
        if (q < cnt) {
          cc = comp;
          const int sg = q % nseg, o = q / nseg;
          if (D == 3) {
            io[0] = o / e[1];
            io[1] = o % e[1];
          } else {
            io[0] = o;
          }
          k0 = sg * SEG;
          len = min(SEG, e[CA] - sg * SEG);
        } else {
          q -= cnt;
        }
      }
    }
  }
  const int v0 = cc == 0 ? 1 : 0, v1 = cc == 1 ? 1 : 0, vc = cc == CA ? 1 : 0;

  // the table entry this thread fills, for every (kGfThreads / TS)-th Gaussian: axis, variant, index
  static_assert(TS <= kGfThreads, "one entry a thread");
  const int te = threadIdx.x % TS, ta = te / (2 * BM), tv = te / BM % 2;
  const int tq = threadIdx.x < kGfThreads / TS * TS ? te % BM : -1;
  const T tpos = gf_pos<T>((ta == 0 ? lo[0] : (ta == 1 ? lo[1] : lo[2])) + tq, tv == 1, dx);

  T acc[SEG];
#pragma unroll
  for (int m = 0; m < SEG; ++m) acc[m] = (T)0;

  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int listed = 0;  // culled Gaussians waiting in the list (uniform across the CTA)
  T cn[D], rn = (T)NAN;  // the next chunk's Gaussian, read ahead (NaN: none)
  const auto ahead = [&](int I) {
    rn = (T)NAN;
    if (I < n) {
#pragma unroll
      for (int a = 0; a < D; ++a) cn[a] = __ldg(cen + (long)I * D + a);
      rn = __ldg(ir + I);
    }
  };
#pragma unroll
  for (int a = 0; a < D; ++a) cn[a] = (T)0;
  ahead(threadIdx.x);
  for (int base = 0; base < n; base += kGfThreads) {
    const int I = base + threadIdx.x;
    T c[D], s[D];
    const T r = rn;
#pragma unroll
    for (int a = 0; a < D; ++a) c[a] = cn[a];
    ahead(I + kGfThreads);
    const bool hit = gf_touches<T, D>(c, r, blo, bhi);
    if (hit)
#pragma unroll
      for (int a = 0; a < D; ++a) s[a] = __ldg(str + (long)I * D + a);
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) s_cnt[w] = __popc(m);
    __syncthreads();
    int off = 0, got = 0;
#pragma unroll
    for (int k = 0; k < kGfWarps; ++k) {
      const int v = s_cnt[k];
      off += k < w ? v : 0;
      got += v;
    }
    if (hit) {  // appended in ascending order after the Gaussians already listed
      const int slot = listed + off + __popc(m & ((1u << lane) - 1u));
#pragma unroll
      for (int a = 0; a < D; ++a) {
        s_c[a][slot] = c[a];
        s_s[a][slot] = s[a];
      }
      s_r[slot] = r;
    }
    __syncthreads();
    listed += got;
    // evaluate once the list could not take another chunk, or at the end
    if (listed > CAP - kGfThreads || base + kGfThreads >= n) {
      const int tot = listed;
      listed = 0;
      for (int sub = 0; sub < tot; sub += SUB) {
        const int cnt = min(SUB, tot - sub);
        if (tq >= 0)
          for (int l = threadIdx.x / TS; l < cnt; l += kGfThreads / TS) {
            const T d = rn_sub(tpos, s_c[ta][sub + l]);
            const T sq = rn_mul(d, d);
            t_sq[l][ta][tv][tq] = sq;
            t_ex[l][ta][tv][tq] = exp(-rn_mul(sq, s_r[sub + l]));
          }
        if (threadIdx.x < cnt) {
          const T rr = s_r[sub + threadIdx.x];
          const bool pos = rr > (T)0;
          t_lo[threadIdx.x] = pos ? (T)(5.0 * (1.0 - kGfMargin)) / rr : (T)INFINITY;
          t_hi[threadIdx.x] = pos ? (T)(5.0 * (1.0 + kGfMargin)) / rr : (T)INFINITY;
        }
        __syncthreads();
        if (cc >= 0) {
          for (int l = 0; l < cnt; ++l) {
            // the other axes once per (column, Gaussian)
            T sxy = t_sq[l][0][v0][io[0]], exy = t_ex[l][0][v0][io[0]];
            if (D == 3) {
              sxy = rn_add(sxy, t_sq[l][1][v1][io[1]]);
              exy = exy * t_ex[l][1][v1][io[1]];
            }
            // dz^2 < A: inside off the boundary; dz^2 > B: outside; between: the exact test
            const T B = t_hi[l] - sxy;
            if (B < (T)0) continue;  // the column misses the support
            const T A = t_lo[l] - sxy, rr = s_r[sub + l];
            const T ev = exy * s_s[cc][sub + l];
            // entries past the segment's end are only added to sums that are not stored
            const T* const psq = &t_sq[l][CA][vc][k0];
            const T* const pex = &t_ex[l][CA][vc][k0];
            T sq[SEG];
            bool near = false;
#pragma unroll
            for (int q0 = 0; q0 < SEG; q0 += 4) {
              if (q0 + 4 > SEG && len <= q0) break;  // 3D: the ninth face, in the last tiles only
              T x4[4], e4[4];
              load4(psq + q0, x4);
              load4(pex + q0, e4);
#pragma unroll
              for (int q = q0; q < SEG && q < q0 + 4; ++q) {
                sq[q] = x4[q - q0];
                const bool in = sq[q] < A;
                if (in) acc[q] += ev * e4[q - q0];
                near |= !in & (sq[q] <= B);
              }
            }
            if (near) {  // rare
#pragma unroll
              for (int q = 0; q < SEG; ++q)
                if (q < len && !(sq[q] < A) && sq[q] <= B) {
                  const T d = sqrt(rn_add(sxy, sq[q]));
                  if (rn_mul(rn_mul(d, d), rr) < (T)5) acc[q] += ev * pex[q];
                }
            }
          }
        }
        __syncthreads();  // the next tables / list entries overwrite what was read
      }
    }
  }

  if (cc >= 0) {
    const Shape fs = face_shape(g, cc);
    T* const o = cc == 0 ? f0 : (cc == 1 ? f1 : f2);
    const long b = D == 3 ? fs.idx(lo[0] + io[0], lo[1] + io[1], lo[2] + k0) : fs.idx(lo[0] + io[0], lo[1] + k0, 0);
    const long st = D == 3 ? 1 : fs.s2;  // the column axis is contiguous (3D: k; 2D: j with s2 == 1)
#pragma unroll
    for (int q = 0; q < SEG; ++q)
      if (q < len) o[b + q * st] = acc[q];
  }
}

// Face-index range along one axis within [lo, hi] (in cells, widened by more than
// the rounding of a face's position).
__device__ __forceinline__ void gf_axis_range(double lo, double hi, bool face_axis, int len, int& i0, int& i1) {
  const double off = face_axis ? 0.0 : 0.5;
  const double a = fmax(ceil(lo - off), 0.0), b = fmin(floor(hi - off), (double)(len - 1));
  if (!(a <= b)) {
    i0 = 1;
    i1 = 0;
    return;
  }
  i0 = (int)a;
  i1 = (int)b;
}

// Offset, its square and exp(-r offset^2) of one face index along an axis.
template <typename T> struct alignas(4 * sizeof(T)) GfAxis {
  T dp, sq, ex, pad;
};
template <typename T>
__device__ __forceinline__ GfAxis<T> gf_axis(int i, bool face, T dx, T c, T r) {
  const T d = rn_sub(gf_pos<T>(i, face, dx), c), sq = rn_mul(d, d);
  return {d, sq, exp(-rn_mul(sq, r)), (T)0};
}

// One warp's piece of a support in the adjoint kernel: 8 faces of the column
// axis from q0 on, at one index of the outer axis (offset d0, its square, its
// factor), times the middle-axis indices ma..mb of the slab.
template <typename T> struct alignas(16) GfTask {
  const T* row;     // the first of the 8 faces, at the slab's start
  unsigned rowst;   // a step along the middle axis
  short q0, last;   // last: of the 8 faces within the range
  short ma, mb, mlast, cc;
  T d0, sq0;
};

// The Gaussian that block b takes: a one-to-one map that puts wide supports
// first, in four classes of radius, so that the last blocks to run are short ones
// (a support of 20 cells is 60 times the work of one of 5).  Every block
// counts the classes for itself: worth it while that is a few loads a thread;
// far more blocks than fit at once even out by themselves.
constexpr int kGfOrderMax = 32 * kGfThreads;
template <typename T>
__device__ __forceinline__ int gf_order(int b, int n, const T* __restrict__ ir) {
  __shared__ T s_min[kGfWarps];
  __shared__ unsigned long long s_cnt[kGfWarps];
  __shared__ int s_pick;
  if (n > kGfOrderMax) return b;
  constexpr unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T least = (T)INFINITY;
  for (int i = threadIdx.x; i < n; i += kGfThreads) {
    const T r = __ldg(ir + i);
    if (r > (T)0) least = min(least, r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) least = min(least, __shfl_xor_sync(all, least, o));
  if (lane == 0) s_min[w] = least;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kGfWarps; ++k) least = min(least, s_min[k]);
  // radii above 3/4, 1/2, 1/4 of the widest; r <= 0 (every face) with the widest, NaN with the narrowest
  const auto bin = [&](T r) { return (r <= least * (T)1.78 ? 0 : (r <= least * (T)4 ? 1 : (r <= least * (T)16 ? 2 : 3))); };
  unsigned packed = 0;  // four counts of at most 32
  for (int i = threadIdx.x; i < n; i += kGfThreads) packed += 1u << (8 * bin(__ldg(ir + i)));
  unsigned long long mine = 0;  // ... in 16 bits each, for the sums over the block
#pragma unroll
  for (int k = 0; k < 4; ++k) mine |= (unsigned long long)(packed >> (8 * k) & 0xff) << (16 * k);
  unsigned long long upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(all, upto, o);
    if (lane >= o) upto += x;
  }
  if (lane == 31) s_cnt[w] = upto;
  __syncthreads();
  unsigned long long total = 0;
#pragma unroll
  for (int k = 0; k < kGfWarps; ++k) {
    if (k < w) upto += s_cnt[k];
    total += s_cnt[k];
  }
  int k = 0, p = b;  // block b is the p-th of class k
  while (k < 3 && p >= (int)(total >> (16 * k) & 0xffff)) p -= (int)(total >> (16 * k++) & 0xffff);
  p -= (int)((upto - mine) >> (16 * k) & 0xffff);
  if (p >= 0 && p < (int)(mine >> (16 * k) & 0xffff))
    for (int i = threadIdx.x; i < n; i += kGfThreads)
      if (bin(__ldg(ir + i)) == k && p-- == 0) s_pick = i;
  __syncthreads();
  return s_pick;
}

// Per-Gaussian sums v[c] adj_strength, v[D+a] adj_center, v[2D+c]
// pen_strength, v[3D+a] pen_center (FP64).
//
// Bound by issue slots: about 19 instructions a face, plus what is done per warp
// and not per face.  So the support, a ball, is split to waste few lanes, and
// what a whole warp would compute alike is computed by one thread each.  A task
// is 8 faces of the column axis (k in 3D, j in 2D; contiguous in memory) at one
// index of the outer axis; its warp walks, 4 faces at a time, the stretch of the
// middle axis that the ball reaches there.  Every thread prepares one task, then
// the warps take them in turn.  The factor of the outer and the column axis stays
// in a register, the middle axis' come from shared memory.  A lane's sums over its
// share of one task are of the run's type, their products with the offsets and the
// sums over tasks are FP64, and a weight is the product of two factors: three (a
// table entry per axis, whose roundings all faces of a plane share) put the FP32 sums
// 1.2 to 1.4 times further from 64 bits.
// 3000 Gaussians of radius 1..9 cells on 128^3 in FP32: 334 us with a lane per column
// (strided loads, 32 unequal columns per warp), 206 us with three factors and FP32 sums
// of up to 32 faces and more, 211 us now.
template <typename T, int D>
__global__ void __launch_bounds__(kGfThreads, sizeof(T) == 4 ? 4 : 2)
    k_gauss_grad(fm_grid g, T dx, int n, const T* __restrict__ cen, const T* __restrict__ ir, const T* __restrict__ str,
                 const T* __restrict__ a0, const T* __restrict__ a1, const T* __restrict__ a2,
                 double* __restrict__ adj_c, double* __restrict__ adj_s, double* __restrict__ pen_c,
                 double* __restrict__ pen_s) {
  constexpr int NV = 4 * D;
  constexpr int CA = D - 1, MA = D - 2;  // column and middle axis
  constexpr int LC = 8, LM = 32 / LC, UN = 2, PAD = LM * UN;
  constexpr int kStretch = 32;           // 2D has no outer axis: middle stretches instead
  static_assert(kStretch % PAD == 0 && kGfTab % kStretch == 0, "stretches end where a step ends");
  __shared__ double s_red[kGfWarps][NV];
  // by variant v (0 cells, 1 faces) of the axis; t_mid is one slab of the axis
  __shared__ GfAxis<T> t_col[2][kGfTab], t_mid[2][kGfTab + PAD];
  __shared__ GfTask<T> s_task[kGfThreads];
  __shared__ int s_i0[D][2], s_len[D][2];  // the support's index range along an axis
  const int I = gf_order<T>(blockIdx.x, n, ir);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T c[D], s[D];
#pragma unroll
  for (int a = 0; a < D; ++a) {
    c[a] = cen[(long)I * D + a];
    s[a] = str[(long)I * D + a];
  }
  const T r = ir[I];
  // NaN or infinite r, or a non-finite centre with r > 0, reaches no face; r <= 0 every face
  bool none = r != r || r == (T)INFINITY;
  if (r > (T)0)
#pragma unroll
    for (int a = 0; a < D; ++a) none = none || !isfinite((double)c[a]);
  if (threadIdx.x < 2 * D) {
    const int a = threadIdx.x >> 1, v = threadIdx.x & 1;
    double lo = -1.0, hi = 1e9;
    if (r > (T)0) {
      // a face's position and its offset from the centre are rounded in the run's type: by up to
      // 2^-23 of the axis in FP32, 0.02 cells at 150000
      const double ulp = sizeof(T) == 4 ? 0x1p-22 : 0x1p-51;
      const double slack = 0.01 + ulp * (a == 0 ? g.n[0] : (a == 1 ? g.n[1] : g.n[2]));
      const double R = sqrt(5.0 / (double)r) * (1.0 + kGfMargin) + slack * (double)dx;
      const double x = (double)(a == 0 ? c[0] : (a == 1 ? c[1] : c[CA]));
      lo = (x - R) / (double)dx;
      hi = (x + R) / (double)dx;
    }
    int b0 = 1, b1 = 0;
    if (!none) gf_axis_range(lo, hi, v == 1, (a == 0 ? g.n[0] : (a == 1 ? g.n[1] : g.n[2])) + v, b0, b1);
    s_i0[a][v] = b0;
    s_len[a][v] = b1 - b0 + 1;
  }
  __syncthreads();
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;

  const T tlo = (T)(5.0 * (1.0 - kGfMargin)) / r, thi = (T)(5.0 * (1.0 + kGfMargin)) / r;
  const T inv = (T)1 / dx;
  // component cc's range; `cols`: its columns fit the table, and there is a ball
  const auto start = [&](int cc, int a) { return s_i0[a][cc == a]; };
  const auto extent = [&](int cc, int a) { return s_len[a][cc == a]; };
  const auto cols = [&](int cc) { return r > (T)0 && extent(cc, CA) <= kGfTab; };
  const int mlen = max(s_len[MA][0], s_len[MA][1]);
  // one component's sums, and which one's
  double S = 0.0, S0 = 0.0, Sm = 0.0, Sc = 0.0, E = 0.0, E0 = 0.0, Em = 0.0, Ec = 0.0;
  int hc = -1;
  const auto flush = [&]() {
    T sc = s[0];
#pragma unroll
    for (int cc = 0; cc < D; ++cc)
      if (hc == cc) {
        sc = s[cc];
        v[cc] += S;
        v[2 * D + cc] += 2.0 * (double)sc * E;
      }
    const double k1 = 2.0 * (double)sc * (double)r, k2 = 2.0 * (double)sc * k1;
    if (D == 3) v[D] += k1 * S0, v[3 * D] += k2 * E0;
    v[D + MA] += k1 * Sm, v[3 * D + MA] += k2 * Em;
    v[D + CA] += k1 * Sc, v[3 * D + CA] += k2 * Ec;
    S = S0 = Sm = Sc = E = E0 = Em = Ec = 0.0;
  };
  for (int m0 = 0; m0 < mlen && r > (T)0; m0 += kGfTab) {  // the middle axis in slabs of the table's length
    if (m0 > 0) __syncthreads();
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      if (m0 == 0)
        for (int q = threadIdx.x; q < min(s_len[CA][f], kGfTab); q += kGfThreads)
          t_col[f][q] = gf_axis<T>(s_i0[CA][f] + q, f == 1, dx, c[CA], r);
      const int ms = min(kGfTab, s_len[MA][f] - m0);
      for (int q = threadIdx.x; q < ms + PAD; q += kGfThreads)
        t_mid[f][q] = q < ms ? gf_axis<T>(s_i0[MA][f] + m0 + q, f == 1, dx, c[MA], r)
                             : GfAxis<T>{(T)0, (T)INFINITY, (T)0, (T)0};  // past the end: outside
    }
    int first[D + 1] = {0};  // each component's first task
#pragma unroll
    for (int cc = 0; cc < D; ++cc) {
      const int ms = min(kGfTab, extent(cc, MA) - m0);
      const int nout = D == 3 ? extent(cc, 0) : (ms + kStretch - 1) / kStretch;
      const bool any = ms > 0 && nout > 0 && cols(cc);
      first[cc + 1] = first[cc] + (any ? (extent(cc, CA) + LC - 1) / LC * nout : 0);
    }
    for (int tb = 0; tb < first[D]; tb += kGfThreads) {
      const int t = tb + threadIdx.x;
      if (t < first[D]) {
        const int cc = t < first[1] ? 0 : (D == 2 || t < first[2] ? 1 : 2);
        const int tt = t - (cc == 0 ? 0 : (cc == 1 ? first[1] : first[2 < D ? 2 : 1]));
        const int ecol = extent(cc, CA), ms = min(kGfTab, extent(cc, MA) - m0);
        const int chunks = (ecol + LC - 1) / LC, o = tt / chunks, q0 = (tt - o * chunks) * LC;
        const T d0 = D == 3 ? rn_sub(gf_pos<T>(start(cc, 0) + o, cc == 0, dx), c[0]) : (T)0, sq0 = rn_mul(d0, d0);
        // the stretch that the ball reaches at the chunk's nearest face, widened
        // to whole indices; the centre in the slab's indices
        const T za = rn_sub(gf_pos<T>(start(cc, CA) + q0, cc == CA, dx), c[CA]);
        const T zb = rn_sub(gf_pos<T>(start(cc, CA) + min(q0 + LC, ecol) - 1, cc == CA, dx), c[CA]);
        const T zm = za > (T)0 ? za : (zb < (T)0 ? zb : (T)0);
        const T rest = thi - sq0 - zm * zm;
        const T half = sqrt(rest) * inv + (T)0.01;
        const T cm = -rn_sub(gf_pos<T>(start(cc, MA) + m0, cc == MA, dx), c[MA]) * inv;
        const T mlo = D == 3 ? (T)0 : (T)(o * kStretch);
        const T mhi = D == 3 ? (T)(ms - 1) : (T)min(ms - 1, o * kStretch + kStretch - 1);
        int ma = 0, mb = -1;
        if (rest >= (T)0) {  // false for NaN
          ma = (int)min(max(floor(cm - half), mlo), mhi + (T)1);
          mb = (int)max(min(ceil(cm + half), mhi), (T)-1);
          if (D == 2) ma &= ~(PAD - 1);  // so that the last step stays within the stretch
        }
        const Shape fs = face_shape(g, cc);
        GfTask<T> k;
        k.row = (cc == 0 ? a0 : (cc == 1 ? a1 : a2)) +
                (D == 3 ? fs.idx(start(cc, 0) + o, start(cc, 1) + m0, start(cc, CA) + q0)
                        : fs.idx(start(cc, 0) + m0, start(cc, 1) + q0, 0));
        k.rowst = D == 3 ? fs.s2 : fs.s1;
        k.q0 = (short)q0, k.last = (short)(min(q0 + LC, ecol) - 1 - q0), k.cc = (short)cc;
        k.ma = (short)ma, k.mb = (short)mb, k.mlast = (short)(ms - 1);
        k.d0 = d0, k.sq0 = sq0;
        s_task[threadIdx.x] = k;
      }
      __syncthreads();
      for (int t = w; t < min(kGfThreads, first[D] - tb); t += kGfWarps) {
        const GfTask<T> k = s_task[t];
        if (k.ma > k.mb) continue;
        const int cc = k.cc;
        if (cc != hc) {
          if (hc >= 0) flush();
          hc = cc;
        }
        const int lc = min(lane & (LC - 1), (int)k.last);
        const GfAxis<T> col = t_col[cc == CA][k.q0 + lc];
        const T zsq = lc == (lane & (LC - 1)) ? col.sq : (T)INFINITY;  // past the end: outside
        const T eoc = D == 3 ? exp(-rn_mul(rn_add(k.sq0, col.sq), r)) : col.ex;
        const T* row = k.row + lc;
        const int mlast = k.mlast;
        const unsigned rowst = k.rowst;
        const GfAxis<T>* const mid = t_mid[cc == MA];
        T P = (T)0, Pm = (T)0, Q = (T)0, Qm = (T)0;
        for (int m = k.ma + lane / LC; m - lane / LC <= k.mb; m += PAD) {
          T av[UN], s2[UN], e[UN], dm[UN];
          bool in[UN], near = false;
#pragma unroll
          for (int h = 0; h < UN; ++h) av[h] = __ldg(row + (unsigned)min(m + h * LM, mlast) * rowst);
#pragma unroll
          for (int h = 0; h < UN; ++h) {
            const GfAxis<T> x = mid[m + h * LM];
            dm[h] = x.dp;
            e[h] = eoc * x.ex;
            // s2 < tlo: inside off the boundary; s2 > thi: outside; between: the exact test
            s2[h] = rn_add(D == 3 ? rn_add(k.sq0, x.sq) : x.sq, zsq);
            in[h] = s2[h] < tlo;
            near |= !in[h] & (s2[h] <= thi);
          }
          if (near) {  // rare
#pragma unroll
            for (int h = 0; h < UN; ++h)
              if (!in[h] && s2[h] <= thi) {
                const T d = sqrt(s2[h]);
                in[h] = rn_mul(rn_mul(d, d), r) < (T)5;
              }
          }
#pragma unroll
          for (int h = 0; h < UN; ++h) {  // selects: a NaN outside stays out
            const T ea = in[h] ? e[h] * av[h] : (T)0, e2 = in[h] ? e[h] * e[h] : (T)0;
            P += ea;
            Pm += ea * dm[h];
            Q += e2;
            Qm += e2 * dm[h];
          }
        }
        const double p = P, q = Q, dc = col.dp;
        S += p, Sm += (double)Pm, Sc += dc * p;
        E += q, Em += (double)Qm, Ec += dc * q;
        if (D == 3) S0 += (double)k.d0 * p, E0 += (double)k.d0 * q;
      }
      __syncthreads();  // the tasks' last readers are done
    }
  }
  if (hc >= 0) flush();
  if (!none) {
#pragma unroll
    for (int cc = 0; cc < D; ++cc) {
      const int e0 = extent(cc, 0), e1 = extent(cc, 1), e2 = D == 3 ? extent(cc, CA) : 1;
      if (cols(cc) || e0 <= 0 || e1 <= 0 || e2 <= 0) continue;
      // per-face path (r <= 0, or a support wider than the table), in the
      // reference's operation order per face
      const Shape fs = face_shape(g, cc);
      const T* const adj = cc == 0 ? a0 : (cc == 1 ? a1 : a2);
      const int i0[3] = {start(cc, 0), start(cc, 1), D == 3 ? start(cc, CA) : 0};
      const T sc = s[cc];
      const unsigned cnt = (unsigned)e0 * (unsigned)e1 * (unsigned)e2;  // < 2^32 (validate_grid)
      for (unsigned q = threadIdx.x; q < cnt; q += kGfThreads) {
        const unsigned ij = q / (unsigned)e2;
        const int k = (int)(q - ij * (unsigned)e2);
        const unsigned ii = ij / (unsigned)e1;
        const int j = (int)(ij - ii * (unsigned)e1), i = (int)ii;
        T p[D], dp[D], e;
        node_pos<T, D>(cc, i0[0] + i, i0[1] + j, i0[2] + k, dx, p);
        if (!gf_weight<T, D>(p, c, r, dp, e)) continue;
        const T av = adj[fs.idx(i0[0] + i, i0[1] + j, i0[2] + k)];
        const T f = rn_mul(e, sc);
        v[cc] += (double)rn_mul(e, av);
        v[2 * D + cc] += (double)rn_mul(rn_mul((T)2, f), e);
        const T ga = rn_mul(rn_mul(sc, e), (T)2);
        const T gp = rn_mul(rn_mul(rn_mul(rn_mul((T)2, f), sc), e), (T)2);
#pragma unroll
        for (int a = 0; a < D; ++a) {
          v[D + a] += (double)rn_mul(rn_mul(rn_mul(ga, dp[a]), r), av);
          v[3 * D + a] += (double)rn_mul(rn_mul(gp, dp[a]), r);
        }
      }
    }
  }
  // fixed-order reduction: butterfly within each warp, then warps in order
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double x = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    v[k] = x;
  }
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) s_red[w][k] = v[k];
  __syncthreads();
  if (threadIdx.x < NV) {
    double x = 0.0;
#pragma unroll
    for (int k = 0; k < kGfWarps; ++k) x += s_red[k][threadIdx.x];
    const int which = threadIdx.x / D, a = threadIdx.x % D;
    double* const o = which == 0 ? adj_s : (which == 1 ? adj_c : (which == 2 ? pen_s : pen_c));
    o[(long)I * D + a] = x;
  }
}

template <typename T>
int gauss_force(const fm_grid& g, double dx, int n, const void* cen, const void* ir, const void* str, void* fx,
                void* fy, void* fz, cudaStream_t s) {
  const T tdx = (T)dx;
  if (g.dim == 2) {
    using Tl = GfTile<2>;
    const unsigned tiles = (unsigned)(((g.n[0] + Tl::B0 - 1) / Tl::B0) * ((g.n[1] + Tl::B1 - 1) / Tl::B1));
    launch(k_gauss_force<T, 2>, tiles, kGfThreads, 0, s, g, tdx, n, (const T*)cen, (const T*)ir, (const T*)str,
           (T*)fx, (T*)fy, (T*)nullptr);
  } else {
    using Tl = GfTile<3>;
    const unsigned tiles = (unsigned)((long)((g.n[0] + Tl::B0 - 1) / Tl::B0) * ((g.n[1] + Tl::B1 - 1) / Tl::B1) *
                                      ((g.n[2] + Tl::B2 - 1) / Tl::B2));
    launch(k_gauss_force<T, 3>, tiles, kGfThreads, 0, s, g, tdx, n, (const T*)cen, (const T*)ir, (const T*)str,
           (T*)fx, (T*)fy, (T*)fz);
  }
  return check_cuda();
}

template <typename T>
int gauss_grad(const fm_grid& g, double dx, int n, const void* cen, const void* ir, const void* str, const void* ax,
               const void* ay, const void* az, double* adj_c, double* adj_s, double* pen_c, double* pen_s,
               cudaStream_t s) {
  if (n == 0) return FM_OK;
  if (g.dim == 2)
    launch(k_gauss_grad<T, 2>, (unsigned)n, kGfThreads, 0, s, g, (T)dx, n, (const T*)cen, (const T*)ir, (const T*)str,
           (const T*)ax, (const T*)ay, (const T*)nullptr, adj_c, adj_s, pen_c, pen_s);
  else
    launch(k_gauss_grad<T, 3>, (unsigned)n, kGfThreads, 0, s, g, (T)dx, n, (const T*)cen, (const T*)ir, (const T*)str,
           (const T*)ax, (const T*)ay, (const T*)az, adj_c, adj_s, pen_c, pen_s);
  return check_cuda();
}

}  // namespace fm

extern "C" {

int fm_gaussian_force(const fm_grid* g, int dtype, double dx, int n, const void* center, const void* inv_radius,
                      const void* strength, void* f_x, void* f_y, void* f_z, void* stream) {
  using namespace fm;
  const int st = validate_grid(g, dtype);
  if (st) return st;
  if (n < 0 || n > kGfMaxN || !(dx > 0)) return FM_ERR_ARG;
  if (n > 0 && (!center || !inv_radius || !strength)) return FM_ERR_ARG;
  if (!f_x || !f_y || (g->dim == 3 && !f_z)) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == FM_F32) return gauss_force<float>(*g, dx, n, center, inv_radius, strength, f_x, f_y, f_z, s);
  return gauss_force<double>(*g, dx, n, center, inv_radius, strength, f_x, f_y, f_z, s);
}

int fm_gaussian_force_grad(const fm_grid* g, int dtype, double dx, int n, const void* center, const void* inv_radius,
                           const void* strength, const void* adj_x, const void* adj_y, const void* adj_z,
                           double* adj_center, double* adj_strength, double* penalty_center,
                           double* penalty_strength, void* stream) {
  using namespace fm;
  const int st = validate_grid(g, dtype);
  if (st) return st;
  if (n < 0 || n > kGfMaxN || !(dx > 0)) return FM_ERR_ARG;
  if (n > 0 && (!center || !inv_radius || !strength || !adj_center || !adj_strength || !penalty_center ||
                !penalty_strength))
    return FM_ERR_ARG;
  if (!adj_x || !adj_y || (g->dim == 3 && !adj_z)) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == FM_F32)
    return gauss_grad<float>(*g, dx, n, center, inv_radius, strength, adj_x, adj_y, adj_z, adj_center, adj_strength,
                             penalty_center, penalty_strength, s);
  return gauss_grad<double>(*g, dx, n, center, inv_radius, strength, adj_x, adj_y, adj_z, adj_center, adj_strength,
                            penalty_center, penalty_strength, s);
}

}  // extern "C"
