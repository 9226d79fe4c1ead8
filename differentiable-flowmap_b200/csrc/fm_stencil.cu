// fm_stencil.cu -- the adjoint source terms as tiled separable stencils.
//
//   calculate_nabla_u_w           r_c = sum_a (d_c u_a)(X_c) w_a(X_c)   (3D/flowmap.py:359-380,
//                                                                        2D/vortex/flowmap.py:361-377)
//   calculate_nabla_scalar_adjoint r_c = (d_c s)(X_c) adj_s(X_c)        (3D/flowmap.py:382-403)
//
// Both interpolate with cubic (3D) / quartic (2D) B-splines at the face nodes
// X_c themselves.  The stencil along an axis (first tap, weights) depends only
// on the node's index along that axis, so the 3D sum factorises across a tile
// of nodes: one CTA loads the tile's input footprint into shared memory once
// and contracts it along k, then j, then i -- O(taps) work per node and each
// input value read from HBM about once, instead of a (taps)^3 gather per node.
// Weights, first taps and the clamp band follow the reference exactly
// (s = clamp(X/dx - BL, 1, len-2-eps), taps iu+lo+t, sample() index clamp);
// only the summation order differs.
#include <cmath>

#include "fm_common.cuh"
#include "fm_internal.h"

namespace fm {

// 3D tile: TI x TJ x TK output nodes (k contiguous); 2D: TI x TJ (j contiguous)
constexpr int kTJ3 = 8, kTK3 = 32;  // the tile height along i is a template parameter (4 or 8)
constexpr int kTJ2 = 64;  // the tile height along i is a template parameter (8, 12 or 16)
constexpr int kStThreads = 256;

template <typename T>
struct StTerm {
  const T* f;  // differentiated along the output face axis
  const T* h;  // interpolated
  int s0, s1, s2;
  T bl0, bl1, bl2;
};
template <typename T>
struct StTerms {
  StTerm<T> t[3];
  int n;
};

template <typename T>
__device__ __forceinline__ StTerm<T> pick_term(const StTerms<T>& ts, int a) {
  return a == 0 ? ts.t[0] : (a == 1 ? ts.t[1] : ts.t[2]);
}

// Per-axis stencil of one output node: unclamped first tap, weights and
// derivative weights of the ORDER+1 taps that can be non-zero.
template <typename T, int ORDER>
__device__ __forceinline__ void axis_stencil(T pos, T dx, T bl, int len, int& base, T* w, T* dw) {
  constexpr int NZ = Taps<ORDER>::nz;
  T u = pos / dx;
  u = u - bl;
  const T hi = (T)((double)len - 2.0 - 1e-6);
  T s = u < hi ? u : hi;
  s = s > (T)1 ? s : (T)1;
  const T iu = floor(s);
  const T f = s - iu;
  int t0;
  if (ORDER == 3) t0 = 1;
  else if (ORDER == 2) t0 = f >= (T)0.5 ? 1 : 0;
  else t0 = f >= (T)0.5 ? 2 : 1;
  base = (int)iu + Taps<ORDER>::lo + t0;
#pragma unroll
  for (int t = 0; t < NZ; ++t) {
    const T x = s - (iu + (T)(Taps<ORDER>::lo + t0 + t));
    bs_eval<T, ORDER>(x, w[t], dw[t]);
  }
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// The two fields of a term side by side: f (differentiated or not) and h, each
// with its own weight.  In FP32 one paired multiply-add (two IEEE FMAs) serves both.
template <typename T>
struct alignas(2 * sizeof(T)) Pair {
  T f, h;
};
__device__ __forceinline__ void pair_fma(Pair<float>& acc, const Pair<float>& x, const Pair<float>& w) {
  const float2 r = __ffma2_rn(make_float2(x.f, x.h), make_float2(w.f, w.h), make_float2(acc.f, acc.h));
  acc.f = r.x;
  acc.h = r.y;
}
__device__ __forceinline__ void pair_fma(Pair<double>& acc, const Pair<double>& x, const Pair<double>& w) {
  acc.f += x.f * w.f;
  acc.h += x.h * w.h;
}
// Weights of one node along one axis.
template <typename T, int NZ>
struct alignas(16) TapWeights {
  Pair<T> v[NZ];
};

template <typename T>
__device__ __forceinline__ void copy_async(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "n"(sizeof(T))
               : "memory");
}

// Shared memory of a 3D tile: footprints, the pairs after the k pass and those after the j
// pass; the latter lie over the footprints where all three do not fit (kOwnB false: FP64
// cubic and quartic tiles 8 high with margins), which then arrive after the i pass
// (nabla_u_w at 40x61x90, order 3 / 4: 80 / 117 us; 111 / 177 by tiles 4 high).
template <typename T, int ORDER, int M, int TI>
struct Fixed3 {
  static constexpr int NZ = Taps<ORDER>::nz;
  static constexpr int FI = TI + NZ - 1 + 2 * M, FJ = kTJ3 + NZ - 1 + 2 * M, FK = kTK3 + NZ - 1 + 2 * M;
  static constexpr size_t front = sizeof(T) * (2 * FI * FJ * FK + 2 * FI * FJ * kTK3), b = sizeof(T) * 2 * FI * kTJ3 * kTK3;
  static constexpr bool kOwnB = front + b <= 227 * 1024 - 8192;  // the tables are static
  static constexpr size_t smem = front + (kOwnB ? b : 0);
};

// Per tile and term, the footprints of both fields are contracted along k (a warp
// per row; a lane's k and so its weights stay in registers), then, as pairs, along
// j and i with one column per thread held in registers: n outputs of a column cost
// n + NZ - 1 shared reads instead of n NZ.  The columns need the first taps of a
// tile to advance by one per node, which fails where the clamp band is inside
// the tile and, with a dx that is no power of two, where a quotient rounds across
// an integer: there every output reads its own taps (a second rule per axis, the
// same operations).  Footprints arrive as asynchronous copies, those of the next
// term while this one is contracted along j and i; the three output grids share a
// launch.  128^3 FP32: nabla_u_w 283 -> 208 us, nabla_scalar_adjoint 108 -> 76 us
// (before: a shared read per tap and weight with four-way conflicts on the k
// weights, footprints through registers one latency at a time).  What bounds it
// now: shared-memory wavefronts (72 % of peak; a fifth of them from copies whose
// source and destination are aligned differently).
template <typename T, int ORDER, int M, int TI3>
__global__ void __launch_bounds__(kStThreads, 2) k_fixed_grad_dot3(fm_grid g, T dx, StTerms<T> terms, MacW<T> outs) {
  constexpr int NZ = Taps<ORDER>::nz;
  constexpr int TI = TI3, TJ = kTJ3, TK = kTK3;
  // footprint: taps from the tile's first base - M (see launch_fixed3)
  using L3 = Fixed3<T, ORDER, M, TI>;
  constexpr int FI = L3::FI, FJ = L3::FJ, FK = L3::FK;
  constexpr int WARPS = kStThreads / 32;
  static_assert(TK == 32 && TJ == WARPS, "a warp is a row along k; an i column per thread");
  using W = TapWeights<T, NZ>;
  using P = Pair<T>;
  // dynamic shared: footprints F, H; pairs A after the k pass, B after the j pass
  extern __shared__ __align__(16) unsigned char st_smem[];
  P* sA = reinterpret_cast<P*>(st_smem);
  P* sB = sA + FI * FJ * TK;
  T* sF = reinterpret_cast<T*>(L3::kOwnB ? sB + FI * TJ * TK : sB);
  T* sH = sF + FI * FJ * FK;
  struct Tables {
    W wI[TI], wJ[TJ], wK[TK];
    int bI[TI], bJ[TJ], bK[TK];
  };
  __shared__ Tables tab[2];

  // one launch for the three output grids: blockIdx.x holds the tile along k and the grid
  const int c = blockIdx.x % 3;
  const Shape so = face_shape(g, c);
  const int i0 = blockIdx.z * TI, j0 = blockIdx.y * TJ, k0 = blockIdx.x / 3 * TK;
  if (i0 >= so.s0 || j0 >= so.s1 || k0 >= so.s2) return;
  T* __restrict__ out = pick(outs, c);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T inv_dx = (T)1 / dx;
  T acc[TI];
#pragma unroll
  for (int e = 0; e < TI; ++e) acc[e] = 0;

  // axis tables of term a (node positions: face axis at i*dx, others at
  // (i+0.5)*dx); along c the field f takes the derivative weights
  auto tables = [&](int a) {
    const StTerm<T> tm = pick_term(terms, a);
    Tables& t = tab[a & 1];
    const int e = threadIdx.x;
    if (e >= TI + TJ + TK) return;
    int ax, loc, len;
    T bl;
    if (e < TI) { ax = 0; loc = e; len = tm.s0; bl = tm.bl0; }
    else if (e < TI + TJ) { ax = 1; loc = e - TI; len = tm.s1; bl = tm.bl1; }
    else { ax = 2; loc = e - TI - TJ; len = tm.s2; bl = tm.bl2; }
    const int node = (ax == 0 ? i0 : (ax == 1 ? j0 : k0)) + loc;
    T fi = (T)node;
    if (ax != c) fi = fi + (T)0.5;
    const T pos = fi * dx;
    int base;
    T w[NZ], dw[NZ];
    axis_stencil<T, ORDER>(pos, dx, bl, len, base, w, dw);
    (ax == 0 ? t.bI : (ax == 1 ? t.bJ : t.bK))[loc] = base;
    W& wt = (ax == 0 ? t.wI : (ax == 1 ? t.wJ : t.wK))[loc];
#pragma unroll
    for (int q = 0; q < NZ; ++q) wt.v[q] = P{ax == c ? dw[q] : w[q], w[q]};
  };
  // footprints of term a (clamped indices: sample()); its tables are visible
  auto load = [&](int a) {
    const StTerm<T> tm = pick_term(terms, a);
    const Tables& t = tab[a & 1];
    const int li = t.bI[0] - M, lj = t.bJ[0] - M, lk = t.bK[0] - M;
    auto row_of = [&](int ii, int jj) {  // fields have fewer than 2^32 entries
      return ((unsigned)clampi(li + ii, 0, tm.s0 - 1) * tm.s1 + clampi(lj + jj, 0, tm.s1 - 1)) * tm.s2;
    };
    const unsigned gk = clampi(lk + lane, 0, tm.s2 - 1);
    static_assert(FJ >= WARPS, "one wrap per step");
    int ii = 0, jj = warp;
    for (int row = warp; row < FI * FJ; row += WARPS) {
      const unsigned q = row_of(ii, jj) + gk;
      copy_async(sF + row * FK + lane, tm.f + q);
      copy_async(sH + row * FK + lane, tm.h + q);
      jj += WARPS;
      if (jj >= FJ) { jj -= FJ; ++ii; }
    }
    constexpr int REST = FK - TK;  // the columns past the first 32
    for (int e = threadIdx.x; e < FI * FJ * REST; e += kStThreads) {
      const int row = e / REST, kk = TK + e - row * REST, ri = row / FJ;
      const unsigned q = row_of(ri, row - ri * FJ) + clampi(lk + kk, 0, tm.s2 - 1);
      copy_async(sF + row * FK + kk, tm.f + q);
      copy_async(sH + row * FK + kk, tm.h + q);
    }
  };

  tables(0);
  __syncthreads();
  load(0);
  for (int a = 0; a < terms.n; ++a) {
    const Tables& t = tab[a & 1];
    const int li = t.bI[0] - M, lj = t.bJ[0] - M, lk = t.bK[0] - M;
    bool col_i = true, col_j = true;  // first taps advance by one per node
#pragma unroll
    for (int q = 1; q < TI; ++q) col_i = col_i && t.bI[q] == t.bI[0] + q;
#pragma unroll
    for (int q = 1; q < TJ; ++q) col_j = col_j && t.bJ[q] == t.bJ[0] + q;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // k pass
    {
      const W w = t.wK[lane];
      const int off = t.bK[lane] - lk;
#pragma unroll 4
      for (int row = warp; row < FI * FJ; row += WARPS) {
        const T* Fr = sF + row * FK + off;
        const T* Hr = sH + row * FK + off;
        P s{0, 0};
#pragma unroll
        for (int q = 0; q < NZ; ++q) pair_fma(s, P{Fr[q], Hr[q]}, w.v[q]);
        sA[row * TK + lane] = s;
      }
    }
    if (a + 1 < terms.n) tables(a + 1);
    __syncthreads();
    if (L3::kOwnB && a + 1 < terms.n) load(a + 1);
    // j pass
    for (int ii = warp; ii < FI; ii += WARPS) {
      const P* Ac = sA + ii * FJ * TK + lane;
      P* Bc = sB + ii * TJ * TK + lane;
      if (col_j) {
        P x[TJ + NZ - 1];
#pragma unroll
        for (int q = 0; q < TJ + NZ - 1; ++q) x[q] = Ac[(M + q) * TK];
#pragma unroll
        for (int j = 0; j < TJ; ++j) {
          const W w = t.wJ[j];
          P s{0, 0};
#pragma unroll
          for (int q = 0; q < NZ; ++q) pair_fma(s, x[j + q], w.v[q]);
          Bc[j * TK] = s;
        }
      } else {
#pragma unroll 1
        for (int j = 0; j < TJ; ++j) {
          const int off = t.bJ[j] - lj;
          const W w = t.wJ[j];
          P s{0, 0};
#pragma unroll
          for (int q = 0; q < NZ; ++q) pair_fma(s, Ac[(off + q) * TK], w.v[q]);
          Bc[j * TK] = s;
        }
      }
    }
    __syncthreads();
    // i pass and product: a thread's TI outputs are a column along i
    const P* Bc = sB + warp * TK + lane;
    if (col_i) {
      P x[TI + NZ - 1];
#pragma unroll
      for (int q = 0; q < TI + NZ - 1; ++q) x[q] = Bc[(M + q) * TJ * TK];
#pragma unroll
      for (int i = 0; i < TI; ++i) {
        const W w = t.wI[i];
        P s{0, 0};
#pragma unroll
        for (int q = 0; q < NZ; ++q) pair_fma(s, x[i + q], w.v[q]);
        acc[i] += (s.f * inv_dx) * s.h;
      }
    } else {
#pragma unroll
      for (int i = 0; i < TI; ++i) {
        const int off = t.bI[i] - li;
        const W w = t.wI[i];
        P s{0, 0};
#pragma unroll
        for (int q = 0; q < NZ; ++q) pair_fma(s, Bc[(off + q) * TJ * TK], w.v[q]);
        acc[i] += (s.f * inv_dx) * s.h;
      }
    }
    if (!L3::kOwnB && a + 1 < terms.n) {
      __syncthreads();  // the i pass has read what the footprints overwrite
      load(a + 1);
    }
  }
  const int k = k0 + lane, j = j0 + warp;
#pragma unroll
  for (int r = 0; r < TI; ++r)
    if (i0 + r < so.s0 && j < so.s1 && k < so.s2) out[so.idx(i0 + r, j, k)] = acc[r];
}

template <typename T, int ORDER, int M, int TI2>
__global__ void __launch_bounds__(kStThreads) k_fixed_grad_dot2(fm_grid g, T dx, int c, StTerms<T> terms,
                                                                  T* __restrict__ out) {
  constexpr int NZ = Taps<ORDER>::nz;
  constexpr int TI = TI2, TJ = kTJ2;
  constexpr int FI = TI + NZ - 1 + 2 * M, FJ = TJ + NZ - 1 + 2 * M;  // taps from the first base - M (fixed3_smem)
  constexpr int NOUT = TI * TJ / kStThreads;
  __shared__ T sF[2 * FI * FJ];
  __shared__ T sA[2 * FI * TJ];
  __shared__ T wI[TI][NZ], dI[TI][NZ], wJ[TJ][NZ], dJ[TJ][NZ];
  __shared__ int bI[TI], bJ[TJ];

  const Shape so = face_shape(g, c);
  const int i0 = blockIdx.y * TI, j0 = blockIdx.x * TJ;
  const T inv_dx = (T)1 / dx;
  T acc[NOUT];
#pragma unroll
  for (int e = 0; e < NOUT; ++e) acc[e] = 0;

  for (int a = 0; a < terms.n; ++a) {
    const StTerm<T> tm = pick_term(terms, a);
    __syncthreads();
    for (int e = threadIdx.x; e < TI + TJ; e += blockDim.x) {
      const int ax = e < TI ? 0 : 1, loc = e < TI ? e : e - TI;
      const int len = ax == 0 ? tm.s0 : tm.s1;
      const T bl = ax == 0 ? tm.bl0 : tm.bl1;
      const int node = (ax == 0 ? i0 : j0) + loc;
      T fi = (T)node;
      if (ax != c) fi = fi + (T)0.5;
      int base;
      T w[NZ], dw[NZ];
      axis_stencil<T, ORDER>(fi * dx, dx, bl, len, base, w, dw);
      (ax == 0 ? bI : bJ)[loc] = base;
      T* wt = ax == 0 ? &wI[0][0] : &wJ[0][0];
      T* dt = ax == 0 ? &dI[0][0] : &dJ[0][0];
#pragma unroll
      for (int t = 0; t < NZ; ++t) { wt[loc * NZ + t] = w[t]; dt[loc * NZ + t] = dw[t]; }
    }
    __syncthreads();
    const int li = bI[0] - M, lj = bJ[0] - M;
    for (int e = threadIdx.x; e < FI * FJ; e += blockDim.x) {
      const int jj = e % FJ, ii = e / FJ;
      const long q = (long)clampi(li + ii, 0, tm.s0 - 1) * tm.s1 + clampi(lj + jj, 0, tm.s1 - 1);
      sF[e] = ldg(tm.f + q);
      sF[FI * FJ + e] = ldg(tm.h + q);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < FI * TJ; e += blockDim.x) {
      const int j = e % TJ, ii = e / TJ;
      const int off = bJ[j] - lj;
      const T* wf = c == 1 ? &dJ[j][0] : &wJ[j][0];
      T af = 0, ah = 0;
#pragma unroll
      for (int t = 0; t < NZ; ++t) {
        af += sF[ii * FJ + off + t] * wf[t];
        ah += sF[FI * FJ + ii * FJ + off + t] * wJ[j][t];
      }
      sA[e] = af;
      sA[FI * TJ + e] = ah;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < NOUT; ++r) {
      const int e = threadIdx.x + r * kStThreads;
      const int j = e % TJ, i = e / TJ;
      const int off = bI[i] - li;
      const T* wf = c == 0 ? &dI[i][0] : &wI[i][0];
      T gf = 0, hh = 0;
#pragma unroll
      for (int t = 0; t < NZ; ++t) {
        gf += sA[(off + t) * TJ + j] * wf[t];
        hh += sA[FI * TJ + (off + t) * TJ + j] * wI[i][t];
      }
      acc[r] += (gf * inv_dx) * hh;
    }
  }
#pragma unroll
  for (int r = 0; r < NOUT; ++r) {
    const int e = threadIdx.x + r * kStThreads;
    const int j = j0 + e % TJ, i = i0 + e / TJ;
    if (i < so.s0 && j < so.s1) out[so.idx(i, j, 0)] = acc[r];
  }
}

// A node's first tap is floor(node position / dx - BL) plus a constant.  With a
// power-of-two dx the quotient is exact and the first taps of a tile of n nodes
// lie within [b0, b0 + n - 1] of the first node's b0 (M = 0).  Otherwise the
// quotient carries a rounding error and they lie within [b0 - 1, b0 + n]: the
// footprints then hold n + NZ + 1 taps from b0 - 1 (M = 1).
static bool power_of_two(double x) {
  int e;
  return x > 0 && std::frexp(x, &e) == 0.5;
}

template <typename T, int ORDER, int M, int TI>
static void launch_fixed3(const fm_grid& g, T dx, const StTerms<T>& terms, const MacW<T>& out, cudaStream_t s) {
  constexpr size_t smem = Fixed3<T, ORDER, M, TI>::smem;
  static_assert(smem <= 227 * 1024 - 8192, "fits a CTA");
  if (!raise_smem_limit(k_fixed_grad_dot3<T, ORDER, M, TI>, smem)) return;
  dim3 grid(3 * ((g.n[2] + kTK3) / kTK3), (g.n[1] + kTJ3) / kTJ3, (g.n[0] + TI) / TI);  // face grids: up to n + 1
  launch(k_fixed_grad_dot3<T, ORDER, M, TI>, grid, kStThreads, smem, s, g, dx, terms, out);
}

// All output grids of one call.  Tile height along i: the autotuner's choice
// (fm_tune_set, FM_TUNE_ADJ_SOURCE_TILE), else 8 in 3D and 16 in 2D; the tile
// changes only the speed, never a result.
template <typename T, int ORDER>
static void launch_fixed(const fm_grid& g, T dx, const StTerms<T>& terms, const MacW<T>& out, cudaStream_t s) {
  const int ti = tuned_value(FM_TUNE_ADJ_SOURCE_TILE, g, g.dim == 3 ? 8 : 16);
  const bool exact = power_of_two((double)dx);
  if (g.dim == 3) {
    if (exact) {
      if (ti == 4) launch_fixed3<T, ORDER, 0, 4>(g, dx, terms, out, s);
      else launch_fixed3<T, ORDER, 0, 8>(g, dx, terms, out, s);
    } else {
      // where the passes share memory an SM holds one CTA, and a wave of tiles 4 high takes 0.7 to 0.8 of the time of
      // one of tiles 8 high: the lower ones where their waves are sooner done (FP64 order 3, us by tiles 8 / 4 high:
      // 35x78x31 in 2 / 2 waves 47 / 42, 24^3 in 1 / 1 33 / 25, 25x49x122 in 3 / 4 74 / 80, 40x61x90 in 3 / 6 79 / 111)
      const auto waves = [&](int t) {
        const long ctas = 3L * ((g.n[2] + kTK3) / kTK3) * ((g.n[1] + kTJ3) / kTJ3) * ((g.n[0] + t) / t);
        return (ctas + 147) / 148;
      };
      if (ti == 4 || (!Fixed3<T, ORDER, 1, 8>::kOwnB && 5 * waves(8) > 4 * waves(4)))
        launch_fixed3<T, ORDER, 1, 4>(g, dx, terms, out, s);
      else launch_fixed3<T, ORDER, 1, 8>(g, dx, terms, out, s);
    }
    return;
  }
  // with margins a 16-row FP64 quartic tile would exceed 48 KB of static shared memory: 12 rows
  for (int c = 0; c < 2; ++c) {
    const Shape so = face_shape(g, c);
    if (ti == 8) {
      dim3 grid((so.s1 + kTJ2 - 1) / kTJ2, (so.s0 + 7) / 8, 1);
      if (exact) launch(k_fixed_grad_dot2<T, ORDER, 0, 8>, grid, kStThreads, 0, s, g, dx, c, terms, out.c[c]);
      else launch(k_fixed_grad_dot2<T, ORDER, 1, 8>, grid, kStThreads, 0, s, g, dx, c, terms, out.c[c]);
    } else if (exact) {
      dim3 grid((so.s1 + kTJ2 - 1) / kTJ2, (so.s0 + 15) / 16, 1);
      launch(k_fixed_grad_dot2<T, ORDER, 0, 16>, grid, kStThreads, 0, s, g, dx, c, terms, out.c[c]);
    } else {
      dim3 grid((so.s1 + kTJ2 - 1) / kTJ2, (so.s0 + 11) / 12, 1);
      launch(k_fixed_grad_dot2<T, ORDER, 1, 12>, grid, kStThreads, 0, s, g, dx, c, terms, out.c[c]);
    }
  }
}

template <typename T>
static int fixed_grad_dot(const fm_grid& g, int order, double dx, const StTerms<T>& terms, void* const* r,
                          cudaStream_t s) {
  const MacW<T> out{{(T*)r[0], (T*)r[1], (T*)r[2]}};
  if (order == 2) launch_fixed<T, 2>(g, (T)dx, terms, out, s);
  else if (order == 3) launch_fixed<T, 3>(g, (T)dx, terms, out, s);
  else launch_fixed<T, 4>(g, (T)dx, terms, out, s);
  return check_cuda();
}

template <typename T>
static int nabla_u_w_t(const fm_grid& g, int order, double dx, const void* const* u, const void* const* w,
                       void* const* r, cudaStream_t s) {
  StTerms<T> terms{};
  terms.n = g.dim;
  for (int a = 0; a < g.dim; ++a) {
    const Shape sa = face_shape(g, a);
    terms.t[a] = StTerm<T>{(const T*)u[a], (const T*)w[a], sa.s0, sa.s1, sa.s2,
                           a == 0 ? (T)0 : (T)0.5, a == 1 ? (T)0 : (T)0.5, a == 2 ? (T)0 : (T)0.5};
  }
  return fixed_grad_dot<T>(g, order, dx, terms, r, s);
}

template <typename T>
static int nabla_scalar_t(const fm_grid& g, double dx, const void* sc, const void* adj, void* const* r,
                          cudaStream_t s) {
  StTerms<T> terms{};
  terms.n = 1;
  const Shape cs = cell_shape(g);
  terms.t[0] = StTerm<T>{(const T*)sc, (const T*)adj, cs.s0, cs.s1, cs.s2, (T)0.5, (T)0.5, (T)0.5};
  return fixed_grad_dot<T>(g, 3, dx, terms, r, s);
}

}  // namespace fm

using namespace fm;

extern "C" {

int fm_nabla_u_w(const fm_grid* g, int dtype, int order, double dx, const void* ux, const void* uy, const void* uz,
                 const void* wx, const void* wy, const void* wz, void* rx, void* ry, void* rz, void* stream) {
  int st = validate_grid(g, dtype);
  if (st) return st;
  const void* u[3] = {ux, uy, uz};
  const void* w[3] = {wx, wy, wz};
  void* r[3] = {rx, ry, rz};
  if (order != 2 && order != 3 && order != 4) return FM_ERR_ARG;
  for (int c = 0; c < g->dim; ++c)
    if (!u[c] || !w[c] || !r[c]) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == FM_F32) return nabla_u_w_t<float>(*g, order, dx, u, w, r, s);
  return nabla_u_w_t<double>(*g, order, dx, u, w, r, s);
}

int fm_nabla_scalar_adjoint(const fm_grid* g, int dtype, double dx, const void* sc, const void* adj, void* rx,
                            void* ry, void* rz, void* stream) {
  int st = validate_grid(g, dtype);
  if (st) return st;
  void* r[3] = {rx, ry, rz};
  if (!sc || !adj) return FM_ERR_ARG;
  for (int c = 0; c < g->dim; ++c)
    if (!r[c]) return FM_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == FM_F32) return nabla_scalar_t<float>(*g, dx, sc, adj, r, s);
  return nabla_scalar_t<double>(*g, dx, sc, adj, r, s);
}

}  // extern "C"
