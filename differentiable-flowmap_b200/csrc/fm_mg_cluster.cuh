// fm_mg_cluster.cuh -- MG levels, and whole PCG solves, resident in the shared
// memory of one thread-block cluster.
//
// Below some size a V-cycle is latency-bound: each RBGS half-sweep, restriction
// and prolongation of the reference (3D/mgpcg.py:157-205) touches a few thousand
// cells but costs a kernel launch of 1-3 us.  Two kernels here run such work in
// one launch of a cluster of NC CTAs:
//   * k_mg_coarse: the levels lc .. L-1 of a V-cycle (down sweeps, restrictions,
//     bottom smoothing, prolongations, up sweeps) of a grid whose finer levels
//     are smoothed by per-level launches;
//   * k_pcg_cluster: the whole preconditioned CG solve of a grid that fits
//     (r, z, p and x in shared memory), the masked solver's included.
//
// Distribution.  The levels l0 .. ld-1 are split along axis 0 into NC slabs (in
// units of planes of level ld, so that every coarse cell's children belong to
// one CTA); z and p carry one ghost plane on each side.  The levels ld .. L-1
// live in CTA 0, each smoothed by as many warps as it has pairs for, with a
// named barrier over those warps.
//
// Exchange.  A cluster barrier with its release fence costs 800-1000 cycles
// (measured, whatever the number of CTAs), so nothing inside a solve uses one.
// Data for another CTA goes by st.async, which counts the bytes on an mbarrier
// of the receiver (about 300 cycles on top of a CTA barrier): edge planes into
// the neighbours' ghost planes after each half-sweep (an mbarrier per colour),
// restricted residuals into CTA 0, its corrections back, CTA sums of the inner
// products to everybody.  Why no push meets a reader: a red half-sweep writes
// red ghosts while the neighbour reads black ones (and vice versa), and a CTA's
// next red values depend on all of the neighbour's black ones; prolongation
// fills only the red ghosts locally (the first up-sweep, of black cells, reads
// no black ghost, and the neighbour's red push needs this CTA's black one); a
// solve's global sums separate one V-cycle's exchanges from the next one's.
//
// Layout.  Each level is stored split by colour: cells of colour c = (i+j+k)&1
// of one row, compacted along the innermost axis (cell k at m = k >> 1), so
// that a warp's loads and stores in a half-sweep hit consecutive banks (an
// interleaved layout strides by two: 2-way conflicts on every access).  The
// neighbours of a colour-c cell (row, m) with s = k & 1 all lie in the other
// colour's array: (row +- 1, m) along the outer axes, (row, m + s) for k + 1
// and (row, m + s - 1) for k - 1.  Rows and planes carry a ring of zeros, so a
// missing neighbour adds +0.0: the sum starts at +0.0 and a round-to-nearest
// sum of +0.0 and anything is never -0.0, so this equals the skipping sum.
// With an obstacle mask the neighbours are selected by per-cell bits instead.
//
// Every arithmetic step is the reference's, in its order, without FMA
// contraction: the V-cycle equals the sequential CPU one bit for bit.  Inner
// products are FP64 sums in a fixed order.
#pragma once

#include <cooperative_groups.h>
#include <stdint.h>

#include "fm_common.cuh"
#include "fm_internal.h"

namespace fm {

constexpr int kClThreads = 1024;
constexpr int kClMaxLevels = 16;
constexpr int kClMaxNC = 16;
constexpr size_t kClMaxSmem = 226 * 1024;  // dynamic shared memory per CTA
constexpr long kClDeepCells = 4096;        // CTA 0 alone smooths the levels of at most this many cells
// Cells a CTA should hold before another CTA pays (whole solves, us for 1 / 2 / 4 / 8 / 16 CTAs: 64^2 151 135 133
// 133 133, 128^2 354 . 266 232 230, 192^2 . . . 480 413, 32^3 . . . 205 184; a sequence of launches: 237, 361, 581, 221).
// Up to where a solve fits the launches are slower: projections, launches / one cluster, 304^2 776 / 612, 368^2 821 /
// 690, 512x272 822 / 764; FP64 176^2 353 / 263, 240^2 847 / 684; see plan_pcg_t for slabs that differ much.
constexpr long kClCellsPerCta = 2048;

// n / d for 0 <= n, d < 2^16 by one multiply: m = ceil(2^32 / d), 0 for d = 1.
struct FastDiv {
  uint32_t m;
  __device__ __forceinline__ int operator()(int n) const { return m ? (int)__umulhi((uint32_t)n, m) : n; }
};
inline FastDiv fast_div(int d) { return FastDiv{d <= 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d)}; }

// One level: shape and shared-memory layout.  Offsets of z, p (with ghost
// planes), r and x (without) are in elements of T, of info and msk in bytes.
struct ClLevel {
  Shape s;
  int rows, nin, M;  // rows per plane, innermost extent, pairs per row
  int sj, si;        // row and plane strides of a colour array
  int pmax;          // planes held (the largest slab)
  int z, r, p, x, info, msk;
  int zin, zinp;     // level ld: this CTA's copy of the corrections of its planes (CTA 0 sends them), planes held
  FastDiv dM, drows, dnin;
  __host__ __device__ __forceinline__ int zsz() const { return (pmax + 2) * si; }
  __host__ __device__ __forceinline__ int rsz() const { return pmax * si; }
  __host__ __device__ __forceinline__ int zinsz() const { return zinp * si; }
};

struct ClArgs {
  ClLevel lv[kClMaxLevels];
  int l0, ld, L;
  int pre_post, bottom, bottom_mode;
  int one_cell;  // the coarsest level is a single cell
  const uint16_t* msk[kClMaxLevels];  // obstacle masks per pair (SOLID), natural row order
};

// info word of a pair (row, m): bits 0-15 offset o of (plane, row, m) in a
// colour array, bit 16 s of the colour-0 cell, 17 / 18 first / last plane of
// the slab, 19-21 / 22-24 neighbour count of the colour-0 / 1 cell, 25 / 26 the
// colour-0 / 1 cell takes part (inside the domain; fluid).
// msk word: per colour c at bit 8c: 0-5 neighbours that are fluid (in the order
// +i -i +j -j +k -k; 2D: +i -i . . +j -j), 6 the cell is fluid.
// A cell that takes no part has count 1, so that its (unused) quotient is cheap.
constexpr uint32_t kClFirst = 1u << 17, kClLast = 1u << 18, kClOnes = (1u << 19) | (1u << 22);

__device__ __forceinline__ int cl_nd(uint32_t f, int c) { return (f >> (19 + 3 * c)) & 7; }
__device__ __forceinline__ bool cl_on(uint32_t f, int c) { return (f >> (25 + c)) & 1; }

// All shared memory is addressed from this array, so that the compiler emits
// shared (not generic) accesses.
extern __shared__ __align__(16) unsigned char cl_smem[];
template <typename T>
__device__ __forceinline__ T* cl_arr() { return reinterpret_cast<T*>(cl_smem); }

// x / nd rounded as the IEEE quotient, without a branch on nd (neighbouring
// lanes have different counts; a divergent branch per count costs several times
// the arithmetic) and with the rare cases after the fact: fast() is stored, and
// replaced by slow() where bad().  FP32: the reciprocal multiply with an FMA
// correction of div_nd, which for a power of two is the exact scaling alone; bad
// outside div_nd's checked range.  FP64: exact scaling by a power of two, else
// the division.
template <typename T>
struct ClQuot;
template <>
struct ClQuot<float> {
  float s, d, rd;
  ClQuot() = default;
  __device__ __forceinline__ explicit ClQuot(int nd) {
    s = (nd == 2 || nd == 6) ? 0.5f : (nd == 4 ? 0.25f : 1.0f);
    d = (nd == 3 || nd == 6) ? 3.0f : (nd == 5 ? 5.0f : (nd == 0 ? 0.0f : 1.0f));
    rd = (nd == 3 || nd == 6) ? (1.0f / 3.0f) : (nd == 5 ? (1.0f / 5.0f) : 1.0f);
  }
  __device__ __forceinline__ float fast(float x) const {
    const float y = __fmul_rn(x, s);
    const float q0 = __fmul_rn(y, rd);
    const float e = __fmaf_rn(-q0, d, y);
    return __fmaf_rn(e, rd, q0);
  }
  template <bool SOLID>
  __device__ __forceinline__ bool bad(float x) const {
    const float ax = fabsf(x);
    return !(ax >= 0x1p-100f && ax <= 0x1p100f) || (SOLID && d == 0.0f);
  }
  __device__ __forceinline__ float slow(float x) const { return x / (d / s); }
};
template <>
struct ClQuot<double> {
  double s, d;
  ClQuot() = default;
  __device__ __forceinline__ explicit ClQuot(int nd) {
    s = nd == 4 ? 0.25 : (nd == 2 ? 0.5 : (nd == 1 ? 1.0 : 0.0));
    d = (double)nd;
  }
  __device__ __forceinline__ double fast(double x) const { return x * s; }
  template <bool SOLID>
  __device__ __forceinline__ bool bad(double) const { return s == 0.0; }
  __device__ __forceinline__ double slow(double x) const { return x / d; }
};

// Sum over the neighbours of the colour-c cell at offset o in the other
// colour's array (at element zo), in the reference's order (+i -i +j -j +k -k).
template <typename T, int D, bool SOLID>
__device__ __forceinline__ T cl_nb(int zo, int o, int s, int si, int sj, unsigned mk) {
  const T* q = cl_arr<T>() + zo + o;
  T v[6];
  v[0] = q[si];
  v[1] = q[-si];
  if (D == 3) {
    v[2] = q[sj];
    v[3] = q[-sj];
  }
  v[4] = q[s];
  v[5] = q[s - 1];
  T nb = 0;
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    if (D == 2 && (a == 2 || a == 3)) continue;
    nb += (!SOLID || ((mk >> a) & 1)) ? v[a] : (T)0;
  }
  return nb;
}

// The two halves of a barrier that orders no memory: it only keeps every CTA in place
// until all have arrived.
__device__ __forceinline__ void cl_cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// shared::cluster addresses and the ghost-plane exchange
__device__ __forceinline__ uint32_t cl_remote(const void* p, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void cl_st_async(uint32_t addr, float v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
               "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cl_st_async(uint32_t addr, double v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}

// The head of the shared memory: mbarriers, whether a wait gave up (which ends
// up as a non-finite outcome), and what the smoothers need of each level.
enum { kBarRed = 0, kBarBlack = 1, kBarSum0 = 2, kBarSum1 = 3, kBarDown = 4, kBarUp = 5, kBarP = 6, kNBars = 7 };

// One level as this CTA sees it.  lo / hi and their mbarriers: shared::cluster
// byte addresses of the neighbours' arrays (0: none).
struct ClRun {
  int z, r, info, msk, si, sj, zsz, rsz, npairs;
  uint32_t lo, hi, lo_bar, hi_bar;
  int lo_shift, hi_shift;  // elements
  uint32_t bytes;          // received per half-sweep
};
struct ClHead {
  uint64_t bar[8];
  int failed, pad[3];
  ClRun run[kClMaxLevels];
  ClArgs args;  // every CTA's copy: indexed loads of kernel parameters miss the constant cache
};
constexpr int kClHead = (sizeof(ClHead) + 127) / 128 * 128;
__device__ __forceinline__ ClHead* cl_head() { return reinterpret_cast<ClHead*>(cl_smem); }
__device__ __forceinline__ const ClArgs& cl_load_args(const ClArgs* __restrict__ a) {
  static_assert(sizeof(ClArgs) % 4 == 0, "copied by words");
  for (int q = threadIdx.x; q < (int)(sizeof(ClArgs) / 4); q += kClThreads)
    reinterpret_cast<uint32_t*>(&cl_head()->args)[q] = reinterpret_cast<const uint32_t*>(a)[q];
  __syncthreads();
  return cl_head()->args;
}

__device__ __forceinline__ uint32_t cl_bar(int b) { return (uint32_t)__cvta_generic_to_shared(cl_head()->bar + b); }
// One thread, once per phase: the bytes this CTA receives in it.
__device__ __forceinline__ void cl_expect(int b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cl_bar(b)), "r"(bytes) : "memory");
}
// Waits for the phase of mbarrier b, at most about a million tries.
__device__ __forceinline__ void cl_wait(int b, uint32_t phase) {
  const uint32_t addr = cl_bar(b), par = (phase >> b) & 1;
  for (int it = 0; it < (1 << 20); ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(addr), "r"(par)
        : "memory");
    if (done) return;
    if (*(volatile int*)&cl_head()->failed) return;
  }
  *(volatile int*)&cl_head()->failed = 1;
}

// End of a half-sweep of colour c; waits: this thread reads ghosts next.
template <bool DIST>
__device__ __forceinline__ void cl_half_end(const ClRun& R, int c, bool waits, int nthr, uint32_t& phase) {
  if constexpr (DIST) {
    if (threadIdx.x == 0) cl_expect(c, R.bytes);
    __syncthreads();
    if (waits) cl_wait(c, phase);
    phase ^= 1u << c;
  } else if (nthr == 32) {
    __syncwarp();
  } else {
    asm volatile("bar.sync 1, %0;" ::"r"(nthr) : "memory");
  }
}

template <typename T>
__device__ __forceinline__ void cl_push_edges(const ClRun& R, uint32_t f, int c, T v) {
  const int q = c * R.zsz + (int)(f & 0xffff);
  if (R.lo && (f & kClFirst)) cl_st_async(R.lo + (uint32_t)sizeof(T) * (q + R.lo_shift), v, R.lo_bar + 8 * c);
  if (R.hi && (f & kClLast)) cl_st_async(R.hi + (uint32_t)sizeof(T) * (q + R.hi_shift), v, R.hi_bar + 8 * c);
}

// `halves` (even) RBGS half-sweeps (3D/mgpcg.py:170-177) of level l, colours
// first, 1 - first, ..., by the first nthr threads (all of them with DIST), U
// pairs per thread; residuals, divisors and addresses stay in registers across
// the half-sweeps (npairs <= U * nthr).  A slot without a pair points at the
// first interior cell and never stores.  zero: z = 0 before the first
// half-sweep, which then reads no neighbours.  In 2D a warp whose cells all take
// part and have four neighbours divides by the one exact multiply.  Returns the
// mbarrier phases.  Out of line: inlined for every level the kernel's code
// outgrows the instruction cache, and a V-cycle runs each only a few
// half-sweeps long.  (One CTA, cycles per half-sweep: 8^2 160, 16^2 190, 64^2
// 430-640, 8^3 260, 16^3 1070; bound by shared-memory wavefronts -- five or
// seven per 32 cells -- at the larger sizes, by the dependent chain of loads,
// the ordered sum, the quotient and the barrier at the smaller ones.)
template <typename T, int D, bool SOLID, bool DIST, int U>
__device__ __noinline__ uint32_t cl_smooth_u(int l, int first, int halves, bool zero, int nthr, uint32_t phase) {
  const ClRun& R = cl_head()->run[l];
  const int si = R.si, sj = R.sj, tid = threadIdx.x;
  const uint32_t* info = reinterpret_cast<const uint32_t*>(cl_smem + R.info);
  const uint16_t* msk = reinterpret_cast<const uint16_t*>(cl_smem + R.msk);
  T* z = cl_arr<T>() + R.z;
  const T* r = cl_arr<T>() + R.r;
  const int npairs = R.npairs, zsz = R.zsz, rsz = R.rsz;
  if (D == 2 && DIST && U == 1 && (tid & ~31) >= npairs) {  // a warp without pairs: only the barriers
    for (int h = 0; h < halves; ++h) cl_half_end<DIST>(R, first ^ (h & 1), h + 2 >= halves, nthr, phase);
    return phase;
  }
  uint32_t f[U];
  unsigned mk[U];
  T rv[U][2];
  T* own[U][2];  // own cell of step t (colour first, then 1 - first)
  const T* row[U][2];  // the k + 1 neighbour (k - 1 before it)
  bool full = D == 2, edge = false;
  constexpr uint32_t both = (3u << 25) | ((uint32_t)(2 * D) << 19) | ((uint32_t)(2 * D) << 22);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int e = tid + u * nthr;
    f[u] = e < npairs ? info[e] : (uint32_t)(si + (D == 3 ? sj : 0) + 1) | kClOnes;
    mk[u] = (SOLID && e < npairs) ? msk[e] : 0;
    const int o = (int)(f[u] & 0xffff);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int c = first ^ t;
      rv[u][t] = r[c * rsz + o - si];
      own[u][t] = z + c * zsz + o;
      row[u][t] = z + (1 - c) * zsz + o + (((f[u] >> 16) & 1) ^ c);
    }
    const bool ed = DIST && (f[u] & (kClFirst | kClLast));
    edge = edge || ed;
    full = full && (f[u] & (0xffu << 19)) == both && !ed;
  }
  if (DIST) edge = __any_sync(0xffffffffu, edge);
  if (D == 2) full = __all_sync(0xffffffffu, full);
  auto nbsum = [&](int u, int t, unsigned m) {
    const T* q = own[u][1 - t];
    T v[6];
    v[0] = q[si];
    v[1] = q[-si];
    if (D == 3) {
      v[2] = q[sj];
      v[3] = q[-sj];
    }
    v[4] = row[u][t][0];
    v[5] = row[u][t][-1];
    T nb = 0;
#pragma unroll
    for (int a = 0; a < 6; ++a) {
      if (D == 2 && (a == 2 || a == 3)) continue;
      nb += (!SOLID || ((m >> a) & 1)) ? v[a] : (T)0;
    }
    return nb;
  };
  if (D == 2 && full) {
    for (int h = 0; h < halves; h += 2) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        T v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const T nb = nbsum(u, t, 63u);
          v[u] = rn_add(rv[u][t], t == 0 && zero ? (T)0 : nb) * (T)0.25;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) *own[u][t] = v[u];
        cl_half_end<DIST>(R, first ^ t, edge || h + 2 >= halves, nthr, phase);
      }
      zero = false;
    }
    return phase;
  }
  ClQuot<T> Q[U][2];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int t = 0; t < 2; ++t) Q[u][t] = ClQuot<T>(cl_nd(f[u], first ^ t));
  for (int h = 0; h < halves; h += 2) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int c = first ^ t;
      T x[U], v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T nb = nbsum(u, t, SOLID ? mk[u] >> (8 * c) : 63u);
        x[u] = rn_add(rv[u][t], t == 0 && zero ? (T)0 : nb);
        v[u] = Q[u][t].fast(x[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (cl_on(f[u], c)) *own[u][t] = v[u];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (Q[u][t].template bad<SOLID>(x[u]) && cl_on(f[u], c)) {
          v[u] = Q[u][t].slow(x[u]);
          *own[u][t] = v[u];
        }
        if (DIST && edge) cl_push_edges(R, f[u], c, v[u]);
      }
      cl_half_end<DIST>(R, c, edge || h + 2 >= halves, nthr, phase);
    }
    zero = false;
  }
  return phase;
}

// Any number of pairs per thread: info words and residuals re-read per half-sweep.
template <typename T, int D, bool SOLID, bool DIST>
__device__ __noinline__ uint32_t cl_smooth_any(int l, int first, int halves, bool zero, int nthr, uint32_t phase) {
  const ClRun& R = cl_head()->run[l];
  const int si = R.si, sj = R.sj, npairs = R.npairs;
  const uint32_t* info = reinterpret_cast<const uint32_t*>(cl_smem + R.info);
  const uint16_t* msk = reinterpret_cast<const uint16_t*>(cl_smem + R.msk);
  constexpr int U = 2;
  for (int h = 0; h < halves; ++h) {
    const int c = first ^ (h & 1);
    const T* rc = cl_arr<T>() + R.r + c * R.rsz - si;
    T* zc = cl_arr<T>() + R.z + c * R.zsz;
    const int zo = R.z + (1 - c) * R.zsz;
    for (int e0 = threadIdx.x; e0 < npairs; e0 += U * nthr) {
      uint32_t f[U];
      T x[U], v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * nthr;
        f[u] = e < npairs ? info[e] : (uint32_t)(si + (D == 3 ? sj : 0) + 1) | kClOnes;
        const unsigned mk = (SOLID && e < npairs) ? msk[e] : 0;
        const int o = f[u] & 0xffff;
        const T nb = cl_nb<T, D, SOLID>(zo, o, (int)((f[u] >> 16) & 1) ^ c, si, sj, mk >> (8 * c));
        x[u] = rn_add(rc[o], zero && h == 0 ? (T)0 : nb);
        v[u] = ClQuot<T>(cl_nd(f[u], c)).fast(x[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const ClQuot<T> Q(cl_nd(f[u], c));
        if (Q.template bad<SOLID>(x[u]) && cl_on(f[u], c)) v[u] = Q.slow(x[u]);
        if (cl_on(f[u], c)) zc[f[u] & 0xffff] = v[u];
        if (DIST) cl_push_edges(R, f[u], c, v[u]);
      }
    }
    cl_half_end<DIST>(R, c, true, nthr, phase);
  }
  return phase;
}

// Everything a CTA knows about its share of the levels.
template <typename T, int D, bool SOLID>
struct ClCta {
  const ClArgs& a;
  int rank, nc, tid;
  int u0, u1;  // units (planes of level ld) of this CTA
  uint32_t phase = 0;  // parities of the mbarriers

  __device__ __forceinline__ ClCta(const ClArgs& args, int rk, int n) : a(args), rank(rk), nc(n), tid(threadIdx.x) {
    u0 = first_unit(rank);
    u1 = first_unit(rank + 1);
  }
  __device__ __forceinline__ int first_unit(int rk) const { return rk * a.lv[a.ld].s.s0 / nc; }
  __device__ __forceinline__ int first_plane(int l) const { return l < a.ld ? u0 << (a.ld - l) : 0; }
  __device__ __forceinline__ int planes(int l) const { return l < a.ld ? (u1 - u0) << (a.ld - l) : a.lv[l].s.s0; }
  __device__ __forceinline__ T* z(int l) const { return cl_arr<T>() + a.lv[l].z; }
  __device__ __forceinline__ T* r(int l) const { return cl_arr<T>() + a.lv[l].r; }
  __device__ __forceinline__ uint32_t* info(int l) const { return reinterpret_cast<uint32_t*>(cl_smem + a.lv[l].info); }
  __device__ __forceinline__ uint16_t* msk(int l) const { return reinterpret_cast<uint16_t*>(cl_smem + a.lv[l].msk); }
  __device__ __forceinline__ int npairs(int l) const { return planes(l) * a.lv[l].rows * a.lv[l].M; }

  // The head; rings and ghosts zero; info (and mask) words of every level this
  // CTA holds.  The caller's next cluster barrier makes it known to the others.
  __device__ __noinline__ void setup() const {
    ClHead* H = cl_head();
    if (tid == 0) {
      H->failed = 0;
      for (int b = 0; b < kNBars; ++b) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_bar(b)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid >= 32 && tid - 32 >= a.l0 && tid - 32 < a.L) {
      const int l = tid - 32;
      const ClLevel& L = a.lv[l];
      ClRun& R = H->run[l];
      const bool dist = l < a.ld;
      R.z = L.z;
      R.r = L.r;
      R.info = L.info;
      R.msk = L.msk;
      R.si = L.si;
      R.sj = L.sj;
      R.zsz = L.zsz();
      R.rsz = L.rsz();
      R.npairs = npairs(l);
      R.lo = dist && rank > 0 ? cl_remote(z(l), rank - 1) : 0;
      R.hi = dist && rank < nc - 1 ? cl_remote(z(l), rank + 1) : 0;
      R.lo_bar = R.lo ? cl_remote(H->bar, rank - 1) : 0;
      R.hi_bar = R.hi ? cl_remote(H->bar, rank + 1) : 0;
      R.lo_shift = rank > 0 ? ((u0 - first_unit(rank - 1)) << (a.ld - l)) * L.si : 0;
      R.hi_shift = -planes(l) * L.si;
      R.bytes = (uint32_t)sizeof(T) * L.rows * L.M * ((R.lo != 0) + (R.hi != 0));
    }
    for (int l = a.l0; l < a.L; ++l) {
      const ClLevel& L = a.lv[l];
      if (l == a.ld)
        for (int q = tid; q < 2 * (L.zinsz()); q += kClThreads) cl_arr<T>()[L.zin + q] = 0;
      if (l >= a.ld && rank != 0) continue;
      T* zl = z(l);
      for (int q = tid; q < 2 * L.zsz(); q += kClThreads) zl[q] = 0;
      const int n = npairs(l), i0 = first_plane(l), np = planes(l), perp = L.rows * L.M;
      uint32_t* inf = info(l);
      for (int e = tid; e < n; e += kClThreads) {
        const int row = L.dM(e), m = e - row * L.M;
        const int p = D == 3 ? L.drows(row) : row, j = D == 3 ? row - p * L.rows : 0;
        const int i = i0 + p;
        const int s0 = (i + j) & 1;
        uint32_t f = (uint32_t)((p + 1) * L.si + (D == 3 ? (j + 1) * L.sj : 0) + m + 1) | ((uint32_t)s0 << 16);
        if (p == 0) f |= kClFirst;
        if (p == np - 1) f |= kClLast;
        unsigned mk = 0;
        if constexpr (SOLID) {
          mk = a.msk[l][i0 * perp + e];
          msk(l)[e] = (uint16_t)mk;
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int k = 2 * m + (s0 ^ c);
          bool on = k < L.nin;
          int nd;
          if constexpr (SOLID) {
            on = on && ((mk >> (8 * c)) & 64);
            nd = __popc((mk >> (8 * c)) & 63);
          } else {
            nd = 2 * D - (i == 0) - (i == L.s.s0 - 1) - (k == 0) - (k == L.nin - 1);
            if (D == 3) nd -= (j == 0) + (j == L.s.s1 - 1);
          }
          f |= (uint32_t)(on ? nd : 1) << (19 + 3 * c);
          if (on) f |= 1u << (25 + c);
        }
        inf[e] = f;
      }
    }
  }

  // Smoothing of level l by the first nthr threads (all of them where the level
  // is distributed).
  template <bool DIST>
  __device__ __forceinline__ void smooth(int l, int first, int halves, bool zero, int nthr) {
    if (halves == 0) return;
    // in 2D each warp by its own pairs: one whose second slot is empty would otherwise compute along on
    // a pair of nobody (FP32 projections with and without that: 384^2 461 / 491 us, 320x448 484 / 511, 192^2
    // 262 / 284, 128^2 240 / 238; in 3D, where more is left of the divergence, 40^3 422 / 407)
    const int n = npairs(l);
    if (n <= (D == 2 ? (tid & ~31) + nthr : nthr)) phase = cl_smooth_u<T, D, SOLID, DIST, 1>(l, first, halves, zero, nthr, phase);
    else if (sizeof(T) == 4 && n <= 2 * nthr) phase = cl_smooth_u<T, D, SOLID, DIST, 2>(l, first, halves, zero, nthr, phase);
    else phase = cl_smooth_any<T, D, SOLID, DIST>(l, first, halves, zero, nthr, phase);
  }

  // Gather-restriction (3D/mgpcg.py:157-163) of the coarse cells below this
  // CTA's planes of level l into its share of level l + 1, or, at l + 1 = ld,
  // into CTA 0.
  __device__ __noinline__ void restrict_to(int l) const {
    const ClLevel& F = a.lv[l];
    const ClLevel& Cc = a.lv[l + 1];
    const T* zf = z(l);
    const T* rf = r(l);
    const uint32_t* inf = info(l);
    const int zsz = F.zsz(), rsz = F.rsz(), cr = Cc.rows, cn = Cc.nin, crsz = Cc.rsz();
    const T scale = (T)1.0 / (T)(D - 1.0);
    const int nP = planes(l) / 2, I0 = first_plane(l) / 2, dst0 = l + 1 == a.ld ? u0 : 0;
    const uint32_t far = l + 1 == a.ld && rank != 0 ? cl_remote(r(l + 1), 0) : 0;
    const uint32_t far_bar = far ? cl_remote(cl_head()->bar + kBarDown, 0) : 0;
    const int n = nP * cr * cn;
    for (int q = tid; q < n; q += kClThreads) {
      const int row = Cc.dnin(q), Kc = q - row * cn;
      const int pI = D == 3 ? Cc.drows(row) : row, J = D == 3 ? row - pI * cr : 0;
      T acc = 0;
#pragma unroll
      for (int di = 0; di < 2; ++di)
#pragma unroll
        for (int dj = 0; dj < (D == 3 ? 2 : 1); ++dj) {
          const int e = ((2 * pI + di) * F.rows + (D == 3 ? 2 * J + dj : 0)) * F.M + Kc;
          const uint32_t f = inf[e];
          const int o = f & 0xffff;
          const unsigned mk = SOLID ? msk(l)[e] : 0u;
#pragma unroll
          for (int dk = 0; dk < 2; ++dk) {
            const int c = (di + dj + dk) & 1;  // the slab starts at an even plane
            const T nb = cl_nb<T, D, SOLID>(F.z + (1 - c) * zsz, o, dk, F.si, F.sj, mk >> (8 * c));
            const T res = rn_sub(rf[c * rsz + o - F.si], rn_sub(rn_mul((T)cl_nd(f, c), zf[c * zsz + o]), nb));
            const T sum = rn_add(acc, rn_mul(res, scale));
            acc = !SOLID || cl_on(f, c) ? sum : acc;
          }
        }
      const int cc = (I0 + pI + J + Kc) & 1;
      const int dst = cc * crsz + (dst0 + pI) * Cc.si + (D == 3 ? (J + 1) * Cc.sj : 0) + (Kc >> 1) + 1;
      if (far) cl_st_async(far + (uint32_t)sizeof(T) * dst, acc, far_bar);
      else r(l + 1)[dst] = acc;
    }
  }

  // CTA 0: the corrections of level ld to the CTAs that prolong them (each its
  // planes and the one beside on either side), into their zin.
  __device__ __noinline__ void send_up() const {
    const ClLevel& L = a.lv[a.ld];
    const int per = 2 * L.rows * L.M;  // cells of a plane
    const int share = kClThreads / nc, rk = tid / share, t0 = tid - rk * share;  // nc is a power of two
    if (rk == 0) return;
    const int f0 = first_unit(rk), f1 = first_unit(rk + 1);
    const int lo = f0 - 1, hi = f1 < L.s.s0 ? f1 + 1 : f1;  // planes lo .. hi-1
    const uint32_t dst = cl_remote(cl_arr<T>() + L.zin, rk), bar = cl_remote(cl_head()->bar + kBarUp, rk);
    for (int q = t0; q < (hi - lo) * per; q += share) {
      const int row2 = L.dM(q), m = q - row2 * L.M;  // rows of both colours
      const int c = row2 & 1, row = row2 >> 1;
      const int pl = D == 3 ? L.drows(row) : row, j = D == 3 ? row - pl * L.rows : 0;
      const int in = (D == 3 ? (j + 1) * L.sj : 0) + m + 1;
      cl_st_async(dst + (uint32_t)sizeof(T) * (c * L.zinsz() + pl * L.si + in),
                  z(a.ld)[c * L.zsz() + (lo + pl + 1) * L.si + in], bar);
    }
  }
  __device__ __forceinline__ uint32_t up_bytes() const {
    const ClLevel& L = a.lv[a.ld];
    return (uint32_t)sizeof(T) * 2 * L.rows * L.M * ((u1 < L.s.s0 ? u1 + 1 : u1) - (u0 - 1));
  }

  // Prolongation z_f += z_c (3D/mgpcg.py:165-168) of level l, one coarse cell
  // (2^(D-1) fine pairs) per thread.  On a distributed level also the red cells
  // of the ghost planes inside the domain, from the coarse planes beside.
  __device__ __noinline__ void prolong_from(int l) const {
    const ClLevel& F = a.lv[l];
    const ClLevel& Cc = a.lv[l + 1];
    const bool dist = l < a.ld, copy = l + 1 == a.ld && rank != 0;
    // coarse colour arrays whose ring plane 0 is global plane cI0 - 1
    const T* zc = copy ? cl_arr<T>() + Cc.zin : z(l + 1);
    const int czsz = copy ? Cc.zinsz() : Cc.zsz(), cI0 = copy ? u0 : (l + 1 < a.ld ? first_plane(l) / 2 : 0);
    T* zf = z(l);
    const int zsz = F.zsz(), np = planes(l), I0 = first_plane(l) / 2;
    const int P_lo = dist && rank > 0 ? -1 : 0, P_hi = np / 2 + (dist && rank < nc - 1 ? 1 : 0);
    const int n = (P_hi - P_lo) * Cc.rows * Cc.nin;
    for (int q = tid; q < n; q += kClThreads) {
      const int row = Cc.dnin(q), K = q - row * Cc.nin;
      const int pl = D == 3 ? Cc.drows(row) : row, J = D == 3 ? row - pl * Cc.rows : 0, P = P_lo + pl;
      const int I = I0 + P, cc = (I + J + K) & 1;
      const T v = zc[cc * czsz + (I - cI0 + 1) * Cc.si + (D == 3 ? (J + 1) * Cc.sj : 0) + (K >> 1) + 1];
#pragma unroll
      for (int di = 0; di < 2; ++di) {
        const int p = 2 * P + di;  // plane of the slab; -1 and np are the ghosts
        if (p < -1 || p > np) continue;
        const bool own = p >= 0 && p < np;
#pragma unroll
        for (int dj = 0; dj < (D == 3 ? 2 : 1); ++dj) {
          const int j = D == 3 ? 2 * J + dj : 0;
          const int o = (p + 1) * F.si + (D == 3 ? (j + 1) * F.sj : 0) + K + 1;
          // with a mask only fluid cells (no other value is ever read)
          uint32_t f = 3u << 25;
          if (SOLID && own) f = info(l)[(p * F.rows + j) * F.M + K];
          if (!SOLID || cl_on(f, 0)) zf[o] = rn_add(zf[o], v);
          if (own && (!SOLID || cl_on(f, 1))) zf[zsz + o] = rn_add(zf[zsz + o], v);
        }
      }
    }
  }

  // A coarsest level of one cell has no neighbours: r / 0, as everywhere (the smoothers'
  // quotients leave that count out).
  __device__ __noinline__ void lone_cell(int sweeps) const {
    const int b = a.L - 1, o = info(b)[0] & 0xffff;
    if (tid == 0 && sweeps > 0) z(b)[o] = div_nd(r(b)[o - a.lv[b].si], 0);
  }

  // Levels l0 .. L-1 of a V-cycle on r(l0) -> z(l0).  Ends with a CTA barrier.
  __device__ __forceinline__ void vcycle() {
    const int ld = a.ld, b = a.L - 1;
    for (int l = a.l0; l < ld; ++l) {
      smooth<true>(l, 0, 2 * a.pre_post, true, kClThreads);
      restrict_to(l);
      __syncthreads();
    }
    if (rank == 0) {
      if (tid == 0) cl_expect(kBarDown, (uint32_t)sizeof(T) * a.lv[ld].rows * a.lv[ld].nin * (a.lv[ld].s.s0 - u1));
      cl_wait(kBarDown, phase);
      phase ^= 1u << kBarDown;
      auto threads_of = [&](int l) {
        const int n = npairs(l);
        return n < kClThreads ? (n + 31) & ~31 : kClThreads;
      };
      for (int l = ld; l < b; ++l) {
        const int nt = threads_of(l);
        if (tid < nt) smooth<false>(l, 0, 2 * a.pre_post, true, nt);
        __syncthreads();
        restrict_to(l);
        __syncthreads();
      }
      // bottom smoothing (3D/mgpcg.py:197-199; mgpcg_solid.py:263-268)
      const int nt = threads_of(b);
      if (tid < nt) {
        const int n = a.bottom_mode == 0 ? a.bottom : a.bottom / 2;
        if (n == 0)
          for (int q = tid; q < 2 * a.lv[b].zsz(); q += nt) z(b)[q] = 0;
        smooth<false>(b, 0, 2 * n, true, nt);
        if (a.bottom_mode == 1) smooth<false>(b, 1, 2 * n, false, nt);
        if (!SOLID && a.one_cell) lone_cell(n);
      }
      __syncthreads();
      for (int l = b - 1; l >= ld; --l) {
        prolong_from(l);
        __syncthreads();
        const int nl = threads_of(l);
        if (tid < nl) smooth<false>(l, 1, 2 * a.pre_post, false, nl);
        __syncthreads();
      }
      send_up();
    } else {
      if (tid == 0) cl_expect(kBarUp, up_bytes());
      cl_wait(kBarUp, phase);
      phase ^= 1u << kBarUp;
    }
    for (int l = ld - 1; l >= a.l0; --l) {
      prolong_from(l);
      __syncthreads();
      smooth<true>(l, 1, 2 * a.pre_post, false, kClThreads);
    }
  }
};

// Levels l0 .. L-1 of a V-cycle whose finer levels run as per-level launches.
template <typename T, int D, typename St>
__global__ void __launch_bounds__(kClThreads, 1) k_mg_coarse(const ClArgs* __restrict__ args, const T* __restrict__ r_top,
                                                             T* __restrict__ z_top, const St* st) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const ClArgs& a = cl_load_args(args);
  ClCta<T, D, false> C(a, (int)cl.block_rank(), (int)cl.num_blocks());
  const int l = a.l0, tid = threadIdx.x;
  const ClLevel& L = a.lv[l];
  C.setup();  // of this CTA's own shared memory only: runs beside the kernel before (128^3 projection: 446 -> 443 us)
  pdl_begin();
  if (st->done) return;  // same value in every CTA of the cluster
  __syncthreads();
  // natural rows -> colour arrays (cell k of a row at m = k >> 1)
  const int rowlen = L.nin, nrows = C.planes(l) * L.rows;
  const long g0 = (long)C.first_plane(l) * L.rows * rowlen;
  T* r = C.r(l);
  for (int q = tid; q < nrows * rowlen; q += kClThreads) {
    const int row = L.dnin(q), k = q - row * rowlen;
    const int p = D == 3 ? L.drows(row) : row, j = D == 3 ? row - p * L.rows : 0;
    const int c = (p + j + k) & 1;  // the slab starts at an even plane
    r[c * L.rsz() + p * L.si + (D == 3 ? (j + 1) * L.sj : 0) + (k >> 1) + 1] = r_top[g0 + q];
  }
  cl_cluster_sync();  // heads and zeroed ghosts everywhere before the first push
  C.vcycle();
  // No CTA exits while another may still send to it: where every wait succeeds none
  // can, but a CTA whose wait gave up runs ahead of its neighbours.  The stores
  // below overlap the barrier (a 128^3 V-cycle: 126.2 us without it, 126.4 so, 126.7 with release and acquire).
  cl_cluster_arrive();
  const T* z = C.z(l);
  for (int q = tid; q < nrows * rowlen; q += kClThreads) {
    const int row = L.dnin(q), k = q - row * rowlen;
    const int p = D == 3 ? L.drows(row) : row, j = D == 3 ? row - p * L.rows : 0;
    const int c = (p + j + k) & 1;
    const T v = z[c * L.zsz() + (p + 1) * L.si + (D == 3 ? (j + 1) * L.sj : 0) + (k >> 1) + 1];
    z_top[g0 + q] = cl_head()->failed ? (T)nan("") : v;  // a wait that gave up ends the solve as non-finite
  }
  cl_cluster_wait();
}

// ---------------------------------------------------------------------------
// whole PCG solve
// ---------------------------------------------------------------------------
struct PcgParams {
  int max_iters;
  double abs_tol, rel_tol, eps;
};
struct PcgOutcome {
  double zTr, tol, rTr, alpha, beta, mean, pAp;
  int it, conv, nonfinite, stepped;
};

// Sums over the cluster's threads, every thread receiving the same values:
// warp shuffles, warp partials in shared memory, CTA partials sent into every
// CTA's slots (two slot buffers and mbarriers in turn, so that a slow reader of
// one sum never meets the next one's).
struct ClSums {
  double warp[2][32];
  double slot[2][2][kClMaxNC];
};
template <int N>
__device__ __forceinline__ void cl_sum(ClSums& S, int& turn, uint32_t& phase, int rank, int nc, double* v) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, bar = kBarSum0 + turn;
#pragma unroll
  for (int k = 0; k < N; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0) S.warp[k][w] = v[k];
  }
  if (threadIdx.x == 0) cl_expect(bar, (uint32_t)sizeof(double) * N * nc);
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      double x = S.warp[k][lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane < nc) cl_st_async(cl_remote(&S.slot[turn][k][rank], lane), x, cl_remote(cl_head()->bar + bar, lane));
    }
  }
  cl_wait(bar, phase);
  phase ^= 1u << bar;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    double x[kClMaxNC];
#pragma unroll
    for (int i = 0; i < kClMaxNC; ++i) x[i] = i < nc ? S.slot[turn][k][i] : 0.0;
#pragma unroll
    for (int h = kClMaxNC / 2; h > 0; h >>= 1)
#pragma unroll
      for (int i = 0; i < h; ++i) x[i] += x[i + h];
    v[k] = x[0];
  }
  turn ^= 1;
}

// PCG (3D/mgpcg.py:207-289; 2D/vortex/mgpcg_solid.py:318-363 with a mask) on the
// right-hand side r_in (natural layout), the solution written to x when the
// solve took a step (x is zero on entry; the kernels before this one clear it).
// The overloads of pcg_skip / pcg_floor / pcg_finish for Ctx connect it to the
// caller's bookkeeping.  With a mask the inner products and the updates of x, r
// and p act on fluid cells, the recentring on all cells.
template <typename T, int D, bool SOLID, typename Ctx>
__global__ void __launch_bounds__(kClThreads, 1) k_pcg_cluster(const ClArgs* __restrict__ args, PcgParams P,
                                                               const T* __restrict__ r_in, T* __restrict__ x_out,
                                                               Ctx st) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ ClSums sums;
  const int rank = (int)cl.block_rank(), nc = (int)cl.num_blocks(), tid = threadIdx.x;
  const ClArgs& a = cl_load_args(args);
  ClCta<T, D, SOLID> C(a, rank, nc);
  const ClLevel& L = a.lv[0];
  const int n = C.npairs(0), si = L.si, sj = L.sj, zsz = L.zsz(), rsz = L.rsz();
  T* z = C.z(0);
  T* r = C.r(0);
  T* p = cl_arr<T>() + L.p;
  T* x = cl_arr<T>() + L.x;
  const bool far_x = L.x < 0;  // no room in shared memory: x stays in x_out (the same thread's cells every time)
  const uint32_t* info = C.info(0);
  const uint16_t* msk = C.msk(0);
  const long g0 = (long)C.first_plane(0) * L.rows * L.nin;  // cell (2m) of pair e is at g0 + 2 e (even rows)
  const double ncell = (double)L.s.size();
  int turn = 0;
  // the set-up writes this CTA's own shared memory and reads constants of the handle: it
  // runs beside the kernel before, unless there are masks, which a kernel packs (256^2
  // projection: 316 -> 313 us)
  if (SOLID) pdl_begin();
  C.setup();
  for (int q = tid; q < 2 * zsz; q += kClThreads) p[q] = 0;
  if (!SOLID) pdl_begin();
  if (pcg_skip(st)) return;  // same value in every CTA of the cluster
  cl_cluster_sync();  // heads and zeroed ghosts everywhere before the first push
  const uint32_t p_lo = rank > 0 ? cl_remote(p, rank - 1) : 0, p_hi = rank < nc - 1 ? cl_remote(p, rank + 1) : 0;
  const ClRun& R0 = cl_head()->run[0];
  // pair e covers cells 2m (colour s0) and 2m + 1 (colour 1 - s0) of its row
  double s[2] = {0, 0};
  for (int e = tid; e < n; e += kClThreads) {
    const uint32_t f = info[e];
    const int o = (int)(f & 0xffff) - si, c0 = (f >> 16) & 1;
    const T v0 = r_in[g0 + 2 * e], v1 = r_in[g0 + 2 * e + 1];
    r[c0 * rsz + o] = v0;
    r[(1 - c0) * rsz + o] = v1;
    s[0] += (double)v0;
    s[0] += (double)v1;
  }
  cl_sum<1>(sums, turn, C.phase, rank, nc, s);
  PcgOutcome R{};
  R.mean = s[0] / ncell;
  for (bool first = true;; first = false) {
    // recentre r, z = M r, z . r
    const T mean = (T)R.mean;
    for (int e = tid; e < n; e += kClThreads) {
      const int o = (int)(info[e] & 0xffff) - si;
      r[o] = r[o] - mean;
      r[rsz + o] = r[rsz + o] - mean;
    }
    __syncthreads();
    C.vcycle();
    s[0] = 0;
    for (int e = tid; e < n; e += kClThreads) {
      const uint32_t f = info[e];
      const int o = f & 0xffff;
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (cl_on(f, c)) s[0] += (double)z[c * zsz + o] * (double)r[c * rsz + o - si];
    }
    cl_sum<1>(sums, turn, C.phase, rank, nc, s);
    if (first) {
      R.zTr = s[0];
      double tol = P.abs_tol;
      if (P.rel_tol > 0 && s[0] * P.rel_tol > tol) tol = s[0] * P.rel_tol;
      const double fl = pcg_floor(st);
      if (fl > tol) tol = fl;
      R.tol = tol;
      if (!SOLID && !isfinite(s[0])) { R.nonfinite = 1; break; }
      if (s[0] == 0.0) { R.conv = 1; break; }  // r = 0: the zero start is the solution
    } else {
      R.beta = s[0] / (R.zTr + P.eps);
      R.zTr = s[0];
      R.it += 1;
      if (R.it >= P.max_iters) break;
    }
    // p = z + beta p, its edge planes into the neighbours' ghosts
    const T beta = (T)R.beta;
    for (int e = tid; e < n; e += kClThreads) {
      const uint32_t f = info[e];
      const int o = f & 0xffff;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int q = c * zsz + o;
        T v = p[q];
        if (cl_on(f, c)) p[q] = v = first ? z[q] : rn_add(z[q], rn_mul(beta, v));
        if (p_lo && (f & kClFirst)) cl_st_async(p_lo + (uint32_t)sizeof(T) * (q + R0.lo_shift), v, R0.lo_bar + 8 * kBarP);
        if (p_hi && (f & kClLast)) cl_st_async(p_hi + (uint32_t)sizeof(T) * (q + R0.hi_shift), v, R0.hi_bar + 8 * kBarP);
      }
    }
    if (tid == 0) cl_expect(kBarP, 2 * R0.bytes);
    __syncthreads();
    cl_wait(kBarP, C.phase);
    C.phase ^= 1u << kBarP;
    // A p (kept in z, which the next V-cycle rewrites) and p . A p
    s[0] = 0;
    for (int e = tid; e < n; e += kClThreads) {
      const uint32_t f = info[e];
      const int o = f & 0xffff;
      const unsigned mk = SOLID ? msk[e] : 0u;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const T pv = p[c * zsz + o];
        const T nb = cl_nb<T, D, SOLID>(L.p + (1 - c) * zsz, o, (int)((f >> 16) & 1) ^ c, si, sj, mk >> (8 * c));
        const T ap = rn_sub(rn_mul((T)cl_nd(f, c), pv), nb);
        if (cl_on(f, c)) {
          z[c * zsz + o] = ap;
          s[0] += (double)pv * (double)ap;
        }
      }
    }
    cl_sum<1>(sums, turn, C.phase, rank, nc, s);
    R.pAp = s[0];
    R.alpha = R.zTr / (s[0] + P.eps);
    // x += alpha p, r -= alpha A p, r . r and the sum of r
    const T alpha = (T)R.alpha;
    s[0] = s[1] = 0;
    for (int e = tid; e < n; e += kClThreads) {
      const uint32_t f = info[e];
      const int o = f & 0xffff;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int q = c * rsz + o - si;
        T rv = r[q];
        if (cl_on(f, c)) {
          const T dx = rn_mul(alpha, p[c * zsz + o]);
          if (far_x) {
            T* xe = x_out + g0 + 2 * e + (((f >> 16) & 1) ^ c);
            *xe = rn_add(first ? (T)0 : *xe, dx);
          } else {
            x[q] = rn_add(first ? (T)0 : x[q], dx);
          }
          rv = rn_sub(rv, rn_mul(alpha, z[c * zsz + o]));
          r[q] = rv;
          s[0] += (double)rv * (double)rv;
        }
        s[1] += (double)rv;
      }
    }
    cl_sum<2>(sums, turn, C.phase, rank, nc, s);
    R.rTr = s[0];
    R.stepped = 1;
    R.mean = s[1] / ncell;
    if (!isfinite(s[0])) { R.nonfinite = 1; break; }
    if (s[0] < R.tol) { R.conv = 1; break; }
  }
  if (R.stepped && !far_x)
    for (int e = tid; e < n; e += kClThreads) {
      const uint32_t f = info[e];
      const int o = (int)(f & 0xffff) - si, c0 = (f >> 16) & 1;
      if (cl_on(f, c0)) x_out[g0 + 2 * e] = x[c0 * rsz + o];
      if (cl_on(f, 1 - c0)) x_out[g0 + 2 * e + 1] = x[(1 - c0) * rsz + o];
    }
  if (tid == 0 && cl_head()->failed) cl.map_shared_rank(cl_head(), 0)->failed = 1;
  cl_cluster_sync();  // no CTA exits while another may still send to it
  if (rank == 0 && tid == 0) {
    if (cl_head()->failed) { R.conv = 0; R.nonfinite = 1; R.rTr = nan(""); }
    pcg_finish(st, R);
  }
}

// ---------------------------------------------------------------------------
// host side: layout of the levels l0 .. L-1 over nc CTAs
// ---------------------------------------------------------------------------
// Fills the level geometry and offsets; returns the shared-memory bytes per
// CTA, or 0 where the split is impossible (fewer units than CTAs, offsets past
// 16 bits).
inline size_t cl_layout(ClArgs& a, const Shape* lv, int l0, int ld, int L, int dim, size_t es, int nc, bool pcg,
                        bool solid, bool x_in = true) {
  a.l0 = l0;
  a.ld = ld;
  a.L = L;
  a.one_cell = lv[L - 1].size() == 1;
  size_t off = kClHead;  // bytes
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 15) & ~size_t(15);
    return o;
  };
  const int units = lv[ld].s0;
  if (units < nc) return 0;
  const int umax = (units + nc - 1) / nc;
  for (int l = 0; l < L; ++l) {
    ClLevel& c = a.lv[l];
    c = ClLevel{};
    c.s = lv[l];
    c.rows = dim == 3 ? lv[l].s1 : 1;
    c.nin = dim == 3 ? lv[l].s2 : lv[l].s1;
    c.M = (c.nin + 1) / 2;
    c.sj = c.M + 2;
    c.si = dim == 3 ? (c.rows + 2) * c.sj : c.sj;
    c.dM = fast_div(c.M);
    c.drows = fast_div(c.rows);
    c.dnin = fast_div(c.nin);
    if (l < l0) continue;
    c.pmax = l < ld ? umax << (ld - l) : lv[l].s0;
    if ((long)(c.pmax + 2) * c.si > 0xffff) return 0;
    if (l == ld) {  // umax planes and one on each side
      c.zinp = umax + 2;
      c.zin = (int)(take(2 * es * c.zinsz()) / es);
    }
    c.z = (int)(take(2 * es * c.zsz()) / es);
    c.r = (int)(take(2 * es * c.rsz()) / es);
    if (pcg && l == 0) {
      c.p = (int)(take(2 * es * c.zsz()) / es);
      c.x = x_in ? (int)(take(2 * es * c.rsz()) / es) : -1;
    }
    c.info = (int)take(sizeof(uint32_t) * (size_t)c.pmax * c.rows * c.M);
    if (solid) c.msk = (int)take(sizeof(uint16_t) * (size_t)c.pmax * c.rows * c.M);
  }
  return off;
}

// Launch as a cluster of nc CTAs (the whole grid), with programmatic dependent launch.
template <typename... KArgs, typename... Args>
inline cudaError_t cl_launch(void (*k)(KArgs...), int nc, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nc, 1, 1);
  cfg.blockDim = dim3(kClThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)nc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_pdl.load(std::memory_order_relaxed) ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, std::forward<Args>(args)...);
  count_launch(1);
  return e;
}

// Whether the device runs `kernel` as a cluster of nc CTAs with this much shared memory.
template <typename Kernel>
inline bool cl_enable(Kernel kernel, int nc, size_t smem) {
  if (!raise_smem_limit(kernel, smem)) return false;
  if (nc > 8 && cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return false;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nc, 1, 1);
  cfg.blockDim = dim3(kClThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)nc;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  return cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
}

// Plans a whole solve in one cluster: returns the CTAs, or 0 (the solve then runs as a
// sequence of launches) where the state does not fit 16 CTAs or level ld has fewer planes
// than the CTAs that the cell count asks for.  With four levels and more that leaves squares
// up to 384^2 (FP64: 240^2, masked 232^2) and cubes of 16^3, 24^3 and 32^3 (FP64: 16^3 and 24^3).
template <typename Kernel>
inline int cl_plan_pcg(ClArgs& a, Kernel kernel, const Shape* lv, int L, const fm_mg_params& P, int dim, size_t es,
                       bool solid, size_t* smem_out) {
  if (P.pre_post < 1 || L < 2) return 0;  // the first sweep of a level is what writes its z
  int ld = 1;
  while (ld < L - 1 && lv[ld].size() > kClDeepCells) ++ld;
  int nc = 1;
  while (nc < kClMaxNC && lv[0].size() > kClCellsPerCta * nc) nc *= 2;
  for (; nc <= kClMaxNC; nc *= 2) {
    size_t smem = cl_layout(a, lv, 0, ld, L, dim, es, nc, true, solid);
    if (smem == 0) return 0;  // too few planes for more CTAs
    if (smem > kClMaxSmem && nc < kClMaxNC) continue;
    if (smem > kClMaxSmem) smem = cl_layout(a, lv, 0, ld, L, dim, es, nc, true, solid, false);
    if (smem > kClMaxSmem) return 0;
    if (!cl_enable(kernel, nc, smem)) break;
    a.pre_post = P.pre_post;
    a.bottom = P.bottom;
    a.bottom_mode = P.bottom_mode;
    *smem_out = smem;
    return nc;
  }
  cudaGetLastError();
  return 0;
}

}  // namespace fm
