// Sub-warp-per-system kernels for n <= 32 (ion-balance systems, n = 2..27 in
// practice, and small macro atoms).
//
// A group of G lanes (G in {4, 8, 16, 32}, so 8/4/2/1 systems per warp) owns
// one system; lane r holds row r of A in registers (NP doubles, NP >= n, all
// indices compile-time after unrolling).  Rows never move: each carries its
// current position `pos`, the pivot search reduces (|a| bits, position) over
// the group, and the pivot row is broadcast through a small shared buffer.
//
// solve  : GSL-exact LU (lu.c:62-288) with the lower triangular sweep of LU_svx
//          riding along, then its row-oriented upper sweep (lu.c:329-360,
//          cblas/source_trsv_r.h) in GSL's operation order, then the reference
//          residual check (matrix_cpu.c:155-187) on the original A held in
//          shared memory.
// invert : in-place Gauss-Jordan whose below-pivot updates are the GSL-exact
//          LU updates (so the pivots, U and the singular test of lu.c:540 are
//          GSL's), above-pivot and already-inverted columns eliminated in the
//          same sweep; columns are unscrambled in reverse pivot order at the end.
#pragma once
#include <type_traits>

#include "ss_common.cuh"

namespace ss {

constexpr int kSmallThreads = 128;

// A solve's shared memory (the mixed path keeps its scales in u, which only its
// exact fallback needs for pivot rows).
template <int NP>
struct __align__(16) SmallSmem {
  static constexpr int S = NP + 1;   // odd row stride (in doubles) avoids bank conflicts
  double stage[NP * S];              // A as loaded, kept for the residual check; comes first
  double u[NP * (NP + 3 - NP / 2)];  // the pivot rows by step (small_urow)
  double xs[NP];                     // solution in natural order
};

// An inverse's: one pivot row at a time.  With a solve's pivot rows beside it fewer
// CTAs fit an SM (20,000 inverses of order 32: 592 us, 390 so).
template <int NP>
struct __align__(16) SmallInvSmem {
  static constexpr int S = NP + 1;
  double stage[NP * S];              // A as loaded, then the rows of the result
  double piv[NP];                    // broadcast pivot row
  int ipiv[NP];                      // position swapped with j at step j
  int csrc[NP];                      // column unscramble map
};

// Start of pivot row j in SmallSmem::u: columns j & ~1 .. NP - 1, the row's
// right-hand side and its pivot's reciprocal (0 if it is not to be used).
template <int NP>
__host__ __device__ constexpr int small_urow(int j) {
  return (j / 2) * 2 * (NP + 3 - j / 2) + (j & 1) * (NP + 2 - (j & ~1));
}

// dynamic shared memory of a launch
template <int KIND, int NP, int G>
constexpr size_t small_smem_bytes() {
  return (KIND == kSolve ? sizeof(SmallSmem<NP>) : sizeof(SmallInvSmem<NP>)) * (kSmallThreads / G);
}

template <int G>
__device__ __forceinline__ unsigned group_mask() {
  const int wlane = threadIdx.x & 31;
  return (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (wlane & ~(G - 1)));
}

// Row stride of a staged system of order n (in doubles): odd, so that a column
// read by rows falls on distinct banks.
__device__ __forceinline__ int small_stride(int n) { return n | 1; }

// Coalesced load of a system into `stage` (rows small_stride(n) apart), every
// load of the lane issued before the first shared-memory store so they are all
// in flight together.  Element e = r n + c goes to e + r for an even n; e / n by
// a 16-bit reciprocal, exact for e < 1024, n <= 32.
template <int NP, int G>
__device__ __forceinline__ void small_stage(double* stage, const double* __restrict__ Ag, int n, int lane, unsigned gmask) {
  constexpr int PER = (NP * NP + G - 1) / G;
  const int nn = n * n;
  double v[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int e = lane + u * G;
    v[u] = (e < nn) ? __ldg(Ag + e) : 0.0;
  }
  const unsigned inv = 65536u / unsigned(n > 0 ? n : 1) + 1u;   // n = 0: an idle group
  const unsigned even = (n & 1) ? 0u : 1u;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const unsigned e = unsigned(lane + u * G);
    if (int(e) < nn) stage[e + even * ((e * inv) >> 16)] = v[u];
  }
  __syncwarp(gmask);
}

// GSL-exact Gauss-Jordan sweep of the row held in a[].  Returns true when U has
// an exact zero on its diagonal.
template <int NP, int G>
__device__ __forceinline__ bool small_exact_gj(SmallInvSmem<NP>& sm, double (&a)[NP], int n, int lane,
                                               unsigned gmask, int& pos, bool& inf_piv) {
  const bool act = lane < n;
  bool done = false;
  bool sing = false;
  inf_piv = false;
  pos = lane;
  double* piv = sm.piv;
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    if (j < n && !sing) {
      // first strict maximum of |a| in current row order (cblas idamax): the
      // eligible rows' keys carry bit 63 and NaN counts as zero; ties go to the
      // smaller position
      const bool elig = act && !done;
      unsigned long long key = 0ull;
      if (elig) {
        const double v = fabs(a[j]);
        key = (v == v) ? (static_cast<unsigned long long>(__double_as_longlong(v)) | (1ull << 63)) : (1ull << 63);
      }
      const unsigned hi = unsigned(key >> 32), lo = unsigned(key);
      const unsigned mh = __reduce_max_sync(gmask, hi);
      const unsigned ml = __reduce_max_sync(gmask, hi == mh ? lo : 0u);
      const int kp = int(__reduce_min_sync(gmask, (elig && hi == mh && lo == ml) ? unsigned(pos) : 0xffffffffu));
      const int p = (__ffs(__ballot_sync(gmask, elig && pos == kp)) - 1) & (G - 1);
      const bool was_done = done;
      if (lane == p) {
        pos = j;
        done = true;
      } else if (pos == j) {
        pos = kp;
      }
      if (lane == 0) sm.ipiv[j] = kp;
      if (lane == p) {
#pragma unroll
        for (int k = 0; k < NP; ++k) piv[k] = a[k];
      }
      __syncwarp(gmask);
      const double ujj = piv[j];
      inf_piv |= isinf(ujj);
      if (ujj == 0.0) {
        sing = true;   // lu.c:540 singular(): the result is decided
      } else {
        const double rinv = __drcp_rn(ujj);   // correctly rounded, = fl(1/ujj)
        if (lane == p) {
#pragma unroll
          for (int k = 0; k < NP; ++k) a[k] = (k == j) ? rinv : mul_rn(a[k], rinv);
        } else if (act) {
          const double l = was_done ? mul_rn(a[j], rinv) : gsl_multiplier(a[j], ujj, rinv);
#pragma unroll
          for (int k = 0; k < NP; ++k)
            if (k != j) a[k] = sub_rn(a[k], mul_rn(l, piv[k]));
          a[j] = -l;
        }
      }
      __syncwarp(gmask);
    }
  }
  return sing;
}

// Reference residual check of x (sm.xs, natural order) against the original
// A (sm.stage), b_i in row i's lane; the first failing row decides
// (matrix_cpu.c:162-187).  Also returns, in *worst, the largest check value over
// all rows.  mask: the lanes that take part, whole groups (n may differ by group).
template <int NP, int G>
__device__ __forceinline__ int small_residual_code(const SmallSmem<NP>& sm, double bi, int n, int lane, unsigned mask,
                                                   double* worst) {
  int code = 0;
  double chk = 0.0;
  if (lane < n) {
    double acc = 0.0;
    const double* arow = sm.stage + lane * small_stride(n);
#pragma unroll
    for (int k = 0; k < NP; ++k)
      if (k < n) acc = add_rn(acc, mul_rn(arow[k], sm.xs[k]));
    const double y = add_rn(0.0, acc);
    if (bi > 0.0) {
      chk = fabs(div_rn(sub_rn(y, bi), y));
      if (chk > kResidEps) code = kResidRel;
    } else {
      chk = fabs(sub_rn(y, bi));
      if (chk > kResidEps) code = kResidAbs;
    }
    if (!(chk == chk)) chk = 1.0e300;   // a NaN check value passes the reference test; flag it
  }
  int first = code ? lane : 0x7fffffff;
  int fcode = code;
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) {
    const int of = __shfl_xor_sync(mask, first, off, G);
    const int oc = __shfl_xor_sync(mask, fcode, off, G);
    const double ow = __shfl_xor_sync(mask, chk, off, G);
    if (of < first) { first = of; fcode = oc; }
    chk = fmax(chk, ow);
  }
  *worst = chk;
  return fcode;
}

// Largest value of each group: a redux per group of the warp, the other groups
// holding zeros (they overlap; a redux under the groups' own masks would run
// one group after another), a butterfly for the smallest groups.
template <int G>
__device__ __forceinline__ unsigned group_max(unsigned mask, unsigned v) {
  if constexpr (G == 32) {
    return __reduce_max_sync(mask, v);
  } else if constexpr (G >= 8) {
    const int own = (threadIdx.x & 31) / G;
    unsigned m = 0u;
#pragma unroll
    for (int q = 0; q < 32 / G; ++q) {
      const unsigned mq = __reduce_max_sync(mask, own == q ? v : 0u);
      m = own == q ? mq : m;
    }
    return m;
  } else {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(mask, v, o, G));
    return v;
  }
}

// The general pivot choice of a step: first strict maximum of |a| in current row
// order (cblas idamax) over the eligible lanes, NaN counting as zero, with the
// multiplier of every lane's row.  Kept out of line: only steps whose pivot is
// zero, tiny, huge or not a number come here.
struct PivotChoice {
  double l;    // this lane's multiplier
  int p;       // the pivot's lane
  int zero;    // an exact zero
};
template <int G>
__device__ __noinline__ PivotChoice small_pivot_general(double v, bool elig, int pos, unsigned mask) {
  unsigned long long key = 0ull;
  if (elig) key = (v == v) ? (static_cast<unsigned long long>(__double_as_longlong(fabs(v))) | (1ull << 63)) : (1ull << 63);
  unsigned at = elig ? unsigned(pos) : 0xffffffffu;
  int p = threadIdx.x & (G - 1);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const unsigned long long k2 = __shfl_xor_sync(mask, key, o, G);
    const unsigned a2 = __shfl_xor_sync(mask, at, o, G);
    const int p2 = __shfl_xor_sync(mask, p, o, G);
    if (k2 > key || (k2 == key && a2 < at)) {
      key = k2;
      at = a2;
      p = p2;
    }
  }
  PivotChoice r;
  r.p = p;
  const double ujj = __shfl_sync(mask, v, p, G);
  r.zero = (ujj == 0.0);
  r.l = gsl_multiplier(v, ujj, __drcp_rn(ujj));
  return r;
}

// The upper sweep by divisions, one lane of each group walking U as GSL does: for
// systems whose quotients div_markstein may not round correctly.  Returns x_lane.
template <int NP, int G>
__device__ __noinline__ double small_upper_general(SmallSmem<NP>& sm, int n, int lane, unsigned mask) {
  __syncwarp(mask);
  if (lane == 0) {
    for (int i = n - 1; i >= 0; --i) {
      const double* ur = sm.u + small_urow<NP>(i) - (i & ~1);
      double u = ur[NP];
      for (int k = i + 1; k < n; ++k) u = sub_rn(u, mul_rn(ur[k], sm.xs[k]));
      sm.xs[i] = div_rn(u, ur[i]);
    }
  }
  __syncwarp(mask);
  return (lane < n) ? sm.xs[lane] : 0.0;
}

// Complete GSL-exact solve of the staged system (sm.stage, kept), b_i in row i's
// lane; writes x unless the system is singular and returns the code.  mask:
// the lanes that call it together, whole groups; n may differ by group (0: an
// idle group), every branch around a warp operation is the same for all of them.
//
// What bounds it is one chain per system, so each step keeps only that chain
// between two pivots, straight-line and in few instructions (the unrolled steps
// are run once per system and have to come through the instruction cache):
//   * the pivot search takes three reductions (high and low words of |a|, then
//     the position: equal magnitudes are common in rate matrices, where a
//     diagonal entry minus its sum leaves the rate itself) and a vote;
//     everything rare goes out of line (small_pivot_general);
//   * every lane forms the reciprocal of its own candidate while the reduction
//     is in flight; the pivot's reciprocal and its next column's entry arrive
//     by shuffle, and only that column is updated before the next search;
//   * the other columns, and the right-hand side as one more column (LU_svx
//     subtracts l_ij y_j from b_i with j ascending, as the update does), follow
//     from the pivot row in shared memory while the next reductions run.  Rows
//     already chosen go through the same update: they are kept in shared memory
//     and what their lanes hold no longer matters.
// The upper sweep's order, x_i = (y_i - U_i,i+1 x_i+1 - U_i,i+2 x_i+2 ...) / U_ii,
// makes a chain of n^2 / 2 subtractions: lane i takes row i of U and all products
// of an x are formed at once, so that the chain holds subtractions alone (one
// lane used to walk it, a load, a product and a difference per entry).
// 4,096 systems of order 27: 66 -> 43 us; 200,000 of the orders one cell carries
// (2-27): 770 -> 522 us.
// CHECK: false leaves the residual check out (code 0 or 4), for callers to whom
// codes 2 and 3 mean nothing.
template <int NP, int G, bool CHECK = true>
__device__ __forceinline__ int small_exact_solve(SmallSmem<NP>& sm, double bi, double* __restrict__ xg, int n,
                                                 int lane, unsigned mask) {
  static_assert(NP % 4 == 0, "pivot rows move in pairs");
  const int gsh = threadIdx.x & 31 & ~(G - 1);
  const unsigned gbits = (G == 32) ? 0xffffffffu : ((1u << (G & 31)) - 1u);
  const int nmax = (G == 32) ? n : int(__reduce_max_sync(mask, unsigned(n)));
  double a[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) a[k] = (lane < n && k < n) ? sm.stage[lane * small_stride(n) + k] : 0.0;
  double t = bi, l = 0.0;
  int pos = lane;
  // sign mask of this lane's magnitudes; 0 once its row is chosen or its system found singular
  unsigned alive = lane < n ? 0x7fffffffu : 0u;
  bool sing = false;
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    if (j < nmax) {
      constexpr unsigned kLo = 0x00200000u, kSpan = 0x7fa00000u;   // 2^-1021 <= |v| < 2^1021
      const int j1 = (j + 1 < NP) ? j + 1 : j;
      const double v = a[j];
      const unsigned key = unsigned(__double2hiint(v)) & alive;
      const unsigned mh = group_max<G>(mask, key);
      const unsigned lo = (key == mh) ? unsigned(__double2loint(v)) : 0u;
      const unsigned ml = group_max<G>(mask, lo);
      const bool cand = key == mh && lo == ml;
      const double rb = rcp_markstein(v);
      // the step before: its columns beyond this one and the right-hand side
      if (j > 0) {
        const double2* pv = reinterpret_cast<const double2*>(sm.u + small_urow<NP>(j - 1));
        const int k0 = (j - 1) & ~1;
#pragma unroll
        for (int k = (j + 1) & ~1; k < NP; k += 2) {
          const double2 w = pv[(k - k0) / 2];
          if (k > j) a[k] = sub_rn(a[k], mul_rn(l, w.x));
          a[k + 1] = sub_rn(a[k + 1], mul_rn(l, w.y));
        }
        t = sub_rn(t, mul_rn(l, pv[(NP - k0) / 2].x));
      }
      // the smallest position among equals; it is the pivot's
      int at = 31 - int(group_max<G>(mask, cand ? 31u - unsigned(pos) : 0u));
      int p = (__ffs((__ballot_sync(mask, cand && pos == at) >> gsh) & gbits) - 1) & (G - 1);
      // a pivot of an unordinary size (0 when every row left is zero there), or a
      // significand that the reciprocal may miss
      bool odd = mh - kLo >= kSpan || ml == 0xffffffffu;
      if (G < 32) odd = __any_sync(mask, odd && j < n && !sing);
      double rinv = __shfl_sync(mask, rb, p, G);
      l = mul_rn(v, rinv);
      if (odd) {
        const PivotChoice ch = small_pivot_general<G>(v, alive != 0u, pos, mask);
        p = ch.p;
        l = ch.l;
        rinv = 0.0;
        at = __shfl_sync(mask, pos, p, G);
        if (ch.zero && j < n) {   // lu.c:540 singular(): the result is decided
          sing = true;
          alive = 0u;
        }
      }
      const double u1 = __shfl_sync(mask, a[j1], p, G);
      if (lane == p && alive) {
        double2* pw = reinterpret_cast<double2*>(sm.u + small_urow<NP>(j));
        const int k0 = j & ~1;
#pragma unroll
        for (int k = k0; k < NP; k += 2) pw[(k - k0) / 2] = make_double2(a[k], a[k + 1]);
        pw[(NP - k0) / 2] = make_double2(t, rinv);
        alive = 0u;
      }
      pos = (lane == p) ? j : (pos == j ? at : pos);
      if (j + 1 < NP) a[j1] = sub_rn(a[j1], mul_rn(l, u1));
      __syncwarp(mask);
    }
  }
  // lane i takes row i of U; the upper sweep turns a[k] from U_ik into the
  // product U_ik x_k, zero for k >= n (u - 0 = u)
  double ri;
  {
    const int row = (lane < NP) ? lane : 0;
    const double* ur = sm.u + small_urow<NP>(row) - (row & ~1);
#pragma unroll
    for (int k = 0; k < NP; k += 2) {
      const double2 w = *reinterpret_cast<const double2*>(ur + k);
      a[k] = w.x;
      a[k + 1] = w.y;
    }
    t = ur[NP];
    ri = ur[NP + 1];
  }
  double xv = 0.0;
  unsigned far = 0u;
#pragma unroll
  for (int i = NP - 1; i >= 0; --i) {
    if (i < nmax) {
      double u = t;
#pragma unroll
      for (int k = i + 1; k < NP; ++k) u = sub_rn(u, a[k]);
      const bool own = lane == i && i < n;
      const double x = div_markstein(own ? u : 1.0, own ? a[i] : 1.0, own ? ri : 1.0, far);
      const double xi = __shfl_sync(mask, x, i & (G - 1), G);
      if (own) xv = x;
      a[i] = (i < n) ? mul_rn(a[i], xi) : 0.0;
    } else {
      a[i] = 0.0;
    }
  }
  if (__any_sync(mask, far >= kDivFar && !sing)) xv = small_upper_general<NP, G>(sm, n, lane, mask);
  int code = kOk;
  if (CHECK) {
    if (lane < n) sm.xs[lane] = xv;
    __syncwarp(mask);
    double worst;
    code = small_residual_code<NP, G>(sm, bi, n, lane, mask, &worst);
  }
  if (lane < n && !sing) xg[lane] = xv;
  return sing ? kSolveSingular : code;
}

// CTAs per SM asked of the register allocator.  Solves: the best of those measured
// (NP = 28 47.2 us at 4, 48.7 at 5; 16 97.0 at 5, 99.7 at 4; 12 61.4 at 6, 64.6 at
// 5); no row is spilled but at NP = 24, 44 bytes at 5.  Inverses: as many as hold
// their rows without spilling; left to itself the allocator takes up to 186
// registers (20,000 of order 16: 104 us at 102 registers, 82 at 80).
template <int KIND, int NP>
constexpr int small_min_blocks() {
  if (KIND != kSolve) return NP > 20 ? 4 : NP > 16 ? 5 : NP > 12 ? 6 : NP > 8 ? 7 : NP > 4 ? 8 : 9;
  return NP > 28 ? 3 : NP > 24 ? 4 : NP > 12 ? 5 : 6;
}

template <int KIND, int NP, int G>
__global__ void __launch_bounds__(kSmallThreads, (small_min_blocks<KIND, NP>()))
small_exact_kernel(BatchView bv) {
  static_assert(G == 4 || G == 8 || G == 16 || G == 32, "group size");
  static_assert(NP <= G, "one row per lane");
  static_assert(small_min_blocks<KIND, NP>() * (small_smem_bytes<KIND, NP, G>() + 1024) <= kSmemPerSm,
                "the CTAs asked for fit an SM");
  constexpr int GPB = kSmallThreads / G;       // groups per block
  extern __shared__ __align__(16) unsigned char small_dsm[];
  using Smem = std::conditional_t<KIND == kSolve, SmallSmem<NP>, SmallInvSmem<NP>>;

  const int grp = threadIdx.x / G;
  const int lane = threadIdx.x % G;
  Smem& sm = reinterpret_cast<Smem*>(small_dsm)[grp];   // [GPB]
  const int count = batch_count(bv);

  if constexpr (KIND == kSolve) {
    // a warp's groups stay together (a group past the list's end idles with
    // n = 0); the next system's place is read, and its matrix brought into L2,
    // while this one is solved
    constexpr int GPW = 32 / G;
    const int sub = (threadIdx.x & 31) / G;
    const int stride = gridDim.x * GPB;
    int first = blockIdx.x * GPB + grp - sub;
    auto system = [&](int it) -> int { return it < count ? bv.list[it] : -1; };
    int s = system(first + sub);
    int n = s >= 0 ? bv.n[s] : 0;
    int64_t oa = s >= 0 ? bv.offA[s] : 0, ov = s >= 0 ? bv.offv[s] : 0;
    static_assert(GPW * G == 32, "whole groups");
    for (; first < count; first += stride) {
      const int s2 = system(first + stride + sub);
      const double bi = (lane < n) ? bv.b[ov + lane] : 0.0;
      small_stage<NP, G>(sm.stage, bv.A + oa, n, lane, 0xffffffffu);
      const int n2 = s2 >= 0 ? bv.n[s2] : 0;
      const int64_t oa2 = s2 >= 0 ? bv.offA[s2] : 0, ov2 = s2 >= 0 ? bv.offv[s2] : 0;
      const int code = small_exact_solve<NP, G>(sm, bi, bv.out + ov, n, lane, 0xffffffffu);
      if (s >= 0 && lane == 0) {
        bv.status[s] = code;
        if (bv.diag) bv.diag[s] = kDiagExact;
      }
      for (int e = 16 * lane; e < n2 * n2; e += 16 * G)
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(bv.A + oa2 + e));
      __syncwarp();
      s = s2;
      n = n2;
      oa = oa2;
      ov = ov2;
    }
  } else {
    constexpr int S = SmallInvSmem<NP>::S;
    const unsigned gmask = group_mask<G>();
    for (int item = blockIdx.x * GPB + grp; item < count; item += gridDim.x * GPB) {
      const int s = bv.list[item];
      const int n = bv.n[s];
      small_stage<NP, G>(sm.stage, bv.A + bv.offA[s], n, lane, gmask);
      const bool act = lane < n;
      double a[NP];
#pragma unroll
      for (int k = 0; k < NP; ++k) a[k] = (act && k < n) ? sm.stage[lane * small_stride(n) + k] : 0.0;
      int pos;
      bool inf_piv;
      const bool sing = small_exact_gj<NP, G>(sm, a, n, lane, gmask, pos, inf_piv);
      // GSL's LU_invx inverts U in place and then finds 1/u_jj = 0 on the
      // diagonal for an infinite pivot: GSL_ESING, output untouched
      const int code = sing ? kInvertSingular : (inf_piv ? kInvertInfPivot : kOk);
      if (code == kOk) {
        // rows of W by position, then the reverse-order column unscramble
        if (act) {
#pragma unroll
          for (int k = 0; k < NP; ++k)
            if (k < n) sm.stage[pos * S + k] = a[k];
        }
        if (lane == 0) {
          for (int c = 0; c < n; ++c) sm.csrc[c] = c;
          for (int j = n - 1; j >= 0; --j) {
            const int q = sm.ipiv[j];
            if (q != j) {
              const int tt = sm.csrc[j];
              sm.csrc[j] = sm.csrc[q];
              sm.csrc[q] = tt;
            }
          }
        }
        __syncwarp(gmask);
        double* __restrict__ Og = bv.out + bv.offA[s];
        for (int e = lane; e < n * n; e += G) {
          const int r = e / n;
          Og[e] = sm.stage[r * S + sm.csrc[e - r * n]];
        }
      }
      if (lane == 0) {
        bv.status[s] = code;
        if (bv.diag) bv.diag[s] = kDiagExact;
      }
      __syncwarp(gmask);
    }
  }
}

}  // namespace ss
