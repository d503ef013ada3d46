// Mixed-precision solve for n <= 32: equilibrated FP32 LU + FP64 iterative
// refinement, with the GSL-exact FP64 solve (kernels_small.cuh) as the
// fallback run in place by the same lane group.
//
//   1. R, C = powers of two that bring every row and then every column of A to
//      a maximum in [0.5, 1); As = fl32(R A C) (scaling by powers of two is exact).
//   2. FP32 LU of As with partial pivoting (rows stay in their lanes).
//   3. x0 = C As^-1 R b, then x += C As^-1 R (b - A x) with the residual in FP64
//      on the original A, until every significant component (|x_j| above
//      `floor` times the sum of |x|) moves by at most tol * |x_j|.
//   4. The FP64 path re-solves the system when: the FP32 factorisation meets a
//      zero / non-finite pivot or a pivot ratio below 1 / cond_limit (condition
//      estimate), a refinement step contracts by less than cond_limit * 4 u32
//      or it runs out of iterations, or the reference's own residual test (matrix_cpu.c:162-187)
//      could land within a factor 256 n u of its 1e-6 threshold for this x, in
//      which case only the exact FP64 solution can decide codes 2 / 3.
// Everything that reaches the caller from the FP32 path therefore has status 0,
// exactly as the reference would report.
#pragma once
#include "kernels_small.cuh"

namespace ss {

__host__ __device__ inline MixedParams default_mixed_params() {
  MixedParams p;
  p.max_iter = 12;
  p.tol = 1.0e-14;
  p.cond_limit = 1.0e3;
  p.resid_margin = 1.0e-8;
  return p;
}

// power of two 2^-e with m * 2^-e in [0.5, 1); 1 for zero / non-finite m
__device__ __forceinline__ double pow2_inv_scale(double m) {
  if (!(m > 0.0) || !isfinite(m)) return 1.0;
  int e;
  frexp(m, &e);
  return ldexp(1.0, -e);
}

// CTAs per SM asked of the register allocator, which without a bound takes the
// registers of one or two of them (order 16, 40,000 rate matrices: 437 us at 114
// registers, 402 at 5 CTAs, 374 at 6; order 32, 4,096: 203 us at 164, 160 at 4).
template <int NP>
constexpr int mixed_min_blocks() {
  return NP > 20 ? 4 : NP > 16 ? 5 : NP > 12 ? 6 : NP > 8 ? 7 : 8;
}

template <int NP, int G>
__global__ void __launch_bounds__(kSmallThreads, (mixed_min_blocks<NP>()))
small_mixed_solve_kernel(BatchView bv, MixedParams mp) {
  constexpr int GPB = kSmallThreads / G;
  static_assert(mixed_min_blocks<NP>() * (small_smem_bytes<kSolve, NP, G>() + 1024) <= kSmemPerSm,
                "the CTAs asked for fit an SM");
  constexpr double kFloor = 1.0e-22;          // significance floor of a component (x_j / sum |x|)
  extern __shared__ __align__(16) unsigned char small_dsm[];
  SmallSmem<NP>* smem_all = reinterpret_cast<SmallSmem<NP>*>(small_dsm);   // [GPB]

  const int grp = threadIdx.x / G;
  const int lane = threadIdx.x % G;
  const unsigned gmask = group_mask<G>();
  SmallSmem<NP>& sm = smem_all[grp];
  // over the space of the fallback's pivot rows: row and column scales, the
  // broadcast pivot row, the row chosen at each step
  double* rsc = sm.u;
  double* csc = rsc + NP;
  float* fpiv = reinterpret_cast<float*>(csc + NP);
  int* lop = reinterpret_cast<int*>(fpiv + NP);
  static_assert(2 * sizeof(double) + sizeof(float) + sizeof(int) <= sizeof(sm.u) / NP, "they fit");

  // a warp's groups stay together, so that their fallbacks run together; a group
  // past the list's end idles with n = 0
  const int count = batch_count(bv);
  const int sub = (threadIdx.x & 31) / G;
  for (int first = blockIdx.x * GPB + grp - sub; first < count; first += gridDim.x * GPB) {
    const bool live = first + sub < count;
    const int s = live ? bv.list[first + sub] : 0;
    const int n = live ? bv.n[s] : 0;
    const int64_t ov = live ? bv.offv[s] : 0;
    const double* __restrict__ bg = bv.b + ov;
    double* __restrict__ xg = bv.out + ov;
    small_stage<NP, G>(sm.stage, bv.A + (live ? bv.offA[s] : 0), n, lane, gmask);
    const bool act = lane < n;
    const int S = small_stride(n);

    // ---- 1. equilibration -------------------------------------------------
    double rmax = 0.0;
    if (act) {
#pragma unroll
      for (int k = 0; k < NP; ++k)
        if (k < n) rmax = fmax(rmax, fabs(sm.stage[lane * S + k]));
    }
    const double rs = pow2_inv_scale(rmax);
    if (act) rsc[lane] = rs;
    __syncwarp(gmask);
    double cmax = 0.0;
    if (act) {
      for (int r = 0; r < n; ++r) cmax = fmax(cmax, fabs(sm.stage[r * S + lane]) * rsc[r]);
    }
    const double cs_own = pow2_inv_scale(cmax);
    if (act) csc[lane] = cs_own;
    __syncwarp(gmask);
    float af[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k)
      af[k] = (act && k < n) ? float(sm.stage[lane * S + k] * rs * csc[k]) : 0.0f;

    // ---- 2. FP32 LU, rows stay in lanes; pstep = step that chose this row --
    bool done = false, bad = false;
    int pstep = 0x7fff;
    float prinv = 0.0f;
    float umax = 0.0f, umin = 3.0e38f;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      if (j < n && !bad) {
        float key = (act && !done) ? fabsf(af[j]) : -1.0f;
        if (!(key == key)) key = 0.0f;
        int kl = lane;
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) {
          const float ok = __shfl_xor_sync(gmask, key, off, G);
          const int ol = __shfl_xor_sync(gmask, kl, off, G);
          if (ok > key || (ok == key && ol < kl)) { key = ok; kl = ol; }
        }
        if (!(key > 0.0f) || !isfinite(key)) {
          bad = true;
        } else {
          umax = fmaxf(umax, key);
          umin = fminf(umin, key);
          const bool was_done = done;
          if (lane == kl) {
            done = true;
            pstep = j;
#pragma unroll
            for (int k = j; k < NP; ++k) fpiv[k] = af[k];
          }
          __syncwarp(gmask);
          const float rinv = 1.0f / fpiv[j];
          if (lane == kl) prinv = rinv;
          if (act && !was_done && lane != kl) {
            const float l = af[j] * rinv;
            af[j] = l;
#pragma unroll
            for (int k = j + 1; k < NP; ++k) af[k] = fmaf(-l, fpiv[k], af[k]);
          }
          __syncwarp(gmask);
        }
      }
    }
    bool fallback = bad || (double(umin) * mp.cond_limit < double(umax));
    int iters = 0;
    int diagbits = 0;
    if (bad || fallback) diagbits |= kDiagIllCond;

    if (live && !fallback) {
      if (act) lop[pstep] = lane;
      __syncwarp(gmask);
      // correction: returns, in lane j, the component j of C As^-1 R v
      auto correct = [&](double v) -> double {
        const double w = v * rs;
        double wmax = act ? fabs(w) : 0.0;
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) wmax = fmax(wmax, __shfl_xor_sync(gmask, wmax, off, G));
        const double sc = pow2_inv_scale(wmax);
        float t = act ? float(w * sc) : 0.0f;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          if (j < n) {
            const float yj = __shfl_sync(gmask, t, lop[j], G);
            if (act && pstep > j) t = fmaf(-af[j], yj, t);
          }
        }
        double dj = 0.0;
#pragma unroll
        for (int j = NP - 1; j >= 0; --j) {
          if (j < n) {
            const float zl = t * prinv;
            const float zj = __shfl_sync(gmask, zl, lop[j], G);
            if (act && pstep < j) t = fmaf(-af[j], zj, t);
            if (lane == j) dj = double(zj);
          }
        }
        return act ? dj * csc[lane] / sc : 0.0;
      };

      double xj = correct(act ? bg[lane] : 0.0);
      double dprev = 0.0;
      bool conv = false;
      for (int it = 0; it < mp.max_iter; ++it) {
        if (act) sm.xs[lane] = xj;
        __syncwarp(gmask);
        double res = 0.0;
        if (act) {
          res = bg[lane];
#pragma unroll
          for (int k = 0; k < NP; ++k)
            if (k < n) res = fma(-sm.stage[lane * S + k], sm.xs[k], res);
        }
        __syncwarp(gmask);
        const double d = correct(res);
        xj += d;
        iters = it + 1;
        // significance-weighted size of the step
        double ax = act ? fabs(xj) : 0.0, sx = ax, dn = act ? fabs(d) : 0.0;
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) sx += __shfl_xor_sync(gmask, sx, off, G);
        double rel = (act && ax > kFloor * sx) ? dn / ax : 0.0;
        double dmax = dn;
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) {
          rel = fmax(rel, __shfl_xor_sync(gmask, rel, off, G));
          dmax = fmax(dmax, __shfl_xor_sync(gmask, dmax, off, G));
        }
        if (!(rel == rel) || !(dmax == dmax)) break;     // non-finite: let FP64 decide
        if (rel <= mp.tol) { conv = true; break; }
        // contraction slower than cond_limit * u32 allows: the estimate was optimistic
        if (it > 0 && dmax > dprev * mp.cond_limit * 2.384185791015625e-07) break;
        dprev = dmax;
      }
      if (!conv) {
        fallback = true;
        diagbits |= kDiagNoConverge;
      } else {
        if (act) sm.xs[lane] = xj;
        __syncwarp(gmask);
        double worst;
        const int code = small_residual_code<NP, G>(sm, act ? bg[lane] : 0.0, n, lane, gmask, &worst);
        // how close could the reference's own residual test come to 1e-6?
        double risk = 0.0;
        if (act) {
          double sabs = 0.0, y = 0.0;
#pragma unroll
          for (int k = 0; k < NP; ++k)
            if (k < n) {
              sabs = fma(fabs(sm.stage[lane * S + k]), fabs(sm.xs[k]), sabs);
              y = fma(sm.stage[lane * S + k], sm.xs[k], y);
            }
          const double bound = 256.0 * n * 1.1102230246251565e-16 * sabs;
          risk = (bg[lane] > 0.0) ? bound / fabs(y) : bound;
          if (!(risk == risk)) risk = 1.0e300;
        }
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) risk = fmax(risk, __shfl_xor_sync(gmask, risk, off, G));
        if (code != 0 || worst > mp.resid_margin || risk > 0.5 * kResidEps) fallback = true;
      }
    }

    // the exact solve of the warp's systems that need it; the others idle in it
    // (under each group's own mask its reductions run one group after another:
    // 4,096 rate matrices of order 8: 39 us, 30 so; 40,000 of order 16: 374,
    // 330 so)
    int code = kOk;
    if (__any_sync(0xffffffffu, fallback)) {
      __syncwarp();
      code = small_exact_solve<NP, G>(sm, act ? bg[lane] : 0.0, xg, fallback ? n : 0, lane, 0xffffffffu);
      if (fallback) diagbits |= kDiagFallback;
    }
    if (!fallback && act) xg[lane] = sm.xs[lane];
    if (live && lane == 0) {
      bv.status[s] = fallback ? code : kOk;
      if (bv.diag) bv.diag[s] = diagbits | (iters & kDiagIterMask);
    }
    __syncwarp();
  }
}

}  // namespace ss
