// The whole n_e iteration of a cell on the GPU (matrix_ion_populations,
// source/matrix_ion.c:219-382), rate matrices assembled where they are solved.
//
// A cell's rounds depend on nothing but that cell, so a CTA takes a cell from a
// queue and runs all of its rounds: each round its warps assemble their
// elements' systems in shared memory (ion_column) and solve them
// (small_exact_solve, a warp per system), then warp 0 floors the populations,
// sums n_e in ion order and decides.  Nothing but the converged n_e and
// populations leaves the SM, and the host takes part only before and after.
// What bounds it is the chain of the largest element's solve, once per round,
// times the rounds of the cell that takes the most.  4,096 cells of five elements
// took 21.5 ms a call with rounds driven by the host (a layout, a plan, five
// launches and four copies each); now 4.9 ms, of which 3 are the 200 rounds of a
// cell that never converges (15 us each) and about 1.5 the copies in and out.
#pragma once
#include "kernels_ionasm.cuh"
#include "kernels_small.cuh"

namespace ss {

struct IonLockView {
  int ncell, h_elem, max_rounds;
  const int* elem_of;      // [nions] element of each ion
  const int* warp_start;   // [warps + 1] each warp's elements, indices into warp_elem
  const int* warp_elem;    // [nelem]
  const double* dens;      // [ncell][nelem] element densities
  double* ne;              // [ncell] in: starting n_e; out: converged
  double* den;             // [ncell][nions] in: starting fractions; out: converged
  int* status;             // [ncell]
  int* iters;              // [ncell]
  int* queue;              // next cell, zeroed before the launch
};

constexpr int kIonLockWarps = 4;         // most warps of one cell
constexpr int kIonLockMaxIons = 4096;    // a cell's populations and terms stay within 64 KB of shared memory
constexpr double kLockDensityMin = 1.0e-20;   // DENSITY_MIN, atomic.h:9
constexpr double kLockFracError = 0.03;       // python.h:1212

// dynamic shared memory: a solve's scratch per warp, then the cell's new
// populations and their terms of n_e
template <int NPM>
constexpr size_t ion_lock_smem(int warps, int nions) {
  return sizeof(SmallSmem<NPM>) * size_t(warps) + sizeof(double) * 2 * size_t(nions);
}

// NPM: padded order that holds every element (<= 32).  Every element goes
// through the same unrolled steps, small ones through the first few of them:
// with a size class each, the warps' code no longer fits the instruction cache
// together and a pivot step at n = 27 takes 740 cycles instead of 430.
template <int NPM>
__global__ void __launch_bounds__(32 * kIonLockWarps, NPM > 28 ? 3 : 4) ion_lockstep_kernel(IonAsmView v, IonLockView lv) {
  extern __shared__ __align__(16) unsigned char lock_dsm[];
  __shared__ int s_cell, s_sing, s_state;    // s_state: 0 another round, 1 converged, 2 singular
  __shared__ double s_ne, s_h1, s_h2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  SmallSmem<NPM>& sm = reinterpret_cast<SmallSmem<NPM>*>(lock_dsm)[warp];
  double* nd = reinterpret_cast<double*>(lock_dsm + sizeof(SmallSmem<NPM>) * size_t(nw));   // [nions]
  double* term = nd + v.nions;                                                              // [nions]

  // neutral and ionised hydrogen densities for charge exchange (matrix_ion.c:228-238)
  auto hydrogen = [&](const double* frac, int cell) {
    double h1 = 0.0, h2 = 0.0;
    if (lv.h_elem >= 0) {
      const double dh = lv.dens[int64_t(cell) * v.nelem + lv.h_elem];
      const int f = v.elem_first[lv.h_elem];
      for (int k = 0; k < v.elem_n[lv.h_elem]; ++k) {
        if (v.ion_istate[f + k] == 1) h1 = mul_rn(frac[f + k], dh);
        if (v.ion_istate[f + k] == 2) h2 = mul_rn(frac[f + k], dh);
      }
    }
    s_h1 = h1;
    s_h2 = h2;
  };

  for (;;) {
    if (threadIdx.x == 0) {
      s_cell = atomicAdd(lv.queue, 1);
      if (s_cell < lv.ncell) {
        s_ne = lv.ne[s_cell];
        s_sing = 0;
        hydrogen(lv.den + int64_t(s_cell) * v.nions, s_cell);
      }
    }
    __syncthreads();
    const int cell = s_cell;
    if (cell >= lv.ncell) break;
    int state = 0, round = 0;
    while (state == 0 && round < lv.max_rounds) {
      ++round;
      const double xne = s_ne, nh1 = s_h1, nh2 = s_h2;
      for (int q = lv.warp_start[warp]; q < lv.warp_start[warp + 1]; ++q) {
        const int e = lv.warp_elem[q], n = v.elem_n[e], f = v.elem_first[e];
        if (lane < n) ion_column(v, cell, f, n, lane, xne, nh1, nh2, sm.stage, small_stride(n));
        __syncwarp();
        // the iteration looks at nothing but code 4: no residual check
        const int code =
            small_exact_solve<NPM, 32, false>(sm, lane == 0 ? 1.0 : 0.0, nd + f, n, lane, 0xffffffffu);
        if (code == kSolveSingular && lane == 0) s_sing = 1;
        __syncwarp();
      }
      __syncthreads();
      if (warp == 0) {
        if (s_sing) {   // matrix_ion.c:295-299: the cell keeps its old populations
          if (lane == 0) s_state = 2;
        } else {
          for (int i = lane; i < v.nions; i += 32) {
            const double x = nd[i] < kLockDensityMin ? kLockDensityMin : nd[i];
            nd[i] = x;
            term[i] = mul_rn(mul_rn(x, double(v.ion_istate[i] - 1)), lv.dens[int64_t(cell) * v.nelem + lv.elem_of[i]]);
          }
          __syncwarp();
          if (lane == 0) {
            double xnew = 0.0;
#pragma unroll 4
            for (int i = 0; i < v.nions; ++i) xnew = add_rn(xnew, term[i]);
            if (xnew < kLockDensityMin) xnew = kLockDensityMin;
            if (fabs(div_rn(sub_rn(xne, xnew), xnew)) < kLockFracError || xnew < 1.e-6) {
              s_state = 1;
              s_ne = xnew;
            } else {
              s_state = 0;
              s_ne = mul_rn(add_rn(xnew, xne), 0.5);
              hydrogen(nd, cell);
            }
          }
        }
      }
      __syncthreads();
      state = s_state;
    }
    // no convergence within the rounds: status -2, inputs kept (matrix_ion.c:366-382)
    if (state == 1)
      for (int i = threadIdx.x; i < v.nions; i += blockDim.x) lv.den[int64_t(cell) * v.nions + i] = nd[i];
    if (threadIdx.x == 0) {
      if (state == 1) lv.ne[cell] = s_ne;
      lv.status[cell] = state == 1 ? 0 : state == 2 ? -1 : -2;
      lv.iters[cell] = round;
    }
    __syncthreads();
  }
}

}  // namespace ss
