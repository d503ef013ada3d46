// Macro-atom epilogue and consumer on the GPU.
//
// After the jumping matrix N = I - Q/Q_norm of every cell is inverted, the
// reference forms B = N^-1 diag(R) (source/macro_accelerate.c:325-334) and, for
// every macro-atom activation, walks one row of B with a running total until it
// reaches a uniform random number z (matom_deactivation_from_matrix,
// macro_accelerate.c:995-1008).  matom_epilogue_kernel forms B in place of the
// inverse and, optionally, the row running totals C[r][c] = sum_{c'<=c} B[r][c'],
// accumulated left to right exactly as that loop accumulates them, so that a
// draw becomes a search of C.  matom_sample_kernel answers a batch of draws.
#pragma once
#include "ss_common.cuh"

namespace ss {

// The systems an epilogue launch serves: all nsys of the batch, or the listed
// ones (list[0 .. count), the count read from count_dev when that is set: a
// list filled on the device by the certified kernel).
struct EpiList {
  const int* list = nullptr;
  int count = 0;
  const int* count_dev = nullptr;
};
__device__ __forceinline__ int epi_count(int nsys, const EpiList& el) {
  if (!el.list) return nsys;
  return el.count_dev ? *el.count_dev : el.count;
}
__device__ __forceinline__ int epi_system(int i, const EpiList& el) { return el.list ? el.list[i] : i; }

// One CTA per system (grid-stride), a warp per 32 rows in 32 x 32 tiles: a tile's
// 32 loads are in flight together, each row of it coalesced; the scaled tile is
// stored as B and passes through shared memory to the lane of its row, which
// adds it to the row's total; the totals leave the same way.  (A thread per row
// straight from global memory, one 8-byte load at a time: 2,550 us for 2,048
// cells of order 200, 470 us now.)  A singular system (status != 0) gets
// B = 0 and C = 0: the reference's output of invert_matrix is a zero-filled
// buffer that the failed call leaves untouched.
__global__ void __launch_bounds__(128) matom_epilogue_kernel(int nsys, const int* __restrict__ n,
                                                             const int64_t* __restrict__ offA,
                                                             const int64_t* __restrict__ offv,
                                                             double* __restrict__ B,
                                                             const double* __restrict__ R,
                                                             double* __restrict__ C,
                                                             const int* __restrict__ status, EpiList el) {
  __shared__ double tiles[4][32 * 33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* tl = tiles[warp];
  const int count = epi_count(nsys, el);
  for (int i = blockIdx.x; i < count; i += gridDim.x) {
    const int s = epi_system(i, el);
    const int ns = n[s];
    const bool ok = status[s] == 0;
    double* __restrict__ Bs = B + offA[s];
    double* __restrict__ Cs = C ? C + offA[s] : nullptr;
    const double* __restrict__ Rs = R + offv[s];
    for (int r0 = 32 * warp; r0 < ns; r0 += 128) {
      double total = 0.0;
      for (int c0 = 0; c0 < ns; c0 += 32) {
        const int c = c0 + lane;
        double* __restrict__ bt = Bs + int64_t(r0) * ns + c;
        const double rc = (c < ns) ? __ldg(Rs + c) : 0.0;
        double v[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = (ok && c < ns && r0 + k < ns) ? bt[int64_t(k) * ns] : 0.0;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          v[k] = ok ? mul_rn(v[k], rc) : 0.0;
          if (c < ns && r0 + k < ns) bt[int64_t(k) * ns] = v[k];
        }
        if (!Cs) continue;
#pragma unroll
        for (int k = 0; k < 32; ++k) tl[k * 33 + lane] = v[k];
        __syncwarp();
        const int cm = min(32, ns - c0);
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = tl[lane * 33 + k];
#pragma unroll
        for (int k = 0; k < 32; ++k)
          if (k < cm) {
            total = add_rn(total, v[k]);
            tl[lane * 33 + k] = total;
          }
        __syncwarp();
        double* __restrict__ ct = Cs + int64_t(r0) * ns + c;
#pragma unroll
        for (int k = 0; k < 32; ++k)
          if (c < ns && r0 + k < ns) ct[int64_t(k) * ns] = tl[k * 33 + lane];
        __syncwarp();
      }
    }
  }
}

// The same for systems whose n x n block fits the dynamic shared memory: the
// block is scaled with coalesced loads and stores, staged in shared memory,
// and each thread runs its row's running total there (the same additions in
// the same order), after which the totals leave with coalesced stores.
__global__ void __launch_bounds__(128) matom_epilogue_tile_kernel(int nsys, const int* __restrict__ n,
                                                                  const int64_t* __restrict__ offA,
                                                                  const int64_t* __restrict__ offv,
                                                                  double* __restrict__ B,
                                                                  const double* __restrict__ R,
                                                                  double* __restrict__ C,
                                                                  const int* __restrict__ status, EpiList el) {
  extern __shared__ double tile[];   // [n][n] of the current system
  const int count = epi_count(nsys, el);
  for (int i = blockIdx.x; i < count; i += gridDim.x) {
    const int s = epi_system(i, el);
    const int ns = n[s];
    const int nn = ns * ns;
    const bool ok = status[s] == 0;
    double* __restrict__ Bs = B + offA[s];
    const double* __restrict__ Rs = R + offv[s];
    for (int e = threadIdx.x; e < nn; e += blockDim.x) {
      const int c = e % ns;
      const double b = ok ? mul_rn(Bs[e], __ldg(Rs + c)) : 0.0;
      Bs[e] = b;
      tile[e] = b;
    }
    if (C) {
      __syncthreads();
      for (int r = threadIdx.x; r < ns; r += blockDim.x) {
        double total = 0.0;
        for (int c = 0; c < ns; ++c) {
          total = add_rn(total, tile[r * ns + c]);
          tile[r * ns + c] = total;
        }
      }
      __syncthreads();
      double* __restrict__ Cs = C + offA[s];
      for (int e = threadIdx.x; e < nn; e += blockDim.x) Cs[e] = tile[e];
    }
    __syncthreads();
  }
}

// Query i draws from row level[i] of system sys[i] with the number z[i]: the
// reference returns 0 when z <= 0 and otherwise the first column whose running
// total is not below z.  target[i] = -1 when the row total stays below z (the
// reference's loop would run past the row), -2 for a system or level out of range.
//
// A draw reads half a row on average, from a row no other draw near it shares:
// what bounds it is the number of loads in flight, then the bytes fetched
// beyond the answer.  A warp serves up to 32 draws, kDrawSlots of them at a time: a
// round reads the next 32 totals of every slot's row, a vote finds the first
// that is not below z, and a slot that is done takes the next draw, so that as
// many loads are in flight at the end of the walks as at their start.
// (A thread per draw walking its row: 373 us for 2^20 draws on 4,096 cells of
// orders 20-200, 1.3 TB/s; the kernel alone now 125 us, about 5 TB/s of lines.
// Four draws to a warp, each to its end, took 282 us: most loads were then those
// of the longest walk.)
constexpr int kDrawThreads = 256, kDrawSlots = 4, kDrawBlocksPerSM = 7;
// Rows that one round covers cost the warp a whole round each; where many of a
// warp's draws have such rows, each is walked by the lane of its draw instead, all
// of them together (4 million draws from rows of 4: 228 us by rounds, 64 walked; of
// 10: 220, 87; of 30: 220, 181; of 32: 222, 270).  With few of them the walk, one load
// at a time, would hold up the warp's other draws (orders 20-200: 125 us against 122).
constexpr int kDrawShort = 31, kDrawShortLanes = 8;

// Draws per warp: 32, or fewer where that would leave warps of the GPU without
// any, but one for every slot.
inline int draws_per_warp(int nq, int sms) {
  const int64_t warps = int64_t(sms) * kDrawBlocksPerSM * (kDrawThreads / 32);
  const int64_t per = (int64_t(nq) + warps - 1) / warps;
  return int(per < kDrawSlots ? kDrawSlots : per > 32 ? 32 : per);
}

__global__ void __launch_bounds__(kDrawThreads, kDrawBlocksPerSM)
matom_sample_kernel(int nq, int per, int nsys, const int* __restrict__ n, const int64_t* __restrict__ offA,
                    const double* __restrict__ C, const int* __restrict__ sys, const int* __restrict__ level,
                    const double* __restrict__ z, int* __restrict__ target) {
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t(blockIdx.x) * (kDrawThreads / 32) + threadIdx.x / 32) * per + lane;
  const bool mine = lane < per && i < nq;
  // this lane's draw
  int64_t off = 0;
  double zl = 0.0;
  int nl = 0, ans = -2;
  if (mine) {
    const int s = sys[i], u = level[i];
    if (s >= 0 && s < nsys) {
      const int ns = n[s];
      if (u >= 0 && u < ns) {
        zl = z[i];
        off = offA[s] + int64_t(u) * ns;
        ans = (0.0 < zl) ? -1 : 0;
        nl = (0.0 < zl) ? ns : 0;
      }
    }
  }
  // rows shorter than a round are walked by their draws' own lanes, together
  const unsigned brief = __ballot_sync(0xffffffffu, nl > 0 && nl <= kDrawShort);
  if (__popc(brief) >= kDrawShortLanes && (brief >> lane & 1u)) {
    for (int c = 0; c < nl; ++c)
      if (!(__ldg(C + off + c) < zl)) {
        ans = c;
        break;
      }
    nl = 0;
  }
  unsigned todo = __ballot_sync(0xffffffffu, nl > 0);
  const double* row[kDrawSlots];   // the next totals of each slot's draw
  double zz[kDrawSlots];
  int left[kDrawSlots], at[kDrawSlots], id[kDrawSlots];   // totals not read yet, columns read, the draw's lane
  auto take = [&](int d) {
    left[d] = 0;
    if (todo == 0u) return;
    id[d] = __ffs(todo) - 1;
    todo &= todo - 1u;
    row[d] = C + __shfl_sync(0xffffffffu, off, id[d]) + lane;
    zz[d] = __shfl_sync(0xffffffffu, zl, id[d]);
    left[d] = __shfl_sync(0xffffffffu, nl, id[d]);
    at[d] = 0;
  };
#pragma unroll
  for (int d = 0; d < kDrawSlots; ++d) {
    row[d] = C;
    zz[d] = 0.0;
    at[d] = id[d] = 0;
    take(d);
  }
  // every branch below is the same for the whole warp
  for (;;) {
    double v[kDrawSlots];
    int open = 0;
#pragma unroll
    for (int d = 0; d < kDrawSlots; ++d) {
      v[d] = (lane < left[d]) ? __ldg(row[d]) : 0.0;
      open |= left[d];
    }
    if (open == 0) break;
#pragma unroll
    for (int d = 0; d < kDrawSlots; ++d) {
      const unsigned hit = __ballot_sync(0xffffffffu, lane < left[d] && !(v[d] < zz[d]));
      if (hit != 0u && lane == id[d]) ans = at[d] + __ffs(hit) - 1;
      row[d] += 32;
      at[d] += 32;
      left[d] = hit != 0u ? 0 : max(0, left[d] - 32);
      if (left[d] == 0) take(d);
    }
  }
  if (mine) target[i] = ans;
}

}  // namespace ss
