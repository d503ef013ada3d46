// Reciprocals and quotients of ss_common.cuh one value at a time, for the test
// that compares them with correctly rounded division (tests/test_gpu_rounding.py).
#include "ss_common.cuh"

namespace {

// q[i] = u[i] / d[i] as a solve forms it: the pivot's reciprocal where
// rcp_covers, else 0; far[i] as div_markstein reports it
__global__ void rounding_kernel(int count, const double* __restrict__ u, const double* __restrict__ d,
                                double* __restrict__ rcp, int* __restrict__ covers, double* __restrict__ q,
                                unsigned* __restrict__ far) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const double r = ss::rcp_markstein(d[i]);
  const bool c = ss::rcp_covers(d[i]);
  unsigned f = 0u;
  rcp[i] = r;
  covers[i] = c;
  q[i] = ss::div_markstein(u[i], d[i], c ? r : 0.0, f);
  far[i] = f;
}

}  // namespace

extern "C" {

unsigned sirocco_check_div_far(void) { return ss::kDivFar; }

// device pointers, `count` elements each; 0 or a CUDA error code
int sirocco_check_rounding(int count, const double* u, const double* d, double* rcp, int* covers, double* q,
                           unsigned* far) {
  if (count < 1) return 0;
  rounding_kernel<<<(count + 255) / 256, 256>>>(count, u, d, rcp, covers, q, far);
  const cudaError_t e = cudaGetLastError();
  return int(e ? e : cudaDeviceSynchronize());
}

}  // extern "C"
