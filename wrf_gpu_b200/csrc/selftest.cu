// Device self-checks of numerical helpers, built as a separate test library
// (libwrfgpu_selftest.so) so the product library exports only its C ABI.
#include <cuda_runtime.h>

#include "dycore_common.cuh"

namespace {

__global__ void k_div_check(const double *a, const double *b, const double *rb, double *q_rcp, double *q_div,
                            long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q_rcp[i] = wg::div_rcp(a[i], b[i], rb[i]);
  q_div[i] = a[i] / b[i];
}

// Groups of three neighbouring quotients as one div_batch.
__global__ void k_div_batch_check(const double *a, const double *b, double *q_batch, double *q_div, long groups) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= groups) return;
  const double n[3] = {a[3 * i], a[3 * i + 1], a[3 * i + 2]}, d[3] = {b[3 * i], b[3 * i + 1], b[3 * i + 2]};
  double q[3];
  wg::div_batch(n, d, q);
  for (int t = 0; t < 3; ++t) {
    q_batch[3 * i + t] = q[t];
    q_div[3 * i + t] = n[t] / d[t];
  }
}

// Largest |1 - b y0| of the reciprocal's seed y0 over the divisors whose high
// word is 1.0's plus i (the instruction reads the high word only, so the ends of the low
// word are the extremes).
__global__ void k_rcp_seed(double *e0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 1 << 20) return;
  double worst = 0.0;
  for (int lo : {0, -1}) {
    const double b = __hiloint2double(0x3ff00000 + i, lo);
    double y0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
    worst = fmax(worst, fabs(__fma_rn(-b, y0, 1.0)));
  }
  e0[i] = worst;
}

}  // namespace

// q_rcp[i] = div_rcp(a[i], b[i], rb[i]) and q_div[i] = a[i] / b[i] (CUDA's
// IEEE division) on device arrays of n doubles.
extern "C" int wrfgpu_selftest_div_rcp(const double *a, const double *b, const double *rb, double *q_rcp,
                                       double *q_div, long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  const int threads = 256;
  const long blocks = (n + threads - 1) / threads;
  k_div_check<<<(unsigned)blocks, threads, 0, stream>>>(a, b, rb, q_rcp, q_div, n);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

// q_batch = div_batch over groups of three and q_div = a / b, on device arrays
// of 3 * groups doubles.
extern "C" int wrfgpu_selftest_div_batch(const double *a, const double *b, double *q_batch, double *q_div,
                                         long groups, cudaStream_t stream) {
  if (groups <= 0) return 0;
  const int threads = 256;
  k_div_batch_check<<<(unsigned)((groups + threads - 1) / threads), threads, 0, stream>>>(a, b, q_batch, q_div, groups);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

// e0 (2^20 doubles) = the seed's error over every high word of [1, 2).
extern "C" int wrfgpu_selftest_rcp_seed(double *e0, cudaStream_t stream) {
  k_rcp_seed<<<(1 << 20) / 256, 256, 0, stream>>>(e0);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}
