// Measured FMA throughput of the CUDA cores (FP32 and FP64 pipes) and of the
// FP64 tensor pipe.
//
// The roofline fractions of the per-centre kernels (expansion, power
// spectrum, pair adjoint) and of the FP64 tile GEMM need the pipe peaks of the
// GPU they run on, under its own clocks and power cap, not datasheet figures.
// This microbenchmark fills every SM with independent FMA chains (eight per
// thread, or per warp eight of the tile GEMM's tensor instructions on register
// operands, enough to cover the pipe latency at full occupancy) and times the
// launch with CUDA events on a private stream; one FMA counts as 2 flops.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "dgemm.cuh"

namespace rgpu {
namespace {

template <typename T>
__global__ void __launch_bounds__(256) fma_chains_kernel(T * __restrict__ out, int iters, T a, T b) {
  T x0 = T(threadIdx.x) * T(1e-3), x1 = x0 + T(1), x2 = x0 + T(2), x3 = x0 + T(3);
  T x4 = x0 + T(4), x5 = x0 + T(5), x6 = x0 + T(6), x7 = x0 + T(7);
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      x0 = fma(x0, a, b);
      x1 = fma(x1, a, b);
      x2 = fma(x2, a, b);
      x3 = fma(x3, a, b);
      x4 = fma(x4, a, b);
      x5 = fma(x5, a, b);
      x6 = fma(x6, a, b);
      x7 = fma(x7, a, b);
    }
  }
  const T s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  // a data-dependent store the compiler cannot drop (a = 1, b = 0 in use,
  // so s stays finite and this branch is never taken)
  if (s == T(-1.2345e30)) out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// Eight chains of m16n8k8 f64 products per warp: 2 x 16 x 8 x 8 flops each.
__global__ void __launch_bounds__(256) dmma_chains_kernel(double * __restrict__ out, int iters, double a, double b) {
  const double av[4] = {a, a, a, a}, bv[2] = {b, b};
  double c[8][4];
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) c[k][e] = double(threadIdx.x + 4 * k + e);
  for (int i = 0; i < iters; ++i)
#pragma unroll
    for (int k = 0; k < 8; ++k) dmma(c[k], av, bv);
  double s = 0.;
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int e = 0; e < 4; ++e) s += c[k][e];
  if (s == -1.2345e30) out[blockIdx.x * blockDim.x + threadIdx.x] = s;  // never taken (a = 1, b = 0 in use)
}

// Best rate (TFLOP/s) of five launches of `kernel` after one to warm up.
template <typename T>
double time_chains(void (*kernel)(T *, int, T, T), int iters, double flops_per_thread) {
  int dev = current_device(), sms = 0, per_sm = 0;
  RGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  RGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0));
  const int blocks = sms * std::max(per_sm, 1);
  cudaStream_t st = nullptr;
  RGPU_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  DevBuf out;
  double best = 0.;
  try {
    RGPU_CUDA(cudaEventCreate(&e0));
    RGPU_CUDA(cudaEventCreate(&e1));
    out.ensure(sizeof(T) * size_t(blocks) * 256);
    const double flops = flops_per_thread * double(iters) * double(blocks) * 256.0;
    for (int rep = 0; rep < 6; ++rep) {  // the first launch warms up
      RGPU_CUDA(cudaEventRecord(e0, st));
      kernel<<<blocks, 256, 0, st>>>(out.as<T>(), iters, T(1), T(0));
      RGPU_LAUNCHED();
      RGPU_CUDA(cudaGetLastError());
      RGPU_CUDA(cudaEventRecord(e1, st));
      RGPU_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      RGPU_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (rep > 0 && ms > 0.f) best = std::max(best, flops / (double(ms) * 1e-3) / 1e12);
    }
  } catch (...) {
    cudaStreamSynchronize(st);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaStreamDestroy(st);
    throw;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(st);
  return best;
}

}  // namespace

double measure_fma_peak(int precision) {
  return precision == RGPU_PRECISION_FP64 ? time_chains<double>(fma_chains_kernel<double>, 4096, 2.0 * 64.0)
                                          : time_chains<float>(fma_chains_kernel<float>, 8192, 2.0 * 64.0);
}

double measure_fp64_tensor_peak() {
  return time_chains<double>(dmma_chains_kernel, 4096, 8 * 2.0 * 16 * 8 * 8 / 32);
}

}  // namespace rgpu
