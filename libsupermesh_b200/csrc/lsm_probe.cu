// Measurement probe (not part of the supermesh API): the FP64 arithmetic
// ceiling that the clipping kernels run against.  The clipper is compiled
// without FMA contraction, so its ceiling is the issue rate of separate
// DADD/DMUL instructions; the probe measures that rate (and, for context,
// the DFMA rate) with long chains of independent operations.  And the
// clippers' quotients and normals on given operands, for comparison with
// divisions (built, like the library, without FMA contraction).
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>

#include "lsm_geom.cuh"

namespace {

constexpr int kChains = 8;
constexpr int kIters = 4096;

__global__ void __launch_bounds__(256) k_dadd_dmul(double seed, double* sink) {
  double x[kChains];
#pragma unroll
  for (int i = 0; i < kChains; ++i) x[i] = seed + i + threadIdx.x * 1e-9;
  const double m = 1.0000000001, a = 1e-12;
  for (int it = 0; it < kIters; ++it) {
#pragma unroll
    for (int i = 0; i < kChains; ++i) {
      x[i] = __dmul_rn(x[i], m);
      x[i] = __dadd_rn(x[i], a);
    }
  }
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < kChains; ++i) s += x[i];
  if (s == 12345.678) sink[0] = s;
}

__global__ void __launch_bounds__(256) k_dfma(double seed, double* sink) {
  double x[kChains];
#pragma unroll
  for (int i = 0; i < kChains; ++i) x[i] = seed + i + threadIdx.x * 1e-9;
  const double m = 1.0000000001, a = 1e-12;
  for (int it = 0; it < kIters; ++it) {
#pragma unroll
    for (int i = 0; i < kChains; ++i) x[i] = __fma_rn(x[i], m, a);
  }
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < kChains; ++i) s += x[i];
  if (s == 12345.678) sink[0] = s;
}

__global__ void __launch_bounds__(256) k_quotients(int64_t n, const double* __restrict__ a,
                                                   const double* __restrict__ b, double* divided, double* by, int* ok) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned range = lsm::div_range(lsm::div_range(0, a[i]), b[i]);
  divided[i] = a[i] / b[i];
  by[i] = lsm::div_by(a[i], b[i], __drcp_rn(b[i]));
  ok[i] = lsm::div_ok(range);
}

__global__ void __launch_bounds__(256) k_normals(int64_t n, const double* __restrict__ uv, double* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* v = uv + 6 * i;
  double* o = out + 4 * i;
  lsm::unit_cross(v[0], v[1], v[2], v[3], v[4], v[5], o[0], o[1], o[2]);
  o[3] = lsm::norm2_3(v[0], v[1], v[2]);
}

}  // namespace

extern "C" {

// a[n] / b[n] by division and by the reciprocal of b (div_by), and whether
// the range check lets the second stand for the first; device arrays.
int lsm_probe_quotients(int64_t n, const double* a, const double* b, double* divided, double* by, int* ok) {
  if (n > 0) k_quotients<<<(unsigned)((n + 255) / 256), 256>>>(n, a, b, divided, by, ok);
  return (int)cudaDeviceSynchronize();
}

// uv[n][6] -> out[n][4]: the unit normal of u x v and the length of u.
int lsm_probe_normals(int64_t n, const double* uv, double* out) {
  if (n > 0) k_normals<<<(unsigned)((n + 255) / 256), 256>>>(n, uv, out);
  return (int)cudaDeviceSynchronize();
}

// Returns FP64 operations per second: mode 0 = separate DADD+DMUL (1 op
// each), mode 1 = DFMA (2 ops each).  Timed with CUDA events, best of
// `reps` launches of blocks_per_sm * SMs blocks of 256 threads.
double lsm_probe_fp64_rate(int mode, int reps) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  double* sink = nullptr;
  if (cudaMalloc(&sink, sizeof(double)) != cudaSuccess) return -1.0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int blocks = sms * 8;
  const double ops_per_thread = (double)kIters * kChains * 2.0;
  double best = 0.0;
  for (int r = 0; r < reps + 1; ++r) {
    cudaEventRecord(e0);
    if (mode == 0)
      k_dadd_dmul<<<blocks, 256>>>(1.0, sink);
    else
      k_dfma<<<blocks, 256>>>(1.0, sink);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (r == 0 || ms <= 0.f) continue;  // first launch warms up
    const double rate = ops_per_thread * blocks * 256.0 / (ms * 1e-3);
    if (rate > best) best = rate;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(sink);
  return cudaGetLastError() == cudaSuccess ? best : -1.0;
}

// Writes `bytes` of zeros to evict the L2 cache between timed steps.
int lsm_probe_flush_l2(void* buf, int64_t bytes, void* stream) {
  return (int)cudaMemsetAsync(buf, 0, (size_t)bytes, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
