// Quotients by a reciprocal beside the division's own, for tests, and the
// FP32 FMA throughput probe: the roofline denominator of the Debye pair
// kernel (FP32-pipe bound).  Eight independent register-resident FFMA chains
// per thread on every SM; FLOP counted as 2 per FMA.
#include <cuda_runtime.h>

#include <algorithm>

#include "device_math.cuh"
#include "engine.hpp"

namespace crab {
namespace {
__global__ void k_quotients(const double* __restrict__ a, const double* __restrict__ b, int64_t n,
                            double* __restrict__ by, double* __restrict__ div) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  by[i] = dev::div_by(a[i], b[i], 1.0 / b[i]);
  div[i] = a[i] / b[i];
}

constexpr int kIter = 4096;
__global__ void k_ffma_peak(float* out, float m, float c, int outer) {
  float a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = threadIdx.x * 1e-3f + k;
  for (int o = 0; o < outer; ++o)
    for (int it = 0; it < kIter; ++it) {
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] = fmaf(a[k], m, c);
    }
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += a[k];
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}
}  // namespace

double measure_fp32_peak(crab_ctx* ctx, double target_ms) {
  const int threads = 256, blocks = ctx->sm_count * 8;
  float* out = (float*)ctx->dev("probe.out", (size_t)threads * blocks * sizeof(float));
  cudaStream_t s = ctx->stream;
  // warm up and calibrate the loop count to roughly target_ms
  k_ffma_peak<<<blocks, threads, 0, s>>>(out, 0.9999f, 1e-4f, 1);
  CRAB_CUDA_CHECK(cudaGetLastError());
  CRAB_CUDA_CHECK(cudaEventRecord(ctx->ev_start, s));
  k_ffma_peak<<<blocks, threads, 0, s>>>(out, 0.9999f, 1e-4f, 1);
  CRAB_CUDA_CHECK(cudaEventRecord(ctx->ev_stop, s));
  CRAB_CUDA_CHECK(cudaEventSynchronize(ctx->ev_stop));
  float ms1 = 0.0f;
  CRAB_CUDA_CHECK(cudaEventElapsedTime(&ms1, ctx->ev_start, ctx->ev_stop));
  const int outer = std::max(1, std::min(1000, (int)(target_ms / std::max(ms1, 1e-3f))));
  double best = 0.0;
  for (int rep = 0; rep < 3; ++rep) {
    CRAB_CUDA_CHECK(cudaEventRecord(ctx->ev_start, s));
    k_ffma_peak<<<blocks, threads, 0, s>>>(out, 0.9999f, 1e-4f, outer);
    CRAB_CUDA_CHECK(cudaEventRecord(ctx->ev_stop, s));
    CRAB_CUDA_CHECK(cudaEventSynchronize(ctx->ev_stop));
    float ms = 0.0f;
    CRAB_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
    const double flop = 2.0 * 8.0 * kIter * (double)outer * threads * (double)blocks;
    best = std::max(best, flop / (ms * 1e-3) / 1e12);
  }
  ctx->launches += 5;
  return best;
}

// by[i] = dev::div_by(a[i], b[i], 1 / b[i]), div[i] = a[i] / b[i].
void probe_quotients(crab_ctx* ctx, const double* a, const double* b, int64_t n, double* by, double* div) {
  if (n == 0) return;
  const size_t bytes = (size_t)n * sizeof(double);
  auto* d = (double*)ctx->dev("probe.quotients", 4 * bytes);
  cudaStream_t s = ctx->stream;
  copy_h2d(ctx, d, a, bytes, s);
  copy_h2d(ctx, d + n, b, bytes, s);
  k_quotients<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d, d + n, n, d + 2 * n, d + 3 * n);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 1;
  copy_d2h(ctx, by, d + 2 * n, bytes, s);
  copy_d2h(ctx, div, d + 3 * n, bytes, s);
  CRAB_CUDA_CHECK(cudaStreamSynchronize(s));
}

}  // namespace crab
