// Exact site–site Debye sums for hydration sites on a voxel lattice.
//
// Hydration sites (crabSAXS src/solvent.rs:208-218, 387-396) are voxel
// centres min + (ix, iy, iz)·spacing, so every site pair is at distance
// spacing·√n with n = Δix² + Δiy² + Δiz² an integer.  The reference sums
// sinc(q r) over all site pairs (solvent.rs:563-570).  Here the pairs are
// counted per n in integer arithmetic (a histogram over all M(M-1)/2 pairs,
// shared-memory atomics), and the sum becomes Σ_n count[n]·sinc(q·spacing·√n)
// evaluated in f64 for the few thousand distinct n.  The result is exact up
// to f64 rounding (the reference's own r differs from spacing·√n by ~1e-15
// relative), and it avoids the coherent FP32 errors a lattice would
// otherwise accumulate: thousands of pairs share each distance.

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>

#include "engine.hpp"

namespace crab {
namespace {

constexpr int kLT = 128;           // sites per tile
constexpr int kSharedBins = 11264; // 44 KB of u32 counters (+2 KB tile: under the 48 KB static limit)

// Counts per squared distance of the tile pairs blockIdx.x, + gridDim.x, ...
// of the upper triangle, two threads per i site (each half of the j tile).  A
// CTA keeps its counters over its tile pairs: one tile pair a CTA spent more
// time clearing and adding up 11,000 counters than on its 16,384 pairs (9,369
// sites: 63 us, 44 so).  At most kLFlush tile pairs between two flushes, so a
// counter stays below 2^30.
constexpr int kLThreads = 2 * kLT;
constexpr int64_t kLFlush = 1 << 16;
__global__ void __launch_bounds__(kLThreads)
    k_lattice_hist(const int4* __restrict__ cells, int64_t m, int64_t n_tiles, int bins,
                   unsigned long long* __restrict__ hist) {
  __shared__ int4 sj[kLT];
  __shared__ unsigned int sh[kSharedBins];
  for (int b = threadIdx.x; b < bins; b += kLThreads) sh[b] = 0u;
  auto flush = [&]() {
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += kLThreads)
      if (sh[b]) {
        atomicAdd(&hist[b], (unsigned long long)sh[b]);
        sh[b] = 0u;
      }
  };
  const int li = threadIdx.x & (kLT - 1), j0 = (threadIdx.x / kLT) * (kLT / 2);
  int64_t since = 0;
  const int64_t n_work = n_tiles * (n_tiles + 1) / 2;
  for (int64_t w = blockIdx.x; w < n_work; w += gridDim.x) {
    // w = tj (tj + 1) / 2 + ti with ti <= tj
    int64_t tj = (int64_t)((sqrt(8.0 * (double)w + 1.0) - 1.0) * 0.5);
    while (tj * (tj + 1) / 2 > w) --tj;
    while ((tj + 1) * (tj + 2) / 2 <= w) ++tj;
    const int64_t ti = w - tj * (tj + 1) / 2;
    if (++since == kLFlush) {
      flush();
      since = 0;
    }
    __syncthreads();
    if (threadIdx.x < kLT) {
      const int64_t j = tj * kLT + threadIdx.x;
      sj[threadIdx.x] = j < m ? cells[j] : make_int4(0, 0, 0, -1);
    }
    __syncthreads();
    const int64_t i = ti * kLT + li;
    if (i >= m) continue;
    const int4 ci = cells[i];
#pragma unroll 4
    for (int j = j0; j < j0 + kLT / 2; ++j) {
      const int4 cj = sj[j];
      if (cj.w < 0 || (ti == tj && j <= li)) continue;  // past the last site, or the pair's other order
      const int dx = ci.x - cj.x, dy = ci.y - cj.y, dz = ci.z - cj.z;
      atomicAdd(&sh[dx * dx + dy * dy + dz * dz], 1u);
    }
  }
  flush();
}

// The same for spans past the shared counters: every pair into device memory,
// a CTA per tile pair (tj, ti) and a thread per i site.  Bound by the L2's
// atomics, which runs of tile pairs on 256 threads as above drive into each
// other (47,663 sites with spans past the line, a call: 24.8 ms, 16.7 so).
__global__ void __launch_bounds__(kLT)
    k_lattice_hist_wide(const int4* __restrict__ cells, int64_t m, unsigned long long* __restrict__ hist) {
  __shared__ int4 sj[kLT];
  const int64_t ti = blockIdx.y, tj = blockIdx.x;
  if (tj < ti) return;  // upper triangle of tile pairs only
  const int64_t j = tj * kLT + threadIdx.x, i = ti * kLT + threadIdx.x;
  sj[threadIdx.x] = j < m ? cells[j] : make_int4(0, 0, 0, -1);
  __syncthreads();
  if (i >= m) return;
  const int4 ci = cells[i];
  for (int k = 0; k < kLT; ++k) {
    const int4 cj = sj[k];
    if (cj.w < 0) break;  // past the last site
    if (ti == tj && k <= (int)threadIdx.x) continue;
    const int dx = ci.x - cj.x, dy = ci.y - cj.y, dz = ci.z - cj.z;
    atomicAdd(&hist[dx * dx + dy * dy + dz * dz], 1ull);
  }
}

// out[d], out[3 + d]: least and largest cell along d (set to INT_MAX and INT_MIN before).
__global__ void __launch_bounds__(256)
    k_lattice_span(const int32_t* __restrict__ cells, int64_t m, int* __restrict__ out) {
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int c = cells[3 * i + d];
      lo[d] = min(lo[d], c);
      hi[d] = max(hi[d], c);
    }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int l = __reduce_min_sync(0xffffffffu, lo[d]), h = __reduce_max_sync(0xffffffffu, hi[d]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(out + d, l);
      atomicMax(out + 3 + d, h);
    }
  }
}

// out[k] = Σ_n count[n] sinc(q_k spacing √n) with the reference sinc
// (|x| < 1e-8 -> 1), one CTA per q.
__global__ void k_lattice_transform(const unsigned long long* __restrict__ hist, int bins, double spacing,
                                    const double* __restrict__ q, double* __restrict__ out) {
  __shared__ double red[32];
  const double qq = q[blockIdx.x];
  double acc = 0.0;
  for (int n = threadIdx.x; n < bins; n += blockDim.x) {
    const unsigned long long c = hist[n];
    if (!c) continue;
    const double x = qq * (spacing * sqrt((double)n));
    acc += (double)c * (fabs(x) < 1e-8 ? 1.0 : sin(x) / x);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < blockDim.x / 32 ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) out[blockIdx.x] = v;
  }
}

}  // namespace

void lattice_plan_init(crab_ctx* ctx, PairPlan& P, const int32_t* cells, int64_t m, double spacing) {
  LatticePart& Lp = P.lattice;
  Lp.m = m;
  Lp.spacing = spacing;
  if (m < 2) {
    Lp.bins = 1;
  } else {
    int lo[3] = {cells[0], cells[1], cells[2]}, hi[3] = {cells[0], cells[1], cells[2]};
    for (int64_t i = 1; i < m; ++i)
      for (int d = 0; d < 3; ++d) {
        lo[d] = std::min(lo[d], cells[3 * i + d]);
        hi[d] = std::max(hi[d], cells[3 * i + d]);
      }
    int64_t nmax = 0;
    for (int d = 0; d < 3; ++d) nmax += (int64_t)(hi[d] - lo[d]) * (hi[d] - lo[d]);
    require(nmax < (int64_t)1 << 30, "hydration lattice too large for the site histogram");
    require((m + kLT - 1) / kLT <= 65535, "too many lattice sites for one histogram launch");
    Lp.bins = (int)nmax + 1;
  }
  std::vector<int4> c4(std::max<int64_t>(m, 1));
  for (int64_t i = 0; i < m; ++i) c4[i] = make_int4(cells[3 * i], cells[3 * i + 1], cells[3 * i + 2], 0);
  Lp.d_cells = (int4*)plan_alloc(ctx, P, P.owned, "lattice_cells", c4.size() * sizeof(int4));
  copy_h2d(ctx, Lp.d_cells, c4.data(), (size_t)m * sizeof(int4), ctx->stream);
  Lp.d_hist = (unsigned long long*)plan_alloc(ctx, P, P.owned, "lattice_hist",
                                               (size_t)Lp.bins * sizeof(unsigned long long));
  Lp.d_out = (double*)plan_alloc(ctx, P, P.owned, "lattice_out", (size_t)std::max<int64_t>(P.nq, 1) * sizeof(double));
  if (!P.d_q) {
    P.d_q = (double*)plan_alloc(ctx, P, P.owned, "lattice_q", (size_t)std::max<int64_t>(P.nq, 1) * sizeof(double));
    copy_h2d(ctx, P.d_q, P.q.data(), (size_t)P.nq * sizeof(double), ctx->stream);
  }
  Lp.active = true;
}

void lattice_plan_init_device(crab_ctx* ctx, PairPlan& P, const int32_t* d_cells, int64_t m, double spacing,
                              const int64_t* span) {
  LatticePart& Lp = P.lattice;
  Lp.m = m;
  Lp.spacing = spacing;
  Lp.bins = 1;
  if (m >= 2) {
    int64_t nmax = 0;
    for (int d = 0; d < 3; ++d) nmax += span[d] * span[d];
    if (nmax >= kSharedBins) {
      // The bound is a cell or two an axis above the cells' own span, which
      // decides between counters in shared and in device memory (294 atoms with
      // 53,353 sites on a 1 Å grid just under the line: 39.4 ms a call by the
      // bound, 1.8 so) and whether the lattice is refused.
      int ext[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
      auto* d_ext = (int*)ctx->dev("lattice.span", sizeof(ext));
      copy_h2d(ctx, d_ext, ext, sizeof(ext), ctx->stream);
      k_lattice_span<<<(unsigned)std::min<int64_t>((m + 255) / 256, ctx->sm_count), 256, 0, ctx->stream>>>(d_cells, m,
                                                                                                         d_ext);
      CRAB_CUDA_CHECK(cudaGetLastError());
      ctx->launches += 1;
      copy_d2h(ctx, ext, d_ext, sizeof(ext), ctx->stream);
      CRAB_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
      nmax = 0;
      for (int d = 0; d < 3; ++d) nmax += (int64_t)(ext[3 + d] - ext[d]) * (ext[3 + d] - ext[d]);
    }
    require(nmax < (int64_t)1 << 30, "hydration lattice too large for the site histogram");
    require((m + kLT - 1) / kLT <= 65535, "too many lattice sites for one histogram launch");
    Lp.bins = (int)nmax + 1;
  }
  Lp.d_cells = (int4*)plan_alloc(ctx, P, P.owned, "lattice_cells", (size_t)std::max<int64_t>(m, 1) * sizeof(int4));
  Lp.d_hist = (unsigned long long*)plan_alloc(ctx, P, P.owned, "lattice_hist",
                                               (size_t)Lp.bins * sizeof(unsigned long long));
  Lp.d_out = (double*)plan_alloc(ctx, P, P.owned, "lattice_out", (size_t)std::max<int64_t>(P.nq, 1) * sizeof(double));
  Lp.active = true;
}

void lattice_plan_launch(crab_ctx* ctx, PairPlan& P, cudaStream_t s) {
  LatticePart& Lp = P.lattice;
  if (!Lp.active || P.nq == 0) return;
  CRAB_CUDA_CHECK(cudaMemsetAsync(Lp.d_hist, 0, (size_t)Lp.bins * sizeof(unsigned long long), s));
  if (Lp.m >= 2) {
    const int64_t nt = (Lp.m + kLT - 1) / kLT;
    if (Lp.bins <= kSharedBins) {
      const unsigned grid = (unsigned)std::min<int64_t>(nt * (nt + 1) / 2, 4 * ctx->sm_count);  // four CTAs an SM
      k_lattice_hist<<<grid, kLThreads, 0, s>>>(Lp.d_cells, Lp.m, nt, Lp.bins, Lp.d_hist);
    } else {
      k_lattice_hist_wide<<<dim3((unsigned)nt, (unsigned)nt), kLT, 0, s>>>(Lp.d_cells, Lp.m, Lp.d_hist);
    }
    CRAB_CUDA_CHECK(cudaGetLastError());
    ctx->launches += 1;
  }
  k_lattice_transform<<<(unsigned)P.nq, 256, 0, s>>>(Lp.d_hist, Lp.bins, Lp.spacing, P.d_q, Lp.d_out);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 1;
}

}  // namespace crab
