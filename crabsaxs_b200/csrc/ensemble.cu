// Batched ensemble scoring (crabSAXS src/ensemble.rs:127-465 and
// src/reweight.rs:84-374 on the device).
//
// The reference's EnsembleFitter::fit_core computes, for each of the 25
// (c1, c2) candidates, a full compute_curve of every conformer (ensemble.rs:
// 244-261): 25·K O(N²·Nq) sums.  c1 and c2 only enter through the amplitude
// recombination, so here:
//   1. one persistent launch of the pair kernel over the work items of every
//      conformer (a batch plan, longest items first across conformers of
//      uneven size) produces each conformer's per-type-pair partials once;
//   2. k_ens_curves recombines them into the curve of every (candidate,
//      conformer) pair;
//   3. k_ens_weights runs, one CTA per candidate, the projected-gradient
//      simplex fit of ensemble.rs:317-381 (250 iterations with the simplex
//      projection of ensemble.rs:449-465);
//   4. k_ens_reweight picks the best candidate, returns ∂χ²/∂(c1, c2) at its
//      weights, and runs the maximum-entropy mirror descent of
//      reweight.rs:84-154 from a uniform prior.
// Steps 1-4 are captured once in a CUDA graph and replayed.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <numeric>
#include <random>

#include "device_math.cuh"
#include "engine.hpp"
#include "ops.hpp"

namespace crab {
namespace {

constexpr int kEW = 256;  // threads whose partial sums the weight fit adds
constexpr int kMaxK = 1024;
constexpr size_t kEnsSmem = 225 * 1024;  // dynamic shared memory of the fit kernels at most

// Raw pair sums of a conformer as partials at q: Σ w w sin(q r)/(q r) of type
// pair ab = (a, b).
struct EnsPartials {
  const double* Pc;       // [ab][nq] of the conformer, at this q
  const double* self_w2;  // [T]
  const double* sum_w;    // [T]
  int nq;
  double qq;
  __device__ __forceinline__ double operator()(int a, int b, int ab) const {
    if (qq == 0.0) return (a == b) ? 0.5 * (sum_w[a] * sum_w[a] - self_w2[a]) : sum_w[a] * sum_w[b];
    return Pc[(size_t)ab * nq] / qq;
  }
};

// term(b, P(a, b)) for b = a .. T - 1 in order, the loads and quotients of eight
// type pairs at a time: one by one they are the kernels' time where a conformer
// has many types (6 conformers of a dozen types, 25 candidates: 110 to 75 us
// each).
template <class Term>
__device__ __forceinline__ void ens_row(const EnsPartials& P, int a, int T, Term term) {
  const int ab0 = a * T - a * (a - 1) / 2 - a;
  if (P.qq == 0.0) {
    for (int b = a; b < T; ++b) term(b, P(a, b, ab0 + b));
    return;
  }
  const double* v = P.Pc + (size_t)ab0 * P.nq;
  int b = a;
  for (; b + 8 <= T; b += 8) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = v[(size_t)(b + u) * P.nq];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = x[u] / P.qq;
#pragma unroll
    for (int u = 0; u < 8; ++u) term(b + u, x[u]);
  }
  for (; b < T; ++b) term(b, v[(size_t)b * P.nq] / P.qq);
}

// curves[cand][k][p] from raw partials [c][ab][p] (Σ w w sin(q r)/r) and the
// per-candidate amplitude tables amp[cand][t][p] (Â_t = V - G E + c2 H).
__global__ void k_ens_curves(const double* __restrict__ raw, const int* __restrict__ sel, const double* __restrict__ q,
                             int nq, int T, const double* __restrict__ amp, const double* __restrict__ self_w2,
                             const double* __restrict__ sum_w, int K, double* __restrict__ curves) {
  const int k = blockIdx.x, cand = blockIdx.y;
  const int c = sel[k];
  const int NP = T * (T + 1) / 2;
  const double* Pc = raw + (size_t)c * NP * nq;
  const double* A = amp + (size_t)cand * T * nq;
  for (int p = threadIdx.x; p < nq; p += blockDim.x) {
    const EnsPartials P{Pc + p, self_w2 + (size_t)c * T, sum_w + (size_t)c * T, nq, q[p]};
    double I = 0.0;
    for (int a = 0; a < T; ++a) {
      const double Aa = A[(size_t)a * nq + p];
      I += Aa * Aa * self_w2[(size_t)c * T + a];
      ens_row(P, a, T, [&](int b, double Pv) { I += 2.0 * Aa * A[(size_t)b * nq + p] * Pv; });
    }
    curves[((size_t)cand * K + k) * nq + p] = fmax(I, 0.0);
  }
}

struct EnsOpts {
  int scale_mode, bg_mode;
  double scale_value, bg_value;
  int uniform;
  double regularization;
  bool operator==(const EnsOpts& o) const {
    return scale_mode == o.scale_mode && bg_mode == o.bg_mode && scale_value == o.scale_value &&
           bg_value == o.bg_value && uniform == o.uniform && regularization == o.regularization;
  }
};

// Sums over p < n of two terms, the terms of index t, t + kEW, ... in thread
// t < kEW, its 32 lanes joined by halving and the warps in order: the same
// additions in the same order whatever the block size.  `red` has two halves
// that alternate, so one barrier is enough (a half is written again after the
// barrier of the sum in between).
struct BlockSums {
  double* red;
  int half = 0;
  template <class F>
  __device__ __forceinline__ double2 sum2(int n, F term) {
    double* r = red + half * (2 * kEW / 32);
    half ^= 1;
    if (threadIdx.x < kEW) {
      double2 v = make_double2(0.0, 0.0);
      for (int p = threadIdx.x; p < n; p += kEW) term(p, v);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if ((threadIdx.x & 31) == 0) {
        r[threadIdx.x >> 5] = v.x;
        r[kEW / 32 + (threadIdx.x >> 5)] = v.y;
      }
    }
    __syncthreads();
    double2 t = make_double2(0.0, 0.0);
#pragma unroll
    for (int w = 0; w < kEW / 32; ++w) {
      t.x += r[w];
      t.y += r[kEW / 32 + w];
    }
    return t;
  }
  template <class F>
  __device__ __forceinline__ double sum(int n, F term) {
    double* r = red + half * (2 * kEW / 32);
    half ^= 1;
    if (threadIdx.x < kEW) {
      double v = 0.0;
      for (int p = threadIdx.x; p < n; p += kEW) term(p, v);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kEW / 32; ++w) t += r[w];
    return t;
  }
};

// Descending bitonic sort of n (power of two) values in smem.
__device__ void bitonic_desc(double* v, int n) {
  for (int size = 2; size <= n; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool desc = (i & size) == 0;
          const double a = v[i], b = v[j];
          if (desc ? (a < b) : (a > b)) {
            v[i] = b;
            v[j] = a;
          }
        }
      }
      __syncthreads();
    }
}

// ensemble.rs:449-465: v = max(v - θ, 0) with θ from the sorted prefix.  Up to
// 128 values are sorted by counting, for each, the values before it (one pass;
// the bitonic network's 28 barriers take three times as long); thread 0 forms
// the running sums, and every thread tests its own index.
__device__ void project_simplex_dev(double* v, int K, double* sorted, int n2, int* rho) {
  const int tid = threadIdx.x;
  if (K <= 128) {
    for (int i = tid; i < n2; i += blockDim.x) sorted[i] = -INFINITY;
    if (tid == 0) *rho = 0;
    __syncthreads();
    for (int i = tid; i < K; i += blockDim.x) {
      const double x = v[i];
      int at = 0;
      for (int j = 0; j < K; ++j) {
        const double u = v[j];
        at += u > x || (!(u < x) && j < i);
      }
      sorted[at] = x;
    }
    __syncthreads();
  } else {
    for (int i = tid; i < n2; i += blockDim.x) sorted[i] = i < K ? v[i] : -INFINITY;
    if (tid == 0) *rho = 0;
    __syncthreads();
    bitonic_desc(sorted, n2);
  }
  double* cum = sorted + n2;
  if (tid == 0) {
    double c = 0.0;
#pragma unroll 8
    for (int i = 0; i < K; ++i) {
      c += sorted[i];
      cum[i] = c;
    }
  }
  __syncthreads();
  for (int i = tid; i < K; i += blockDim.x)
    if (sorted[i] + (1.0 - cum[i]) / (double)(i + 1) > 0.0) atomicMax(rho, i + 1);
  __syncthreads();
  const int r = *rho;
  const double theta = ((r > 0 ? cum[r - 1] : 0.0) - 1.0) / (double)max(r, 1);
  for (int i = tid; i < K; i += blockDim.x) v[i] = fmax(v[i] - theta, 0.0);
  __syncthreads();
}

// The weight kernel's shared memory, in doubles: weights, gradients and
// proposals, the sorted values and their running sums; per q the mixture, the
// weighted residual, y, sigma, 1/sigma and 1/sigma²; two chunks of gradient
// terms; and the curves, where they fit.
constexpr int kWT = 512;  // threads of k_ens_weights
__host__ __device__ inline int ew_pow2(int K) {
  int n2 = 1;
  while (n2 < K) n2 <<= 1;
  return n2;
}
// q per chunk of gradient terms (a power of two up to 32)
__host__ __device__ inline int ew_chunk(int K) { return K <= 256 ? 32 : 8; }
__host__ __device__ inline size_t ew_full(int K, int nq) {
  return (size_t)4 * K + ew_pow2(K) + 6 * (size_t)nq + 2 * (size_t)ew_chunk(K) * (K | 1);
}
// Very long q grids keep only the mixture and the residual there, and one q
// of gradient terms at a time.
__host__ __device__ inline bool ew_lean(int K, int nq) { return ew_full(K, nq) * sizeof(double) > kEnsSmem; }
__host__ __device__ inline size_t ew_doubles(int K, int nq) {
  return ew_lean(K, nq) ? (size_t)4 * K + ew_pow2(K) + 2 * (size_t)nq + 2 * (size_t)(K | 1) : ew_full(K, nq);
}
__host__ __device__ inline bool ew_on_chip(int K, int nq) {
  return (ew_doubles(K, nq) + (size_t)K * nq) * sizeof(double) <= kEnsSmem;
}

// Σ_p (rs[p] cv[k][p]) / sg[p] for every k into out[k], each in the order of p.
// The terms of a chunk of P q are formed, one chunk ahead, by the warps beyond
// the K threads that add them up (by all warps if those are too many), a lane
// for each q of the chunk.
__device__ __forceinline__ void ew_gradient(const double* cv, int K, int nq, const double* rs, const double* sg,
                                            const double* isg, bool plain, int P, double* terms, double* out) {
  const int tid = threadIdx.x, kp = (K + 31) & ~31, ks = K | 1;
  const bool apart = kp <= kWT / 2;
  const int t0 = apart ? tid - kp : tid, tn = apart ? kWT - kp : kWT;
  const int lp = t0 & (P - 1), k_first = t0 / P, k_step = tn / P;
  auto form = [&](int q0, double* to) {
    const int p = q0 + lp;
    if (t0 < 0 || p >= nq) return;
    const double r = rs[p], b = sg[p], y = plain ? 0.0 : isg[p];
    const double* c = cv + k_first * nq + p;
    double* d = to + lp * ks + k_first;
#pragma unroll 2
    for (int k = k_first; k < K; k += k_step, c += k_step * nq, d += k_step) {
      const double a = r * *c;
      *d = plain ? a / b : dev::div_by(a, b, y);
    }
  };
  double acc[kMaxK / kWT] = {0.0, 0.0};
  form(0, terms);
  __syncthreads();
  int buf = 0;
  for (int q0 = 0; q0 < nq; q0 += P, buf ^= 1) {
    const double* t = terms + buf * P * ks;
    if (q0 + P < nq) form(q0 + P, terms + (buf ^ 1) * P * ks);
    const int n = min(P, nq - q0);
#pragma unroll
    for (int j = 0; j < kMaxK / kWT; ++j) {
      const int k = tid + j * kWT;
      if (k >= K) break;
      if (n == 32) {
#pragma unroll
        for (int p = 0; p < 32; ++p) acc[j] += t[p * ks + k];
      } else {
        for (int p = 0; p < n; ++p) acc[j] += t[p * ks + k];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < kMaxK / kWT; ++j)
    if (tid + j * kWT < K) out[tid + j * kWT] = acc[j];
  __syncthreads();
}

// One CTA per candidate: ensemble.rs:317-381.  Bound by latency: 250 steps, each
// a chain of sums.  Every sum keeps its terms and their order (the final
// iterate depends on the last bits), but the terms are formed in parallel: 41
// us a step became 13 us for 48 curves of 300 q (one thread per curve ran the
// gradient's 300 dependent divisions, and one thread the projection's).
__global__ void __launch_bounds__(kWT)
    k_ens_weights(const double* __restrict__ curves, int K, int nq, const double* __restrict__ y,
                  const double* __restrict__ sg, EnsOpts o, double* __restrict__ weights, double* __restrict__ fit,
                  double* __restrict__ fitted, double* __restrict__ grad_w) {
  extern __shared__ double sm[];
  const int n2 = ew_pow2(K), tid = threadIdx.x;
  double* w = sm;                // K
  double* g = w + K;             // K
  double* prop = g + K;          // K
  double* sorted = prop + K;     // n2, then K running sums
  double* mix = sorted + n2 + K; // nq
  double* rs = mix + nq;         // nq: residual / sigma x scale
  const bool lean = ew_lean(K, nq);
  const int P = lean ? 1 : ew_chunk(K);
  double* terms = rs + nq;       // 2 x P x (K | 1)
  double* perq = terms + 2 * (size_t)P * (K | 1);
  double* isg = perq;            // nq: 1 / sigma
  double* ww = perq + nq;        // nq: 1 / sigma²
  const double* ys = lean ? y : perq + 2 * (size_t)nq;
  const double* sgs = lean ? sg : perq + 3 * (size_t)nq;
  double* cvs = perq + (lean ? 0 : 4 * (size_t)nq);
  __shared__ double red[4 * kEW / 32];
  __shared__ int rho, plain_s;
  const int cand = blockIdx.x;
  const double* cv = curves + (size_t)cand * K * nq;
  if (tid == 0) plain_s = lean ? 1 : 0;
  __syncthreads();
  for (int p = tid; p < nq && !lean; p += kWT) {
    const double v = sg[p];
    perq[2 * nq + p] = y[p];
    perq[3 * nq + p] = v;
    isg[p] = 1.0 / v;
    ww[p] = 1.0 / (v * v);
    if (!(v > 1e-100 && v < 1e100)) plain_s = 1;
  }
  BlockSums bs{red};
  auto wgt = [&](int p) { return lean ? 1.0 / (sg[p] * sg[p]) : ww[p]; };
  if (ew_on_chip(K, nq)) {
    for (int i = tid; i < K * nq; i += kWT) cvs[i] = cv[i];
    cv = cvs;
  }
  for (int k = tid; k < K; k += kWT) w[k] = 1.0 / (double)K;
  __syncthreads();
  const bool plain = plain_s != 0;
  const double d2 =
      o.bg_mode == CRAB_BG_FIT ? bs.sum(nq, [&](int p, double& v) { v += wgt(p); }) : 0.0;
  // mixture, then scale and background (ensemble.rs:383-434)
  double s, b;
  auto mixture = [&]() {
    for (int p = tid; p < nq; p += kWT) {
      double m = 0.0;
      const double* c = cv + p;
#pragma unroll 8
      for (int k = 0; k < K; ++k, c += nq) m += *c * w[k];
      mix[p] = m;
    }
    __syncthreads();
    const double2 nd = bs.sum2(nq, [&](int p, double2& v) {
      const double q = wgt(p);
      v.x += mix[p] * ys[p] * q;
      v.y += mix[p] * mix[p] * q;
    });
    s = o.scale_mode == CRAB_SCALE_FIT ? (nd.y > 0.0 ? nd.x / nd.y : 0.0) : o.scale_value;
    s = fmax(s, 0.0);
    b = 0.0;
    if (o.bg_mode == CRAB_BG_FIT) {
      const double n2s = bs.sum(nq, [&](int p, double& v) { v += (ys[p] - s * mix[p]) * wgt(p); });
      b = d2 > 0.0 ? n2s / d2 : 0.0;
    } else if (o.bg_mode == CRAB_BG_FIXED) {
      b = o.bg_value;
    }
  };
  const int iters = o.uniform ? 0 : 250;
  for (int it = 0; it < iters; ++it) {
    mixture();
    for (int p = tid; p < nq; p += kWT) rs[p] = (s * mix[p] + b - ys[p]) / sgs[p] * s;
    __syncthreads();
    ew_gradient(cv, K, nq, rs, sgs, isg, plain, P, terms, g);
    for (int k = tid; k < K; k += kWT) {
      const double acc = g[k];
      g[k] = 2.0 * acc + 2.0 * o.regularization * (w[k] - 1.0 / (double)K);
    }
    __syncthreads();
    double nrm = bs.sum(K, [&](int k, double& v) { v += g[k] * g[k]; });
    nrm = fmax(sqrt(nrm), 1.0);
    for (int k = tid; k < K; k += kWT) prop[k] = w[k] - 0.05 * g[k] / nrm;
    __syncthreads();
    project_simplex_dev(prop, K, sorted, n2, &rho);
    const double delta = bs.sum(K, [&](int k, double& v) { v += fabs(prop[k] - w[k]); });
    for (int k = tid; k < K; k += kWT) w[k] = prop[k];
    __syncthreads();
    if (delta < 1e-8) break;
  }
  mixture();
  const double chi = bs.sum(nq, [&](int p, double& v) {
                       const double r = (s * mix[p] + b - ys[p]) / sgs[p];
                       v += r * r;
                     }) /
                     (double)max(nq - 1, 1);
  for (int p = tid; p < nq; p += kWT) {
    fitted[(size_t)cand * nq + p] = s * mix[p] + b;
    rs[p] = (s * mix[p] + b - ys[p]) / sgs[p] * s;
  }
  __syncthreads();
  // ∂χ²_red/∂w_k at the final weights (scale and background held)
  ew_gradient(cv, K, nq, rs, sgs, isg, plain, P, terms, g);
  for (int k = tid; k < K; k += kWT) {
    const double acc = g[k];
    grad_w[(size_t)cand * K + k] = 2.0 * acc / (double)max(nq - 1, 1);
    weights[(size_t)cand * K + k] = w[k];
  }
  if (tid == 0) {
    fit[4 * cand] = s;
    fit[4 * cand + 1] = b;
    fit[4 * cand + 2] = chi;
    fit[4 * cand + 3] = (double)iters;
  }
}

struct RwOpts {
  double kl, step, tol, floor;
  int max_iter, scale_mode, bg_mode;
  double scale_value, bg_value;
  bool operator==(const RwOpts& o) const {
    return kl == o.kl && step == o.step && tol == o.tol && floor == o.floor && max_iter == o.max_iter &&
           scale_mode == o.scale_mode && bg_mode == o.bg_mode && scale_value == o.scale_value &&
           bg_value == o.bg_value;
  }
};

// ---- KL reweighting -------------------------------------------------------
// reweight.rs:84-154 on the best candidate's K curves, bound by the latency of
// its 500 steps, each with a line search of up to 14 evaluations.  Every CTA
// holds all K weights, gradients and proposals and does all work on them, so
// that an evaluation needs one exchange at most: with the curves split over a
// cluster of CL CTAs (CTA r keeps the rows [r kr, (r+1) kr) in its shared
// memory), the partial mixtures of all CTAs, added in rank order, and once per
// step the gradients of their rows.  All CTAs therefore hold the same values and
// take the same branches.  CL is one where the curves fit one CTA's shared
// memory: a step of 48 curves of 300 q (five evaluations on average) then has
// block barriers only, and takes 19 us (100 us on 8 CTAs that split the weights
// too, with a cluster barrier for each of the six sums of an evaluation).
// Where the buffers fit too, SP = kRwCluster such CTAs, each with all curves,
// evaluate the next SP step lengths of the line search at once; the first one
// that decreases the objective is taken from the CTA that has it, so that the
// steps and their values are those of the search one by one (500 steps: 9.5 to
// 4.1 ms).
constexpr int kRwCluster = 8;
constexpr int kRwHalvings = 14;  // step lengths of a line search
namespace cg = cooperative_groups;

// Threads of a CTA: about one per q, and a warp more for the K logarithms, or
// one per curve.
inline int rw_threads(int K, int nq) {
  return std::min(512, std::max({128, (nq + 31) / 32 * 32 + 64, (K + 31) / 32 * 32}));
}

// Sums over the block of N values per thread (a fixed tree, then the warps in
// order); the two halves of `red` alternate, as in BlockSums.
struct RwSums {
  double* red;  // [2][4 x 16]
  int half = 0;
  template <int N>
  __device__ __forceinline__ void operator()(double (&v)[N]) {
    double* r = red + half * 64;
    half ^= 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
      for (int i = 0; i < N; ++i) r[i * 16 + (threadIdx.x >> 5)] = v[i];
    __syncthreads();
    const int warps = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = 0.0;
#pragma unroll 4
    for (int w = 0; w < warps; ++w)
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] += r[i * 16 + w];
  }
  __device__ __forceinline__ double max(double v) {
    double* r = red + half * 64;
    half ^= 1;
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = v;
    __syncthreads();
    v = r[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = fmax(v, r[w]);
    return v;
  }
};

__host__ __device__ inline int rw_rows(int K, int cl) { return (K + cl - 1) / cl; }
// Shared memory in doubles without the curves: weights, gradients, proposals
// and the logarithms of both; per q the mixture (then the gradient's factor), y
// and 1/sigma²; in a cluster the partial mixtures (two halves) and the
// gradients (two halves) that its CTAs exchange.
__host__ __device__ inline size_t rw_doubles(int K, int nq, int cl) {
  return 5 * (size_t)K + 3 * (size_t)nq + (cl > 1 ? 2 * (size_t)nq : 0) + 2 * (size_t)rw_rows(K, cl);
}
__host__ __device__ inline bool rw_on_chip(int K, int nq, int cl) {
  return (rw_doubles(K, nq, cl) + (size_t)rw_rows(K, cl) * nq) * sizeof(double) <= kEnsSmem;
}
__host__ __device__ inline size_t rw_smem(int K, int nq, int cl) {
  return (rw_doubles(K, nq, cl) + (rw_on_chip(K, nq, cl) ? (size_t)rw_rows(K, cl) * nq : 0)) * sizeof(double);
}

// Doubles more of a CTA that searches step lengths in a cluster: two halves of
// proposal, logarithms, mixture, and of the cluster's (χ², KL, scale, background).
__host__ __device__ inline size_t rw_search_doubles(int K, int nq) {
  return 2 * (2 * (size_t)K + (size_t)nq + 4 * kRwCluster);
}

// Best candidate, ∂χ²/∂(c1, c2) there, then reweight.rs:84-154.
// out: [0] best candidate, [1] scale, [2] bg, [3] reduced chi2, [4] KL,
// [5] iterations, [6] converged, [7] dchi/dc1, [8] dchi/dc2.
template <int CL, int SP>
__global__ void __launch_bounds__(512, 1)
    k_ens_reweight(const double* __restrict__ curves, const double* __restrict__ fitc, int n_cand, int K, int nq,
                   const double* __restrict__ y, const double* __restrict__ sg, const double* __restrict__ weights,
                   const double* __restrict__ dcurves, RwOpts o, double* __restrict__ w_out,
                   double* __restrict__ out) {
  extern __shared__ double sm[];
  __shared__ double red[2 * 64];
  __shared__ int best;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int back = nt - 1 - tid;  // the K-wide work of an evaluation starts at the last warp
  int rank = 0;
  static_assert(CL == 1 || SP == 1, "the cluster splits the curves or the step lengths");
  if constexpr (CL > 1) rank = (int)cg::this_cluster().block_rank();
  int srank = 0;
  if constexpr (SP > 1) srank = (int)cg::this_cluster().block_rank();
  const int kr = rw_rows(K, CL), k0 = min(K, rank * kr), nk = min(K, k0 + kr) - k0;
  double* w = sm;              // K
  double* g = w + K;           // K
  double* pr = g + K;          // K
  double* lw = pr + K;         // K: log(w / prior)
  double* lp = lw + K;         // K: log(pr / prior)
  double* mix = lp + K;        // nq
  double* ys = mix + nq;       // nq
  double* ww = ys + nq;        // nq
  double* own = ww + nq;       // 2 x nq: this CTA's partial mixture (in a cluster)
  double* gx = own + (CL > 1 ? 2 * (size_t)nq : 0);  // 2 x kr
  double* found = gx + 2 * (size_t)kr;  // the search's two halves
  const size_t half_doubles = SP > 1 ? rw_search_doubles(K, nq) / 2 : 0;
  double* cvs = found + 2 * half_doubles;
  RwSums sums{red};
  if (tid == 0) {
    best = 0;
    for (int c = 1; c < n_cand; ++c)
      if (fitc[4 * c + 2] < fitc[4 * best + 2]) best = c;
  }
  for (int p = tid; p < nq; p += nt) {
    ys[p] = y[p];
    ww[p] = 1.0 / (sg[p] * sg[p]);
  }
  __syncthreads();
  const double* cvr = curves + ((size_t)best * K + k0) * nq;  // this CTA's rows
  const double dof = (double)max(nq - 1, 1);
  // ∂χ²/∂c1 and ∂χ²/∂c2 at the best candidate's weights, scale and background
  if (rank == 0 && srank == 0) {
    const double s = fitc[4 * best], b = fitc[4 * best + 1];
    const double* wb = weights + (size_t)best * K;
    const double* cb = curves + (size_t)best * K * nq;
    const double* d1c = dcurves + (size_t)(2 * best) * K * nq;
    const double* d2c = dcurves + (size_t)(2 * best + 1) * K * nq;
    double v[2] = {0.0, 0.0};
    for (int p = tid; p < nq; p += nt) {
      double m = 0.0, d1 = 0.0, d2 = 0.0;
#pragma unroll 4
      for (int k = 0; k < K; ++k) {
        m += cb[(size_t)k * nq + p] * wb[k];
        d1 += d1c[(size_t)k * nq + p] * wb[k];
        d2 += d2c[(size_t)k * nq + p] * wb[k];
      }
      const double wgt = 2.0 * (s * m + b - ys[p]) * ww[p] / dof * s;
      v[0] += wgt * d1;
      v[1] += wgt * d2;
    }
    sums(v);
    if (tid == 0) {
      out[7] = v[0];
      out[8] = v[1];
    }
  }
  if (rw_on_chip(K, nq, CL)) {
    for (int i = tid; i < nk * nq; i += nt) cvs[i] = cvr[i];
    cvr = cvs;
  }
  const double prior = 1.0 / (double)K, residual = 1.0 - o.floor * (double)K;
  double sw, sy;  // Σ 1/σ², Σ y/σ²
  {
    double v[3] = {0.0, 0.0, 0.0};
    for (int p = tid; p < nq; p += nt) {
      v[0] += ww[p];
      v[1] += ww[p] * ys[p];
    }
    for (int k = tid; k < K; k += nt) v[2] += prior;
    sums(v);
    sw = v[0];
    sy = v[1];
    const double all = fmax(v[2], 1e-300);
    for (int k = tid; k < K; k += nt) w[k] = o.floor <= 0.0 ? prior / all : o.floor + residual * prior / all;
  }
  __syncthreads();
  int par = 0, gpar = 0;
  double s, b, chi, kl;
  // log(wv / prior) into lv; the mixture of wv, then scale and background
  // (reweight.rs:236-301), χ² and the KL term
  auto evaluate = [&](const double* wv, double* lv, double* mix) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};  // Σ m/σ², Σ m²/σ², Σ m y/σ², Σ w log(w/prior)
    for (int k = back; k < K; k += nt) {
      const double l = log(wv[k] / prior);
      lv[k] = l;
      v[3] += wv[k] * l;
    }
    double* mine = CL > 1 ? own + (size_t)par * nq : mix;
    auto moments = [&](int p, double m) {
      v[0] += ww[p] * m;
      v[1] += ww[p] * m * m;
      v[2] += ww[p] * m * ys[p];
    };
    for (int p = tid; p < nq; p += nt) {
      double m = 0.0, m1 = 0.0;
      const double* c = cvr + p;
      int k = 0;
#pragma unroll 4
      for (; k + 1 < nk; k += 2, c += 2 * nq) {
        m += c[0] * wv[k0 + k];
        m1 += c[nq] * wv[k0 + k + 1];
      }
      if (k < nk) m += c[0] * wv[k0 + k];
      m += m1;
      mine[p] = m;
      if (CL == 1) moments(p, m);
    }
    if constexpr (CL > 1) {
      cg::this_cluster().sync();
      for (int p = tid; p < nq; p += nt) {
        double m = 0.0;
#pragma unroll
        for (int r = 0; r < CL; ++r) m += cg::this_cluster().map_shared_rank(mine, r)[p];
        mix[p] = m;
        moments(p, m);
      }
      par ^= 1;  // the barrier of the next exchange releases this half
    }
    sums(v);
    const double sx = v[0], sxx = v[1], sxy = v[2];
    kl = v[3];
    auto fscale = [&](double bb) { return sxx > 0.0 ? fmax((sxy - bb * sx) / sxx, 0.0) : 0.0; };
    auto fbg = [&](double ss) { return sw > 0.0 ? (sy - ss * sx) / sw : 0.0; };
    if (o.scale_mode == CRAB_SCALE_FIXED) {
      s = fmax(o.scale_value, 0.0);
      b = o.bg_mode == CRAB_BG_FIXED ? o.bg_value : (o.bg_mode == CRAB_BG_FIXED_ZERO ? 0.0 : fbg(s));
    } else if (o.bg_mode == CRAB_BG_FIXED) {
      s = fscale(o.bg_value);
      b = o.bg_value;
    } else if (o.bg_mode == CRAB_BG_FIXED_ZERO) {
      s = fscale(0.0);
      b = 0.0;
    } else {
      const double det = sxx * sw - sx * sx;
      s = fabs(det) > 1e-20 ? fmax((sxy * sw - sx * sy) / det, 0.0) : 0.0;
      b = fbg(s);
    }
    double e[1] = {0.0};
    for (int p = tid; p < nq; p += nt) {
      const double r = s * mix[p] + b - ys[p];
      e[0] += r * r * ww[p];
    }
    sums(e);
    chi = e[0] / dof;
  };
  int iterations = 0, converged = 0;
  if constexpr (SP > 1) cg::this_cluster().sync();  // every CTA runs before one writes into another
  evaluate(w, lw, mix);
  for (int it = 0; it < o.max_iter; ++it) {
    iterations = it + 1;
    // gradient at w, whose mixture, scale and background the last evaluation left
    for (int p = tid; p < nq; p += nt) mix[p] = 2.0 * ((s * mix[p] + b) - ys[p]) * s * ww[p] / dof;
    __syncthreads();
    double* gown = gx + gpar * kr;
    for (int k = tid >> 5; k < nk; k += nt >> 5) {  // a warp per curve
      double dg = 0.0;
      const double* c = cvr + k * nq;
#pragma unroll 4
      for (int p = tid & 31; p < nq; p += 32) dg += mix[p] * c[p];
#pragma unroll
      for (int q = 16; q > 0; q >>= 1) dg += __shfl_xor_sync(0xffffffffu, dg, q);
      if ((tid & 31) == 0) gown[k] = dg;
    }
    if constexpr (CL > 1) cg::this_cluster().sync();
    else __syncthreads();
    double gmax = 0.0;
    for (int k = tid; k < K; k += nt) {
      double v;
      if constexpr (CL > 1) v = cg::this_cluster().map_shared_rank(gown, k / kr)[k % kr];
      else v = gown[k];
      v += o.kl * (lw[k] + 1.0);
      g[k] = v;
      gmax = fmax(gmax, fabs(v));
    }
    gpar ^= 1;
    gmax = fmax(sums.max(gmax), 1e-12);
    double step = o.step / gmax;
    const double objective = chi + o.kl * kl;
    // proposal exp(log w - step g), normalised and floored (w is at most one,
    // and |step g| at most o.step: the largest exponent needs no search
    // unless the step is very long)
    auto propose = [&](double step, double* pr) {
      double mx = o.step;
      if (o.step > 100.0) {
        mx = -INFINITY;
        for (int k = tid; k < K; k += nt) mx = fmax(mx, lw[k] - step * g[k]);
        mx = sums.max(mx);
      }
      double t[1] = {0.0};
      for (int k = tid; k < K; k += nt) {
        const double e = w[k] > 0.0 ? exp(lw[k] - step * g[k] - mx) : 0.0;
        pr[k] = e;
        t[0] += e;
      }
      sums(t);
      const double all = fmax(t[0], 1e-300);
      for (int k = tid; k < K; k += nt) pr[k] = fmax(o.floor, 0.0) + residual * (pr[k] / all);
      __syncthreads();
    };
    bool accepted = false;
    const double *np = pr, *nl = lp;  // the accepted weights and their logarithms
    if constexpr (SP > 1) {
      for (int h0 = 0; h0 < kRwHalvings && !accepted; h0 += SP) {
        double* mine = found + par * half_doubles;  // proposal, logarithms, mixture, table
        double* table = mine + 2 * K + nq;
        par ^= 1;  // a half is written again only after the barrier that follows its readers
        double length = step;
        for (int h = 0; h < h0 + srank; ++h) length *= 0.5;
        if (h0 + srank < kRwHalvings) {
          propose(length, mine);
          evaluate(mine, mine + K, mine + 2 * K);
          if (tid < SP) {
            double* t = cg::this_cluster().map_shared_rank(table, tid) + 4 * srank;
            t[0] = chi;
            t[1] = kl;
            t[2] = s;
            t[3] = b;
          }
        }
        cg::this_cluster().sync();
        for (int r = 0; r < SP && h0 + r < kRwHalvings && !accepted; ++r)
          if (table[4 * r] + o.kl * table[4 * r + 1] <= objective + 1e-12) {
            accepted = true;
            chi = table[4 * r];
            kl = table[4 * r + 1];
            s = table[4 * r + 2];
            b = table[4 * r + 3];
            np = cg::this_cluster().map_shared_rank(mine, r);
            nl = np + K;
            for (int p = tid; p < nq; p += nt) mix[p] = np[2 * K + p];
          }
      }
    } else {
      for (int h = 0; h < kRwHalvings && !accepted; ++h) {
        propose(step, pr);
        evaluate(pr, lp, mix);
        if (chi + o.kl * kl <= objective + 1e-12) accepted = true;
        else step *= 0.5;
      }
    }
    if (!accepted) {
      evaluate(w, lw, mix);  // back at the last accepted weights
      break;
    }
    double t[1] = {0.0};
    for (int k = tid; k < K; k += nt) {
      const double v = np[k];
      t[0] += fabs(v - w[k]);
      w[k] = v;
      lw[k] = nl[k];
    }
    sums(t);
    if (t[0] <= o.tol) {
      converged = 1;
      break;
    }
  }
  if (rank == 0 && srank == 0) {
    for (int k = tid; k < K; k += nt) w_out[k] = w[k];
    if (tid == 0) {
      out[0] = best;
      out[1] = s;
      out[2] = b;
      out[3] = chi;
      out[4] = kl;
      out[5] = iterations;
      out[6] = converged;
    }
  }
  if constexpr (CL * SP > 1) cg::this_cluster().sync();  // no CTA leaves while a peer may still read its shared memory
}

template <int CL, int SP>
void launch_reweight(cudaStream_t s, size_t smem, const double* curves, const double* fitc, int n_cand, int K, int nq,
                     const double* y, const double* sg, const double* weights, const double* dcurves, RwOpts o,
                     double* w_out, double* out) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL * SP);
  cfg.blockDim = dim3(rw_threads(K, nq));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL * SP;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CL * SP > 1 ? 1 : 0;
  CRAB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k_ens_reweight<CL, SP>, curves, fitc, n_cand, K, nq, y, sg, weights, dcurves, o,
                                     w_out, out));
}

// Derivative curves dI/dc1 and dI/dc2 of every conformer at every candidate:
// dcurves[2*cand + m][k][p] (m = 0: c1, 1: c2) from dÂ tables damp.
__global__ void k_ens_dcurves(const double* __restrict__ raw, const int* __restrict__ sel,
                              const double* __restrict__ q, int nq, int T, const double* __restrict__ amp,
                              const double* __restrict__ damp, const double* __restrict__ self_w2,
                              const double* __restrict__ sum_w, int K, const double* __restrict__ curves,
                              double* __restrict__ dcurves) {
  const int k = blockIdx.x, cm = blockIdx.y, cand = cm >> 1;
  const int c = sel[k];
  const int NP = T * (T + 1) / 2;
  const double* Pc = raw + (size_t)c * NP * nq;
  const double* A = amp + (size_t)cand * T * nq;
  const double* dA = damp + (size_t)cm * T * nq;
  for (int p = threadIdx.x; p < nq; p += blockDim.x) {
    const EnsPartials P{Pc + p, self_w2 + (size_t)c * T, sum_w + (size_t)c * T, nq, q[p]};
    double d = 0.0;
    for (int a = 0; a < T; ++a) {
      const double Aa = A[(size_t)a * nq + p], dAa = dA[(size_t)a * nq + p];
      d += 2.0 * Aa * dAa * self_w2[(size_t)c * T + a];
      ens_row(P, a, T, [&](int b, double Pv) {
        d += 2.0 * (dAa * A[(size_t)b * nq + p] + Aa * dA[(size_t)b * nq + p]) * Pv;
      });
    }
    // the clamp at zero has no derivative
    dcurves[((size_t)cm * K + k) * nq + p] = curves[((size_t)cand * K + k) * nq + p] > 0.0 ? d : 0.0;
  }
}

}  // namespace

// ------------------------------------------------------------------ host side

struct EnsemblePlan {
  crab_ctx* ctx = nullptr;
  int K = 0, T = 0, n_cand = 0;
  int64_t nq = 0;
  std::vector<double> q, cand;
  std::vector<AtomClass> classes;
  bool implicit = true;
  crab_solvent solvent{};
  std::unique_ptr<PairPlan> pair;
  std::vector<double> self_w2, sum_w;  // [K][T]
  std::vector<double> amp, damp;       // [n_cand][T][nq], [2 n_cand][T][nq]
  std::vector<void*> owned;
  double* d_partials = nullptr;  // raw pair sums [K][T(T+1)/2][nq]: the pair plan's output, or uploaded
  double *d_q = nullptr, *d_amp = nullptr, *d_damp = nullptr, *d_self = nullptr, *d_sumw = nullptr;
  double *d_curves = nullptr, *d_dcurves = nullptr;
  int* d_sel = nullptr;
  // fit state
  double *d_y = nullptr, *d_sg = nullptr, *d_weights = nullptr, *d_fit = nullptr, *d_fitted = nullptr,
         *d_gradw = nullptr, *d_wkl = nullptr, *d_out = nullptr;
  cudaGraphExec_t graph = nullptr;
  // what the graph's nodes hold by value
  int graph_k = -1, graph_budget = 0;
  EnsOpts graph_fit{};
  RwOpts graph_reweight{};
  int64_t graph_kernels = 0;
  ~EnsemblePlan() {
    if (graph) cudaGraphExecDestroy(graph);
    for (void* p : owned) cudaFree(p);
  }
  template <class T_>
  T_* alloc(size_t n) {
    void* p = nullptr;
    CRAB_CUDA_CHECK(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T_)));
    owned.push_back(p);
    return (T_*)p;
  }
};

// Scattering classes of the whole ensemble (sorted) and their type indices:
// every conformer uses the same types.
static std::map<AtomClass, int> ensemble_class_index(crab_struct* const* sts, int K, bool implicit) {
  std::map<AtomClass, int> index;
  for (int c = 0; c < K; ++c) {
    require(sts[c] && sts[c]->n > 0, "ensemble must contain non-empty conformers");
    for (int64_t i = 0; i < sts[c]->n; ++i)
      index[AtomClass{sts[c]->elem[i], implicit ? (int)sts[c]->group[i] : -1}] = 0;
  }
  int T = 0;
  for (auto& kv : index) kv.second = T++;
  return index;
}

static std::vector<int32_t> conformer_types(const crab_struct* st, const std::map<AtomClass, int>& index,
                                            bool implicit) {
  std::vector<int32_t> type(st->n);
  for (int64_t i = 0; i < st->n; ++i) type[i] = index.at(AtomClass{st->elem[i], implicit ? (int)st->group[i] : -1});
  return type;
}

// Doubles per conformer in a gathered partials buffer: the raw pair sums
// [T(T+1)/2][nq], then Σw² and Σw per type.
static size_t partials_block(int T, int64_t nq) { return (size_t)(T * (T + 1) / 2) * nq + 2 * (size_t)T; }

// With `given` (a gathered buffer of K partials blocks) the pair sums are
// uploaded instead of computed, and no pair plan is built.
static std::unique_ptr<EnsemblePlan> make_ensemble_plan(crab_ctx* ctx, crab_struct* const* sts, int K, const double* q,
                                                        int64_t nq, const crab_solvent& s, bool implicit,
                                                        const double* cand, int n_cand,
                                                        const double* given = nullptr) {
  require(K > 0 && K <= kMaxK, "ensemble size must be between 1 and 1024");
  require(n_cand > 0, "at least one (c1, c2) candidate");
  require(s.hydration_model == CRAB_HYD_ANALYTIC, "the batched ensemble covers the analytic hydration model");
  for (int c = 0; c < n_cand; ++c)
    require(std::isfinite(cand[2 * c]) && cand[2 * c] > 0.0 && std::isfinite(cand[2 * c + 1]),
            "candidate c1 must be finite and positive, c2 finite");
  std::unique_ptr<EnsemblePlan> E(new EnsemblePlan());
  E->ctx = ctx;
  E->K = K;
  E->nq = nq;
  E->n_cand = n_cand;
  E->q.assign(q, q + nq);
  E->cand.assign(cand, cand + 2 * n_cand);
  E->implicit = implicit;
  E->solvent = s;
  // shared scattering types over the whole ensemble
  const std::map<AtomClass, int> index = ensemble_class_index(sts, K, implicit);
  for (const auto& kv : index) E->classes.push_back(kv.first);
  const int T = (int)index.size();
  E->T = T;
  E->self_w2.assign((size_t)K * T, 0.0);
  E->sum_w.assign((size_t)K * T, 0.0);
  if (!given) {
    std::vector<Layout> parts;
    for (int c = 0; c < K; ++c) {
      const crab_struct* st = sts[c];
      const std::vector<int32_t> type = conformer_types(st, index, implicit);
      parts.push_back(build_layout(st->xyz.data(), st->occ.data(), type.data(), st->n, T, false));
      for (int a = 0; a < T; ++a) {
        E->self_w2[(size_t)c * T + a] = parts.back().self_w2[a];
        E->sum_w[(size_t)c * T + a] = parts.back().sum_w[a];
      }
    }
    E->pair = make_batch_pair_plan(ctx, std::move(parts), q, nq);
    E->d_partials = E->pair->d_out;
  } else {
    const size_t P = (size_t)(T * (T + 1) / 2), block = partials_block(T, nq);
    std::vector<double> raw((size_t)K * P * nq);
    for (int c = 0; c < K; ++c) {
      const double* b = given + (size_t)c * block;
      std::copy(b, b + P * nq, raw.begin() + (size_t)c * P * nq);
      for (int a = 0; a < T; ++a) {
        E->self_w2[(size_t)c * T + a] = b[P * nq + a];
        E->sum_w[(size_t)c * T + a] = b[P * nq + T + a];
      }
    }
    E->d_partials = E->alloc<double>(raw.size());
    copy_h2d(ctx, E->d_partials, raw.data(), raw.size() * sizeof(double), ctx->stream);
  }
  // amplitude tables per candidate and their c1/c2 derivatives
  E->amp.assign((size_t)n_cand * T * nq, 0.0);
  E->damp.assign((size_t)2 * n_cand * T * nq, 0.0);
  for (int a = 0; a < T; ++a)
    for (int64_t p = 0; p < nq; ++p) {
      double v, e, h;
      debye_class_amplitudes(E->classes[a], implicit, q[p], s.bulk_density, s.shell_thickness, &v, &e, &h);
      for (int c = 0; c < n_cand; ++c) {
        const double c1 = cand[2 * c], c2 = cand[2 * c + 1];
        const double G = excluded_volume_scale(q[p], c1);
        const double dG = G * (3.0 / c1 - 2.0 * c1 * (1.62 * 1.62) * q[p] * q[p] / 4.0);
        E->amp[((size_t)c * T + a) * nq + p] = v - G * e + c2 * h;
        E->damp[((size_t)(2 * c) * T + a) * nq + p] = -dG * e;
        E->damp[((size_t)(2 * c + 1) * T + a) * nq + p] = h;
      }
    }
  cudaStream_t sm = ctx->stream;
  E->d_q = E->alloc<double>(nq);
  E->d_amp = E->alloc<double>(E->amp.size());
  E->d_damp = E->alloc<double>(E->damp.size());
  E->d_self = E->alloc<double>(E->self_w2.size());
  E->d_sumw = E->alloc<double>(E->sum_w.size());
  E->d_sel = E->alloc<int>(K);
  E->d_curves = E->alloc<double>((size_t)n_cand * K * nq);
  E->d_dcurves = E->alloc<double>((size_t)2 * n_cand * K * nq);
  copy_h2d(ctx, E->d_q, q, nq * sizeof(double), sm);
  copy_h2d(ctx, E->d_amp, E->amp.data(), E->amp.size() * sizeof(double), sm);
  copy_h2d(ctx, E->d_damp, E->damp.data(), E->damp.size() * sizeof(double), sm);
  copy_h2d(ctx, E->d_self, E->self_w2.data(), E->self_w2.size() * sizeof(double), sm);
  copy_h2d(ctx, E->d_sumw, E->sum_w.data(), E->sum_w.size() * sizeof(double), sm);
  std::vector<int> all(K);
  std::iota(all.begin(), all.end(), 0);
  copy_h2d(ctx, E->d_sel, all.data(), K * sizeof(int), sm);
  CRAB_CUDA_CHECK(cudaStreamSynchronize(sm));
  return E;
}

static void ensemble_launch_curves(EnsemblePlan& E, int Ksel) {
  crab_ctx* ctx = E.ctx;
  k_ens_curves<<<dim3(Ksel, E.n_cand), 128, 0, ctx->stream>>>(E.d_partials, E.d_sel, E.d_q, (int)E.nq, E.T, E.d_amp,
                                                             E.d_self, E.d_sumw, Ksel, E.d_curves);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 1;
}

static size_t weights_smem(int K, int64_t nq) {
  return (ew_doubles(K, (int)nq) + (ew_on_chip(K, (int)nq) ? (size_t)K * nq : 0)) * sizeof(double);
}

// Cluster of the reweighting: one CTA (or eight that search step lengths) while
// its shared memory holds the curves and the search's buffers, else eight that
// split the curves (1,000 of 20 q, which alone would fit one CTA: 500 steps 14 ms,
// 65 there), unless they are few (20 of 1,200 q: 12 ms, 10 there).
static bool rw_search(int K, int64_t nq) {
  return rw_smem(K, (int)nq, 1) + rw_search_doubles(K, (int)nq) * sizeof(double) <= kEnsSmem;
}
static int rw_cluster(int K, int64_t nq) {
  return rw_on_chip(K, (int)nq, 1) && (K <= 32 || rw_search(K, nq)) ? 1 : kRwCluster;
}

static void ensemble_fit_buffers(EnsemblePlan& E, const double* y, const double* sg) {
  crab_ctx* ctx = E.ctx;
  // shared-memory opt-in of both kernels, done before any graph capture
  require(weights_smem(E.K, E.nq) <= kEnsSmem && rw_smem(E.K, (int)E.nq, rw_cluster(E.K, E.nq)) <= kEnsSmem,
          "ensemble too large for the on-chip weight fit");
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_ens_weights, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEnsSmem));
  constexpr auto smem_max = cudaFuncAttributeMaxDynamicSharedMemorySize;
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_ens_reweight<1, 1>, smem_max, (int)kEnsSmem));
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_ens_reweight<1, kRwCluster>, smem_max, (int)kEnsSmem));
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_ens_reweight<kRwCluster, 1>, smem_max, (int)kEnsSmem));
  if (!E.d_y) {
    E.d_y = E.alloc<double>(E.nq);
    E.d_sg = E.alloc<double>(E.nq);
    E.d_weights = E.alloc<double>((size_t)E.n_cand * E.K);
    E.d_gradw = E.alloc<double>((size_t)E.n_cand * E.K);
    E.d_fit = E.alloc<double>((size_t)4 * E.n_cand);
    E.d_fitted = E.alloc<double>((size_t)E.n_cand * E.nq);
    E.d_wkl = E.alloc<double>(E.K);
    E.d_out = E.alloc<double>(16);
  }
  copy_h2d(ctx, E.d_y, y, E.nq * sizeof(double), ctx->stream);
  copy_h2d(ctx, E.d_sg, sg, E.nq * sizeof(double), ctx->stream);
}

// fit_core (ensemble.rs:234-299) on the selected conformers, all on the device.
static void ensemble_launch_fit(EnsemblePlan& E, int Ksel, const EnsOpts& eo, const RwOpts* ro) {
  crab_ctx* ctx = E.ctx;
  cudaStream_t sm = ctx->stream;
  ensemble_launch_curves(E, Ksel);
  const size_t shm = weights_smem(Ksel, E.nq);
  k_ens_weights<<<E.n_cand, kWT, shm, sm>>>(E.d_curves, Ksel, (int)E.nq, E.d_y, E.d_sg, eo, E.d_weights, E.d_fit,
                                            E.d_fitted, E.d_gradw);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 1;
  if (ro) {
    k_ens_dcurves<<<dim3(Ksel, 2 * E.n_cand), 128, 0, sm>>>(E.d_partials, E.d_sel, E.d_q, (int)E.nq, E.T, E.d_amp,
                                                           E.d_damp, E.d_self, E.d_sumw, Ksel, E.d_curves,
                                                           E.d_dcurves);
    CRAB_CUDA_CHECK(cudaGetLastError());
    const int cl = rw_cluster(Ksel, E.nq);
    size_t shr = rw_smem(Ksel, (int)E.nq, cl);
    const bool search = cl == 1 && rw_search(Ksel, E.nq);
    if (search) shr += rw_search_doubles(Ksel, (int)E.nq) * sizeof(double);
    auto* go = cl > 1 ? launch_reweight<kRwCluster, 1> : search ? launch_reweight<1, kRwCluster> : launch_reweight<1, 1>;
    go(sm, shr, E.d_curves, E.d_fit, E.n_cand, Ksel, (int)E.nq, E.d_y, E.d_sg, E.d_weights, E.d_dcurves, *ro, E.d_wkl,
       E.d_out);
    CRAB_CUDA_CHECK(cudaGetLastError());
    ctx->launches += 2;
  }
}

// The full scoring pass of a plan as one CUDA graph: pair sums of every
// conformer, curves at every candidate, weight fits, ∂χ²/∂(c1,c2), KL
// reweighting.  Captured on first use and replayed while the options and the
// wait budget, which its nodes hold, stay the same.
static void ensemble_graph_launch(EnsemblePlan& E, const EnsOpts& eo, const RwOpts& ro) {
  crab_ctx* ctx = E.ctx;
  if (!E.graph || E.graph_k != E.K || E.graph_budget != ctx->wait_budget || !(E.graph_fit == eo) ||
      !(E.graph_reweight == ro)) {
    if (E.graph) {
      cudaGraphExecDestroy(E.graph);
      E.graph = nullptr;
    }
    cudaGraph_t g = nullptr;
    const int64_t before = ctx->launches;
    CRAB_CUDA_CHECK(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    try {
      if (E.pair) pair_plan_launch(ctx, *E.pair, ctx->stream, false);
      ensemble_launch_fit(E, E.K, eo, &ro);
    } catch (...) {
      cudaStreamEndCapture(ctx->stream, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    CRAB_CUDA_CHECK(cudaStreamEndCapture(ctx->stream, &g));
    CRAB_CUDA_CHECK(cudaGraphInstantiate(&E.graph, g, 0));
    cudaGraphDestroy(g);
    E.graph_k = E.K;
    E.graph_budget = ctx->wait_budget;
    E.graph_fit = eo;
    E.graph_reweight = ro;
    E.graph_kernels = ctx->launches - before;  // kernels recorded into the graph
    ctx->launches = before;
  }
  CRAB_CUDA_CHECK(cudaGraphLaunch(E.graph, ctx->stream));
  ctx->launches += E.graph_kernels;
}

// Throws when a wait of the plan's pair kernel ran out; waits for the pair sums.
static void check_pair_status(EnsemblePlan& E) {
  if (!E.pair) return;
  int status = 0;
  copy_d2h(E.ctx, &status, E.pair->d_status, sizeof(int), E.ctx->stream);
  CRAB_CUDA_CHECK(cudaStreamSynchronize(E.ctx->stream));
  if (status) throw Error(status, "pair kernel: a bounded wait on a j-tile copy ran out");
}

static EnsOpts ens_opts(const crab_fit_options* fo, bool uniform, double reg) {
  EnsOpts o;
  o.scale_mode = fo ? fo->scale_mode : CRAB_SCALE_FIT;
  o.bg_mode = fo ? fo->bg_mode : CRAB_BG_FIT;
  o.scale_value = fo ? fo->scale_value : 0.0;
  o.bg_value = fo ? fo->bg_value : 0.0;
  o.uniform = uniform ? 1 : 0;
  o.regularization = reg;
  return o;
}

}  // namespace crab

using namespace crab;

struct crab_ensemble_plan {
  std::unique_ptr<crab::EnsemblePlan> plan;
};

extern "C" {

int crab_ensemble_curves(crab_ctx* ctx, crab_struct* const* structures, int32_t k, const double* q, int64_t nq,
                         const crab_solvent* solvent, int implicit_hydrogen, const double* cand, int32_t n_cand,
                         double* curves) {
  if (!ctx || !structures || k <= 0 || !q || nq <= 0 || !solvent || !cand || n_cand <= 0 || !curves)
    return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() {
    validate_q(q, nq);
    validate_solvent(*solvent);
    auto E = make_ensemble_plan(ctx, structures, k, q, nq, *solvent, implicit_hydrogen != 0, cand, n_cand);
    pair_plan_launch(ctx, *E->pair, ctx->stream, false);
    ensemble_launch_curves(*E, k);
    check_pair_status(*E);
    copy_d2h(ctx, curves, E->d_curves, (size_t)n_cand * k * nq * sizeof(double), ctx->stream);
    CRAB_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
  });
}

int crab_ensemble_plan_create(crab_ctx* ctx, crab_struct* const* structures, int32_t k, const double* q, int64_t nq,
                              const crab_solvent* solvent, int implicit_hydrogen, const double* cand, int32_t n_cand,
                              crab_ensemble_plan** out) {
  if (!ctx || !structures || k <= 0 || !q || nq <= 0 || !solvent || !cand || n_cand <= 0 || !out) return CRAB_EINVAL;
  *out = nullptr;
  return guarded_impl(ctx, [&]() {
    validate_q(q, nq);
    validate_solvent(*solvent);
    crab_ensemble_plan* p = new crab_ensemble_plan();
    p->plan = make_ensemble_plan(ctx, structures, k, q, nq, *solvent, implicit_hydrogen != 0, cand, n_cand);
    *out = p;
  });
}

int crab_ensemble_plan_autotune(crab_ctx* ctx, crab_ensemble_plan* plan, int32_t* chosen) {
  if (!ctx || !plan) return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() {
    if (plan->plan->graph) {  // first: the tuner frees tables that it holds, also where it fails later
      cudaGraphExecDestroy(plan->plan->graph);
      plan->plan->graph = nullptr;
    }
    const int c = pair_plan_autotune(ctx, *plan->plan->pair, nullptr, nullptr, 0, nullptr);
    if (chosen) *chosen = c;
  });
}

int crab_ensemble_plan_score(crab_ctx* ctx, crab_ensemble_plan* plan, const double* y, const double* sigma,
                             const crab_fit_options* fopt, const crab_reweight_options* ropt, double* elapsed_ms,
                             double* best_fit, double* weights, double* grad_w, double* kl_weights,
                             double* reweight_out) {
  if (!ctx || !plan || !y || !sigma) return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() {
    EnsemblePlan& E = *plan->plan;
    for (int64_t p = 0; p < E.nq; ++p)
      require(std::isfinite(y[p]) && std::isfinite(sigma[p]) && sigma[p] > 0.0, "invalid experimental curve");
    ensemble_fit_buffers(E, y, sigma);
    const EnsOpts eo = ens_opts(fopt, false, 0.0);
    RwOpts ro{1.0, 0.5, 1e-8, 1e-10, 500, CRAB_SCALE_FIT, CRAB_BG_FIT, 0.0, 0.0};
    if (ropt) {
      ro = RwOpts{ropt->kl_strength, ropt->step_size, ropt->tolerance, ropt->min_weight, ropt->max_iterations,
                  ropt->scale_mode, ropt->bg_mode, ropt->scale_value, ropt->bg_value};
      require(ro.max_iter > 0 && ro.step > 0.0 && ro.tol > 0.0 && ro.floor >= 0.0 && ro.floor * E.K < 1.0 &&
                  ro.kl >= 0.0,
              "maximum-entropy options are invalid");
    }
    CRAB_CUDA_CHECK(cudaEventRecord(ctx->ev_start, ctx->stream));
    ensemble_graph_launch(E, eo, ro);
    CRAB_CUDA_CHECK(cudaEventRecord(ctx->ev_stop, ctx->stream));
    std::vector<double> fit((size_t)4 * E.n_cand), out(16);
    copy_d2h(ctx, fit.data(), E.d_fit, fit.size() * sizeof(double), ctx->stream);
    copy_d2h(ctx, out.data(), E.d_out, 9 * sizeof(double), ctx->stream);
    CRAB_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    float ms = 0.0f;
    CRAB_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
    check_pair_status(E);
    if (elapsed_ms) *elapsed_ms = ms;
    const int best = (int)out[0];
    if (best_fit) {
      best_fit[0] = best;
      best_fit[1] = E.cand[2 * best];
      best_fit[2] = E.cand[2 * best + 1];
      best_fit[3] = fit[4 * best];
      best_fit[4] = fit[4 * best + 1];
      best_fit[5] = fit[4 * best + 2];
      best_fit[6] = out[7];
      best_fit[7] = out[8];
    }
    if (weights) copy_d2h(ctx, weights, E.d_weights + (size_t)best * E.K, E.K * sizeof(double), ctx->stream);
    if (grad_w) copy_d2h(ctx, grad_w, E.d_gradw + (size_t)best * E.K, E.K * sizeof(double), ctx->stream);
    if (kl_weights) copy_d2h(ctx, kl_weights, E.d_wkl, E.K * sizeof(double), ctx->stream);
    if (reweight_out)
      for (int i = 0; i < 6; ++i) reweight_out[i] = out[1 + i];
    CRAB_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
  });
}

int crab_ensemble_plan_destroy(crab_ensemble_plan* plan) {
  if (!plan) return CRAB_OK;
  if (plan->plan && plan->plan->ctx) cudaSetDevice(plan->plan->ctx->device);
  delete plan;
  return CRAB_OK;
}

}  // extern "C"

// ensemble.rs:302-315: the 5 x 5 (c1, c2) candidate grid.
static std::vector<double> fit_candidates(const crab_fit_options* fopt) {
  std::vector<double> cand;
  for (int i = 0; i < 5; ++i)
    for (int j = 0; j < 5; ++j) {
      cand.push_back(fopt->c1_lo + (fopt->c1_hi - fopt->c1_lo) * (double)i / 4.0);
      cand.push_back(fopt->c2_lo + (fopt->c2_hi - fopt->c2_lo) * (double)j / 4.0);
    }
  return cand;
}

static void check_ensemble_inputs(const crab_ensemble_options& eo, const double* y, const double* sigma, int64_t nq) {
  require(std::isfinite(eo.regularization) && eo.regularization >= 0.0 && std::isfinite(eo.min_weight) &&
              eo.min_weight >= 0.0 && eo.min_weight <= 1.0 && eo.max_conformers >= 0 && eo.bootstrap >= 0,
          "ensemble regularization and pruning options are invalid");
  for (int64_t p = 0; p < nq; ++p)
    require(std::isfinite(y[p]) && std::isfinite(sigma[p]) && sigma[p] > 0.0, "invalid experimental curve");
}

// EnsembleFitter::fit (ensemble.rs:127-232) once the pair sums are on the
// device: fit_core for every pruning round, the optional residual
// bootstrap, and the outputs.
static void ensemble_fit_rounds(crab_ctx* ctx, std::unique_ptr<EnsemblePlan>& E, const std::vector<double>& cand,
                                const double* y, const double* sigma, int64_t nq, const crab_ensemble_options& eo,
                                const crab_fit_options* fopt, crab_ensemble_result* result, int32_t* selected_out,
                                double* weights_out, double* fitted_out, double* intervals_out,
                                double* bootstrap_chi2_out) {
  ensemble_fit_buffers(*E, y, sigma);
  const EnsOpts o = ens_opts(fopt, eo.uniform || !eo.fit_weights, eo.regularization);
  struct Core {
    std::vector<double> w, fitted;
    double scale, bg, chi2, c1, c2;
  };
  auto fit_core = [&](const std::vector<int>& sel, const double* yy) {
    copy_h2d(ctx, E->d_sel, sel.data(), sel.size() * sizeof(int), ctx->stream);
    copy_h2d(ctx, E->d_y, yy, nq * sizeof(double), ctx->stream);
    ensemble_launch_fit(*E, (int)sel.size(), o, nullptr);
    std::vector<double> fit(4 * 25);
    copy_d2h(ctx, fit.data(), E->d_fit, fit.size() * sizeof(double), ctx->stream);
    CRAB_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    int best = 0;
    for (int c = 1; c < 25; ++c)
      if (fit[4 * c + 2] < fit[4 * best + 2]) best = c;
    Core core;
    core.w.resize(sel.size());
    core.fitted.resize(nq);
    copy_d2h(ctx, core.w.data(), E->d_weights + (size_t)best * sel.size(), sel.size() * sizeof(double), ctx->stream);
    copy_d2h(ctx, core.fitted.data(), E->d_fitted + (size_t)best * nq, nq * sizeof(double), ctx->stream);
    CRAB_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    core.scale = fit[4 * best];
    core.bg = fit[4 * best + 1];
    core.chi2 = fit[4 * best + 2];
    core.c1 = cand[2 * best];
    core.c2 = cand[2 * best + 1];
    return core;
  };
  std::vector<int> selected(E->K);
  std::iota(selected.begin(), selected.end(), 0);
  Core core = fit_core(selected, y);
  for (bool changed = true; changed;) {
    changed = false;
    std::vector<int> keep;
    for (size_t i = 0; i < selected.size(); ++i)
      if (core.w[i] + 1e-12 >= eo.min_weight) keep.push_back(selected[i]);
    if (keep.empty())
      keep.push_back(selected[std::max_element(core.w.begin(), core.w.end()) - core.w.begin()]);
    if (eo.max_conformers > 0 && (int)keep.size() > eo.max_conformers) {
      std::vector<std::pair<double, int>> ranked;
      for (size_t i = 0; i < selected.size(); ++i) ranked.push_back({core.w[i], selected[i]});
      std::stable_sort(ranked.begin(), ranked.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
      keep.clear();
      for (int i = 0; i < eo.max_conformers; ++i) keep.push_back(ranked[i].second);
    }
    std::sort(keep.begin(), keep.end());
    if (keep != selected) {
      selected = keep;
      core = fit_core(selected, y);
      changed = true;
    }
  }
  // weight intervals from a residual bootstrap (ensemble.rs:174-216); the
  // resampling indices come from a seeded std::mt19937_64 stream (the
  // reference draws them from ChaCha8, so individual replicates differ)
  const size_t ns = selected.size();
  std::vector<std::vector<double>> samples(ns);
  if (eo.bootstrap > 0) {
    std::mt19937_64 rng(eo.seed);
    std::vector<double> resid(nq), synth(nq);
    for (int64_t p = 0; p < nq; ++p) resid[p] = (y[p] - core.fitted[p]) / sigma[p];
    for (int b = 0; b < eo.bootstrap; ++b) {
      for (int64_t p = 0; p < nq; ++p) synth[p] = core.fitted[p] + resid[rng() % (uint64_t)nq] * sigma[p];
      Core rep = fit_core(selected, synth.data());
      for (size_t i = 0; i < ns; ++i) samples[i].push_back(rep.w[i]);
      if (bootstrap_chi2_out) bootstrap_chi2_out[b] = rep.chi2;
    }
    copy_h2d(ctx, E->d_y, y, nq * sizeof(double), ctx->stream);
  }
  if (intervals_out) {
    auto quantile = [](const std::vector<double>& v, double prob) {
      const double pos = std::min(std::max(prob, 0.0), 1.0) * (double)(v.size() - 1);
      const size_t lo = (size_t)std::floor(pos), hi = (size_t)std::ceil(pos);
      return v[lo] + (v[hi] - v[lo]) * (pos - (double)lo);
    };
    for (size_t i = 0; i < ns; ++i) {
      if (eo.bootstrap > 0) {
        std::sort(samples[i].begin(), samples[i].end());
        intervals_out[3 * i] = quantile(samples[i], 0.5);
        intervals_out[3 * i + 1] = quantile(samples[i], 0.025);
        intervals_out[3 * i + 2] = quantile(samples[i], 0.975);
      } else {
        intervals_out[3 * i] = intervals_out[3 * i + 1] = intervals_out[3 * i + 2] = core.w[i];
      }
    }
  }
  const double dof = (double)std::max<int64_t>(nq - 1, 1);
  result->scale = core.scale;
  result->background = core.bg;
  result->c1 = core.c1;
  result->c2 = core.c2;
  result->reduced_chi2 = core.chi2;
  result->chi2 = core.chi2 * dof;
  result->iterations = 250;
  result->n_selected = (int)selected.size();
  if (selected_out)
    for (size_t i = 0; i < selected.size(); ++i) selected_out[i] = selected[i];
  if (weights_out) std::copy(core.w.begin(), core.w.end(), weights_out);
  if (fitted_out) std::copy(core.fitted.begin(), core.fitted.end(), fitted_out);
}

extern "C" {

// EnsembleFitter::fit (ensemble.rs:127-232): partials once, fit_core on the
// device for every pruning round, optional residual bootstrap.
int crab_ensemble_fit(crab_ctx* ctx, crab_struct* const* structures, int32_t k, const double* q, const double* y,
                      const double* sigma, int64_t nq, const crab_ensemble_options* eopt, const crab_fit_options* fopt,
                      crab_ensemble_result* result, int32_t* selected_out, double* weights_out, double* fitted_out,
                      double* intervals_out, double* bootstrap_chi2_out) {
  if (!ctx || !structures || k <= 0 || !q || !y || !sigma || nq <= 0 || !eopt || !fopt || !result) return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() {
    validate_q(q, nq);
    validate_solvent(fopt->solvent);
    check_ensemble_inputs(*eopt, y, sigma, nq);
    const std::vector<double> cand = fit_candidates(fopt);
    auto E = make_ensemble_plan(ctx, structures, k, q, nq, fopt->solvent, fopt->implicit_hydrogen != 0, cand.data(), 25);
    pair_plan_launch(ctx, *E->pair, ctx->stream, false);
    check_pair_status(*E);
    ensemble_fit_rounds(ctx, E, cand, y, sigma, nq, *eopt, fopt, result, selected_out, weights_out, fitted_out,
                        intervals_out, bootstrap_chi2_out);
  });
}

int crab_ensemble_partials(crab_ctx* ctx, crab_struct* const* structures, int32_t k, const double* q, int64_t nq,
                           int implicit_hydrogen, int shard, int n_shards, int32_t* n_types, double* out,
                           int64_t capacity) {
  if (!ctx || !structures || k <= 0 || !q || nq <= 0 || !n_types || n_shards < 1 || shard < 0 || shard >= n_shards)
    return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() {
    validate_q(q, nq);
    require(k <= kMaxK, "ensemble size must be between 1 and 1024");
    const bool implicit = implicit_hydrogen != 0;
    const std::map<AtomClass, int> index = ensemble_class_index(structures, k, implicit);
    const int T = (int)index.size();
    *n_types = T;
    if (!out) return;
    const size_t P = (size_t)(T * (T + 1) / 2), block = partials_block(T, nq);
    if (capacity < 0 || (uint64_t)capacity < block * (size_t)k) throw Error(CRAB_ECAPACITY, "partials buffer too small");
    std::fill(out, out + block * (size_t)k, 0.0);
    // conformers longest first by N², then the greedy owners
    std::vector<int> order(k);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return structures[a]->n > structures[b]->n; });
    std::vector<int64_t> cost(k);
    for (int i = 0; i < k; ++i) cost[i] = structures[order[i]]->n * structures[order[i]]->n;
    const std::vector<int32_t> owner = shard_owners(cost.data(), k, n_shards);
    std::vector<int> mine;
    for (int i = 0; i < k; ++i)
      if (owner[i] == shard) mine.push_back(order[i]);
    std::sort(mine.begin(), mine.end());
    if (mine.empty()) return;
    std::vector<Layout> parts;
    for (int c : mine) {
      const crab_struct* st = structures[c];
      const std::vector<int32_t> type = conformer_types(st, index, implicit);
      parts.push_back(build_layout(st->xyz.data(), st->occ.data(), type.data(), st->n, T, false));
      double* b = out + (size_t)c * block;
      for (int a = 0; a < T; ++a) {
        b[P * nq + a] = parts.back().self_w2[a];
        b[P * nq + T + a] = parts.back().sum_w[a];
      }
    }
    auto plan = make_batch_pair_plan(ctx, std::move(parts), q, nq);
    pair_plan_launch(ctx, *plan, ctx->stream, false);
    std::vector<double> raw(mine.size() * P * (size_t)nq);
    int status = 0;
    copy_d2h(ctx, raw.data(), plan->d_out, raw.size() * sizeof(double), ctx->stream);
    copy_d2h(ctx, &status, plan->d_status, sizeof(int), ctx->stream);
    CRAB_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    if (status) throw Error(status, "pair kernel: a bounded wait on a j-tile copy ran out");
    for (size_t i = 0; i < mine.size(); ++i)
      std::copy(raw.begin() + i * P * nq, raw.begin() + (i + 1) * P * nq, out + (size_t)mine[i] * block);
  });
}

int crab_ensemble_fit_partials(crab_ctx* ctx, crab_struct* const* structures, int32_t k, const double* q,
                               const double* y, const double* sigma, int64_t nq, const crab_ensemble_options* eopt,
                               const crab_fit_options* fopt, const double* partials, int32_t n_types,
                               crab_ensemble_result* result, int32_t* selected_out, double* weights_out,
                               double* fitted_out, double* intervals_out, double* bootstrap_chi2_out) {
  if (!ctx || !structures || k <= 0 || !q || !y || !sigma || nq <= 0 || !eopt || !fopt || !partials || !result)
    return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() {
    validate_q(q, nq);
    validate_solvent(fopt->solvent);
    check_ensemble_inputs(*eopt, y, sigma, nq);
    require((int)ensemble_class_index(structures, k, fopt->implicit_hydrogen != 0).size() == n_types,
            "partials were computed for another set of atom types");
    const std::vector<double> cand = fit_candidates(fopt);
    auto E = make_ensemble_plan(ctx, structures, k, q, nq, fopt->solvent, fopt->implicit_hydrogen != 0, cand.data(), 25,
                                partials);
    ensemble_fit_rounds(ctx, E, cand, y, sigma, nq, *eopt, fopt, result, selected_out, weights_out, fitted_out,
                        intervals_out, bootstrap_chi2_out);
  });
}

}  // extern "C"
