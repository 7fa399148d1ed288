// Coordinate pair-distance distribution P(r) (crabSAXS src/metrics.rs:475-541).
//
// The reference takes dmax as the square root of the largest squared pair
// distance d2 = dx*dx + dy*dy + dz*dz (f64, left to right), sets
// step = dmax / bins, and adds w_i*w_j for every pair i < j to bin
// min(floor(sqrt(d2) / step), bins - 1).  On the device:
//
//   k_pr_far     farthest atom from the first one, then from that one: a pair,
//                whose distance bounds dmax from below; then the largest
//                distance R of an atom from the pair's middle, and from where
//                Ritter's sphere moves it to
//   k_pr_rim     the atoms that can belong to a longer pair: an atom at distance
//                d from the centre is in no pair longer than d + R
//   k_pr_dmax    the exact f64 maximum of d2 over the pairs of those (a few per
//                cent of a globule's atoms)
//   k_pr_edges   per bin k the smallest f64 d2 that the reference's
//                floor(sqrt(d2) / step) maps to k or above: a binary search
//                over the bit patterns of non-negative doubles, with the same
//                IEEE-rounded sqrt and division.  A pair's bin is the number
//                of edges at or below its d2
//   k_pr_place   the atoms of each weight class into its tiles, centred, in
//                units of the step, FP32
//   k_pr_count   (up to 64 distinct weights) per pair the bin coordinate
//                x = r / step from those.  When x is farther than a proven error
//                bound delta from every integer, floor(x) is the reference's
//                bin, counted in shared memory per class pair; otherwise (about
//                2*delta of the pairs) the pair goes to its warp's queue, and 32
//                of them at a time are placed by their f64 d2, computed with the
//                reference's operation order (no fused multiply-add), against
//                the exact edges
//   k_pr_hist    (more weights) the same per tile of spatially ordered atoms,
//                adding the f64 products w_i*w_j to per-warp shared histograms,
//                or, with very many bins, to a row per block in device memory
//   k_pr_combine hist[k] = Σ over class pairs (in order) of count * w_a * w_b
//   k_pr_reduce  (weighted modes) the per-block rows summed in block order
//
// k_pr_count's bound is instruction issue.  The tiles' four i atoms a lane are
// held doubled, so that one packed f32x2 instruction serves two j atoms as they
// lie; the counters of a bin are 32 words, one a lane (4 with over 1,500 bins),
// so that neighbouring atoms, whose distances to one j atom fall into the same
// bins, never meet in a word.
// 100,000 atoms, 160 bins: 5.0e9 pairs in 2.94 ms (1.70e12 a second, issue slots
// 79 % busy, 17 instructions a pair), where one i atom a thread, a copy of the
// counters per warp and a branch around each near-edge pair took 5.4 ms (23
// instructions a pair).  The call went from 10.3 to 3.6 ms: dmax takes 0.1 ms
// (0.9 ms over spatially ordered tiles), the order itself and the packing of the
// tiles, 3.6 ms of host work, are gone.

#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "device_math.cuh"
#include "engine.hpp"
#include "ops.hpp"
#include "tile_rows.cuh"

namespace crab {
namespace {

constexpr int kPrThreads = kTile;         // one i atom per thread
constexpr size_t kPrDynSmem = 96 * 1024;  // edges + histograms
constexpr int64_t kPrMaxBins = 1 << 24;
constexpr int kPrMaxClasses = 64;                 // weight classes for integer counting
constexpr size_t kPrMaxCountBytes = 256u << 20;   // u64 counts [class pairs][bins]
constexpr int kPrFlushItems = 1 << 18;            // u32 counters: units of 8192 pairs between flushes

enum PrMode { kPrCounts = 0, kPrWeighted = 1, kPrWeightedGlobal = 2 };

struct PrParams {
  double step;
  float inv_step;
  float delta;     // bound on |x_fp32 - x_exact| in bins; FLT_MAX: always exact
  int degenerate;  // every pair distance is zero: no histogram
  int pad;
};

__device__ __forceinline__ double pr_sqdist(const double4& a, const double4& b) {
  const double dx = __dsub_rn(a.x, b.x), dy = __dsub_rn(a.y, b.y), dz = __dsub_rn(a.z, b.z);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Work item w of the upper triangle of tile pairs, column-major: (a, b), a <= b.
__device__ __forceinline__ void pr_tri_decode(int64_t w, int& a, int& b) {
  int64_t bb = (int64_t)((sqrt(8.0 * (double)w + 1.0) - 1.0) * 0.5);
  while (bb > 0 && bb * (bb + 1) / 2 > w) --bb;
  while ((bb + 1) * (bb + 2) / 2 <= w) ++bb;
  b = (int)bb;
  a = (int)(w - bb * (bb + 1) / 2);
}

constexpr int kPrFarBlocks = 148;
constexpr int kPrMaxSteps = 5;
constexpr int64_t kPrEvery = 4096;  // atoms up to which every pair is looked at for the longest
struct PrFar {  // of a block: largest squared distance and its atom
  double d2;
  long long at;
};

__device__ __forceinline__ double pr_sqdist3(const double* a, const double* b) {
  const double dx = __dsub_rn(a[0], b[0]), dy = __dsub_rn(a[1], b[1]), dz = __dsub_rn(a[2], b[2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// The farther of two, the lower atom among equals.
__device__ __forceinline__ PrFar pr_farther(const PrFar& a, const PrFar& b) {
  return b.d2 > a.d2 || (b.d2 == a.d2 && b.at < a.at) ? b : a;
}
__device__ __forceinline__ PrFar pr_block_far(PrFar v, PrFar* red) {
  for (int o = 16; o > 0; o >>= 1) {
    PrFar w;
    w.d2 = __shfl_xor_sync(0xffffffffu, v.d2, o);
    w.at = __shfl_xor_sync(0xffffffffu, v.at, o);
    v = pr_farther(v, w);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int k = 1; k < (int)(blockDim.x >> 5); ++k) v = pr_farther(v, red[k]);
  return v;
}

// The farthest atom that step k found; `steps` holds the steps' results, one
// run of kPrFarBlocks after the other.
__device__ __forceinline__ PrFar pr_step_far(const PrFar* __restrict__ steps, int k, PrFar* red) {
  PrFar v{-1.0, 0};
  for (int i = threadIdx.x; i < kPrFarBlocks; i += blockDim.x) v = pr_farther(v, steps[k * kPrFarBlocks + i]);
  return pr_block_far(v, red);
}

// Centre of step `step` (2 or more): the middle of the pair of steps 0 and 1,
// moved towards the farthest atom of each step between as far as a ball needs
// that covers the pair, or the last ball, and that atom (Ritter's sphere).
__device__ __forceinline__ void pr_centre(const double* __restrict__ xyz, const PrFar* __restrict__ steps, int step,
                                          PrFar* red, double (&c)[3]) {
  const PrFar e0 = pr_step_far(steps, 0, red), e1 = pr_step_far(steps, 1, red);
  for (int d = 0; d < 3; ++d) c[d] = 0.5 * (xyz[3 * e0.at + d] + xyz[3 * e1.at + d]);
  double r = 0.5 * sqrt(e1.d2);
  for (int k = 2; k < step; ++k) {
    const PrFar f = pr_step_far(steps, k, red);
    const double R = sqrt(f.d2);
    if (R > r) {
      const double move = 0.5 * (R - r) / R;
      for (int d = 0; d < 3; ++d) c[d] += move * (xyz[3 * f.at + d] - c[d]);
      r = 0.5 * (R + r);
    }
  }
}

// far[block]: the farthest atom from atom 0 (step 0), from the farthest of
// step 0 (step 1), or from the step's centre (the given one, if it is given).
// Step 0 also flags a coordinate that is not finite or 1e100 and over.
__global__ void __launch_bounds__(256) k_pr_far(const double* __restrict__ xyz, int64_t n, int step, int given,
                                                const double* __restrict__ centre, PrFar* __restrict__ steps,
                                                unsigned* __restrict__ invalid) {
  __shared__ PrFar red[8];
  double base[3] = {xyz[0], xyz[1], xyz[2]};
  if (step == 1) {
    const int64_t at = pr_step_far(steps, 0, red).at;
    for (int d = 0; d < 3; ++d) base[d] = xyz[3 * at + d];
  } else if (step > 1 && given) {
    for (int d = 0; d < 3; ++d) base[d] = centre[d];
  } else if (step > 1) {
    pr_centre(xyz, steps, step, red, base);
  }
  PrFar v{-1.0, 0};
  bool fine = true;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* p = xyz + 3 * i;
    if (step == 0) fine = fine && fabs(p[0]) < 1e100 && fabs(p[1]) < 1e100 && fabs(p[2]) < 1e100;
    v = pr_farther(v, PrFar{pr_sqdist3(base, p), (long long)i});
  }
  if (!fine) *invalid = 1u;
  v = pr_block_far(v, red);
  if (threadIdx.x == 0) steps[step * kPrFarBlocks + blockIdx.x] = v;
}

// count, then list: the atoms that may belong to a pair at least as long as
// the known one, from the step (2 .. n_steps - 1) whose centre has the atoms
// nearest; radius[0]: the largest distance R from it.  Distances are f64 with
// relative errors below 1e-14; 1e-9 of R covers them.
__global__ void __launch_bounds__(256) k_pr_rim(const double* __restrict__ xyz, int64_t n, int n_steps, int given,
                                                const PrFar* __restrict__ steps, double* __restrict__ centre,
                                                int* __restrict__ list,
                                                unsigned* __restrict__ count, unsigned long long* __restrict__ dmax2,
                                                double* __restrict__ radius) {
  __shared__ PrFar red[8];
  const PrFar v = pr_step_far(steps, 1, red);
  int use = 2;
  double r2 = pr_step_far(steps, 2, red).d2;
  for (int k = 3; k < n_steps; ++k) {
    const double k2 = pr_step_far(steps, k, red).d2;
    if (k2 < r2) {
      r2 = k2;
      use = k;
    }
  }
  double c[3];
  if (given)
    for (int d = 0; d < 3; ++d) c[d] = centre[d];
  else
    pr_centre(xyz, steps, use, red, c);
  const double R = sqrt(r2);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *radius = R;
    if (!given)
      for (int d = 0; d < 3; ++d) centre[d] = c[d];
    atomicMax(dmax2, (unsigned long long)__double_as_longlong(v.d2));
  }
  const double least = sqrt(v.d2) - R * (1.0 + 1e-9);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (sqrt(pr_sqdist3(c, xyz + 3 * i)) >= least) list[atomicAdd(count, 1u)] = (int)i;
}

// The f64 maximum of d2 over the listed atoms' pairs, tile pairs taken in turn.
// FP32 first: with coordinates from the centre, each within R, a squared
// distance (at most 4 R²) is off by less than 2^-20 R² x 4, and pairs that are
// below the longest known one by 1e-5 R² are left out; eight at a time, so that
// an f64 pair (a few in a million) costs no branch per pair.  With eleven f64
// instructions a pair and the first pair's middle as the centre, 100,000 atoms
// of a ball took 60 to 470 us, depending on the first pair; so 66 where they
// took 470.
__global__ void __launch_bounds__(kPrThreads)
    k_pr_dmax(const double* __restrict__ xyz, const int* __restrict__ list, const unsigned* __restrict__ count,
              const double* __restrict__ centre, const double* __restrict__ radius, unsigned long long* out) {
  __shared__ double sj[3][kPrThreads];
  __shared__ float4 fj[kPrThreads];
  const int m = (int)*count, tid = threadIdx.x;
  const int64_t nt = (m + kPrThreads - 1) / kPrThreads, n_work = nt * (nt + 1) / 2;
  const double c[3] = {centre[0], centre[1], centre[2]}, R = *radius;
  auto atom = [&](int k) { return list ? (int64_t)list[k] : (int64_t)k; };  // no list: every atom
  const bool narrow = R > 1e-15 && R < 1e15;  // squares well inside FP32's range
  double best = 0.0;
  for (int64_t w = blockIdx.x; w < n_work; w += gridDim.x) {
    int a, b;
    pr_tri_decode(w, a, b);
    const int nb = min(kPrThreads, m - b * kPrThreads), i = a * kPrThreads + tid;
    __syncthreads();
    if (tid < nb) {
      const double* p = xyz + 3 * atom(b * kPrThreads + tid);
      for (int d = 0; d < 3; ++d) sj[d][tid] = p[d];
    }
    // past the end: the last atom again
    {
      const double* p = xyz + 3 * atom(b * kPrThreads + min(tid, nb - 1));
      fj[tid] = make_float4((float)(p[0] - c[0]), (float)(p[1] - c[1]), (float)(p[2] - c[2]), 0.0f);
    }
    __syncthreads();
    if (i < m) {
      const double* p = xyz + 3 * atom(i);
      const double pi[3] = {p[0], p[1], p[2]};
      const float fx = (float)(pi[0] - c[0]), fy = (float)(pi[1] - c[1]), fz = (float)(pi[2] - c[2]);
      const double known = fmax(best, __longlong_as_double((long long)__ldcg(out)));
      const float least = narrow ? (float)(known - 1e-5 * R * R) * (1.0f - 1e-6f) : -1.0f;
      for (int j0 = 0; j0 < nb; j0 += 8) {
        float far = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 f = fj[j0 + j];
          const float dx = fx - f.x, dy = fy - f.y, dz = fz - f.z;
          far = fmaxf(far, fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
        }
        if (far >= least)
          for (int j = j0; j < min(j0 + 8, nb); ++j) {
            const double pj[3] = {sj[0][j], sj[1][j], sj[2][j]};
            best = fmax(best, pr_sqdist3(pi, pj));
          }
      }
    }
    // the next tiles know what this one found
    const double top = __longlong_as_double((long long)__ldcg(out));
    if (best > top) atomicMax(out, (unsigned long long)__double_as_longlong(best));  // non-negative doubles order as their bits
  }
}

// metrics.rs:515-516: floor(sqrt(d2) / step) as usize, capped at bins - 1
// (the cast saturates and sends NaN to 0).
__device__ __forceinline__ int64_t pr_bin_of(double d2, double step, int64_t bins) {
  const double v = floor(sqrt(d2) / step);
  if (!(v >= 0.0)) return 0;
  if (v >= (double)bins) return bins - 1;
  return (int64_t)v < bins - 1 ? (int64_t)v : bins - 1;
}

// rim_radius: the largest distance of an atom from the centre of the FP32
// coordinates.  The kernels take FP32 coordinates scaled by inv_step = fl(1/step)
// and x = sqrt.approx(d2f) in bins.  With
// R = radius / step and d = sqrt(d2) / step, x differs from d by at most
//   sqrt(3) * 2^-22 * R + 11.5 * 2^-24 * d
// (per coordinate the rounding to float and the scaling, 2 * 2^-24 * R each
// side of the difference; the difference, the sum of squares, a 4-ulp
// sqrt.approx and the rounded reciprocal step relative to d).  delta is four
// times that with d <= bins + 1; when delta would exceed a quarter bin, or
// above 2^20 bins, every pair takes the exact path.  So it does where 1/step is
// not a normal FP32 number (steps above 8e37 or below 3e-39): x is then off by
// any factor, and the bin of a counted pair is an address.
__global__ void k_pr_edges(const unsigned long long* __restrict__ dmax2_bits, int64_t bins,
                           const double* __restrict__ rim_radius, const unsigned* __restrict__ invalid,
                           double* __restrict__ edges, PrParams* __restrict__ par) {
  const double radius = *rim_radius * (1.0 + 1e-6) + 1e-30;  // of the FP32 coordinates
  const double dmax2 = __longlong_as_double((long long)*dmax2_bits);
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (!(dmax2 > 0.0) || *invalid) {
    if (k == 0) par->degenerate = 1;
    return;
  }
  const double step = sqrt(dmax2) / (double)bins;
  if (k == 0) {
    par->step = step;
    par->inv_step = (float)fmin(1.0 / step, (double)FLT_MAX);
    const double bound = (1.7320508075688772 * 0x1p-22 * radius / step + 11.5 * 0x1p-24 * (double)(bins + 1));
    par->delta = bins > (1 << 20) ? FLT_MAX : (float)fmin(4.0 * bound, 0.25);
    if (4.0 * bound > 0.25 || !(1.0 / step >= (double)FLT_MIN && 1.0 / step <= (double)FLT_MAX)) par->delta = FLT_MAX;
    par->degenerate = 0;
  }
  if (k > bins) return;
  if (k == 0) { edges[0] = 0.0; return; }
  if (k == bins) { edges[bins] = __longlong_as_double(0x7FF0000000000000ll); return; }
  // smallest d2 with bin >= k: bin(+0) = 0 < k and bin(+inf) = bins - 1 >= k
  unsigned long long lo = 0ull, hi = 0x7FF0000000000000ull;
  while (hi - lo > 1ull) {
    const unsigned long long mid = lo + (hi - lo) / 2;
    if (pr_bin_of(__longlong_as_double((long long)mid), step, bins) >= k) hi = mid;
    else lo = mid;
  }
  edges[k] = __longlong_as_double((long long)hi);
}

__device__ __forceinline__ float pr_sqrt_approx(float v) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// Bin coordinate of a pair from FP32 coordinates already in bins.
__device__ __forceinline__ float pr_bin_coord(const float4& fi, const float4& fj) {
  const float fx = fi.x - fj.x, fy = fi.y - fj.y, fz = fi.z - fj.z;
  return pr_sqrt_approx(fx * fx + fy * fy + fz * fz);
}

// The reference's bin of a pair from its exact f64 d2, starting the search at
// the FP32 estimate x.
__device__ __forceinline__ int pr_exact_bin(const double4& pi, const double4& pj, float x, const double* E, int bins) {
  int e = (int)fminf(fmaxf(x, 0.0f), (float)(bins - 1));
  const double d2 = pr_sqdist(pi, pj);
  while (e + 1 < bins && d2 >= E[e + 1]) ++e;
  while (e > 0 && d2 < E[e]) --e;
  return e;
}

constexpr float kPrMagic = 12582912.0f;  // 1.5 * 2^23: x + kPrMagic holds floor(x) in its low bits
constexpr int kPrMagicBits = 0x4B400000;

// Packed f32x2 arithmetic (two pairs per instruction, each lane rounded as
// the scalar operation).
__device__ __forceinline__ unsigned long long pr_pack(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void pr_unpack(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long pr_sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long pr_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long pr_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long pr_add2_rd(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Two pairs (i, j) and (i, j+1) from the packed j tile: their bin coordinates
// x, x + kPrMagic rounded down (whose bits are kPrMagicBits + floor(x)), and
// whether each is within delta of a bin edge.
struct PrTwo {
  float xa, xb, ta, tb;
  bool edge_a, edge_b;
};
__device__ __forceinline__ PrTwo pr_two(unsigned long long fx2, unsigned long long fy2, unsigned long long fz2,
                                        const float4& xy, const float2& zz, unsigned long long magic2,
                                        unsigned long long half2, float near_edge) {
  const unsigned long long dx = pr_sub2(fx2, pr_pack(xy.x, xy.y));
  const unsigned long long dy = pr_sub2(fy2, pr_pack(xy.z, xy.w));
  const unsigned long long dz = pr_sub2(fz2, pr_pack(zz.x, zz.y));
  const unsigned long long d2 = pr_fma2(dx, dx, pr_fma2(dy, dy, pr_mul2(dz, dz)));
  float d2a, d2b;
  pr_unpack(d2, d2a, d2b);
  PrTwo r;
  r.xa = pr_sqrt_approx(d2a);
  r.xb = pr_sqrt_approx(d2b);
  const unsigned long long x2 = pr_pack(r.xa, r.xb);
  const unsigned long long t2 = pr_add2_rd(x2, magic2);
  const unsigned long long c2 = pr_sub2(pr_sub2(x2, pr_sub2(t2, magic2)), half2);  // frac - 0.5
  float ca, cb;
  pr_unpack(t2, r.ta, r.tb);
  pr_unpack(c2, ca, cb);
  r.edge_a = fabsf(ca) > near_edge;
  r.edge_b = fabsf(cb) > near_edge;
  return r;
}

// ---- counting (few distinct weights) ----
constexpr int kPcT = 1024, kPcWarps = kPcT / 32;
constexpr int kPcQueue = 96;  // near-edge pairs a warp holds: up to 31 left over and 64 new ones
constexpr size_t kPcSmem = 225 * 1024;
__host__ __device__ inline size_t pc_smem(int64_t bins, int columns) {
  return (size_t)(bins + 1) * 8 + (size_t)bins * columns * 4 + (size_t)kPcWarps * kPcQueue * sizeof(int2);
}

// Word of an atom: class << 24 | rank in it.  Writes its scaled FP32
// coordinates into the class's tiles and its index into slot order.
__global__ void k_pr_place(const double* __restrict__ xyz, const uint32_t* __restrict__ word,
                           const int* __restrict__ tile0, int64_t n, const double* __restrict__ centre,
                           const PrParams* __restrict__ par, unsigned char* __restrict__ pts, int* __restrict__ atom) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || par->degenerate) return;
  const double scale = (double)par->inv_step;
  const uint32_t w = word[i], rank = w & 0xffffffu;
  const int64_t tile = tile0[w >> 24] + (rank >> 7);
  const int s = rank & 127, e = s & 63;
  float* c = reinterpret_cast<float*>(pts + (tile * 2 + (s >> 6)) * kHistChunkBytes);
  c[(e >> 1) * 4 + (e & 1)] = (float)((xyz[3 * i] - centre[0]) * scale);
  c[(e >> 1) * 4 + 2 + (e & 1)] = (float)((xyz[3 * i + 1] - centre[1]) * scale);
  c[128 + e] = (float)((xyz[3 * i + 2] - centre[2]) * scale);
  atom[tile * kTile + s] = (int)i;
}

// One warp's near-edge pairs (slots of both atoms), placed 32 at a time.
struct PrQueue {
  int2* q;
  int n;
  const double* xyz;
  const int* atom;
  const double* E;
  unsigned* col;  // this lane's counter of bin 0
  int bins, columns;
  float inv_step;
  __device__ __forceinline__ void place(int k) {
    const double* a = xyz + 3 * (int64_t)atom[q[k].x];
    const double* b = xyz + 3 * (int64_t)atom[q[k].y];
    const double d2 = pr_sqdist3(a, b);
    int e = (int)fminf((float)sqrt(d2) * inv_step, (float)(bins - 1));
    while (e + 1 < bins && d2 >= E[e + 1]) ++e;
    while (e > 0 && d2 < E[e]) --e;
    atomicAdd(col + e * columns, 1u);
  }
  __device__ __forceinline__ void push(bool mine, int i, int j) {
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (mine) q[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = make_int2(i, j);
    n += __popc(m);
    __syncwarp();
    if (n >= 64) drain(32);
  }
  // places the last pairs until fewer than `keep` are left (keep 32), or all (keep 1)
  __device__ __forceinline__ void drain(int keep) {
    const int lane = threadIdx.x & 31;
    while (n >= keep) {
      const int take = min(n, 32);
      if (lane < take) place(n - take + lane);
      n -= take;
      __syncwarp();
    }
  }
};

// The NI groups of 32 i atoms from slot i0 on against nj atoms of a half tile
// (slots j0 on, jslot in the tile); DIAG: one tile with itself, j > i only.
// FULL: all NI * 32 i atoms are there.
template <int NI, bool DIAG, bool FULL, int SH>
__device__ __forceinline__ void pc_unit(const unsigned char* __restrict__ itile, const unsigned char* __restrict__ ch,
                                        int i0, int cnt_i, int nj, int jslot, int islots, int jslots, float thr,
                                        unsigned base, PrQueue& Q) {
  using namespace dev;
  i0 += threadIdx.x & 31;
  unsigned long long nx[NI], ny[NI], nz[NI];
  bool on[NI];
#pragma unroll
  for (int g = 0; g < NI; ++g) {
    const int s = i0 + g * 32;
    const unsigned char* c = itile + (s >> 6) * kHistChunkBytes;
    const float* xy = reinterpret_cast<const float*>(c) + ((s & 63) >> 1) * 4 + (s & 1);
    const float* z = reinterpret_cast<const float*>(c + 512) + (s & 63);
    const float x = -xy[0], y = -xy[2], zz = -z[0];
    nx[g] = pack2(x, x);
    ny[g] = pack2(y, y);
    nz[g] = pack2(zz, zz);
    on[g] = FULL || s < cnt_i;
  }
  const float4* jxy = reinterpret_cast<const float4*>(ch);
  const float2* jz = reinterpret_cast<const float2*>(ch + 512);
  const unsigned long long tiny = pack2(1e-12f, 1e-12f), nhalf = pack2(-0.5f, -0.5f), magic = pack2(kPrMagic, kPrMagic),
                           nmagic = pack2(-kPrMagic, -kPrMagic), minus = pack2(-1.0f, -1.0f);
  unsigned marks = 0u;  // bit 2 g + half of the current entry, 8 bits an entry
  auto entry = [&](int e, int at, bool second) {
    const float4 a = __ldg(jxy + e);
    const float2 b = __ldg(jz + e);
    const unsigned long long jx = pack2(a.x, a.y), jy = pack2(a.z, a.w), jz2 = pack2(b.x, b.y);
#pragma unroll
    for (int g = 0; g < NI; ++g) {
      unsigned long long dx, dy, dz, d2, x, t, u;
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dx) : "l"(jx), "l"(nx[g]));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dy) : "l"(jy), "l"(ny[g]));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dz) : "l"(jz2), "l"(nz[g]));
      asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d2) : "l"(dz), "l"(tiny));
      asm("fma.rn.f32x2 %0, %1, %1, %0;" : "+l"(d2) : "l"(dy));
      asm("fma.rn.f32x2 %0, %1, %1, %0;" : "+l"(d2) : "l"(dx));
      float va, vb, xa, xb, ta, tb, ua, ub;
      unpack2(d2, va, vb);
      asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(xa) : "f"(va));
      asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(xb) : "f"(vb));
      // x - 1/2 (the root as d2 rsqrt(d2)) rounds to floor(x) but for the edges
      // themselves; u = x - floor(x) - 1/2
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(x) : "l"(d2), "l"(pack2(xa, xb)), "l"(nhalf));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(x), "l"(magic));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(u) : "l"(t), "l"(nmagic));
      asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(u) : "l"(minus), "l"(x));
      unpack2(t, ta, tb);
      unpack2(u, ua, ub);
      const unsigned aa = base + (__float_as_uint(ta) << SH), ab = base + (__float_as_uint(tb) << SH);
      if constexpr (FULL && !DIAG) {
        // counted, or near an edge: marked
        asm volatile(
            "{\n .reg .pred p;\n .reg .f32 v;\n abs.f32 v, %2;\n setp.gt.f32 p, v, %3;\n"
            " @!p red.shared.add.u32 [%1], 1;\n @p or.b32 %0, %0, %4;\n}"
            : "+r"(marks)
            : "r"(aa), "f"(ua), "f"(thr), "r"(1u << (at * 8 + 2 * g))
            : "memory");
        if (second)
          asm volatile(
              "{\n .reg .pred p;\n .reg .f32 v;\n abs.f32 v, %2;\n setp.gt.f32 p, v, %3;\n"
              " @!p red.shared.add.u32 [%1], 1;\n @p or.b32 %0, %0, %4;\n}"
              : "+r"(marks)
              : "r"(ab), "f"(ub), "f"(thr), "r"(2u << (at * 8 + 2 * g))
              : "memory");
      } else {
        bool oa = on[g], ob = on[g] && second;
        if constexpr (DIAG) {
          oa = oa && jslot + 2 * e > i0 + g * 32;
          ob = ob && jslot + 2 * e + 1 > i0 + g * 32;
        }
        const bool fa = fabsf(ua) > thr, fb = fabsf(ub) > thr;
        if (oa && !fa) asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(aa) : "memory");
        if (ob && !fb) asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(ab) : "memory");
        if (oa && fa) marks |= 1u << (at * 8 + 2 * g);
        if (ob && fb) marks |= 2u << (at * 8 + 2 * g);
      }
    }
  };
  // four entries at a time, then their marked pairs
  for (int e = 0; 2 * e < nj; e += 4) {
    if (2 * e + 8 <= nj) {
#pragma unroll
      for (int k = 0; k < 4; ++k) entry(e + k, k, true);
    } else {
      for (int k = 0; 2 * (e + k) < nj; ++k) entry(e + k, k, 2 * (e + k) + 1 < nj);
    }
    while (__any_sync(0xffffffffu, marks != 0u)) {
      const int bit = __ffs(marks) - 1;  // -1: none of this lane's
      const int k = bit >> 3, g = (bit & 7) >> 1, half = bit & 1;
      Q.push(marks != 0u, islots + i0 + g * 32, jslots + 2 * (e + k) + half);
      marks &= marks - 1u;
    }
  }
}

// counts[row][bin]: pairs of the class pair per bin.  Shared: edges, counters
// (columns words a bin), the warps' queues.
template <int SH>
__global__ void __launch_bounds__(kPcT, 1)
    k_pr_count(const unsigned char* __restrict__ pts, const int* __restrict__ tile_cnt, const int* __restrict__ atom,
               const double* __restrict__ xyz, const HistRow* __restrict__ rows, const int2* __restrict__ cta,
               const double* __restrict__ edges, const PrParams* __restrict__ par, int bins,
               unsigned long long* __restrict__ counts) {
  constexpr int kColumns = 1 << (SH - 2);
  extern __shared__ double pr_dyn[];
  if (par->degenerate) return;
  unsigned* hist = reinterpret_cast<unsigned*>(pr_dyn + bins + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int k = tid; k <= bins; k += kPcT) pr_dyn[k] = edges[k];
  for (int k = tid; k < bins * kColumns; k += kPcT) hist[k] = 0u;
  __syncthreads();
  // a pair is near an edge when its fractional bin coordinate is within delta
  // of 0 or 1: |frac - 0.5| > 0.5 - delta (always, when delta is FLT_MAX)
  const float thr = 0.5f - par->delta;
  const unsigned col = (unsigned)(lane & (kColumns - 1));
  const unsigned base =
      (unsigned)__cvta_generic_to_shared(hist + col) - ((unsigned)kPrMagicBits << SH);  // 32-bit wrap-around
  PrQueue Q{reinterpret_cast<int2*>(hist + (size_t)bins * kColumns) + warp * kPcQueue, 0, xyz, atom, pr_dyn,
            hist + col, bins, kColumns, par->inv_step};
  const int2 first = cta[blockIdx.x], last = cta[blockIdx.x + 1];
  for (int row = first.x; row <= last.x; ++row) {
    const HistRow R = rows[row];
    const int begin = row == first.x ? first.y : 0;
    const int end = row == last.x ? last.y : hist_units(R);
    if (begin >= end) continue;
    const int per = 2 * R.split;
    // at most 2^31 pairs of a row between flushes of its 32-bit counters
    for (int u0 = begin; u0 < end; u0 += kPrFlushItems * R.split) {
      const int u1 = min(end, u0 + kPrFlushItems * R.split);
      for (int u = u0 + warp; u < u1; u += kPcWarps) {
        const int2 t = hist_tiles(R, u / per);
        const int half = u % per / R.split, sub = u % R.split, jslot = half * kHistChunkAtoms;
        const int nj = min(kHistChunkAtoms, tile_cnt[t.y] - jslot), ni = tile_cnt[t.x];
        if (nj <= 0) continue;
        const unsigned char* it = pts + (size_t)t.x * 2 * kHistChunkBytes;
        const unsigned char* ch = pts + ((size_t)t.y * 2 + half) * kHistChunkBytes;
        const int groups = (ni + 31) >> 5, g0 = R.igroups ? sub : 0, g1 = R.igroups ? min(groups, g0 + 1) : groups;
        const int is = t.x * kTile, js = t.y * kTile + jslot;
        if (R.diag && t.x == t.y) {
          for (int g = g0; g < g1; ++g) pc_unit<1, true, false, SH>(it, ch, g * 32, ni, nj, jslot, is, js, thr, base, Q);
        } else if (g1 - g0 < 4) {
          for (int g = g0; g < g1; ++g) pc_unit<1, false, false, SH>(it, ch, g * 32, ni, nj, jslot, is, js, thr, base, Q);
        } else {
          if (ni == kTile) pc_unit<4, false, true, SH>(it, ch, 0, ni, nj, jslot, is, js, thr, base, Q);
          else pc_unit<4, false, false, SH>(it, ch, 0, ni, nj, jslot, is, js, thr, base, Q);
        }
      }
      Q.drain(1);
      __syncthreads();
      if constexpr (kColumns == 32) {
        for (int k = warp; k < bins; k += kPcWarps) {  // a warp per bin
          const unsigned c = hist[k * 32 + lane];
          hist[k * 32 + lane] = 0u;
          // 32-bit halves of the sum of 32 counters
          const unsigned lo = __reduce_add_sync(0xffffffffu, c & 0xffffu), hi = __reduce_add_sync(0xffffffffu, c >> 16);
          const unsigned long long all = (unsigned long long)lo + ((unsigned long long)hi << 16);
          if (lane == 0 && all) atomicAdd(&counts[(size_t)R.acc * bins + k], all);
        }
      } else {
        // a thread per bin: there are thousands, and with a warp for each the
        // flushes were a small structure's time (344 atoms of three weights, 7,296
        // bins: 202 to 127 us a call; 150 of 58, 6,386 bins: 774 to 425)
        uint2* four = reinterpret_cast<uint2*>(hist);
        for (int k = tid; k < bins; k += kPcT) {
          const uint2 a = four[2 * k], b = four[2 * k + 1];
          four[2 * k] = four[2 * k + 1] = make_uint2(0u, 0u);
          const unsigned long long all = (unsigned long long)a.x + a.y + b.x + b.y;
          if (all) atomicAdd(&counts[(size_t)R.acc * bins + k], all);
        }
      }
      __syncthreads();
    }
  }
}

struct PrAcc {
  double* w;
  __device__ __forceinline__ void add(int e, double wij) const { atomicAdd(&w[e], wij); }
};

// Shared layout: kPrWeighted: edges[bins + 1] (f64), then copies x f64[bins]; kPrWeightedGlobal: no dynamic
// shared memory (edges and the block's row in device memory).
template <int kMode>
__global__ void __launch_bounds__(kPrThreads, 8)
    k_pr_hist(const double4* __restrict__ pos, const float4* __restrict__ pos32, const int2* __restrict__ tiles,
              int n_tiles, int64_t chunk, const double* __restrict__ edges,
              const PrParams* __restrict__ par, int bins, int copies, double* __restrict__ rows) {
  extern __shared__ double pr_dyn[];
  __shared__ double4 sj[kPrThreads];
  __shared__ float4 sj32[kPrThreads];
  // the j tile in bins as pairs of atoms: {x_j, x_j+1, y_j, y_j+1} and {z_j, z_j+1}
  __shared__ float4 sjp[kPrThreads / 2];
  __shared__ float2 sjz[kPrThreads / 2];
  if (par->degenerate) return;
  const float inv_step = par->inv_step;
  // a pair is near an edge when its fractional bin coordinate is within delta
  // of 0 or 1: |frac - 0.5| > 0.5 - delta (always, when delta is FLT_MAX)
  const float near_edge = 0.5f - par->delta;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int si = lane * 4 + warp;  // this thread's slot in the i tile
  const double* E = kMode == kPrWeightedGlobal ? edges : pr_dyn;
  double* Hw = kMode == kPrWeightedGlobal ? rows + (size_t)blockIdx.x * bins : pr_dyn + bins + 1;
  if constexpr (kMode != kPrWeightedGlobal) {
    for (int k = threadIdx.x; k <= bins; k += kPrThreads) pr_dyn[k] = edges[k];
    for (int k = threadIdx.x; k < copies * bins; k += kPrThreads) Hw[k] = 0.0;
  }
  PrAcc acc;
  acc.w = kMode == kPrWeightedGlobal ? Hw : Hw + (size_t)(warp % copies) * bins;
  const int top = kPrMagicBits + bins - 1;  // floor(x) capped at bins - 1, in magic bits
  const int64_t n_work = (int64_t)n_tiles * (n_tiles + 1) / 2;
  int64_t w = (int64_t)blockIdx.x * chunk;
  const int64_t w_end = min(w + chunk, n_work);
  int a = 0, b = 0;
  if (w < w_end) pr_tri_decode(w, a, b);
  int cur_b = -1;

  for (; w < w_end; ++w) {
    const int2 ta = tiles[a], tb = tiles[b];
    if (b != cur_b) {
      __syncthreads();
      if ((int)threadIdx.x < tb.y) {
        const int64_t g = (int64_t)b * kPrThreads + threadIdx.x;
        const float4 f = pos32[g];
        sj[threadIdx.x] = pos[g];
        const float4 fs = make_float4(f.x * inv_step, f.y * inv_step, f.z * inv_step, 0.0f);
        sj32[threadIdx.x] = fs;
        float* xy = reinterpret_cast<float*>(&sjp[threadIdx.x >> 1]);
        float* z = reinterpret_cast<float*>(&sjz[threadIdx.x >> 1]);
        const int h = threadIdx.x & 1;
        xy[h] = fs.x;
        xy[2 + h] = fs.y;
        z[h] = fs.z;
      }
      __syncthreads();
      cur_b = b;
    }
    if (si < ta.y) {
      const int64_t gi = (int64_t)a * kPrThreads + si;
      float4 fi = pos32[gi];
      fi = make_float4(fi.x * inv_step, fi.y * inv_step, fi.z * inv_step, 0.0f);
      const double wi = pos[gi].w;
      if (a != b && tb.y == kPrThreads) {
        // full off-diagonal tile: 32 pairs per chunk without branches, two
        // pairs per packed instruction; pairs near an edge are marked and
        // placed exactly after the chunk
        const unsigned long long fx2 = pr_pack(fi.x, fi.x), fy2 = pr_pack(fi.y, fi.y), fz2 = pr_pack(fi.z, fi.z);
        const unsigned long long magic2 = pr_pack(kPrMagic, kPrMagic), half2 = pr_pack(0.5f, 0.5f);
#pragma unroll 1
        for (int jc = 0; jc < kPrThreads; jc += 32) {
          unsigned marked = 0u;
#pragma unroll
          for (int jj = 0; jj < 32; jj += 2) {
            const PrTwo r = pr_two(fx2, fy2, fz2, sjp[(jc + jj) >> 1], sjz[(jc + jj) >> 1], magic2, half2, near_edge);
            marked |= ((r.edge_a ? 1u : 0u) | (r.edge_b ? 2u : 0u)) << jj;
            if (!r.edge_a) acc.add(min(__float_as_int(r.ta), top) - kPrMagicBits, wi * sj[jc + jj].w);
            if (!r.edge_b) acc.add(min(__float_as_int(r.tb), top) - kPrMagicBits, wi * sj[jc + jj + 1].w);
          }
          while (marked) {
            const int j = jc + __ffs(marked) - 1;
            marked &= marked - 1u;
            const double4 pj = sj[j];
            acc.add(pr_exact_bin(pos[gi], pj, pr_bin_coord(fi, sj32[j]), E, bins), wi * pj.w);
          }
        }
      } else {
        for (int j = (a == b) ? si + 1 : 0; j < tb.y; ++j) {
          const float x = pr_bin_coord(fi, sj32[j]);
          const float t = __fadd_rd(x, kPrMagic);
          const float frac = x - (t - kPrMagic);
          const double4 pj = sj[j];
          int e;
          if (fabsf(frac - 0.5f) > near_edge) e = pr_exact_bin(pos[gi], pj, x, E, bins);
          else e = min(__float_as_int(t), top) - kPrMagicBits;
          acc.add(e, wi * pj.w);
        }
      }
    }
    if (++a > b) {
      a = 0;
      ++b;
    }
  }
  if constexpr (kMode == kPrWeighted) {
    __syncthreads();
    for (int k = threadIdx.x; k < bins; k += kPrThreads) {
      double sum = 0.0;
      for (int c = 0; c < copies; ++c) sum += Hw[(size_t)c * bins + k];
      rows[(size_t)blockIdx.x * bins + k] = sum;
    }
  }
}

// hist[k] = Σ_pairs counts[pair][k] * wprod[pair], pairs in order.
__global__ void k_pr_combine(const unsigned long long* __restrict__ counts, const double* __restrict__ wprod,
                             int n_pairs, int bins, const PrParams* __restrict__ par, double* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= bins) return;
  double s = 0.0;
  if (!par->degenerate)
    for (int p = 0; p < n_pairs; ++p) s += (double)counts[(size_t)p * bins + k] * wprod[p];
  out[k] = s;
}

__global__ void k_pr_reduce(const double* __restrict__ rows, int n_rows, int bins, const PrParams* __restrict__ par,
                            double* __restrict__ out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= bins) return;
  double s = 0.0;
  if (!par->degenerate)
    for (int g = 0; g < n_rows; ++g) s += rows[(size_t)g * bins + k];
  out[k] = s;
}

template <int kMode>
int pr_blocks_per_sm(size_t dyn) {
  // of the function, whatever context sets it: always the same value
  if (dyn)
    CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_pr_hist<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPrDynSmem));
  int per_sm = 0;
  CRAB_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pr_hist<kMode>, kPrThreads, dyn));
  return std::max(per_sm, 1);
}

}  // namespace

namespace {

// Weight classes of the atoms: distinct weights, the atoms of each, and per
// atom class << 24 | rank in it (in the context's pinned buffer).  More than
// kPrMaxClasses weights: `few` is false and the rest is not complete.
struct PrClasses {
  uint32_t* word = nullptr;
  std::vector<double> w;
  std::vector<int64_t> n;
  bool few = true;
  int ids[256];  // open addressing over the weights' bits: never more than a quarter full
  PrClasses() { std::fill(ids, ids + 256, -1); }
  int add(double weight) {  // the class of this weight's bits, a new one if there is none
    uint64_t key;
    std::memcpy(&key, &weight, sizeof key);
    uint32_t h = (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> 56);
    for (; ids[h] >= 0; h = (h + 1) & 255)
      if (std::memcmp(&w[ids[h]], &weight, sizeof weight) == 0) return ids[h];
    if (w.size() == kPrMaxClasses) {
      few = false;
      return 0;
    }
    ids[h] = (int)w.size();
    w.push_back(weight);
    n.push_back(0);
    return ids[h];
  }
  void put(int64_t i, int k) { word[i] = (uint32_t)k << 24 | ((uint32_t)n[k]++ & 0xffffffu); }
};

double histogram_of(crab_ctx* ctx, const double* xyz, PrClasses& C, const std::function<const double*()>& weights,
                    int64_t n, int64_t bins, double* hist, const std::function<void()>& meanwhile);

}  // namespace

double pair_distance_histogram(crab_ctx* ctx, const double* xyz, const double* w, int64_t n, int64_t bins,
                               double* hist) {
  require(bins >= 1 && bins <= kPrMaxBins, "bins must be in [1, 16777216]");
  require(n >= 0, "negative atom count");
  for (int64_t i = 0; i < n; ++i) require(std::isfinite(w[i]), "weights must be finite");
  PrClasses C;
  C.word = (uint32_t*)ctx->host("pr.word", (size_t)std::max<int64_t>(n, 1) * sizeof(uint32_t));
  int last = -1;
  for (int64_t i = 0; i < n && C.few; ++i) {
    if (last < 0 || std::memcmp(&C.w[last], &w[i], sizeof(double)) != 0) last = C.add(w[i]);
    if (C.few) C.put(i, last);
  }
  return histogram_of(ctx, xyz, C, [&]() { return w; }, n, bins, hist, []() {});
}

namespace {

double histogram_of(crab_ctx* ctx, const double* xyz, PrClasses& C, const std::function<const double*()>& weights,
                    int64_t n, int64_t bins, double* hist, const std::function<void()>& meanwhile) {
  TraceScope trace("pr.histogram");
  const std::vector<double>& class_w = C.w;
  const std::vector<int64_t>& class_n = C.n;
  std::fill(hist, hist + bins, 0.0);
  ctx->last_pr_ms = ctx->last_pr_hist_ms = 0.0;
  ctx->last_pr_mode = -1;
  ctx->last_pr_pairs = (double)n * (double)(n > 0 ? n - 1 : 0) * 0.5;
  if (n < 2) {
    for (int64_t i = 0; i < 3 * n; ++i)
      require(std::fabs(xyz[i]) < 1e100, "coordinates must be finite and below 1e100");
    meanwhile();
    return 0.0;
  }
  cudaStream_t s = ctx->stream;
  auto* hx = (double*)ctx->host("pr.xyz", (size_t)n * 3 * sizeof(double));
  std::memcpy(hx, xyz, (size_t)n * 3 * sizeof(double));
  auto* d_xyz = (double*)ctx->dev("pr.xyz", (size_t)n * 3 * sizeof(double));
  copy_h2d(ctx, d_xyz, hx, (size_t)n * 3 * sizeof(double), s);
  const int T = (int)class_w.size();
  trace_mark("pr.copied");
  const int n_pairs = T * (T + 1) / 2;
  const size_t edge_bytes = (size_t)(bins + 1) * sizeof(double);
  // counting: pairs per class pair and bin in whole numbers, 32 counters a bin
  // (4 where those do not fit)
  const int columns = pc_smem(bins, 32) <= kPcSmem ? 32 : 4;
  int mode = kPrWeightedGlobal, copies = 1;
  std::vector<HistRow> rows;
  std::vector<double> row_pairs;
  std::vector<int> tile_cnt, tile0;
  bool fits = C.few && (size_t)n_pairs * bins * 8 <= kPrMaxCountBytes &&
              edge_bytes + (size_t)bins * 4 <= kPrDynSmem && n < (1 << 24);
  if (fits) {
    for (int a = 0; a < T; ++a) {
      tile0.push_back((int)tile_cnt.size());
      for (int64_t at = 0; at < class_n[a]; at += kTile)
        tile_cnt.push_back((int)std::min<int64_t>(kTile, class_n[a] - at));
    }
    tile0.push_back((int)tile_cnt.size());
    int64_t units = 0;
    for (int a = 0; a < T; ++a)
      for (int b = a; b < T; ++b) {
        HistRow r{tile0[a], tile0[a + 1] - tile0[a], tile0[b], tile0[b + 1] - tile0[b], a == b, (int)bins, 1, 0, 0,
                  0.0f, pair_index(a, b, T)};
        fits = hist_row_units(r, class_n[a], false, 8 * kPcWarps, &units) && fits;
        rows.push_back(r);
        row_pairs.push_back(a == b ? 0.5 * (double)class_n[a] * (double)(class_n[a] - 1)
                                   : (double)class_n[a] * (double)class_n[b]);
      }
  }
  if (fits) {
    mode = kPrCounts;
  } else if (edge_bytes + (size_t)bins * 8 <= kPrDynSmem) {
    mode = kPrWeighted;
    copies = (int)std::min<size_t>(kPrThreads / 32, (kPrDynSmem - edge_bytes) / ((size_t)bins * 8));
  }
  // dmax, bin edges
  struct Misc {  // one buffer: what the kernels share and the host reads back
    unsigned long long dmax2;
    unsigned rim, invalid;
    PrParams par;
    double radius, centre[3];
  };
  auto* h_misc = (Misc*)ctx->host("pr.misc", sizeof(Misc));
  std::memset(h_misc, 0, sizeof(Misc));
  // few atoms: looking at all their pairs takes less than the four passes that
  // leave some out (354 atoms, 444 bins: 146 us a call with the passes, 128
  // without; 4,000 atoms, 160 bins: 168 and 155)
  const bool every = n <= kPrEvery;
  if (mode != kPrCounts || every) {  // the weighted kernels' tiles are centred on the host
    double lo[3] = {xyz[0], xyz[1], xyz[2]}, hi[3] = {xyz[0], xyz[1], xyz[2]};
    for (int64_t i = 0; i < n; ++i)
      for (int d = 0; d < 3; ++d) {
        const double v = xyz[3 * i + d];
        require(std::fabs(v) < 1e100, "coordinates must be finite and below 1e100");
        lo[d] = min_num(lo[d], v);
        hi[d] = max_num(hi[d], v);
      }
    for (int d = 0; d < 3; ++d) h_misc->centre[d] = 0.5 * (lo[d] + hi[d]);
  }
  if (every) {
    const double* c = h_misc->centre;
    double r2 = 0.0;
    for (int64_t i = 0; i < n; ++i) {
      const double dx = xyz[3 * i] - c[0], dy = xyz[3 * i + 1] - c[1], dz = xyz[3 * i + 2] - c[2];
      r2 = max_num(r2, dx * dx + dy * dy + dz * dz);
    }
    h_misc->radius = std::sqrt(r2) * (1.0 + 1e-12);
    h_misc->rim = (unsigned)n;
  }
  auto* d_misc = (Misc*)ctx->dev("pr.misc", sizeof(Misc));
  auto* d_far = (PrFar*)ctx->dev("pr.far", kPrMaxSteps * kPrFarBlocks * sizeof(PrFar));
  auto* d_rim = (int*)ctx->dev("pr.rim", (size_t)n * sizeof(int));
  auto* d_edges = (double*)ctx->dev("pr.edges", edge_bytes);
  auto* d_out = (double*)ctx->dev("pr.out", (size_t)bins * sizeof(double));
  copy_h2d(ctx, d_misc, h_misc, sizeof(Misc), s);
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  struct EvGuard {
    cudaEvent_t* e;
    ~EvGuard() {
      for (int i = 0; i < 3; ++i)
        if (e[i]) cudaEventDestroy(e[i]);
    }
  } ev_guard{ev};
  for (auto& e : ev) CRAB_CUDA_CHECK(cudaEventCreate(&e));
  CRAB_CUDA_CHECK(cudaEventRecord(ev[0], s));
  double* d_centre = d_misc->centre;
  PrParams* d_par = &d_misc->par;
  if (!every) {
    // two moves of the centre (7 us each) where the rim's pairs can take more than that
    const int given = mode != kPrCounts, steps = !given && n >= 8192 ? kPrMaxSteps : 3;
    for (int step = 0; step < steps; ++step)
      k_pr_far<<<kPrFarBlocks, 256, 0, s>>>(d_xyz, n, step, given, d_centre, d_far, &d_misc->invalid);
    k_pr_rim<<<kPrFarBlocks, 256, 0, s>>>(d_xyz, n, steps, given, d_far, d_centre, d_rim, &d_misc->rim, &d_misc->dmax2,
                                          &d_misc->radius);
    ctx->launches += steps + 1;
  }
  k_pr_dmax<<<8 * ctx->sm_count, kPrThreads, 0, s>>>(d_xyz, every ? nullptr : d_rim, &d_misc->rim, d_centre,
                                                     &d_misc->radius, &d_misc->dmax2);
  k_pr_edges<<<(unsigned)((bins + 1 + 127) / 128), 128, 0, s>>>(&d_misc->dmax2, bins, &d_misc->radius, &d_misc->invalid,
                                                                d_edges, d_par);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 2;
  const int ibins = (int)bins;
  if (mode == kPrCounts) {
    // tables in one copy: weight products, words, tile starts and counts, rows, CTA starts
    double all_pairs = 0.0;
    for (double p : row_pairs) all_pairs += p;
    const int grid = (int)std::max<int64_t>(
        1, std::min<int64_t>(ctx->sm_count, std::max<int64_t>(n_pairs, (int64_t)(all_pairs / 8192.0) + 1)));
    const std::vector<int2> starts = hist_starts(rows, row_pairs, 0, rows.size(), grid, 0, 1, 2.0);
    auto at16 = [](size_t v) { return (v + 15) / 16 * 16; };
    const size_t o_rows = at16((size_t)n_pairs * 8), o_start = at16(o_rows + rows.size() * sizeof(HistRow)),
                 o_tile0 = at16(o_start + starts.size() * sizeof(int2)), o_cnt = at16(o_tile0 + tile0.size() * 4),
                 all = o_cnt + tile_cnt.size() * 4;
    auto* h = (unsigned char*)ctx->host("pr.tables", all);
    for (int a = 0; a < T; ++a)
      for (int b = a; b < T; ++b) ((double*)h)[pair_index(a, b, T)] = class_w[a] * class_w[b];
    std::memcpy(h + o_rows, rows.data(), rows.size() * sizeof(HistRow));
    std::memcpy(h + o_start, starts.data(), starts.size() * sizeof(int2));
    std::memcpy(h + o_tile0, tile0.data(), tile0.size() * 4);
    std::memcpy(h + o_cnt, tile_cnt.data(), tile_cnt.size() * 4);
    auto* d = (unsigned char*)ctx->dev("pr.tables", all);
    copy_h2d(ctx, d, h, all, s);
    auto* d_word = (uint32_t*)ctx->dev("pr.word", (size_t)n * sizeof(uint32_t));
    copy_h2d(ctx, d_word, C.word, (size_t)n * sizeof(uint32_t), s);
    auto* d_pts = (unsigned char*)ctx->dev("pr.pts", tile_cnt.size() * 2 * kHistChunkBytes);
    auto* d_atom = (int*)ctx->dev("pr.atom", tile_cnt.size() * kTile * sizeof(int));
    auto* d_counts = (unsigned long long*)ctx->dev("pr.counts", (size_t)n_pairs * bins * 8);
    CRAB_CUDA_CHECK(cudaMemsetAsync(d_counts, 0, (size_t)n_pairs * bins * 8, s));
    k_pr_place<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_xyz, d_word, (const int*)(d + o_tile0), n, d_centre, d_par, d_pts, d_atom);
    CRAB_CUDA_CHECK(cudaEventRecord(ev[1], s));
    const size_t dyn = pc_smem(bins, columns);
    auto* kernel = columns == 32 ? k_pr_count<7> : k_pr_count<4>;
    CRAB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPcSmem));
    kernel<<<grid, kPcT, dyn, s>>>(d_pts, (const int*)(d + o_cnt), d_atom, d_xyz, (const HistRow*)(d + o_rows),
                                   (const int2*)(d + o_start), d_edges, d_par, ibins, d_counts);
    CRAB_CUDA_CHECK(cudaGetLastError());
    CRAB_CUDA_CHECK(cudaEventRecord(ev[2], s));
    k_pr_combine<<<(ibins + 127) / 128, 128, 0, s>>>(d_counts, (const double*)d, n_pairs, ibins, d_par, d_out);
  } else {
    const std::vector<int32_t> type(n, 0);
    const double* w = weights();
    Layout L;
    {
      TraceScope t2("pr.layout");
      L = build_layout(xyz, w, type.data(), n, 1, false, true);
    }
    const int n_tiles = L.n_tiles;
    const int64_t n_pad = L.n_pad;
    auto* h_pos = (double4*)ctx->host("pr.pos", (size_t)n_pad * sizeof(double4));
    auto* h_tiles = (int2*)ctx->host("pr.tiles", (size_t)n_tiles * sizeof(int2));
    for (int64_t k = 0; k < n_pad; ++k) {
      const int64_t src = L.source[k];
      h_pos[k] = src >= 0 ? make_double4(xyz[3 * src], xyz[3 * src + 1], xyz[3 * src + 2], w[src])
                          : make_double4(0.0, 0.0, 0.0, 0.0);
      // centred on the box, as the edges' error bound has it
      for (int d = 0; d < 3 && src >= 0; ++d)
        L.atoms[4 * k + d] = (float)(xyz[3 * src + d] - h_misc->centre[d]);
    }
    for (int t = 0; t < n_tiles; ++t) {
      int cnt = 0;
      while (cnt < kTile && L.source[(int64_t)t * kTile + cnt] >= 0) ++cnt;
      h_tiles[t] = make_int2(L.tile_type[t], cnt);
    }
    trace_mark("pr.pack");
    auto* d_pos = (double4*)ctx->dev("pr.pos", (size_t)n_pad * sizeof(double4));
    auto* d_pos32 = (float4*)ctx->dev("pr.pos32", (size_t)n_pad * sizeof(float4));
    auto* d_tiles = (int2*)ctx->dev("pr.tiles", (size_t)n_tiles * sizeof(int2));
    copy_h2d(ctx, d_pos, h_pos, (size_t)n_pad * sizeof(double4), s);
    copy_h2d(ctx, d_pos32, L.atoms.data(), (size_t)n_pad * sizeof(float4), s);
    copy_h2d(ctx, d_tiles, h_tiles, (size_t)n_tiles * sizeof(int2), s);
    size_t dyn = 0;
    int per_sm = 1;
    if (mode == kPrWeighted) {
      dyn = edge_bytes + (size_t)copies * bins * 8;
      per_sm = pr_blocks_per_sm<kPrWeighted>(dyn);
    } else {
      per_sm = pr_blocks_per_sm<kPrWeightedGlobal>(0);
    }
    const int64_t n_work = (int64_t)n_tiles * (n_tiles + 1) / 2;
    // one f64 row per block: at most 256 MB of rows
    const int64_t max_rows = std::max<int64_t>(1, (int64_t)(256u << 20) / (bins * 8));
    const int64_t grid0 = std::max<int64_t>(1, std::min({(int64_t)ctx->sm_count * per_sm, n_work, max_rows}));
    const int64_t chunk = (n_work + grid0 - 1) / grid0;
    const int grid = (int)((n_work + chunk - 1) / chunk);
    auto* d_rows = (double*)ctx->dev("pr.rows", (size_t)grid * bins * 8);
    if (mode == kPrWeightedGlobal) CRAB_CUDA_CHECK(cudaMemsetAsync(d_rows, 0, (size_t)grid * bins * 8, s));
    CRAB_CUDA_CHECK(cudaEventRecord(ev[1], s));
    if (mode == kPrWeighted)
      k_pr_hist<kPrWeighted><<<grid, kPrThreads, dyn, s>>>(d_pos, d_pos32, d_tiles, n_tiles, chunk, d_edges, d_par,
                                                           ibins, copies, d_rows);
    else
      k_pr_hist<kPrWeightedGlobal><<<grid, kPrThreads, 0, s>>>(d_pos, d_pos32, d_tiles, n_tiles, chunk, d_edges,
                                                               d_par, ibins, 1, d_rows);
    CRAB_CUDA_CHECK(cudaGetLastError());
    CRAB_CUDA_CHECK(cudaEventRecord(ev[2], s));
    k_pr_reduce<<<(ibins + 127) / 128, 128, 0, s>>>(d_rows, grid, ibins, d_par, d_out);
  }
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += mode == kPrCounts ? 3 : 2;
  auto* h_out = (double*)ctx->host("pr.out", (size_t)bins * sizeof(double));
  copy_d2h(ctx, h_misc, d_misc, sizeof(Misc), s);
  copy_d2h(ctx, h_out, d_out, (size_t)bins * sizeof(double), s);
  trace_mark("pr.launch");
  meanwhile();
  CRAB_CUDA_CHECK(cudaStreamSynchronize(s));
  trace_mark("pr.device");
  require(!h_misc->invalid, "coordinates must be finite and below 1e100");
  std::memcpy(hist, h_out, (size_t)bins * sizeof(double));
  float t_all = 0.f, t_hist = 0.f;
  CRAB_CUDA_CHECK(cudaEventElapsedTime(&t_hist, ev[1], ev[2]));
  CRAB_CUDA_CHECK(cudaEventElapsedTime(&t_all, ev[0], ev[2]));
  ctx->last_pr_ms = t_all;
  ctx->last_pr_hist_ms = t_hist;
  ctx->last_pr_mode = mode;
  double dmax2;
  std::memcpy(&dmax2, &h_misc->dmax2, sizeof dmax2);
  if (!(dmax2 > 0.0)) {
    std::fill(hist, hist + bins, 0.0);
    return 0.0;
  }
  return std::sqrt(dmax2);
}

// metrics.rs:550-583 normalize_distribution, in place on (r, p): trapezoid
// area to one, rg = sqrt(max(moment / 2, 0)) from the trapezoid of r^2 p,
// dmax = r at the last p above 1 % of the maximum (NaN stands for None).
// False when the area is not finite and positive.
bool normalize_distribution(int64_t m, const double* r, double* p, double* rg, double* dmax) {
  if (m <= 0) return false;
  double area = 0.0;
  for (int64_t i = 0; i + 1 < m; ++i) area += 0.5 * (r[i + 1] - r[i]) * (p[i] + p[i + 1]);
  if (!std::isfinite(area) || area <= 0.0) return false;
  for (int64_t i = 0; i < m; ++i) p[i] /= area;
  double moment = 0.0;
  for (int64_t i = 0; i + 1 < m; ++i)
    moment += 0.5 * (r[i + 1] - r[i]) * (r[i] * r[i] * p[i] + r[i + 1] * r[i + 1] * p[i + 1]);
  const double g = std::sqrt(std::fmax(moment / 2.0, 0.0));
  *rg = std::isfinite(g) ? g : NAN;
  double maximum = 0.0;
  for (int64_t i = 0; i < m; ++i) maximum = std::fmax(maximum, p[i]);
  *dmax = NAN;
  for (int64_t i = m - 1; i >= 0; --i)
    if (p[i] > maximum * 0.01) {
      *dmax = r[i];
      break;
    }
  return true;
}

}  // namespace

void coordinate_features(crab_ctx* ctx, const crab_struct* st, int64_t bins, double* rg, double* dmax, double* r,
                         double* p, int64_t* m, double* pr_rg, double* pr_dmax) {
  TraceScope trace("pr.features");
  require(st->n > 0, "coordinate features require a non-empty structure");
  bins = std::max<int64_t>(bins, 16);
  const int64_t n = st->n;
  const double* xyz = st->xyz.data();
  // metrics.rs:245-266: |form factor at q = 0| with implicit hydrogens, floored at 1e-6
  // one weight per (element, group) at full occupancy; occupancy scales the
  // form factor as form_factor_for_atom does (formfactor.rs:425-439)
  double ff0[CRAB_EL_OTHER + 1][15];
  int cls[CRAB_EL_OTHER + 1][15];
  bool have[CRAB_EL_OTHER + 1][15] = {};
  auto weight = [&](int64_t i) {
    const int el = st->elem[i], g = st->group[i] + 1;
    const double f = (el == CRAB_EL_H) ? 0.0 : st->occ[i] * ff0[el][g];
    return std::fmax(std::fabs(f), 1e-6);
  };
  PrClasses C;
  C.word = (uint32_t*)ctx->host("pr.word", (size_t)n * sizeof(uint32_t));
  for (int64_t i = 0; i < n; ++i) {
    const int el = st->elem[i], g = st->group[i] + 1;
    if (!have[el][g]) {
      ff0[el][g] = form_factor(el, g - 1, 1.0, true, 0.0);
      cls[el][g] = -1;
      have[el][g] = true;
    }
    if (!C.few) continue;
    int& full = cls[el][g];
    if (st->occ[i] != 1.0) {
      const int k = C.add(weight(i));
      if (C.few) C.put(i, k);
    } else {
      if (full < 0) full = C.add(weight(i));
      if (C.few) C.put(i, full);
    }
  }
  std::vector<double> hist(bins), all_w;
  auto weights = [&]() {
    all_w.resize(n);
    for (int64_t i = 0; i < n; ++i) all_w[i] = weight(i);
    return (const double*)all_w.data();
  };
  const double dm = histogram_of(ctx, xyz, C, weights, n, bins, hist.data(), [&]() {
    double total = 0.0, c[3] = {0.0, 0.0, 0.0};  // each sum in the reference's order
    const bool words = C.few;
    auto w_of = [&](int64_t i) { return words ? C.w[C.word[i] >> 24] : weight(i); };
    for (int64_t i = 0; i < n; ++i) {
      const double w = w_of(i);
      total += w;
      for (int d = 0; d < 3; ++d) c[d] = c[d] + xyz[3 * i + d] * w;
    }
    for (int d = 0; d < 3; ++d) c[d] = c[d] / total;
    double acc = 0.0;
    for (int64_t i = 0; i < n; ++i) {
      const double dx = xyz[3 * i] - c[0], dy = xyz[3 * i + 1] - c[1], dz = xyz[3 * i + 2] - c[2];
      acc += w_of(i) * (((0.0 + dx * dx) + dy * dy) + dz * dz);
    }
    *rg = std::sqrt(acc / total);
  });
  *dmax = dm;
  if (dm <= 0.0) {  // metrics.rs:489-498
    r[0] = 0.0; p[0] = 1.0; *m = 1; *pr_rg = 0.0; *pr_dmax = 0.0;
    return;
  }
  const double step = dm / (double)bins;
  for (int64_t k = 0; k < bins; ++k) {
    r[k] = ((double)k + 0.5) * step;
    p[k] = hist[k];
  }
  *m = bins;
  if (!normalize_distribution(bins, r, p, pr_rg, pr_dmax)) {  // metrics.rs:527-532
    r[0] = step * 0.5; p[0] = 1.0; *m = 1; *pr_rg = 0.0; *pr_dmax = dm;
  }
}

}  // namespace crab

using namespace crab;

extern "C" {

int crab_pair_distance_histogram(crab_ctx* ctx, const double* xyz, const double* w, int64_t n, int64_t bins,
                                 double* dmax, double* hist) {
  if (!ctx || !dmax || !hist || (n > 0 && (!xyz || !w))) return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() { *dmax = pair_distance_histogram(ctx, xyz, w, n, bins, hist); });
}

int crab_coordinate_features(crab_ctx* ctx, crab_struct* st, int64_t bins, double* rg, double* dmax, double* r,
                             double* p, int64_t* m, double* pr_rg, double* pr_dmax) {
  if (!ctx || !st || !rg || !dmax || !r || !p || !m || !pr_rg || !pr_dmax) return CRAB_EINVAL;
  return guarded_impl(ctx, [&]() { coordinate_features(ctx, st, bins, rg, dmax, r, p, m, pr_rg, pr_dmax); });
}

int crab_pr_last_timing(crab_ctx* ctx, double* total_ms, double* histogram_ms, double* pairs, int32_t* mode) {
  if (!ctx) return CRAB_EINVAL;
  std::lock_guard<std::mutex> g(ctx->mu);
  if (total_ms) *total_ms = ctx->last_pr_ms;
  if (histogram_ms) *histogram_ms = ctx->last_pr_hist_ms;
  if (pairs) *pairs = ctx->last_pr_pairs;
  if (mode) *mode = ctx->last_pr_mode;
  return CRAB_OK;
}

}  // extern "C"
