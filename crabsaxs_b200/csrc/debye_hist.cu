// Debye pair sums by distance: every pair is deposited once into a fine
// distance histogram of its class pair, and the histogram, not the pairs,
// meets the q grid.
//
// The recurrence kernels of debye.cu spend about 1.5 packed FP32 steps on
// every pair and every q point.  But Σ w_i w_j sin(q r_ij)/r_ij depends on a
// pair only through r_ij, and as a function of r it is band-limited by q.  So
// with bins of width h, q_max h <= kHistStep, a pair at r = (b + u) h,
// |u| <= 1/2, needs two numbers per bin, the pair count and Σ u:
//     sin(q r)/r  ~  f(q, b h) + h² f''(q, b h)/24  +  u h f'(q, b h),
// the least-squares straight line over the bin (f(q, r) = sin(q r)/r).  Its
// remainder h² f''/2 (u² - 1/12) has zero mean over the bin and an RMS of
// 0.037 (q h)² of f's amplitude: 9e-7 at q_max h = 0.005, the size of the phase
// error q δr that the FP32 coordinates carry at 45 Å, and like it uncorrelated
// from pair to pair.  What follows, per class pair and q, is the f64 sum
//     Σ_b count_b (f + h² f''/24) + (Σu)_b h f'
// over the bins, the same for every pair of atoms however many there are.
//
// k_hist_pairs: one CTA of 32 warps per SM keeps the histogram of one class
// pair in shared memory (two u32 words per bin: the count, and Σ u as fixed
// point of 2^-11, the low bits of a float, summed modulo 2^32).  A warp takes
// a unit of 128 i atoms (four a lane) by 64 j atoms; the j atoms come by bulk
// copies into its own double buffer as pairs (x0, x1, y0, y1), (z0, z1), so
// that one packed f32x2 instruction serves two pairs.  Per pair: 8 packed
// half-instructions for r and its fixed-point split, one MUFU reciprocal root,
// one address and two `red.shared.add.u32`.  Every CTA owns a contiguous run
// of units, sorted by class pair, so it adds its histogram into the one in
// device memory (u64 counts, i64 Σu) once per class pair that it meets and at
// the latest every kHistFlush units.  All sums are integers: the result does
// not depend on the order of anything.
// Atoms whose weight (occupancy) is not the commonest of their type cannot be
// counted; their pairs go through the same kernel into w_i w_j and w_i w_j u
// in 64-bit fixed point, in shared memory while the bins fit (20,000 atoms of
// distinct weights: 1.07 ms, 4.4 ms with adds into device memory).
// k_hist_transform: the sum over the bins for 16 class pairs and 128 q per CTA,
// over a slice of the bins; k_hist_reduce adds the slices in order.
//
// Bound: issue slots and the shared-memory atomics.  On random points, 4.3e8
// pairs and 13,000 bins (B200, 1965 MHz), the inner loop takes 0.41 ms, 0.28 ms
// without its atomics, and 1.05 ms with one 64-bit atomic per pair instead of
// two 32-bit ones; four i atoms a lane take 0.41 ms, two 0.44, one 0.50.
// 20,000 atoms with 9,369 sites at 500 q: k_hist_pairs 0.36 to 0.41 ms (1e12 pairs/s),
// transform and reduction 0.02 ms, against 18 ms for the recurrence kernel.
// The error against the FP64 kernel falls from 1.2e-9 to 9e-11 of the basis
// (2-norm), as counts do not round.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>

#include "device_math.cuh"
#include "engine.hpp"
#include "tile_rows.cuh"

namespace crab {
namespace {

using namespace dev;

constexpr int kHT = 1024;                     // threads of a pair CTA
constexpr int kHWarps = kHT / 32;
constexpr int kChunkAtoms = kHistChunkAtoms;  // j atoms of a unit
constexpr int kChunkBytes = kHistChunkBytes;  // 32 x {x0,x1,y0,y1}, then 32 x {z0,z1}
constexpr int kHistMaxBins = 22400;           // 2 words per bin beside the warps' double buffers in 227 KB
constexpr double kHistStep = 0.005;           // q_max h aimed at
constexpr double kHistMaxStep = 0.0075;       // beyond it (q_max x extent > 168) the recurrence kernels run
constexpr double kHistMaxReach = 1e18;        // squares of distances below FP32's largest number
constexpr int64_t kHistMaxBytes = (int64_t)8 << 30;  // sums of a plan in device memory
constexpr size_t kHistKeepBytes = (size_t)256 << 20;     // of a slot of one-shot calls, kept between them
constexpr int kHistFlush = 224;               // units between flushes: less than 2^21 pairs, |Σu| 2^11 < 2^31 in one bin
constexpr int kHistStagingBytes = kHWarps * 2 * kChunkBytes;
constexpr int kHistBarBytes = kHWarps * 2 * 8;
constexpr int kHistSumOffset = kHistMaxBins * 4;  // Σu words after the counts
static_assert((long long)kHistFlush * 128 * kChunkAtoms < (1ll << 21), "Σu of one bin must stay below 2^31");
static_assert(kHistFlush % kHWarps == 0, "the warps of a CTA take equal shares");
constexpr float kMagicBin = 12582912.0f;      // 1.5 x 2^23: adding it rounds to an integer in the low bits
constexpr unsigned kMagicBinBits = 0x4B400000u;
constexpr float kMagicU = 6144.0f;            // 1.5 x 2^12: low bits in units of 2^-11
constexpr unsigned kMagicUBits = 0x45C00000u;
constexpr int kLooseMaxBins = 11424;          // 64-bit sums in shared memory; wider rows add into device memory
constexpr int kLooseSumOffset = kLooseMaxBins * 8;
enum { kCounts = 0, kLooseShared = 1, kLooseGlobal = 2 };  // where the pairs of a launch go
// Dynamic shared memory of a launch: staging, barriers and the sums that its
// mode keeps there.
template <int MODE>
constexpr int hist_smem() {
  return kHistStagingBytes + kHistBarBytes +
         2 * (MODE == kCounts ? kHistSumOffset : MODE == kLooseShared ? kLooseSumOffset : 0);
}
static_assert(hist_smem<kCounts>() <= 232448, "histogram and staging exceed the shared memory of an SM");
static_assert(hist_smem<kLooseShared>() <= 232448, "loose sums and staging exceed the shared memory of an SM");
constexpr int kHistQ = 128, kHistR = 16;      // q and type pairs of a transform CTA
constexpr int kHistW = 16, kHistM = 5;        // bins of a wide bin, and its moments
constexpr int kHistB = 16;                    // wide bins per step of the transform

__device__ __forceinline__ unsigned long long hfma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long hadd2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long hmul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Of two pairs (j0, j1 against one i): the bin as kMagicBin's low bits and
// u = r/h - bin.  r comes from one MUFU reciprocal root refined with an FMA
// residual (within half an ulp, unbiased, as in the recurrence kernels); the
// bin and u each take one rounding of r/h.
struct HistTwo {
  float ba, bb, ua, ub;
};
__device__ __forceinline__ HistTwo hist_two(unsigned long long jx, unsigned long long jy, unsigned long long jz,
                                            unsigned long long nix, unsigned long long niy, unsigned long long niz,
                                            unsigned long long ih2) {
  const unsigned long long dx = hadd2(jx, nix), dy = hadd2(jy, niy), dz = hadd2(jz, niz);
  const unsigned long long x = hfma2(dx, dx, hfma2(dy, dy, hfma2(dz, dz, pack2(1e-12f, 1e-12f))));
  float xa, xb, ya, yb;
  unpack2(x, xa, xb);
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(ya) : "f"(xa));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yb) : "f"(xb));
  const unsigned long long y = pack2(ya, yb);
  const unsigned long long s = hmul2(x, y);
  const unsigned long long e = hfma2(hmul2(s, pack2(-1.0f, -1.0f)), s, x);  // x - s²
  const unsigned long long r = hfma2(e, hmul2(y, pack2(0.5f, 0.5f)), s);
  const unsigned long long b = hfma2(r, ih2, pack2(kMagicBin, kMagicBin));
  const unsigned long long nb = hfma2(b, pack2(-1.0f, -1.0f), pack2(kMagicBin, kMagicBin));  // minus the bin
  const unsigned long long u = hfma2(r, ih2, nb);
  HistTwo t;
  unpack2(b, t.ba, t.bb);
  unpack2(u, t.ua, t.ub);
  return t;
}

// Where a warp's pairs go: base is the shared address of bin 0 less that of
// bin kMagicBinBits (32-bit wrap-around); cnt and sum the row's sums in device
// memory.
struct HistSink {
  unsigned base;
  unsigned long long *cnt, *sum;
};

// ww: the pair's weight in fixed-point steps (loose pairs only).
template <int MODE>
__device__ __forceinline__ void deposit(const HistSink& k, float bin, float u, bool on, double ww) {
  if (!on) return;
  if constexpr (MODE == kCounts) {
    const unsigned addr = k.base + (__float_as_uint(bin) << 2);
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr) : "memory");
    asm volatile("red.shared.add.u32 [%0+%2], %1;" ::"r"(addr), "r"(__float_as_uint(u + kMagicU)), "n"(kHistSumOffset)
                 : "memory");
  } else {
    const unsigned long long v = (unsigned long long)__double2ll_rn(ww);
    const unsigned long long m = (unsigned long long)__double2ll_rn(ww * (double)u);
    if constexpr (MODE == kLooseShared) {
      const unsigned addr = k.base + (__float_as_uint(bin) << 3);
      asm volatile("red.shared.add.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
      asm volatile("red.shared.add.u64 [%0+%2], %1;" ::"r"(addr), "l"(m), "n"(kLooseSumOffset) : "memory");
    } else {
      const unsigned b = __float_as_uint(bin) - kMagicBinBits;
      atomicAdd(&k.cnt[b], v);
      atomicAdd(&k.sum[b], m);
    }
  }
}

// The NI * 32 atoms of the i tile from slot i0 on (those below cnt_i) against
// nj atoms of the chunk at `ch` from its entry e0 (slots jslot) on.  DIAG: both are of the same
// tile, pairs with slot j > i only.
template <int NI, bool DIAG, int MODE>
__device__ __forceinline__ void hist_unit(const unsigned char* ch, int e0, int nj, int jslot, const unsigned char* itile,
                                          int i0, int cnt_i, unsigned long long ih2, const HistSink& sink,
                                          const double* wi, const double* wj, double sc) {
  i0 += threadIdx.x & 31;  // this lane's first slot
  unsigned long long nx[NI], ny[NI], nz[NI];
  bool on[NI];
  double w[NI];
#pragma unroll
  for (int g = 0; g < NI; ++g) {
    const int s = i0 + g * 32;
    const unsigned char* c = itile + (s >> 6) * kChunkBytes;
    const float* xy = reinterpret_cast<const float*>(c) + ((s & 63) >> 1) * 4 + (s & 1);
    const float* z = reinterpret_cast<const float*>(c + 512) + (s & 63);
    const float x = -xy[0], y = -xy[2], zz = -z[0];
    nx[g] = pack2(x, x);
    ny[g] = pack2(y, y);
    nz[g] = pack2(zz, zz);
    on[g] = s < cnt_i;
    w[g] = MODE != kCounts ? wi[s] * sc : 1.0;
  }
  const float4* jxy = reinterpret_cast<const float4*>(ch) + e0;
  const float2* jz = reinterpret_cast<const float2*>(ch + 512) + e0;
  auto entry = [&](int e, bool second) {
    const float4 a = jxy[e];
    const float2 b = jz[e];
    const unsigned long long jx2 = pack2(a.x, a.y), jy2 = pack2(a.z, a.w), jz2 = pack2(b.x, b.y);
    double wa = 1.0, wb = 1.0;
    if constexpr (MODE != kCounts) {
      wa = wj[2 * e];
      wb = wj[2 * e + 1];
    }
#pragma unroll
    for (int g = 0; g < NI; ++g) {
      const HistTwo t = hist_two(jx2, jy2, jz2, nx[g], ny[g], nz[g], ih2);
      bool oa = on[g], ob = on[g] && second;
      if constexpr (DIAG) {
        oa = oa && jslot + 2 * e > i0 + g * 32;
        ob = ob && jslot + 2 * e + 1 > i0 + g * 32;
      }
      deposit<MODE>(sink, t.ba, t.ua, oa, w[g] * wa);
      deposit<MODE>(sink, t.bb, t.ub, ob, w[g] * wb);
    }
  };
  const int full = nj >> 1;
#pragma unroll 2
  for (int e = 0; e < full; ++e) entry(e, true);
  if (nj & 1) entry(full, false);
}

template <int MODE>
__global__ void __launch_bounds__(kHT, 1)
    k_hist_pairs(const unsigned char* __restrict__ pts, const int* __restrict__ tile_cnt,
                 const double* __restrict__ weight, const HistRow* __restrict__ rows, const int2* __restrict__ cta,
                 unsigned long long* __restrict__ cnt, unsigned long long* __restrict__ sum, int max_bins, double sc,
                 int* __restrict__ status, int budget) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* stage = sm + warp * 2 * kChunkBytes;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kHistStagingBytes) + warp * 2;
  unsigned* hist = reinterpret_cast<unsigned*>(sm + kHistStagingBytes + kHistBarBytes);
  unsigned long long* hist64 = reinterpret_cast<unsigned long long*>(hist);
  if (lane == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  for (int b = threadIdx.x; b < max_bins; b += kHT) {
    if constexpr (MODE == kCounts) hist[b] = hist[b + kHistMaxBins] = 0u;
    if constexpr (MODE == kLooseShared) hist64[b] = hist64[b + kLooseMaxBins] = 0ull;
  }
  __syncthreads();
  if (budget < 0) budget = kWaitBudget;
  bool ok = true;
  unsigned phase = 0u;  // bit b: parity of the next completion of bar[b]
  HistSink sink;
  sink.base = (unsigned)__cvta_generic_to_shared(hist) - (kMagicBinBits << (MODE == kCounts ? 2 : 3));
  const int2 first = cta[blockIdx.x], last = cta[blockIdx.x + 1];
  for (int row = first.x; row <= last.x; ++row) {
    const HistRow R = rows[row];
    const int begin = row == first.x ? first.y : 0;
    const int end = row == last.x ? last.y : hist_units(R);
    if (begin >= end) continue;
    const int bins = R.bins, per = 2 * R.split, flush = kHistFlush * R.split;
    const unsigned long long ih2 = pack2(R.inv_h, R.inv_h);
    sink.cnt = cnt + R.acc;
    sink.sum = sum + R.acc;
    for (int u0 = begin; u0 < end; u0 += flush) {
      const int u1 = min(end, u0 + flush);
      // a unit: its tile pair, half of the j tile, and (split rows) group of i atoms;
      // the j half comes by one bulk copy (768 bytes, 16-byte aligned)
      auto fetch = [&](int u, int buf) {
        if (lane == 0) {
          const int2 t = hist_tiles(R, u / per);
          const int half = u % per / R.split;
          mbar_expect_tx(&bar[buf], kChunkBytes);
          bulk_g2s(stage + buf * kChunkBytes, pts + ((size_t)t.y * 2 + half) * kChunkBytes, kChunkBytes, &bar[buf]);
        }
      };
      int u = u0 + warp, buf = 0;
      if (ok && u < u1) fetch(u, 0);
      for (; ok && u < u1; u += kHWarps) {
        const bool more = u + kHWarps < u1;
        if (more) fetch(u + kHWarps, buf ^ 1);
        const bool mine = mbar_wait(&bar[buf], (phase >> buf) & 1u, budget);
        ok = __all_sync(0xffffffffu, mine);
        if (!ok) {
          if (lane == 0) {  // leave only after this warp's copies have landed
            atomicExch(status, CRAB_ETIMEOUT);
            mbar_wait(&bar[buf], (phase >> buf) & 1u, kDrainBudget);
            if (more) mbar_wait(&bar[buf ^ 1], (phase >> (buf ^ 1)) & 1u, kDrainBudget);
          }
          break;
        }
        phase ^= 1u << buf;
        const int2 t = hist_tiles(R, u / per);
        const int sub = u % R.split, quarter = R.quarters ? sub / R.igroups * 16 : 0;  // first j atom in the chunk
        const int jslot = u % per / R.split * kChunkAtoms + quarter;
        const int nj = min(R.quarters ? 16 : kChunkAtoms, tile_cnt[t.y] - jslot), ni = tile_cnt[t.x];
        if (nj > 0) {
          const unsigned char* it = pts + (size_t)t.x * 2 * kChunkBytes;
          const unsigned char* ch = stage + buf * kChunkBytes;
          const double* wi = MODE != kCounts ? weight + (size_t)t.x * kTile : nullptr;
          const double* wj = MODE != kCounts ? weight + (size_t)t.y * kTile + jslot : nullptr;
          const int groups = (ni + 31) >> 5, g0 = R.igroups ? sub % R.igroups : 0,
                    g1 = R.igroups ? min(groups, g0 + 1) : groups;
          if (R.diag && t.x == t.y) {
            for (int g = g0; g < g1; ++g)
              if (jslot + nj > g * 32 + 1)  // some j beyond the group's first i
                hist_unit<1, true, MODE>(ch, quarter >> 1, nj, jslot, it, g * 32, ni, ih2, sink, wi, wj, sc);
          } else if (MODE != kCounts || g1 - g0 < 4) {
            for (int g = g0; g < g1; ++g)
              hist_unit<1, false, MODE>(ch, quarter >> 1, nj, jslot, it, g * 32, ni, ih2, sink, wi, wj, sc);
          } else {
            hist_unit<4, false, MODE>(ch, 0, nj, jslot, it, 0, ni, ih2, sink, wi, wj, sc);
          }
        }
        __syncwarp();  // every lane has read the buffer before its next copy
        buf ^= 1;
      }
      if constexpr (MODE != kLooseGlobal) {
        __syncthreads();
        for (int b = threadIdx.x; b < bins; b += kHT) {
          if constexpr (MODE == kCounts) {
            const unsigned c = hist[b];
            if (c) {
              const int s = (int)(hist[b + kHistMaxBins] - c * kMagicUBits);
              atomicAdd(&sink.cnt[b], (unsigned long long)c);
              atomicAdd(&sink.sum[b], (unsigned long long)(long long)s);
              hist[b] = hist[b + kHistMaxBins] = 0u;
            }
          } else {
            const unsigned long long c = hist64[b], s = hist64[b + kLooseMaxBins];
            if (c | s) {
              atomicAdd(&sink.cnt[b], c);
              atomicAdd(&sink.sum[b], s);
              hist64[b] = hist64[b + kLooseMaxBins] = 0ull;
            }
          }
        }
        __syncthreads();
      }
    }
  }
}

// part[slice][row][k] = Σ over the slice's bins of what a bin holds times f(q_k, .).
// kHistW bins are first joined to one wide bin of width H: its moments
//     M_m = Σ x^m,  x = (r - r0)/H in [-1/2, 1/2],  m < kHistM,
// follow from the bins' counts and Σu (and, for the second moment of u inside
// a bin, count/12), and f(q, r) = Σ_m x^m H^m f^(m)(q, r0)/m! with
//     f^(0) = sin(q r)/r,  f^(m) = (q^m sin(q r + m pi/2) - m f^(m-1))/r.
// With q H <= 0.08 (0.12 at the coarsest) five terms leave 1e-10 (4e-10) of f's
// amplitude, and 32 numbers become five: a sixth of the f64 multiply-adds and
// a sixteenth of the sines of a sum over the bins themselves.  The
// derivatives' rounding is that of f times (H/2r)^m, at most about one.
// One q per thread, kHistR rows per CTA, which read their moments from shared
// memory as broadcasts.
__global__ void __launch_bounds__(kHistQ)
    k_hist_transform(const unsigned long long* __restrict__ cnt, const unsigned long long* __restrict__ sum,
                     const unsigned long long* __restrict__ lcnt, const unsigned long long* __restrict__ lsum,
                     const HistOut* __restrict__ rows, const HistBlock* __restrict__ blocks, int n_rows, int slice,
                     double inv_sc, const double* __restrict__ q, int nq, double* __restrict__ part) {
  __shared__ double mo[kHistB][kHistM][kHistR];
  __shared__ double rinv[kHistB];
  const HistBlock blk = blocks[blockIdx.z];
  const int bins = blk.bins, row0 = blk.out0, nr = blk.n;
  const double h = blk.h, H = h * kHistW;
  const int wide = bins / kHistW;
  if ((int)blockIdx.x * slice >= wide) return;
  const int k = blockIdx.y * kHistQ + threadIdx.x;
  const double qk = q[min(k, nq - 1)];
  const int w_end = min(wide, ((int)blockIdx.x + 1) * slice);
  double acc[kHistR];
#pragma unroll
  for (int r = 0; r < kHistR; ++r) acc[r] = 0.0;
  for (int w0 = blockIdx.x * slice; w0 < w_end; w0 += kHistB) {
    int any = 0;
    for (int idx = threadIdx.x; idx < kHistB * kHistR; idx += kHistQ) {
      const int r = idx / kHistB, w = w0 + idx % kHistB;
      double m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0, m4 = 0.0;
      if (r < nr && w < w_end) {
        const HistOut o = rows[row0 + r];
        double c[kHistW], u[kHistW];  // all loads in flight together
        if (o.uniform >= 0) {
          const ulonglong2* pc = reinterpret_cast<const ulonglong2*>(cnt + o.uniform + (int64_t)w * kHistW);
          const ulonglong2* ps = reinterpret_cast<const ulonglong2*>(sum + o.uniform + (int64_t)w * kHistW);
#pragma unroll
          for (int i = 0; i < kHistW; i += 2) {
            const ulonglong2 x = pc[i / 2], y = ps[i / 2];
            any |= (x.x | x.y) != 0;
            c[i] = o.ww * (double)x.x;
            c[i + 1] = o.ww * (double)x.y;
            u[i] = o.ww * ((double)(long long)y.x * (1.0 / 2048.0));
            u[i + 1] = o.ww * ((double)(long long)y.y * (1.0 / 2048.0));
          }
        } else {
#pragma unroll
          for (int i = 0; i < kHistW; ++i) c[i] = u[i] = 0.0;
        }
        if (o.loose >= 0) {
          const ulonglong2* pc = reinterpret_cast<const ulonglong2*>(lcnt + o.loose + (int64_t)w * kHistW);
          const ulonglong2* ps = reinterpret_cast<const ulonglong2*>(lsum + o.loose + (int64_t)w * kHistW);
#pragma unroll
          for (int i = 0; i < kHistW; i += 2) {
            const ulonglong2 x = pc[i / 2], y = ps[i / 2];
            any |= (x.x | x.y | y.x | y.y) != 0;
            c[i] += (double)(long long)x.x * inv_sc;
            c[i + 1] += (double)(long long)x.y * inv_sc;
            u[i] += (double)(long long)y.x * inv_sc;
            u[i + 1] += (double)(long long)y.y * inv_sc;
          }
        }
#pragma unroll
        for (int i = 0; i < kHistW; ++i) {
          const double d = ((double)i - 0.5 * (kHistW - 1)) * (1.0 / kHistW), d2 = d * d;
          const double s = u[i] * (1.0 / kHistW);                    // Σ (x - d)
          const double v = c[i] * (1.0 / (12.0 * kHistW * kHistW));  // Σ (x - d)²
          m0 += c[i];
          m1 += fma(c[i], d, s);
          m2 += fma(c[i], d2, fma(2.0 * d, s, v));
          m3 += d * fma(c[i], d2, fma(3.0 * d, s, 3.0 * v));
          m4 += d2 * fma(c[i], d2, fma(4.0 * d, s, 6.0 * v));
        }
      }
      double* dst = &mo[idx % kHistB][0][r];
      dst[0] = m0;
      dst[kHistR] = m1 * H;
      dst[2 * kHistR] = m2 * (H * H / 2.0);
      dst[3 * kHistR] = m3 * (H * H * H / 6.0);
      dst[4 * kHistR] = m4 * (H * H * H * H / 24.0);
    }
    if (threadIdx.x < kHistB)
      rinv[threadIdx.x] = 1.0 / (h * ((double)(w0 + threadIdx.x) * kHistW + 0.5 * (kHistW - 1)));
    if (__syncthreads_or(any)) {
      double sn, cn, ss, sc;
      sincos(qk * (h * ((double)w0 * kHistW + 0.5 * (kHistW - 1))), &sn, &cn);
      sincos(qk * H, &ss, &sc);
      const int n = min(kHistB, w_end - w0);
#pragma unroll 1
      for (int i = 0; i < n; ++i) {
        const double ri = rinv[i];
        double p = qk * cn, f[kHistM];
        f[0] = sn * ri;
        f[1] = (p - f[0]) * ri;
        p = -qk * qk * sn;
        f[2] = fma(-2.0, f[1], p) * ri;
        p = -qk * qk * qk * cn;
        f[3] = fma(-3.0, f[2], p) * ri;
        p = qk * qk * (qk * qk) * sn;
        f[4] = fma(-4.0, f[3], p) * ri;
#pragma unroll
        for (int m = 0; m < kHistM; ++m)
#pragma unroll
          for (int r = 0; r < kHistR; ++r) acc[r] = fma(mo[i][m][r], f[m], acc[r]);
        const double t = fma(sn, sc, cn * ss);  // one wide bin on
        cn = fma(cn, sc, -sn * ss);
        sn = t;
      }
    }
    __syncthreads();
  }
  if (k < nq)
    for (int r = 0; r < nr; ++r) part[((size_t)blockIdx.x * n_rows + row0 + r) * nq + k] = acc[r];
}

// out[row's type pair][k] = the slices of part: thread row y takes the slices
// y, y + 8, ... in order, then row 0 adds the eight sums in order.
__global__ void __launch_bounds__(256) k_hist_reduce(const double* __restrict__ part, const HistOut* __restrict__ rows,
                                                     int n_rows, int slice, int nq, double* __restrict__ out) {
  __shared__ double red[8][32];
  const int64_t n = (int64_t)n_rows * nq, i = (int64_t)blockIdx.x * 32 + threadIdx.x;
  double s = 0.0;
  if (i < n) {
    const int slices = ((rows[i / nq].bins + kHistW - 1) / kHistW + slice - 1) / slice;
#pragma unroll 4
    for (int p = threadIdx.y; p < slices; p += 8) s += part[(size_t)p * n + i];
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && i < n) {
    s = 0.0;
    for (int y = 0; y < 8; ++y) s += red[y][threadIdx.x];
    out[rows[i / nq].out * (int64_t)nq + i % nq] = s;
  }
}

constexpr double kRowCost = 8.0;  // of a row's flush, in units of 8192 pairs
constexpr int kSplitUnits = 8 * kHWarps;

// The plan's host arrays as one block, uploaded in one copy.
struct HistBlob {
  std::vector<unsigned char> bytes;
  template <class T>
  size_t add(const T* v, size_t n) {
    const size_t at = (bytes.size() + 255) / 256 * 256;
    bytes.resize(at + n * sizeof(T));
    if (n) std::memcpy(bytes.data() + at, v, n * sizeof(T));
    return at;
  }
  template <class T>
  size_t add(const std::vector<T>& v) {
    return add(v.data(), v.size());
  }
};

}  // namespace

// Bins for this reach (largest distance) and q_max; 0: more than an SM's
// shared memory holds at the coarsest step, or nothing to resolve.
int hist_bins(double reach, double qmax) {
  if (!(qmax > 0.0) || !std::isfinite(reach * qmax)) return 0;
  double want = reach * qmax / kHistStep;
  if (want > kHistMaxBins - 8) {
    if (reach * qmax / kHistMaxStep > kHistMaxBins - 8) return 0;
    want = kHistMaxBins - 8;
  }
  return ((int)std::max(want, (double)kHistMinBins - 8.0) + 8 + kHistW - 1) / kHistW * kHistW;
}

// A pair's bin is an address as it stands, so nothing may come here whose FP32
// distance is not a number: beyond kHistMaxReach the squares overflow, and
// coordinates or weights that are not finite go to the recurrence kernels,
// whose addresses do not depend on them.
bool hist_structure_bins(double reach, double qmax, int* bins, float* inv_h) {
  if (!(reach < kHistMaxReach)) return false;
  reach = std::max(reach, 1e-3) * 1.0001 + 1e-3;
  *bins = std::min(hist_bins(reach, qmax), kHistMaxBins);
  if (*bins == 0) return false;
  *inv_h = (float)((double)(*bins - 4) / reach);  // every r/h stays below bins - 2 after its roundings
  return true;
}

// What the histogram of these classes takes beside its launches, in us: a row's
// bins are cleared and transformed, those that its pairs hit flushed, and rows
// with loose members do so a second time; loose pairs, whose sums are 64 bits
// wide, cost themselves.  Fitted to 1,670 plans of 1 to 400 types and 2 to 20,000
// atoms at 4 to 500 q: half of them within 17 %.
double hist_us(const HistShape& X, int T, bool skip_last, int64_t nq, double* n_rows) {
  const double blocks = std::ceil((double)nq / kHistQ);
  double us = 0.0;
  *n_rows = 0.0;
  for (int c = 0; c < X.S; ++c) {
    double types = 0.0, loose_types = 0.0, counted = 0.0, loose = 0.0;
    for (int a = 0; a < T; ++a) {
      const double u = (double)X.uni[(size_t)c * T + a].atoms, l = (double)X.loose[(size_t)c * T + a].atoms;
      types += u + l > 0.0;
      loose_types += l > 0.0;
      counted += u;
      loose += l;
    }
    const double bins = X.bins[c], rows = 0.5 * types * (types + 1.0) - (skip_last ? 1.0 : 0.0);
    // each loose class against the loose and the counted atoms of the others
    const double loose_rows = loose_types * (types + 1.0) * (counted > loose ? 1.0 : 0.5);
    const double loose_pairs = loose * (counted + 0.5 * loose);
    const double hit = std::min(bins, 0.5 * (counted + loose) * (counted + loose) / std::max(rows, 1.0));
    us += std::min(0.03 * loose_pairs, 25.0) + 6e-6 * loose_pairs +
          rows * (bins * (6e-6 + 1.35e-5 * blocks) + 6e-6 * hit) + loose_rows * (2e-6 * bins + 1.2e-5 * hit);
    *n_rows += rows + loose_rows;
  }
  return us;
}

// if_faster: only where the recurrence kernels would take longer.  They are the
// better ones for many types of few atoms and for few q, where the bins of every
// class pair cost more than its pairs (kernel time, histogram against
// recurrence: 14 types, 1,400 atoms with weights of their own, 8 q 107 / 31 us;
// 213 types, 20,000 atoms, 12 q 5.8 / 1.7 ms; 250 types, 2,500 atoms, 100 q 4.7 /
// 0.37 ms).  The choice depends on the problem alone, not on the shard or the
// device, so that all parts of one sum take the same kernels.
bool hist_plan_init(crab_ctx* ctx, PairPlan& P, bool if_faster) {
  double qmax = 0.0;
  for (double v : P.q) qmax = std::max(qmax, v);
  const Layout& L = P.L;
  const int T = L.T;
  const std::vector<int> seg = P.segments.empty() ? std::vector<int>{0, L.n_tiles} : P.segments;
  const int S = (int)seg.size() - 1;
  HistShape X;
  X.S = S;
  // every structure's own bins: they span its largest distance, h being the
  // inverse of an FP32 number so that r/h carries no common error
  X.bins.resize(S);
  X.inv_h.resize(S);
  for (int c = 0; c < S; ++c)
    if (!hist_structure_bins(P.segments.empty() ? L.extent : P.seg_extent[c], qmax, &X.bins[c], &X.inv_h[c]))
      return false;
  X.uni.resize((size_t)S * T);
  X.loose.resize((size_t)S * T);
  std::vector<HistRange>&uni = X.uni, &loose = X.loose;
  std::vector<int>& tcnt = X.tile_cnt;
  double& sumw = X.sum_abs_w;
  if (if_faster) {
    // atoms by tile, and the share of loose ones in a sample (three atoms of a
    // tile against its first): what the choice needs without a pass over all
    for (int c = 0; c < S; ++c) {
      const int every = std::max(1, (seg[c + 1] - seg[c]) / 256);
      int64_t seen = 0, odd = 0;
      for (int t = seg[c]; t < seg[c + 1]; ++t) {
        const float* w = L.atoms.data() + 4 * (size_t)t * kTile + 3;
        int n = kTile;
        while (n > 0 && w[4 * (n - 1)] == 0.0f) --n;
        uni[(size_t)c * T + L.tile_type[t]].atoms += n;
        if (n < 2 || t % every) continue;
        for (const int k : {n / 3, 2 * n / 3, n - 1})
          if (k > 0) {
            odd += w[4 * k] != w[0];
            ++seen;
          }
      }
      for (int a = 0; a < T && odd; ++a) {
        HistRange &U = uni[(size_t)c * T + a], &Lo = loose[(size_t)c * T + a];
        Lo.atoms = (int64_t)((double)U.atoms * (double)odd / (double)seen + 0.5);
        U.atoms -= Lo.atoms;
      }
    }
    double rows;
    const double us = hist_us(X, T, P.skip_last, P.nq, &rows);
    // 15 us: its launches above the recurrence's one, of which a plan of one call
    // gets ten back from the shorter tables; 0.05 us a row and 0.01 us an atom:
    // its tables and points on the host
    const double extra = (P.pooled ? 5.0 : 15.0) + 0.05 * rows + 0.01 * (double)L.n;
    if (!(us + extra < 0.8 * recurrence_us(X, T, P.skip_last, P.q))) return false;
    for (HistRange& r : uni) r.atoms = 0;
    for (HistRange& r : loose) r.atoms = 0;
  }
  // a type's atoms: the commonest weight if it has a majority, else whichever the vote leaves
  struct Run {
    size_t range;
    const float* a;
    int64_t m;
  };
  std::vector<Run> runs;
  for (int c = 0; c < S; ++c) {
    double s1 = 0.0;
    for (int t0 = seg[c]; t0 < seg[c + 1];) {
      const int ty = L.tile_type[t0];
      int t1 = t0 + 1;
      while (t1 < seg[c + 1] && L.tile_type[t1] == ty) ++t1;
      const Run r{(size_t)c * T + ty, L.atoms.data() + (size_t)t0 * kTile * 4, (int64_t)(t1 - t0) * kTile};
      const float* a = r.a;
      float major = 0.0f;
      int64_t votes = 0;
      for (int64_t i = 0; i < r.m; ++i) {
        const float w = a[4 * i + 3];
        if (!std::isfinite(a[4 * i]) || !std::isfinite(a[4 * i + 1]) || !std::isfinite(a[4 * i + 2]) ||
            !std::isfinite(w))
          return false;
        if (w == 0.0f) continue;  // padding, or an atom without weight
        if (votes == 0) major = w;
        votes += w == major ? 1 : -1;
        s1 += std::fabs((double)w);
      }
      uni[r.range].w = (double)major;
      for (int64_t i = 0; i < r.m; ++i)
        if (a[4 * i + 3] != 0.0f) ++(a[4 * i + 3] == major ? uni : loose)[r.range].atoms;
      X.any_loose = X.any_loose || loose[r.range].atoms > 0;
      runs.push_back(r);
      t0 = t1;
    }
    sumw = std::max(sumw, s1);
  }
  std::vector<unsigned char> pts;
  pts.reserve((size_t)(L.n_tiles + 2 * S) * 2 * kChunkBytes);
  std::vector<double> weight;
  auto append = [&](HistRange& R, const float* a, double w, int64_t& fill) {
    if (fill % kTile == 0) {
      pts.resize(pts.size() + 2 * kChunkBytes, 0);
      tcnt.push_back(0);
      weight.resize(weight.size() + kTile, 0.0);
      if (fill == 0) R.t0 = (int)tcnt.size() - 1;
      ++R.n;
    }
    const int s = (int)(fill % kTile);
    float* c = reinterpret_cast<float*>(pts.data() + pts.size() - 2 * kChunkBytes + (s >> 6) * kChunkBytes);
    const int e = s & 63;
    c[(e >> 1) * 4 + (e & 1)] = a[0];
    c[(e >> 1) * 4 + 2 + (e & 1)] = a[1];
    c[128 + e] = a[2];
    weight[weight.size() - kTile + s] = w;
    ++tcnt.back();
    ++fill;
    ++R.atoms;
  };
  for (const Run& r : runs) {
    // the class's loose tiles, then right after them its counted ones
    for (HistRange* R : {&loose[r.range], &uni[r.range]}) {
      int64_t fill = 0;
      R->atoms = 0;
      for (int64_t i = 0; i < r.m; ++i) {
        const float w = r.a[4 * i + 3];
        if (w != 0.0f && ((double)w == uni[r.range].w) == (R == &uni[r.range])) append(*R, r.a + 4 * i, w, fill);
      }
    }
  }
  return hist_build(ctx, P, X, &pts, &weight);
}

bool hist_build(crab_ctx* ctx, PairPlan& P, HistShape& X, const std::vector<unsigned char>* pts,
                const std::vector<double>* weight) {
  typedef HistRange Range;
  // all of the plan's part or nothing: an allocation that fails leaves no half
  // of it to be taken as built
  HistPart H;
  struct Undo {
    PairPlan& P;
    size_t kept;
    bool on = true;
    ~Undo() {
      for (; on && P.owned.size() > kept; P.owned.pop_back()) cudaFree(P.owned.back());
    }
  } undo{P, P.owned.size()};
  const int T = P.L.T, S = X.S;
  const std::vector<Range>&uni = X.uni, &loose = X.loose;
  const std::vector<int>& bins = X.bins;
  const std::vector<float>& inv_h = X.inv_h;
  const std::vector<int>& tcnt = X.tile_cnt;
  const bool any_loose = X.any_loose;
  const double sumw = X.sum_abs_w;
  // rows: class pairs of uniform tiles, and the tile sets with a loose member
  std::vector<HistRow> rows, lrows;
  std::vector<double> pairs, lpairs;  // of every row
  std::vector<HistOut> outs;
  int64_t loose_bins = 0, all_units = 0;
  int widest = 0;
  bool fits = true;
  auto row_of = [&](const Range& x, const Range& y, int diag, int c, int64_t acc, bool split) {
    HistRow r{x.t0, x.n, y.t0, y.n, diag, bins[c], 1, 0, 0, inv_h[c], acc};
    fits = hist_row_units(r, x.atoms, split, split ? (int64_t)1 << 20 : kSplitUnits, &all_units) && fits;
    widest = std::max(widest, bins[c]);
    return r;
  };
  auto pairs_of = [](const Range& x, const Range& y, int diag) {
    return diag ? 0.5 * (double)x.atoms * (double)(x.atoms - 1) : (double)x.atoms * (double)y.atoms;
  };
  for (int c = 0; c < S; ++c)
    for (int a = 0; a < T; ++a)
      for (int b = a; b < T; ++b) {
        if (P.skip_last && a == T - 1 && b == T - 1) continue;
        const Range &ua = uni[(size_t)c * T + a], &ub = uni[(size_t)c * T + b];
        const Range &la = loose[(size_t)c * T + a], &lb = loose[(size_t)c * T + b];
        HistOut o;
        o.uniform = o.loose = -1;
        o.out = c * P.n_pairs + pair_index(a, b, T);
        o.bins = bins[c];
        o.seg = c;
        o.ww = ua.w * ub.w;
        if (ua.n && ub.n) {
          o.uniform = (int64_t)rows.size();  // row number for now, then the row's sums
          rows.push_back(row_of(ua, ub, a == b, c, 0, false));
          pairs.push_back(pairs_of(ua, ub, a == b));
        }
        auto add = [&](const Range& x, const Range& y, int diag) {
          if (!x.n || !y.n) return;
          lrows.push_back(row_of(x, y, diag, c, loose_bins, true));
          lpairs.push_back(pairs_of(x, y, diag));
          o.loose = loose_bins;
        };
        // each loose atom against every atom of the other class, once
        if (a == b) {
          add(la, la, 1);
          add(la, ua, 0);
        } else {
          add(la, Range{lb.n ? lb.t0 : ub.t0, lb.n + ub.n, lb.atoms + ub.atoms, 0.0}, 0);
          add(lb, ua, 0);
        }
        if (o.loose >= 0) loose_bins += bins[c];
        if (o.uniform >= 0 || o.loose >= 0) outs.push_back(o);
      }
  if (any_loose && !std::isfinite(sumw * sumw)) return false;  // no fixed-point scale
  // unit numbers are 32-bit, and with loose members all rows are resident
  if (outs.empty() || !fits || loose_bins > (int64_t)1 << 27) return false;
  // loose sums: the largest power of two that keeps Σ|w w| below 2^61 steps
  int ex = 0;
  std::frexp(std::max(sumw * sumw, 1e-300), &ex);
  H.scale = std::ldexp(1.0, std::max(-1000, std::min(1000, 61 - ex)));
  // groups of rows whose sums (16 bytes a bin) stay in the L2 together; each
  // group is one launch of every kernel
  int64_t acc_bins = 0;
  size_t part_rows = 0;
  const int qblocks = (int)((P.nq + kHistQ - 1) / kHistQ);
  std::vector<HistRow> drows;
  std::vector<double> dpairs;
  std::vector<int2> starts;
  // one CTA per SM, but at least half a tile pair's pairs for each, unless it
  // has a row of its own
  auto grid_of = [&](const std::vector<HistRow>& r, const std::vector<double>& n, size_t r0, size_t r1) {
    double all = 0.0;
    for (size_t k = r0; k < r1; ++k) all += n[k];
    const int64_t want = std::max<int64_t>((int64_t)(r1 - r0), (int64_t)(all / (128 * kChunkAtoms)) / P.n_shards + 1);
    return (int)std::min<int64_t>(ctx->sm_count, want);
  };
  std::vector<HistBlock> blocks;
  const bool one = !lrows.empty();  // with loose rows: all in one group
  for (size_t o0 = 0; o0 < outs.size();) {
    HistGroup g;
    g.out0 = (int)o0;
    g.row0 = (int)drows.size();
    g.block0 = (int)blocks.size();
    int64_t used = 0, steps = 0;
    size_t o1 = o0;
    for (; o1 < outs.size(); ++o1) {
      HistOut& v = outs[o1];
      if (!one && o1 > o0 && (size_t)(used + v.bins) * 16 > kHistGroupBytes) break;
      if (v.uniform >= 0) {
        const size_t v_row = (size_t)v.uniform;
        HistRow r = rows[v_row];
        r.acc = v.uniform = used;
        used += v.bins;
        dpairs.push_back(pairs[v_row]);
        drows.push_back(r);
      }
      if ((int)blocks.size() == g.block0 || blocks.back().n == kHistR || outs[o1 - 1].seg != v.seg) {
        blocks.push_back(HistBlock{(int)(o1 - o0), 0, v.bins, 1.0 / (double)inv_h[v.seg]});
        steps += (v.bins / kHistW + kHistB - 1) / kHistB;
      }
      ++blocks.back().n;
    }
    g.n_out = (int)(o1 - o0);
    g.n_rows = (int)drows.size() - g.row0;
    g.n_blocks = (int)blocks.size() - g.block0;
    if (g.n_rows) {
      g.grid = grid_of(drows, dpairs, g.row0, drows.size());
      g.start0 = (int)starts.size();
      const std::vector<int2> st =
          hist_starts(drows, dpairs, g.row0, g.row0 + g.n_rows, g.grid, P.shard, P.n_shards, kRowCost);
      starts.insert(starts.end(), st.begin(), st.end());
    }
    // slices of the transform: about four CTAs per SM, whole steps of kHistB bins
    g.slice = (int)std::max<int64_t>(1, steps * qblocks / (4 * ctx->sm_count)) * kHistB;  // in wide bins
    g.slices = (widest / kHistW + g.slice) / g.slice;
    acc_bins = std::max(acc_bins, used);
    part_rows = std::max(part_rows, (size_t)g.n_out * g.slices);
    H.groups.push_back(g);
    o0 = o1;
  }
  if (!lrows.empty()) {
    H.loose_start0 = (int)starts.size();
    H.loose_row0 = (int)drows.size();
    drows.insert(drows.end(), lrows.begin(), lrows.end());
    dpairs.insert(dpairs.end(), lpairs.begin(), lpairs.end());
    H.loose_grid = grid_of(drows, dpairs, H.loose_row0, drows.size());
    const std::vector<int2> st =
        hist_starts(drows, dpairs, H.loose_row0, drows.size(), H.loose_grid, P.shard, P.n_shards, kRowCost);
    starts.insert(starts.end(), st.begin(), st.end());
  }
  if ((acc_bins + loose_bins) * 16 > kHistMaxBytes) return false;
  HistBlob blob;
  blob.bytes.reserve((pts ? pts->size() + weight->size() * 8 : 0) + drows.size() * 64 + outs.size() * 64 + 65536);
  const size_t o_cnt = blob.add(tcnt), o_rows = blob.add(drows), o_outs = blob.add(outs), o_blocks = blob.add(blocks),
               o_start = blob.add(starts), o_q = blob.add(P.q), o_pts = pts ? blob.add(*pts) : 0,
               o_w = pts && any_loose ? blob.add(*weight) : 0, o_more = blob.add(X.more);
  auto* d = (unsigned char*)plan_alloc(ctx, P, P.owned, "hist_in", blob.bytes.size());
  copy_h2d(ctx, d, blob.bytes.data(), blob.bytes.size(), ctx->stream);
  H.d_pts = pts ? d + o_pts : (unsigned char*)plan_alloc(ctx, P, P.owned, "hist_pts", tcnt.size() * 2 * kChunkBytes);
  H.d_weight = !any_loose ? nullptr
               : pts      ? (double*)(d + o_w)
                          : (double*)plan_alloc(ctx, P, P.owned, "hist_w", tcnt.size() * kTile * sizeof(double));
  H.d_more = d + o_more;
  H.d_tile_cnt = (int*)(d + o_cnt);
  H.d_rows = (HistRow*)(d + o_rows);
  H.d_outs = (HistOut*)(d + o_outs);
  H.d_blocks = (HistBlock*)(d + o_blocks);
  H.d_start = (int2*)(d + o_start);
  H.acc_bins = acc_bins;
  H.widest = widest;
  H.loose_bins = loose_bins;
  H.d_acc = (unsigned long long*)plan_alloc(ctx, P, P.owned, "hist_acc", (size_t)(acc_bins + loose_bins) * 16);
  H.d_part = (double*)plan_alloc(ctx, P, P.owned, "hist_part", part_rows * (size_t)P.nq * sizeof(double));
  constexpr auto smem_max = cudaFuncAttributeMaxDynamicSharedMemorySize;
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_hist_pairs<kCounts>, smem_max, hist_smem<kCounts>()));
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_hist_pairs<kLooseShared>, smem_max, hist_smem<kLooseShared>()));
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_hist_pairs<kLooseGlobal>, smem_max, hist_smem<kLooseGlobal>()));
  H.active = true;
  P.hist = std::move(H);
  if (!P.d_q) P.d_q = (double*)(d + o_q);
  undo.on = false;
  return true;
}

// The sums of a one-shot call reach 8 GB (hundreds of types with odd weights),
// which its context would keep for good; such a call takes 10 ms and more, a new
// allocation about one.
HistPoolRelease::~HistPoolRelease() {
  for (auto it = ctx->bufs.lower_bound("pair.hist"); it != ctx->bufs.end() && it->first.compare(0, 9, "pair.hist") == 0;) {
    if (it->second.bytes > kHistKeepBytes) {
      cudaFree(it->second.ptr);
      it = ctx->bufs.erase(it);
    } else {
      ++it;
    }
  }
}

void hist_plan_launch(crab_ctx* ctx, PairPlan& P, cudaStream_t s) {
  HistPart& H = P.hist;
  const int nq = (int)P.nq, qblocks = (nq + kHistQ - 1) / kHistQ;
  unsigned long long* cnt = H.d_acc;
  unsigned long long* sum = cnt + H.acc_bins;
  unsigned long long* lcnt = sum + H.acc_bins;
  unsigned long long* lsum = lcnt + H.loose_bins;
  for (size_t i = 0; i < H.groups.size(); ++i) {
    const HistGroup& g = H.groups[i];
    CRAB_CUDA_CHECK(cudaMemsetAsync(H.d_acc, 0, (size_t)(H.acc_bins + H.loose_bins) * 16, s));
    if (g.n_rows) {
      k_hist_pairs<kCounts><<<g.grid, kHT, hist_smem<kCounts>(), s>>>(
          H.d_pts, H.d_tile_cnt, nullptr, H.d_rows + g.row0, H.d_start + g.start0, cnt, sum, H.widest, 1.0, P.d_status,
          ctx->wait_budget);
      CRAB_CUDA_CHECK(cudaGetLastError());
      ctx->launches += 1;
    }
    if (H.loose_grid) {  // with loose rows there is one group
      if (H.widest <= kLooseMaxBins)
        k_hist_pairs<kLooseShared><<<H.loose_grid, kHT, hist_smem<kLooseShared>(), s>>>(
            H.d_pts, H.d_tile_cnt, H.d_weight, H.d_rows + H.loose_row0, H.d_start + H.loose_start0, lcnt, lsum,
            H.widest, H.scale, P.d_status, ctx->wait_budget);
      else
        k_hist_pairs<kLooseGlobal><<<H.loose_grid, kHT, hist_smem<kLooseGlobal>(), s>>>(
            H.d_pts, H.d_tile_cnt, H.d_weight, H.d_rows + H.loose_row0, H.d_start + H.loose_start0, lcnt, lsum, 0,
            H.scale, P.d_status, ctx->wait_budget);
      CRAB_CUDA_CHECK(cudaGetLastError());
      ctx->launches += 1;
    }
    k_hist_transform<<<dim3(g.slices, qblocks, g.n_blocks), kHistQ, 0, s>>>(cnt, sum, lcnt, lsum, H.d_outs + g.out0,
                                                                           H.d_blocks + g.block0, g.n_out, g.slice,
                                                                           1.0 / H.scale, P.d_q, nq, H.d_part);
    CRAB_CUDA_CHECK(cudaGetLastError());
    k_hist_reduce<<<(unsigned)(((int64_t)g.n_out * nq + 31) / 32), dim3(32, 8), 0, s>>>(H.d_part, H.d_outs + g.out0, g.n_out,
                                                                                 g.slice, nq, P.d_out);
    CRAB_CUDA_CHECK(cudaGetLastError());
    ctx->launches += 2;
  }
}

}  // namespace crab
