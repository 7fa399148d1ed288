// Hydration-shell site placement on a voxel grid, bit-exact against the
// reference.
//
// Adaptive coarse shell (crabSAXS src/solvent.rs:121-223): a voxel centre is a
// site when it lies within the outer radius (clearance + shell width) of some
// atom and not within the clearance of any atom; sites are listed in z→y→x
// voxel order.  Exterior shell (src/solvent.rs:259-401): voxels inside a vdW +
// probe sphere are molecular, the unknown voxels 6-connected to the box
// boundary are exterior, and exterior voxels within vdW + probe + thickness of
// an atom are sites.
//
// Exactness: every per-voxel decision in the reference is an OR over atoms of
// (voxel inside the atom's clipped bounding box) AND (squared distance <=
// r² + 1e-10), and the flood fill's result is the connected component of the
// boundary, independent of visiting order.  The device evaluates the same f64
// expressions in the same order with explicitly rounded intrinsics (no fused
// multiply-add), so the site set and its order equal the reference's.  The
// O(N) prologue (centroid, Rg, bounding box) runs on the host in the
// reference's sequential order.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "engine.hpp"

namespace crab {
namespace {

struct Box {
  double mn[3];
  double spacing;
  uint64_t n[3];
};

__device__ __forceinline__ double norm2_rn(double dx, double dy, double dz) {
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// One end of the clipped voxel range of one atom along d (solvent.rs:187-194 /
// 322-329): of p - radius (up 0) or p + radius (up 1).
__device__ __forceinline__ uint32_t range_end(const Box& b, double p, double radius, int d, bool up) {
  const double t = __ddiv_rn(__dsub_rn(up ? __dadd_rn(p, radius) : __dsub_rn(p, radius), b.mn[d]), b.spacing);
  if (!up) return (uint32_t)fmax(floor(__dsub_rn(t, 1e-10)), 0.0);
  const double c = ceil(__dadd_rn(t, 1e-10));
  const uint64_t cu = c > 0.0 ? (uint64_t)c : 0ull;
  return (uint32_t)(cu < b.n[d] - 1 ? cu : b.n[d] - 1);
}

// The voxels x of [lo, hi] on the row at (dy, dz) from the atom whose squared
// distance passes the threshold.  The distance is monotone in |x - p| also as
// rounded (every rounding is), so they are an interval: its ends come from the
// square root, and only a voxel closer to an end than the rounding of that
// estimate can move it is tested itself.  False: none.
__device__ __forceinline__ bool row_interval(const Box& b, double inv_spacing, double p, double radius, double thr,
                                             double dy, double dz, uint32_t lo, uint32_t hi, uint32_t& first,
                                             uint32_t& last) {
  const double dyz = __dadd_rn(__dmul_rn(dy, dy), __dmul_rn(dz, dz));
  const double left = thr - dyz;  // error below 1e-15 (thr + dyz)
  if (left < -1e-13 * thr) return false;
  const double half = sqrt(fmax(left, 0.0));
  // half is within 1e-6 of the radius (left near zero), voxel positions within
  // a few roundings of the coordinates
  double margin = 1e-3 + (1e-6 * radius + 1e-14 * (fabs(p) + fabs(b.mn[0]))) * inv_spacing;
  if (!isfinite(left)) margin = __longlong_as_double(0x7ff0000000000000ll);  // every voxel is tested
  const double t0 = (p - half - b.mn[0]) * inv_spacing, t1 = (p + half - b.mn[0]) * inv_spacing;
  const double f = ceil(t0 - margin), l = floor(t1 + margin);
  int64_t i = f > (double)lo ? (f > (double)hi ? (int64_t)hi + 1 : (int64_t)f) : (int64_t)lo;
  int64_t j = l < (double)hi ? (l < (double)lo ? (int64_t)lo - 1 : (int64_t)l) : (int64_t)hi;
  auto pass = [&](int64_t v) {
    const double px = __dadd_rn(b.mn[0], __dmul_rn((double)v, b.spacing));
    return norm2_rn(__dsub_rn(px, p), dy, dz) <= thr;
  };
  while (i <= j && !((double)i >= t0 + margin) && !pass(i)) ++i;
  while (i <= j && !((double)j <= t1 - margin) && !pass(j)) --j;
  first = (uint32_t)i;
  last = (uint32_t)j;
  return i <= j;
}

// Sets bits c0 .. c1; words that have them already are left alone (most of the
// rows inside the molecule).
__device__ __forceinline__ void set_bits(uint32_t* mask, uint32_t c0, uint32_t c1) {
  for (uint32_t w = c0 >> 5; w <= c1 >> 5; ++w) {
    uint32_t m = 0xffffffffu;
    if (w == c0 >> 5) m &= 0xffffffffu << (c0 & 31u);
    if (w == c1 >> 5) m &= 0xffffffffu >> (31u - (c1 & 31u));
    if (m & ~__ldcg(mask + w)) atomicOr(mask + w, m);
  }
}

// One warp per atom, a lane per row (y, z) of the atom's box: marks the row's
// voxels within the outer radius in one bitmap and those of the inner radius'
// own box within the inner radius in a second one (bit c for voxel c, in voxel
// order).  The ends of the ranges are one f64 division each, a lane for each.
// A test and a byte store per voxel was bound by its instructions (20,000
// atoms at 1 Angstrom: 35 us for the inner and 144 us for the outer spheres;
// 58,870 at 4, both spheres: 49 us); a row is one square root and one or two
// words (29, and 61 us for both of the exterior grid's spheres at once; 53 us
// at 4 Angstrom, where a warp's fixed part is most of it).  Voxel numbers fit 32 bits: a grid has at most 4e9 voxels.
__global__ void k_rasterize(const double* __restrict__ xyz, const double* __restrict__ radius_per_atom,
                            double outer_add, double inner_add, int64_t n, Box b, double inv, uint32_t* __restrict__ outer,
                            uint32_t* __restrict__ inner) {
  const int lane = threadIdx.x & 31;
  const int64_t atom = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (atom >= n) return;
  const double p[3] = {xyz[3 * atom], xyz[3 * atom + 1], xyz[3 * atom + 2]};
  const double ro = radius_per_atom ? __dadd_rn(radius_per_atom[atom], outer_add) : outer_add;
  const double ri = radius_per_atom ? __dadd_rn(radius_per_atom[atom], inner_add) : inner_add;
  const double to = __dadd_rn(__dmul_rn(ro, ro), 1e-10), ti = __dadd_rn(__dmul_rn(ri, ri), 1e-10);
  // lane 6 w + 3 u + d: end u along d of the outer (w 0) or inner range
  const int d = lane % 3, w = lane / 6;
  const double pd = d == 0 ? p[0] : (d == 1 ? p[1] : p[2]);
  const uint32_t end = lane < 12 ? range_end(b, pd, w ? ri : ro, d, lane % 6 >= 3) : 0u;
  uint32_t lo[3], hi[3], li[3], hj[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = __shfl_sync(0xffffffffu, end, k);
    hi[k] = __shfl_sync(0xffffffffu, end, 3 + k);
    li[k] = __shfl_sync(0xffffffffu, end, 6 + k);
    hj[k] = __shfl_sync(0xffffffffu, end, 9 + k);
  }
  if (hi[0] < lo[0] || hi[1] < lo[1] || hi[2] < lo[2]) return;  // then so is the inner range
  const uint32_t nx = (uint32_t)b.n[0], ny = (uint32_t)b.n[1];
  const uint32_t ey = hi[1] - lo[1] + 1, ez = hi[2] - lo[2] + 1;
  // this lane's first row, and the step of 32 rows in the same radices
  const uint32_t sy = 32u % ey, sz = 32u / ey;
  uint32_t y = (uint32_t)lane % ey, z = (uint32_t)lane / ey;
  while (z < ez) {
    const uint32_t vy = lo[1] + y, vz = lo[2] + z;
    const double dy = __dsub_rn(__dadd_rn(b.mn[1], __dmul_rn((double)vy, b.spacing)), p[1]);
    const double dz = __dsub_rn(__dadd_rn(b.mn[2], __dmul_rn((double)vz, b.spacing)), p[2]);
    const uint32_t row = (vz * ny + vy) * nx;
    uint32_t i, j;
    if (row_interval(b, inv, p[0], ro, to, dy, dz, lo[0], hi[0], i, j)) set_bits(outer, row + i, row + j);
    if (vy >= li[1] && vy <= hj[1] && vz >= li[2] && vz <= hj[2] && li[0] <= hj[0] &&
        row_interval(b, inv, p[0], ri, ti, dy, dz, li[0], hj[0], i, j))
      set_bits(inner, row + i, row + j);
    y += sy;
    z += sz;
    if (y >= ey) {
      y -= ey;
      ++z;
    }
  }
}

// Words of a bitmap, with one more that is read past the last (fill_row).
__host__ __device__ inline uint64_t mask_words(uint64_t count) { return (count + 31) / 32 + 1; }

// Sites among voxels 32 w .. 32 w + 31: in a and not in b (adaptive: outer and
// inner bitmaps) or in both (exterior: exterior and outer bitmaps).
__device__ __forceinline__ uint32_t site_bits(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                                              uint64_t w, uint64_t words, int both) {
  if (w >= words) return 0u;
  return a[w] & (both ? b[w] : ~b[w]);
}

constexpr int kScanThreads = 256;
constexpr int kChunk = kScanThreads * 32;  // voxels; a word per thread

__global__ void k_count(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint64_t words, int both,
                        uint32_t* __restrict__ chunk_count) {
  __shared__ uint32_t s[kScanThreads / 32];
  uint32_t c = __popc(site_bits(a, b, (uint64_t)blockIdx.x * kScanThreads + threadIdx.x, words, both));
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) t += s[w];
    chunk_count[blockIdx.x] = t;
  }
}

// Exclusive scan of chunk counts in one block of 1024 threads; total at offsets[n].
__global__ void k_scan_chunks(const uint32_t* __restrict__ cnt, uint64_t n, uint64_t* __restrict__ offsets) {
  __shared__ uint64_t warp_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t per = (n + blockDim.x - 1) / blockDim.x;
  const uint64_t b0 = threadIdx.x * per, b1 = min(n, b0 + per);
  uint64_t s = 0;
  for (uint64_t i = b0; i < b1; ++i) s += cnt[i];
  uint64_t incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  uint64_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < 32; ++w) {
    if (w < warp) before += warp_sum[w];
    all += warp_sum[w];
  }
  if (threadIdx.x == 0) offsets[n] = all;
  uint64_t run = before + incl - s;
  for (uint64_t i = b0; i < b1; ++i) {
    offsets[i] = run;
    run += cnt[i];
  }
}

// Position of a thread's first site: sites of the blocks before, of the warps
// before and of the lanes before (voxel order).
__device__ __forceinline__ uint64_t site_position(uint32_t c, const uint64_t* __restrict__ offsets) {
  __shared__ uint32_t warp_tot[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += warp_tot[w];
  return offsets[blockIdx.x] + before + incl - c;
}

__global__ void k_emit(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint64_t words, int both, Box bx,
                       const uint64_t* __restrict__ offsets, double* __restrict__ sites, int32_t* __restrict__ cells) {
  const uint64_t w = (uint64_t)blockIdx.x * kScanThreads + threadIdx.x;
  uint32_t bits = site_bits(a, b, w, words, both);
  uint64_t pos = site_position(__popc(bits), offsets);
  const uint32_t nx = (uint32_t)bx.n[0], ny = (uint32_t)bx.n[1];  // a grid has fewer than 2^32 voxels
  for (; bits; bits &= bits - 1u, ++pos) {
    const uint32_t v = (uint32_t)(w * 32) + (uint32_t)(__ffs(bits) - 1);
    const uint32_t row = v / nx, x = v - row * nx, z = row / ny, y = row - z * ny;
    sites[3 * pos] = __dadd_rn(bx.mn[0], __dmul_rn((double)x, bx.spacing));
    sites[3 * pos + 1] = __dadd_rn(bx.mn[1], __dmul_rn((double)y, bx.spacing));
    sites[3 * pos + 2] = __dadd_rn(bx.mn[2], __dmul_rn((double)z, bx.spacing));
    cells[3 * pos] = (int32_t)x;
    cells[3 * pos + 1] = (int32_t)y;
    cells[3 * pos + 2] = (int32_t)z;
  }
}

// Bits x0 .. x0 + 31 of the row whose first voxel is c, of a bitmap in voxel
// order (the caller clears those past the row's end).
__device__ __forceinline__ uint32_t fill_row(const uint32_t* __restrict__ bits, uint64_t c) {
  return __funnelshift_r(bits[c >> 5], bits[(c >> 5) + 1], (uint32_t)(c & 31));
}

// Exterior flood fill on bits, in shared memory: a cluster of kFillCtas CTAs,
// each holding a slab of z planes as two bitmaps of rows, 32 voxels along x a
// word (open: not molecular; ext: exterior).  A round carries the exterior
// label both ways along x (runs of open bits filled by one addition per word
// and direction), along y (32 lines a word, a warp per column of words: the
// maps of the label through the lanes' parts compose in a shuffle scan) and
// along z (a thread per column, across slabs from the neighbours' boundary
// planes), until a round changes nothing in any slab.  The result is the
// 6-connected component of the boundary's open voxels, as k_sweep's fixed
// point is.  Every round but the last labels a voxel, so there are no more
// rounds than voxels.  Rows are an odd number of words apart and so are the
// lanes' parts along y: a warp's words lie in different banks.  One launch
// instead of three per round of sweeps over bytes: 20,000 atoms, 1.17 million
// voxels, few rounds: 250 us in the sweeps' launches, 138 us with a thread per
// line of words along y and rows a multiple of four words apart, 26 us so; a box
// of 1.28 million whose pockets take eleven rounds 97 us (450 with the sweeps).
constexpr int kFillCtas = 8, kFillThreads = 1024;
constexpr size_t kFillSmem = 220 * 1024;
__host__ __device__ inline uint64_t fill_row_words(const Box& b) { return ((b.n[0] + 31) / 32) | 1; }
__host__ __device__ inline uint64_t fill_words(const Box& b) {  // of one bitmap of a slab
  return ((b.n[2] + kFillCtas - 1) / kFillCtas) * b.n[1] * fill_row_words(b);
}

// Bits of the runs of m from each seed (a subset of m) upwards: the addition's
// carry runs from a run's lowest seed to the run's end.
__device__ __forceinline__ uint32_t fill_up(uint32_t m, uint32_t seed) { return (((m + seed) ^ m) & m) | seed; }

// mol: bitmap of the molecular voxels; exterior: cleared bitmap, set here.
__global__ void __cluster_dims__(kFillCtas, 1, 1) __launch_bounds__(kFillThreads, 1)
    k_flood_fill(const uint32_t* __restrict__ mol, uint32_t* __restrict__ exterior, Box b) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ uint32_t fill_smem[];
  __shared__ int changed[2];
  const int rank = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t nx = (uint32_t)b.n[0], ny = (uint32_t)b.n[1], nz = (uint32_t)b.n[2], nw = (nx + 31) / 32;
  const uint32_t rw = (uint32_t)fill_row_words(b), plane = ny * rw;
  const uint32_t slab = (nz + kFillCtas - 1) / kFillCtas, z0 = min(nz, rank * slab), zs = min(nz, z0 + slab) - z0;
  uint32_t* open = fill_smem;
  uint32_t* ext = fill_smem + (size_t)slab * plane;
  // a thread per word, boundary voxels seeded
#pragma unroll 4
  for (uint32_t w = tid; w < zs * ny * nw; w += kFillThreads) {
    const uint32_t r = w / nw, k = w - r * nw, z = z0 + r / ny, y = r % ny, left = nx - 32 * k;
    const uint32_t valid = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
    const uint32_t m = ~fill_row(mol, ((uint64_t)z * ny + y) * nx + 32 * k) & valid;
    uint32_t edge = y == 0 || y + 1 == ny || z == 0 || z + 1 == nz ? 0xffffffffu : 0u;
    if (k == 0) edge |= 1u;
    if (left <= 32) edge |= 1u << (left - 1);
    open[r * rw + k] = m;
    ext[r * rw + k] = m & edge;
  }
  if (tid < 2) changed[tid] = 0;
  cl.sync();
  const uint32_t part = ((ny + 31) / 32) | 1;  // rows of a lane along y
  for (uint32_t round = 0;; ++round) {
    int any = 0;
    // x: a thread per row
    for (uint32_t r = tid; r < zs * ny; r += kFillThreads) {
      uint32_t* e = ext + (size_t)r * rw;
      const uint32_t* m = open + (size_t)r * rw;
      uint32_t carry = 0;
      for (uint32_t k = 0; k < nw; ++k) {
        const uint32_t old = e[k], v = fill_up(m[k], (old | carry) & m[k]);
        if (v != old) {
          e[k] = v;
          any = 1;
        }
        carry = v >> 31;
      }
      carry = 0;
      for (uint32_t k = nw; k-- > 0;) {
        const uint32_t old = e[k], mr = __brev(m[k]);
        const uint32_t v = __brev(fill_up(mr, (__brev(old) | carry) & mr));
        if (v != old) {
          e[k] = v;
          any = 1;
        }
        carry = v & 1u;
      }
    }
    __syncthreads();
    // y: a warp per column of words of a plane, lanes in order of y
    for (uint32_t l = warp; l < zs * nw; l += kFillThreads / 32) {
      const uint32_t at = (l / nw) * plane + l % nw, y0 = min(ny, lane * part), y1 = min(ny, y0 + part);
#pragma unroll
      for (int dir = 0; dir < 2; ++dir) {
        // the label after this lane's rows is g | (label before & t)
        uint32_t g = 0u, t = 0xffffffffu;
#pragma unroll 4
        for (uint32_t k = y0; k < y1; ++k) {
          const uint32_t i = at + (dir == 0 ? k : y1 - 1 - (k - y0)) * rw, m = open[i];
          g = ext[i] | (g & m);
          t &= m;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t pg = dir == 0 ? __shfl_up_sync(0xffffffffu, g, o) : __shfl_down_sync(0xffffffffu, g, o);
          const uint32_t pt = dir == 0 ? __shfl_up_sync(0xffffffffu, t, o) : __shfl_down_sync(0xffffffffu, t, o);
          if (dir == 0 ? lane >= o : lane + o < 32) {
            g |= pg & t;
            t &= pt;
          }
        }
        uint32_t c = dir == 0 ? __shfl_up_sync(0xffffffffu, g, 1) : __shfl_down_sync(0xffffffffu, g, 1);
        if (lane == (dir == 0 ? 0 : 31)) c = 0u;
#pragma unroll 4
        for (uint32_t k = y0; k < y1; ++k) {
          const uint32_t i = at + (dir == 0 ? k : y1 - 1 - (k - y0)) * rw, old = ext[i];
          c = old | (c & open[i]);
          if (c != old) {
            ext[i] = c;
            any = 1;
          }
        }
        __syncwarp();
      }
    }
    // the neighbours' boundary planes are read as they stand: a label that is
    // missed now was set since the last agreement, which then is not the last one
    cl.sync();
    const uint32_t* below = rank > 0 ? cl.map_shared_rank(ext, rank - 1) + (size_t)(slab - 1) * plane : nullptr;
    const uint32_t* above = rank + 1 < kFillCtas && z0 + zs < nz ? cl.map_shared_rank(ext, rank + 1) : nullptr;
    if (zs)
      for (uint32_t l = tid; l < ny * nw; l += kFillThreads) {
        const uint32_t at = (l / nw) * rw + l % nw;
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
          uint32_t c = dir == 0 ? (below ? below[at] : 0u) : (above ? above[at] : 0u);
#pragma unroll 8
          for (uint32_t k = 0; k < zs; ++k) {
            const uint32_t i = at + (dir == 0 ? k : zs - 1 - k) * plane, old = ext[i];
            c = old | (c & open[i]);
            if (c != old) {
              ext[i] = c;
              any = 1;
            }
          }
        }
      }
    if (__syncthreads_or(any) && tid == 0)
      for (int r = 0; r < kFillCtas; ++r) *cl.map_shared_rank(&changed[round & 1], r) = 1;
    cl.sync();
    const int go = changed[round & 1];
    if (tid == 0) changed[(round & 1) ^ 1] = 0;  // of the next round, which sets it after its barriers
    if (!go) break;
  }
  for (uint32_t w = tid; w < zs * ny * nw; w += kFillThreads) {
    const uint32_t r = w / nw, k = w - r * nw, v = ext[r * rw + k];
    const uint64_t c = ((uint64_t)(z0 + r / ny) * ny + r % ny) * nx + 32 * k;
    const uint32_t sh = (uint32_t)(c & 31);
    if (v << sh) atomicOr(exterior + (c >> 5), v << sh);
    if (sh && v >> (32 - sh)) atomicOr(exterior + (c >> 5) + 1, v >> (32 - sh));
  }
  cl.sync();  // no CTA leaves while a neighbour may still read its slab
}

// Voxel states of the sweeps from the molecular bitmap (0 unknown, 1
// molecular), and the exterior (2) voxels' bitmap from the states.
__global__ void k_fill_states(const uint32_t* __restrict__ mol, uint64_t count, uint8_t* __restrict__ s) {
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < count; c += (uint64_t)gridDim.x * blockDim.x)
    s[c] = (uint8_t)(mol[c >> 5] >> (c & 31) & 1u);
}

__global__ void k_fill_bits(const uint8_t* __restrict__ s, uint64_t count, uint32_t* __restrict__ exterior) {
  // whole warps: the loop's bound is a multiple of 32
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < (count + 31) / 32 * 32;
       c += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t bits = __ballot_sync(0xffffffffu, c < count && s[c] == 2);
    if ((c & 31) == 0) exterior[c >> 5] = bits;
  }
}

// Exterior flood fill: boundary seeds, then line sweeps along x, y and z that
// carry the exterior label (2) through unknown voxels (0), repeated until no
// voxel changes.  The fixed point is the 6-connected component of the
// boundary's unknown voxels, i.e. the reference's BFS result.
__global__ void k_seed_boundary(uint8_t* __restrict__ s, Box b) {
  const uint64_t count = b.n[0] * b.n[1] * b.n[2];
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < count; c += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t x = c % b.n[0], y = (c / b.n[0]) % b.n[1], z = c / (b.n[0] * b.n[1]);
    const bool edge = x == 0 || x + 1 == b.n[0] || y == 0 || y + 1 == b.n[1] || z == 0 || z + 1 == b.n[2];
    if (edge && s[c] == 0) s[c] = 2;
  }
}

// Voxels of a line a thread loads before it carries the label through them:
// one memory latency per batch instead of one per voxel.
constexpr int kSweepBatch = 16;
// Sweep rounds enqueued between two reads of the change flag by the host.
constexpr int kRoundsPerSync = 6;

// One thread per line; axis 0: lines along x (one per (y,z)); 1: along y;
// 2: along z.  A forward and a backward pass each carry the exterior label
// through runs of unknown voxels.  Lines of one axis are disjoint, so threads
// never touch the same voxel.  The round returns at once when the previous
// round changed nothing (*prev_changed == 0): the fixed point is reached.
__global__ void k_sweep(uint8_t* __restrict__ s, Box b, int axis, const int* __restrict__ prev_changed,
                        int* __restrict__ changed) {
  if (prev_changed && *prev_changed == 0) return;
  const uint64_t nx = b.n[0], ny = b.n[1], nz = b.n[2];
  uint64_t lines, len, stride;
  if (axis == 0) { lines = ny * nz; len = nx; stride = 1; }
  else if (axis == 1) { lines = nx * nz; len = ny; stride = nx; }
  else { lines = nx * ny; len = nz; stride = nx * ny; }
  const uint64_t l = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= lines) return;
  uint64_t start;
  if (axis == 0) start = l * nx;                       // l = z*ny + y
  else if (axis == 1) start = (l / nx) * nx * ny + (l % nx);  // l = z*nx + x
  else start = l;                                       // l = y*nx + x
  uint8_t* line = s + start;
  int any = 0;
  bool carry = false;
  // voxels past either end read as molecular (1): never written, stop the carry
  for (uint64_t i0 = 0; i0 < len; i0 += kSweepBatch) {
    uint8_t v[kSweepBatch];
#pragma unroll
    for (int k = 0; k < kSweepBatch; ++k) v[k] = i0 + k < len ? line[(i0 + k) * stride] : (uint8_t)1;
#pragma unroll
    for (int k = 0; k < kSweepBatch; ++k) {
      if (v[k] == 2) carry = true;
      else if (v[k] == 0) {
        if (carry) {
          line[(i0 + k) * stride] = 2;
          any = 1;
        }
      } else carry = false;
    }
  }
  carry = false;
  for (uint64_t e = len; e > 0;) {
    const uint64_t i0 = e - 1;  // this batch covers i0, i0 - 1, ..., down to index 0 at most
    uint8_t v[kSweepBatch];
#pragma unroll
    for (int k = 0; k < kSweepBatch; ++k) v[k] = (uint64_t)k <= i0 ? line[(i0 - k) * stride] : (uint8_t)1;
#pragma unroll
    for (int k = 0; k < kSweepBatch; ++k) {
      if (v[k] == 2) carry = true;
      else if (v[k] == 0) {
        if (carry) {
          line[(i0 - k) * stride] = 2;
          any = 1;
        }
      } else carry = false;
    }
    e = e > (uint64_t)kSweepBatch ? e - kSweepBatch : 0;
  }
  if (any) atomicOr(changed, 1);
}

// Lines of at most kWarpLine voxels are swept by one warp each: lane l holds
// voxels 4l .. 4l+3 (past the end of the line: molecular, never written).
// The forward pass carries the label through a voxel by one of three maps of
// the carry (exterior: set, molecular: clear, unknown: unchanged), and maps of
// this kind compose as "the later constant wins"; an inclusive shuffle scan of
// the lanes' composed maps gives every lane its incoming carry, and the lane
// then steps through its four voxels as the sequential pass does.  The
// backward pass does the same from the right on the updated voxels, so the
// line ends as k_sweep's forward and backward passes leave it.
constexpr int kWarpLine = 128;

// Carry map of four voxels in the given order: (constant?, value).
__device__ __forceinline__ void carry_map(const uint8_t (&v)[4], bool forward, int& is_const, int& value) {
  is_const = 0;
  value = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint8_t x = v[forward ? e : 3 - e];
    if (x == 2) { is_const = 1; value = 1; }
    else if (x != 0) { is_const = 1; value = 0; }
  }
}

__global__ void k_sweep_warp(uint8_t* __restrict__ s, Box b, int axis, const int* __restrict__ prev_changed,
                             int* __restrict__ changed) {
  if (prev_changed && *prev_changed == 0) return;
  const uint64_t nx = b.n[0], ny = b.n[1], nz = b.n[2];
  uint64_t lines, len, stride;
  if (axis == 0) { lines = ny * nz; len = nx; stride = 1; }
  else if (axis == 1) { lines = nx * nz; len = ny; stride = nx; }
  else { lines = nx * ny; len = nz; stride = nx * ny; }
  const uint64_t l = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // one line per warp
  if (l >= lines) return;  // the whole warp
  const int lane = threadIdx.x & 31;
  uint64_t start;
  if (axis == 0) start = l * nx;
  else if (axis == 1) start = (l / nx) * nx * ny + (l % nx);
  else start = l;
  uint8_t* line = s + start;
  uint8_t v[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint64_t k = (uint64_t)(4 * lane + e);
    v[e] = k < len ? line[k * stride] : (uint8_t)1;
  }
  unsigned wrote = 0u;  // bit e: voxel e became exterior
  // forward: lanes in increasing order
  int c, val;
  carry_map(v, true, c, val);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int pc = __shfl_up_sync(0xffffffffu, c, o), pv = __shfl_up_sync(0xffffffffu, val, o);
    if (lane >= o && !c) { c = pc; val = pv; }
  }
  int carry = __shfl_up_sync(0xffffffffu, val, 1);
  if (lane == 0) carry = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (v[e] == 2) carry = 1;
    else if (v[e] == 0) {
      if (carry) { v[e] = 2; wrote |= 1u << e; }
    } else carry = 0;
  }
  // backward: lanes in decreasing order, on the updated voxels
  carry_map(v, false, c, val);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int pc = __shfl_down_sync(0xffffffffu, c, o), pv = __shfl_down_sync(0xffffffffu, val, o);
    if (lane + o < 32 && !c) { c = pc; val = pv; }
  }
  carry = __shfl_down_sync(0xffffffffu, val, 1);
  if (lane == 31) carry = 0;
#pragma unroll
  for (int e = 3; e >= 0; --e) {
    if (v[e] == 2) carry = 1;
    else if (v[e] == 0) {
      if (carry) { v[e] = 2; wrote |= 1u << e; }
    } else carry = 0;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (wrote & (1u << e)) line[(uint64_t)(4 * lane + e) * stride] = 2;
  if (__any_sync(0xffffffffu, wrote != 0u) && lane == 0) atomicOr(changed, 1);
}

// Grid buffers live in the context's pool ("grid." slots), so repeated calls
// allocate nothing.  A slot above kGridKeepBytes (a box of more than 2^28
// voxels) is released when the build ends, so a one-off large box does not
// keep its memory; a build that leaves its sites and their cells on the device
// keeps those slots, which trim_grid_pool releases once they are read.
constexpr size_t kGridKeepBytes = 256ull << 20;

template <class T>
T* pool(crab_ctx* ctx, const char* name, size_t count) {
  return (T*)ctx->dev(name, std::max<size_t>(count, 1) * sizeof(T));
}

void trim_slots(crab_ctx* ctx, bool keep_sites) {
  for (auto it = ctx->bufs.lower_bound("grid."); it != ctx->bufs.end() && it->first.compare(0, 5, "grid.") == 0;) {
    if (it->second.bytes > kGridKeepBytes &&
        !(keep_sites && (it->first == "grid.sites" || it->first == "grid.cells"))) {
      cudaFree(it->second.ptr);
      it = ctx->bufs.erase(it);
    } else {
      ++it;
    }
  }
}

struct GridPoolTrim {
  crab_ctx* ctx;
  bool keep_sites;
  ~GridPoolTrim() { trim_slots(ctx, keep_sites); }
};

GridResult compact_sites(crab_ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t count, int both,
                         const Box& bx, bool to_host) {
  cudaStream_t s = ctx->stream;
  const uint64_t chunks = (count + kChunk - 1) / kChunk, words = (count + 31) / 32;
  uint32_t* d_cnt = pool<uint32_t>(ctx, "grid.chunk_count", chunks);
  uint64_t* d_off = pool<uint64_t>(ctx, "grid.chunk_offset", chunks + 1);
  k_count<<<(unsigned)chunks, kScanThreads, 0, s>>>(a, b, words, both, d_cnt);
  CRAB_CUDA_CHECK(cudaGetLastError());
  k_scan_chunks<<<1, 1024, 0, s>>>(d_cnt, chunks, d_off);
  CRAB_CUDA_CHECK(cudaGetLastError());
  uint64_t m = 0;
  copy_d2h(ctx, &m, d_off + chunks, sizeof(uint64_t), s);
  CRAB_CUDA_CHECK(cudaStreamSynchronize(s));
  trace_mark("sites counted");
  GridResult r;
  r.spacing = bx.spacing;
  r.m = (int64_t)m;
  r.build = ctx->grid_builds;
  if (m) {
    require(bx.n[0] < (1ull << 31) && bx.n[1] < (1ull << 31) && bx.n[2] < (1ull << 31), "grid axis too long");
    double* d_sites = pool<double>(ctx, "grid.sites", 3 * m);
    int32_t* d_cells = pool<int32_t>(ctx, "grid.cells", 3 * m);
    k_emit<<<(unsigned)chunks, kScanThreads, 0, s>>>(a, b, words, both, bx, d_off, d_sites, d_cells);
    CRAB_CUDA_CHECK(cudaGetLastError());
    r.d_sites = d_sites;
    r.d_cells = d_cells;
    if (to_host) {
      r.sites.resize(3 * m);
      r.cells.resize(3 * m);
      copy_d2h(ctx, r.sites.data(), d_sites, 3 * m * sizeof(double), s);
      copy_d2h(ctx, r.cells.data(), d_cells, 3 * m * sizeof(int32_t), s);
    }
    CRAB_CUDA_CHECK(cudaStreamSynchronize(s));
  }
  ctx->launches += m ? 4 : 3;
  return r;
}

const double* upload_xyz(crab_ctx* ctx, const double* xyz, int64_t n) {
  double* d = pool<double>(ctx, "grid.xyz", 3 * n);
  copy_h2d(ctx, d, xyz, 3 * n * sizeof(double), ctx->stream);
  return d;
}

// Box set-up shared by both grids (solvent.rs:160-176 / 290-306).
bool make_box(const AtomSweep& w, double pad, double spacing, Box* b, uint64_t* count) {
  double mx[3];
  for (int d = 0; d < 3; ++d) {
    b->mn[d] = w.mn[d] - pad;
    mx[d] = w.mx[d] + pad;
  }
  b->spacing = spacing;
  unsigned __int128 total = 1;
  for (int d = 0; d < 3; ++d) {
    const double span = std::ceil(((mx[d] - b->mn[d]) / spacing) - 1e-10);
    if (!(span < 9.0e18)) return false;
    b->n[d] = (uint64_t)std::max(span, 0.0) + 1;
    total *= b->n[d];
    if (total > (unsigned __int128)UINT64_MAX) return false;
  }
  *count = (uint64_t)total;
  return true;
}

}  // namespace

GridResult adaptive_grid_device(crab_ctx* ctx, const double* xyz, int64_t n, double spacing, double clearance,
                                double padding, bool to_host, const GridAtoms& have) {
  GridResult r;
  if (n == 0) {
    r.voxel_volume = adaptive_site_volume(spacing);
    return r;
  }
  require(std::isfinite(spacing) && spacing > 0.0 && std::isfinite(clearance) && clearance > 0.0 &&
              std::isfinite(padding) && padding >= 0.0,
          "adaptive hydration-grid dimensions must be finite and positive");
  AtomSweep own;
  if (!have.sweep) {
    sweep_box(xyz, n, own);
    sweep_radii(xyz, n, own);
  }
  const AtomSweep& w = have.sweep ? *have.sweep : own;
  const double inner = clearance, outer = clearance + adaptive_shell_width(w.rg);
  Box b;
  uint64_t count = 0;
  require(make_box(w, padding, spacing, &b, &count), "adaptive hydration grid is too large");
  require(count <= (uint64_t)4000000000ull, "adaptive hydration grid exceeds 4e9 voxels");
  TraceScope trace("adaptive_grid");
  ++ctx->grid_builds;
  GridPoolTrim trim{ctx, !to_host};
  cudaStream_t s = ctx->stream;
  const uint64_t words = mask_words(count);
  uint32_t* shell = pool<uint32_t>(ctx, "grid.masks", 2 * words);
  uint32_t* mol = shell + words;
  const double* d_xyz = have.d_xyz ? have.d_xyz : upload_xyz(ctx, xyz, n);
  CRAB_CUDA_CHECK(cudaMemsetAsync(shell, 0, 2 * words * sizeof(uint32_t), s));
  const unsigned blocks = (unsigned)((n * 32 + 255) / 256);
  k_rasterize<<<blocks, 256, 0, s>>>(d_xyz, nullptr, outer, inner, n, b, 1.0 / spacing, shell, mol);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 1;
  r = compact_sites(ctx, shell, mol, count, 0, b, to_host);
  r.voxel_volume = adaptive_site_volume(spacing);
  r.outer = outer;
  return r;
}

GridResult exterior_grid_device(crab_ctx* ctx, const double* xyz, const int8_t* elem, int64_t n, double spacing,
                                double probe, double thickness, bool to_host, const GridAtoms& have) {
  GridResult r;
  if (n == 0) {
    r.voxel_volume = (spacing * spacing) * spacing;
    return r;
  }
  require(std::isfinite(spacing) && spacing > 0.0 && std::isfinite(probe) && probe >= 0.0 &&
              std::isfinite(thickness) && thickness > 0.0,
          "solvent-grid dimensions must be finite and positive");
  double vmax = 0.0;
  std::vector<double> radius(n);
  for (int64_t i = 0; i < n; ++i) {
    radius[i] = vdw_radius(elem[i]);
    vmax = max_num(vmax, radius[i]);
  }
  const double margin = vmax + probe + thickness + spacing;
  AtomSweep own;
  if (!have.sweep) sweep_box(xyz, n, own);
  Box b;
  uint64_t count = 0;
  require(make_box(have.sweep ? *have.sweep : own, margin, spacing, &b, &count), "solvent grid is too large");
  if (count > 250000000ull)
    throw Error(CRAB_EINVAL, "solvent grid requires " + std::to_string(count) + " voxels; limit is 250000000");
  TraceScope trace("exterior_grid");
  ++ctx->grid_builds;
  GridPoolTrim trim{ctx, !to_host};
  cudaStream_t s = ctx->stream;
  // bitmaps: near an atom, molecular, exterior
  const uint64_t words = mask_words(count);
  uint32_t* near = pool<uint32_t>(ctx, "grid.masks", 3 * words);
  uint32_t* mol = near + words;
  uint32_t* exterior = mol + words;
  const double* d_xyz = have.d_xyz ? have.d_xyz : upload_xyz(ctx, xyz, n);
  double* d_rad = pool<double>(ctx, "grid.radius", n);
  CRAB_CUDA_CHECK(cudaMemsetAsync(near, 0, 3 * words * sizeof(uint32_t), s));
  copy_h2d(ctx, d_rad, radius.data(), n * sizeof(double), s);
  const unsigned blocks = (unsigned)((n * 32 + 255) / 256);
  k_rasterize<<<blocks, 256, 0, s>>>(d_xyz, d_rad, probe + thickness, probe, n, b, 1.0 / spacing, near, mol);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 1;
  // on bits in a cluster's shared memory while a slab of both bitmaps fits
  // (6 million voxels), else by sweeps over the states, a byte each
  if (2 * fill_words(b) * sizeof(uint32_t) <= kFillSmem) {
    CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_flood_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFillSmem));
    k_flood_fill<<<kFillCtas, kFillThreads, 2 * fill_words(b) * sizeof(uint32_t), s>>>(mol, exterior, b);
    CRAB_CUDA_CHECK(cudaGetLastError());
    ctx->launches += 1;
  } else {
    uint8_t* state = pool<uint8_t>(ctx, "grid.states", count);
    int* d_changed = pool<int>(ctx, "grid.changed", kRoundsPerSync);
    const unsigned wide = (unsigned)std::min<uint64_t>((count + 255) / 256, 65535);
    k_fill_states<<<wide, 256, 0, s>>>(mol, count, state);
    CRAB_CUDA_CHECK(cudaGetLastError());
    k_seed_boundary<<<wide, 256, 0, s>>>(state, b);
    CRAB_CUDA_CHECK(cudaGetLastError());
    ctx->launches += 2;
    // Sweep rounds until the fixed point, kRoundsPerSync rounds per read of the
    // flag: round k writes d_changed[k] and returns at once when round k - 1
    // changed nothing, so the last flag of a batch is 0 exactly when the fill
    // has converged.  Every productive round labels at least one voxel, so the
    // number of rounds cannot exceed the number of voxels.
    for (uint64_t round = 0; round <= count; round += kRoundsPerSync) {
      CRAB_CUDA_CHECK(cudaMemsetAsync(d_changed, 0, kRoundsPerSync * sizeof(int), s));
      for (int k = 0; k < kRoundsPerSync; ++k) {
        const int* prev = k ? d_changed + k - 1 : nullptr;
        for (int axis = 0; axis < 3; ++axis) {
          const uint64_t lines = axis == 0 ? b.n[1] * b.n[2] : axis == 1 ? b.n[0] * b.n[2] : b.n[0] * b.n[1];
          if (b.n[axis] <= (uint64_t)kWarpLine)  // one warp per line
            k_sweep_warp<<<(unsigned)((lines + 3) / 4), 128, 0, s>>>(state, b, axis, prev, d_changed + k);
          else  // one thread per line
            k_sweep<<<(unsigned)((lines + 127) / 128), 128, 0, s>>>(state, b, axis, prev, d_changed + k);
          CRAB_CUDA_CHECK(cudaGetLastError());
          ctx->launches += 1;
        }
      }
      int changed = 0;
      copy_d2h(ctx, &changed, d_changed + kRoundsPerSync - 1, sizeof(int), s);
      CRAB_CUDA_CHECK(cudaStreamSynchronize(s));
      if (!changed) break;
    }
    k_fill_bits<<<wide, 256, 0, s>>>(state, count, exterior);
    CRAB_CUDA_CHECK(cudaGetLastError());
    ctx->launches += 1;
  }
  trace_mark("flood fill");
  r = compact_sites(ctx, exterior, near, count, 1, b, to_host);
  r.voxel_volume = (spacing * spacing) * spacing;
  r.outer = vmax + probe + thickness;
  return r;
}

void trim_grid_pool(crab_ctx* ctx) { trim_slots(ctx, false); }

}  // namespace crab

// ------------------------------------------------------- no-allocation variant
//
// crab_hydration_grid_adaptive_noalloc is for callers that cannot allocate
// device memory through the CUDA runtime (a host runtime whose own allocator
// owns the device, a process that must keep its memory budget fixed, code
// running inside a callback where cudaMalloc is not allowed).  It takes
// device pointers for the atoms and the site output and keeps every
// temporary (voxel masks, chunk counts, offsets, the box header) in one
// file-scope __device__ array of fixed size, so it calls no cudaMalloc,
// cudaFree or allocating library routine.

#include <mutex>

namespace crab {
namespace {

constexpr uint64_t kNoAllocMaxVoxels = CRAB_NOALLOC_MAX_VOXELS;
static_assert(kNoAllocMaxVoxels % kChunk == 0, "voxel limit must be a whole number of scan chunks");
constexpr uint64_t kNoAllocChunks = kNoAllocMaxVoxels / kChunk;

struct NoAllocHeader {
  Box box;
  uint64_t count;
  double inner, outer;
  int status;  // 0 ok, 1 grid larger than the static scratch, 2 a coordinate not finite
};
static_assert(sizeof(NoAllocHeader) <= 256, "header must fit its 256-byte slot");

constexpr size_t kHdrBytes = 256;
constexpr size_t kShellOff = kHdrBytes;
constexpr size_t kMolOff = kShellOff + kNoAllocMaxVoxels / 8;
constexpr size_t kCntOff = kMolOff + kNoAllocMaxVoxels / 8;
constexpr size_t kOffOff = kCntOff + kNoAllocChunks * sizeof(uint32_t);
constexpr size_t kNoAllocBytes = kOffOff + (kNoAllocChunks + 1) * sizeof(uint64_t);

// The scratch shared by every call on a device; it keeps the last call's
// contents, and calls whose kernels overlap on the GPU race on it.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Single-thread prologue in the reference's sequential order
// (solvent.rs:144-176): centroid, radius of gyration, shell radii, padded box.
__global__ void k_noalloc_prologue(const double* __restrict__ xyz, int64_t n, double spacing, double clearance,
                                   double padding, NoAllocHeader* hdr) {
  double c[3] = {0.0, 0.0, 0.0};
  bool finite = true;  // the allocating entry point rejects the same input (crab_structure_create)
  for (int64_t i = 0; i < n; ++i)
    for (int d = 0; d < 3; ++d) {
      finite = finite && isfinite(xyz[3 * i + d]);
      c[d] = __dadd_rn(c[d], xyz[3 * i + d]);
    }
  if (!finite) {
    hdr->status = 2;
    hdr->count = 0ull;
    return;
  }
  for (int d = 0; d < 3; ++d) c[d] = __ddiv_rn(c[d], (double)n);
  double acc = 0.0;
  for (int64_t i = 0; i < n; ++i) {
    const double dx = __dsub_rn(xyz[3 * i], c[0]), dy = __dsub_rn(xyz[3 * i + 1], c[1]),
                 dz = __dsub_rn(xyz[3 * i + 2], c[2]);
    acc = __dadd_rn(acc, norm2_rn(dx, dy, dz));
  }
  const double rg = sqrt(__ddiv_rn(acc, (double)n));
  const double width = rg <= 15.0 ? 3.0 : (rg >= 20.0 ? 5.0 : __dadd_rn(3.0, __dmul_rn(0.4, __dsub_rn(rg, 15.0))));
  hdr->inner = clearance;
  hdr->outer = __dadd_rn(clearance, width);
  double mn[3] = {xyz[0], xyz[1], xyz[2]}, mx[3] = {xyz[0], xyz[1], xyz[2]};
  for (int64_t i = 1; i < n; ++i)
    for (int d = 0; d < 3; ++d) {
      mn[d] = fmin(mn[d], xyz[3 * i + d]);
      mx[d] = fmax(mx[d], xyz[3 * i + d]);
    }
  double total = 1.0;
  for (int d = 0; d < 3; ++d) {
    hdr->box.mn[d] = __dsub_rn(mn[d], padding);
    const double hi = __dadd_rn(mx[d], padding);
    const double span = ceil(__dsub_rn(__ddiv_rn(__dsub_rn(hi, hdr->box.mn[d]), spacing), 1e-10));
    const double nd = fmax(span, 0.0) + 1.0;
    total *= nd;
    hdr->box.n[d] = nd < 9.0e15 ? (uint64_t)nd : 0ull;
  }
  hdr->box.spacing = spacing;
  hdr->status = total > (double)kNoAllocMaxVoxels ? 1 : 0;
  hdr->count = hdr->status ? 0ull : hdr->box.n[0] * hdr->box.n[1] * hdr->box.n[2];
}

// k_emit restricted to the caller's capacity; no voxel indices.
__global__ void k_noalloc_emit(const uint32_t* __restrict__ shell, const uint32_t* __restrict__ mol, uint64_t words,
                               Box bx, const uint64_t* __restrict__ offsets, double* __restrict__ sites,
                               uint64_t capacity) {
  const uint64_t w = (uint64_t)blockIdx.x * kScanThreads + threadIdx.x;
  uint32_t bits = site_bits(shell, mol, w, words, 0);
  uint64_t pos = site_position(__popc(bits), offsets);
  const uint32_t nx = (uint32_t)bx.n[0], ny = (uint32_t)bx.n[1];
  for (; bits && pos < capacity; bits &= bits - 1u, ++pos) {
    const uint32_t v = (uint32_t)(w * 32) + (uint32_t)(__ffs(bits) - 1);
    const uint32_t row = v / nx, x = v - row * nx, z = row / ny, y = row - z * ny;
    sites[3 * pos] = __dadd_rn(bx.mn[0], __dmul_rn((double)x, bx.spacing));
    sites[3 * pos + 1] = __dadd_rn(bx.mn[1], __dmul_rn((double)y, bx.spacing));
    sites[3 * pos + 2] = __dadd_rn(bx.mn[2], __dmul_rn((double)z, bx.spacing));
  }
}

// Device address of the scratch array, looked up once per device (the name
// g_noalloc_scratch is only a host-side handle; kernels need this address).
// The cached address belongs to the device's current CUDA context: after a
// cudaDeviceReset of that device it is stale, so a process that resets a
// device must not call the entry point on it again.
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_dev[256] = {};

cudaError_t noalloc_scratch(unsigned char** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 256) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  if (!g_noalloc_dev[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_dev[dev] = (unsigned char*)p;
  }
  *out = g_noalloc_dev[dev];
  return cudaSuccess;
}

}  // namespace
}  // namespace crab

extern "C" int crab_hydration_grid_adaptive_noalloc(const double* d_xyz, int64_t n, double spacing, double clearance,
                                                    double padding, double* d_sites, int64_t capacity, int64_t* m,
                                                    double* voxel_volume, void* stream) {
  using namespace crab;
  if (n < 0 || capacity < 0 || !m || (n > 0 && !d_xyz) || (capacity > 0 && !d_sites)) return CRAB_EINVAL;
  if (!std::isfinite(spacing) || spacing <= 0.0 || !std::isfinite(clearance) || clearance <= 0.0 ||
      !std::isfinite(padding) || padding < 0.0)
    return CRAB_EINVAL;
  if (voxel_volume) *voxel_volume = adaptive_site_volume(spacing);
  *m = 0;
  if (n == 0) return CRAB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  unsigned char* base = nullptr;
  if (noalloc_scratch(&base) != cudaSuccess) return CRAB_ECUDA;
  NoAllocHeader* hdr = (NoAllocHeader*)base;
  k_noalloc_prologue<<<1, 1, 0, s>>>(d_xyz, n, spacing, clearance, padding, hdr);
  if (cudaGetLastError() != cudaSuccess) return CRAB_ECUDA;
  NoAllocHeader h;
  if (cudaMemcpyAsync(&h, hdr, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess) return CRAB_ECUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return CRAB_ECUDA;
  if (h.status) return CRAB_EINVAL;  // a coordinate not finite, or a grid larger than CRAB_NOALLOC_MAX_VOXELS
  uint32_t* shell = (uint32_t*)(base + kShellOff);
  uint32_t* mol = (uint32_t*)(base + kMolOff);
  uint32_t* cnt = (uint32_t*)(base + kCntOff);
  uint64_t* off = (uint64_t*)(base + kOffOff);
  // the masks keep the previous call's voxels: clear the part this grid uses
  const uint64_t words = (h.count + 31) / 32;
  if (cudaMemsetAsync(shell, 0, words * sizeof(uint32_t), s) != cudaSuccess ||
      cudaMemsetAsync(mol, 0, words * sizeof(uint32_t), s) != cudaSuccess)
    return CRAB_ECUDA;
  const unsigned blocks = (unsigned)((n * 32 + 255) / 256);
  k_rasterize<<<blocks, 256, 0, s>>>(d_xyz, nullptr, h.outer, h.inner, n, h.box, 1.0 / spacing, shell, mol);
  const uint64_t chunks = (h.count + kChunk - 1) / kChunk;
  k_count<<<(unsigned)chunks, kScanThreads, 0, s>>>(shell, mol, words, 0, cnt);
  k_scan_chunks<<<1, 1024, 0, s>>>(cnt, chunks, off);
  if (cudaGetLastError() != cudaSuccess) return CRAB_ECUDA;
  uint64_t total = 0;
  if (cudaMemcpyAsync(&total, off + chunks, sizeof(total), cudaMemcpyDeviceToHost, s) != cudaSuccess) return CRAB_ECUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return CRAB_ECUDA;
  *m = (int64_t)total;
  if (total > 0 && capacity > 0) {
    k_noalloc_emit<<<(unsigned)chunks, kScanThreads, 0, s>>>(shell, mol, words, h.box, off, d_sites,
                                                            (uint64_t)capacity);
    if (cudaGetLastError() != cudaSuccess) return CRAB_ECUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return CRAB_ECUDA;
  }
  return (capacity > 0 && (int64_t)total > capacity) ? CRAB_ECAPACITY : CRAB_OK;
}
