// Work units of the kernels that visit every pair of a class pair's tiles
// (Debye distance histogram, P(r)): rows, their tile pairs, and the split of a
// row list over CTAs.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "engine.hpp"

namespace crab {

__host__ __device__ __forceinline__ int hist_units(const HistRow& r) {
  return 2 * r.split * (r.diag ? r.ni * (r.ni + 1) / 2 : r.ni * r.nj);
}

// Tile pair p of a row: i tile and j tile, j fastest; on the diagonal row the
// pairs i <= j in the order of j(j+1)/2 + i.
__device__ __forceinline__ int2 hist_tiles(const HistRow& r, int p) {
  if (!r.diag) return make_int2(r.i0 + p / r.nj, r.j0 + p % r.nj);
  int j = (int)((sqrtf(8.0f * (float)p + 1.0f) - 1.0f) * 0.5f);
  while ((long long)j * (j + 1) / 2 > p) --j;
  while ((long long)(j + 1) * (j + 2) / 2 <= p) ++j;
  return make_int2(r.i0 + (p - j * (j + 1) / 2), r.j0 + j);
}

// Units of a row: halves of its tile pairs, or where those are too few for the
// warps of a CTA (below `least`) each by igroups groups of 32 i atoms, and
// with `quarters` by four quarters of the j atoms.  False past 2^30 units.
inline bool hist_row_units(HistRow& r, int64_t i_atoms, bool quarters, int64_t least, int64_t* total) {
  const int64_t units = 2 * (r.diag ? (int64_t)r.ni * (r.ni + 1) / 2 : (int64_t)r.ni * r.nj);
  r.split = 1;
  r.igroups = r.quarters = 0;
  if (units < least) {
    r.igroups = r.ni == 1 ? (int)((i_atoms + 31) / 32) : 4;
    r.quarters = quarters ? 1 : 0;
    r.split = r.igroups * (quarters ? 4 : 1);
  }
  *total += units * r.split;
  return *total <= (int64_t)1 << 30;
}

// CTA starts over the rows r0 .. r1: equal shares of the cost.  A row costs its
// pairs in units of 8192, 0.1 per unit for empty tile space, and row_cost for
// its flush and the wait for its last units.  (The units of a row come first, so
// that the first part of a split owns some.)
inline std::vector<int2> hist_starts(const std::vector<HistRow>& rows, const std::vector<double>& pairs, size_t r0,
                                     size_t r1, int grid, int shard, int shards, double row_cost) {
  auto work = [&](size_t r) {
    return pairs[r] / (128.0 * kHistChunkAtoms) + 0.1 * hist_units(rows[r]) / rows[r].split;
  };
  double total = 0.0;
  for (size_t r = r0; r < r1; ++r) total += row_cost + work(r);
  const int parts = grid * shards;
  std::vector<int2> out;
  size_t row = r0;
  double before = 0.0;  // cost of the rows before `row`
  for (int p = 0; p <= grid; ++p) {
    const double at = total * (double)(shard * grid + p) / parts;
    while (row + 1 < r1 && before + row_cost + work(row) <= at) before += row_cost + work(row++);
    const int n = hist_units(rows[row]);
    const double in = std::min(1.0, std::max(0.0, (at - before) / work(row)));
    int u = (int)std::ceil(in * n);
    // rows of less than a share are not cut: each cut costs another flush
    if (work(row) + row_cost < total / parts) u = in > 0.5 ? n : 0;
    if (shards > 1) u -= u % (2 * rows[row].split);  // shards take whole tile pairs
    if (shard * grid + p == parts) {
      row = r1 - 1;
      u = hist_units(rows[row]);
    }
    out.push_back(make_int2((int)(row - r0), u));
  }
  return out;
}

}  // namespace crab
