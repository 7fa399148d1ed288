// Debye terms of one structure, from its atoms to the six curves, on the device.
//
// The host makes one pass over elements, groups and occupancies (which
// scattering class an atom belongs to, and its place in the class's run of
// tiles: one 32-bit word per atom) and two over the coordinates (box, largest
// distance from its centre).  Everything that is as long as the atom list times
// anything else happens here:
//   k_front_points   centred FP32 coordinates into the histogram's tiles
//   k_front_sites    the hydration sites, which never leave the device, and
//                    their lattice cells
//   (debye_hist.cu)  the pair sums
//   k_debye_terms    amplitudes per class and q (solvent.rs:454-488) and the
//                    quadratic forms of solvent.rs:533-577 from the pair sums
// What comes back is the result.  Before, the same call typed the atoms into
// three arrays, laid them out in tiles twice, formed the amplitude tables and
// the six quadratic forms per q on one host core, and copied every type pair's
// partial sums back: of 290 us for 1,000 atoms of 14 classes at 100 q, 40 were
// kernels.  One call now takes 112 us there (with the histogram alone 291), 0.34
// ms for 7,321 atoms on a measured 333-q grid (1.00 ms), and 0.87 ms for 20,000
// atoms with their grid at 500 q (1.56 ms), half of it the pair kernel.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "engine.hpp"
#include "ops.hpp"

namespace crab {
namespace {

constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr uint32_t kDropped = 0xFFFFFFFFu, kLooseBit = 1u << 23, kRankMask = kLooseBit - 1;
constexpr int kCodes = 256;  // element * 16 + group + 1
constexpr int kFrontClasses = 200;  // scattering classes at most, sites among them

// Word of an atom: class << 24 | loose << 23 | rank among its class's counted
// or loose atoms.  tile0[2 c], tile0[2 c + 1]: first counted and loose tile.
__global__ void k_front_points(const double* __restrict__ xyz, const uint32_t* __restrict__ word,
                               const double* __restrict__ occ, const int* __restrict__ tile0, int64_t n, double cx,
                               double cy, double cz, unsigned char* __restrict__ pts, double* __restrict__ weight) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t w = word[i];
  if (w == kDropped) return;
  const uint32_t rank = w & kRankMask;
  const int64_t tile = tile0[2 * (w >> 24) + ((w & kLooseBit) ? 1 : 0)] + (rank >> 7);
  const int s = rank & 127, e = s & 63;
  float* c = reinterpret_cast<float*>(pts + (tile * 2 + (s >> 6)) * kHistChunkBytes);
  c[(e >> 1) * 4 + (e & 1)] = (float)(xyz[3 * i] - cx);
  c[(e >> 1) * 4 + 2 + (e & 1)] = (float)(xyz[3 * i + 1] - cy);
  c[128 + e] = (float)(xyz[3 * i + 2] - cz);
  if (weight) weight[tile * kTile + s] = occ[i];
}

__global__ void k_front_sites(const double* __restrict__ sites, const int32_t* __restrict__ cells, int64_t m, int tile0,
                              double cx, double cy, double cz, unsigned char* __restrict__ pts,
                              double* __restrict__ weight, int4* __restrict__ lattice) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int64_t tile = tile0 + (i >> 7);
  const int s = (int)(i & 127), e = s & 63;
  float* c = reinterpret_cast<float*>(pts + (tile * 2 + (s >> 6)) * kHistChunkBytes);
  c[(e >> 1) * 4 + (e & 1)] = (float)(sites[3 * i] - cx);
  c[(e >> 1) * 4 + 2 + (e & 1)] = (float)(sites[3 * i + 1] - cy);
  c[128 + e] = (float)(sites[3 * i + 2] - cz);
  if (weight) weight[tile * kTile + s] = 1.0;
  lattice[i] = make_int4(cells[3 * i], cells[3 * i + 1], cells[3 * i + 2], 0);
}

struct TermsArg {
  const ClassAmp* cls;   // [T]; cls[T] holds the hydrogen's form factor for water
  const double* sums;    // per type Σw², then Σw
  const double* raw;     // [T(T+1)/2][nq] Σ w w sin(q r)/r
  const double* lattice; // [nq] site-site sums, or null
  const double* q;
  int T, nq, terms, shard;  // terms: 6, or 1 for the vacuum
  double density, site_volume;
};
constexpr int kTQ = 8, kTR = 32;  // q and row groups of a CTA

__device__ __forceinline__ double gauss_sum(const ClassAmp& c, double q) {
  const double s = q / (4.0 * kPi), s2 = s * s;
  double v = 0.0;
#pragma unroll
  for (int k = 0; k < 5; ++k) v += c.a[k] * exp(-c.b[k] * s2);
  return v + c.c;
}

// Σ_ab of the quadratic forms X_a Y_b at 8 q per CTA: the amplitudes of all
// classes go to shared memory, 32 threads per q take every 32nd type pair each
// (partials read in runs of 8 q), and their sums are added in order.  A chain
// of exponentials and pairs per thread, so few q a CTA
// (14 classes, 100 q: 8.7 us; 15 at 32 q a CTA and 8 threads per q).
__global__ void __launch_bounds__(kTQ * kTR) k_debye_terms(TermsArg A, double* __restrict__ out) {
  extern __shared__ double amp[];  // [3][T][kTQ]
  __shared__ double red[kTR][6][kTQ];
  const int lane = threadIdx.x, y = threadIdx.y, T = A.T, tid = y * kTQ + lane;
  const int k = blockIdx.x * kTQ + lane, kc = min(k, A.nq - 1);
  const double qk = A.q[kc];
  double *V = amp, *E = V + T * kTQ, *H = E + T * kTQ;
  for (int a = y; a < T; a += kTR) {
    const ClassAmp& c = A.cls[a];
    double v = gauss_sum(c, qk), e = 0.0, h = 0.0;
    if (c.water) {
      const double x = qk * 0.9572;
      h = A.density / 10.0 * A.site_volume *
          (v + 2.0 * gauss_sum(A.cls[T], qk) * (fabs(x) < 1e-8 ? 1.0 : sin(x) / x));
      v = 0.0;
    } else if (A.terms > 1) {
      e = A.density * (c.volume * exp(-c.pv * qk * qk / (4.0 * kPi)));
      if (c.shell > 0.0) h = A.density * 0.1 * (c.shell * exp(-c.ps * qk * qk / (4.0 * kPi)));
    }
    V[a * kTQ + lane] = v;
    E[a * kTQ + lane] = e;
    H[a * kTQ + lane] = h;
  }
  __syncthreads();
  double t[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const double inv = qk != 0.0 ? 1.0 / qk : 0.0;
  int a = 0, left = y;  // type pair y, y + kTR, ... as (a, a + left)
  for (int ab = y; ab < T * (T + 1) / 2; ab += kTR) {
    while (left >= T - a) left -= T - a++;
    const int b = a + left;
    double P;
    if (A.lattice && a == T - 1) P = A.lattice[kc];
    else if (qk != 0.0) P = A.raw[(size_t)ab * A.nq + kc] * inv;
    else if (A.shard != 0) P = 0.0;
    else P = a == b ? 0.5 * (A.sums[T + a] * A.sums[T + a] - A.sums[a]) : A.sums[T + a] * A.sums[T + b];
    const double va = V[a * kTQ + lane], vb = V[b * kTQ + lane];
    t[0] += 2.0 * va * vb * P;
    if (A.terms > 1) {
      const double ea = E[a * kTQ + lane], eb = E[b * kTQ + lane], ha = H[a * kTQ + lane], hb = H[b * kTQ + lane];
      t[1] += 2.0 * ea * eb * P;
      t[2] += 2.0 * ha * hb * P;
      t[3] += (va * eb + vb * ea) * P;
      t[4] += (va * hb + vb * ha) * P;
      t[5] += (ea * hb + eb * ha) * P;
    }
    left += kTR;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) red[y][i][lane] = t[i];
  __syncthreads();
  for (int i = tid; i < A.terms * kTQ; i += kTQ * kTR) {
    const int term = i / kTQ, l = i % kTQ, kk = blockIdx.x * kTQ + l;
    double s = 0.0;
    for (int g = 0; g < kTR; ++g) s += red[g][term][l];
    if (A.shard == 0)
      for (int c = 0; c < T; ++c) {
        const double v = V[c * kTQ + l], e = E[c * kTQ + l], h = H[c * kTQ + l];
        const double x = term == 0 || term > 2 ? (term == 5 ? e : v) : (term == 1 ? e : h);
        const double z = term < 3 ? x : (term == 3 ? e : h);
        s += x * z * A.sums[c];
      }
    if (kk < A.nq) out[(size_t)term * A.nq + kk] = s;
  }
}

// Whether a call of these classes is faster here than on the general path, whose
// tables, layout and quadratic forms one host core makes and whose sites come
// back to the host.  For few q, or few atoms of many classes with weights of
// their own, it is not (vacuum calls: 36 classes, 2,790 atoms, 2 q 379 us here, 178
// there; four classes, 737 atoms, 10 q 119 / 99 us; 1,000 atoms of 14 classes, 100 q
// 112 / 291).  Fitted with hist_us to 664 calls of 1 to 42 classes, 2 to 4,000 atoms
// and 2 to 300 q.
bool front_pays(const HistShape& X, int T, bool grid, const crab_solvent* solvent, const std::vector<double>& q,
                int64_t n) {
  if (solvent && solvent->hydration_model == CRAB_HYD_GRID) return true;  // 1.05 to 7 times faster at any size
  const double nq = (double)q.size();
  double rows;
  const double us = hist_us(X, T, false, (int64_t)q.size(), &rows);
  const double types = T - (grid ? 1 : 0);
  const double host = nq * (0.027 * types + 0.0016 * types * (types + 1.0) * (solvent ? 3.2 : 1.0)) +
                      (grid ? 40.0 + 0.02 * (double)n : 0.0);
  const double least = 5.7e-8 * (double)n * (double)n * nq;  // of the recurrence, without a look at the q grid
  return us < host + 0.8 * least + 1.0 || us < host + 0.8 * recurrence_us(X, T, false, q) + 1.0;
}

}  // namespace

// The six solvent terms (out [6][nq]), or with solvent null the vacuum curve's
// unclamped sum (out [nq]); false where the histogram does not apply or does not
// pay (nothing done, the caller takes the general path).
bool debye_terms_device(crab_ctx* ctx, const crab_struct* st, const double* q, int64_t nq, const crab_solvent* solvent,
                        bool implicit, double* out, int shard, int n_shards, FrontKeep* keep) {
  const int64_t n = st->n;
  if (ctx->pair_variant || n == 0 || nq == 0 || n >= (int64_t)kRankMask) return false;
  const bool grid = solvent && solvent->hydration_model != CRAB_HYD_ANALYTIC;
  double qmax = 0.0;
  for (int64_t k = 0; k < nq; ++k) qmax = std::max(qmax, q[k]);
  // classes present, in (element, group) order
  const int8_t *el = st->elem.data(), *gr = st->group.data();
  int64_t part[4][kCodes] = {};
  const int gmask = implicit ? 0xff : 0;
  for (int64_t i = 0; i < n; ++i) ++part[i & 3][el[i] * 16 + ((gr[i] + 1) & gmask)];
  int cls_of[kCodes];
  std::vector<AtomClass> cls;
  std::vector<int64_t> count;
  for (int code = 0; code < kCodes; ++code) {
    const int64_t m = part[0][code] + part[1][code] + part[2][code] + part[3][code];
    const AtomClass k{code / 16, code % 16 - 1};
    const bool drop = m == 0 || class_dropped(k, implicit, !solvent ? TermSet::Vacuum
                                                          : grid   ? TermSet::SolventGrid
                                                                   : TermSet::SolventAnalytic);
    cls_of[code] = drop ? -1 : (int)cls.size();
    if (!drop) {
      cls.push_back(k);
      count.push_back(m);
    }
  }
  const int TA = (int)cls.size(), T = TA + (grid ? 1 : 0);
  if (TA == 0 || T > kFrontClasses) return false;
  const double* x = st->xyz.data();
  const double* occ = st->occ.data();
  HistShape X;
  X.bins.assign(1, kHistMinBins);
  X.inv_h.resize(1);
  X.uni.resize(T);
  X.loose.resize(T);
  const std::vector<double> qs(q, q + nq);
  // the share of loose atoms in a sample decides, before anything is as long as
  // the atom list but the classes; with the fewest bins first
  std::vector<double> w0(TA, 0.0);
  const int64_t stride = std::max<int64_t>(1, n / 256);
  int64_t seen = 0, odd = 0;
  for (int64_t i = 0; i < n; i += stride) {
    const int k = cls_of[el[i] * 16 + ((gr[i] + 1) & gmask)];
    if (k < 0 || occ[i] == 0.0) continue;
    if (w0[k] == 0.0) w0[k] = occ[i];
    odd += occ[i] != w0[k];
    ++seen;
  }
  const double share = seen ? (double)odd / (double)seen : 0.0;
  for (int k = 0; k < TA; ++k) {
    X.loose[k].atoms = (int64_t)(share * (double)count[k] + 0.5);
    X.uni[k].atoms = count[k] - X.loose[k].atoms;
  }
  if (!front_pays(X, T, grid, solvent, qs, n)) return false;
  // box, centre and the largest distance from it
  double lo[3] = {x[0], x[1], x[2]}, hi[3] = {x[0], x[1], x[2]}, c[3], r2 = 0.0;
  for (int64_t i = 0; i < n; ++i)
    for (int d = 0; d < 3; ++d) {
      lo[d] = min_num(lo[d], x[3 * i + d]);
      hi[d] = max_num(hi[d], x[3 * i + d]);
    }
  for (int d = 0; d < 3; ++d) c[d] = 0.5 * (lo[d] + hi[d]);
  for (int64_t i = 0; i < n; ++i) {
    const double dx = x[3 * i] - c[0], dy = x[3 * i + 1] - c[1], dz = x[3 * i + 2] - c[2];
    r2 = max_num(r2, dx * dx + dy * dy + dz * dz);
  }
  const double rmax = std::sqrt(r2);
  // the sites lie within a shell of 16 Å at most around the atoms; refused here
  // rather than after the grid is built
  if (!hist_structure_bins(2.0 * (rmax + (grid ? 16.0 : 0.0)), qmax, &X.bins[0], &X.inv_h[0])) return false;
  if (X.bins[0] > kHistMinBins && !front_pays(X, T, grid, solvent, qs, n)) return false;
  auto* hx = (double*)ctx->host("front.xyz", (size_t)n * 3 * sizeof(double));
  std::memcpy(hx, x, (size_t)n * 3 * sizeof(double));
  auto* d_xyz = (double*)ctx->dev("front.xyz", (size_t)n * 3 * sizeof(double));
  copy_h2d(ctx, d_xyz, hx, (size_t)n * 3 * sizeof(double), ctx->stream);
  GridResult g;
  GridPoolRelease grid_release{ctx, grid};
  if (grid) {
    TraceScope tg("hydration_sites");
    g = solvent->hydration_model == CRAB_HYD_ADAPTIVE
            ? adaptive_grid_device(ctx, x, n, solvent->grid_spacing, 3.0, 12.0, false, GridAtoms{d_xyz, nullptr})
            : exterior_grid_device(ctx, x, el, n, 1.0, 1.4, solvent->shell_thickness, false, GridAtoms{d_xyz, nullptr});
    if (!hist_structure_bins(2.0 * (rmax + g.outer), qmax, &X.bins[0], &X.inv_h[0])) return false;
  }
  // words: a class's candidate for its counted weight is the weight of its
  // first atom; should that turn out rarer than half, the majority vote's
  auto* word = (uint32_t*)ctx->host("front.word", (size_t)n * sizeof(uint32_t));
  std::fill(w0.begin(), w0.end(), 0.0);
  std::vector<int64_t> nu(TA), nl(TA);
  std::vector<double> sw(T, 0.0), sw2(T, 0.0);
  double s_abs = 0.0;
  for (int round = 0; round < 2; ++round) {
    std::fill(nu.begin(), nu.end(), 0);
    std::fill(nl.begin(), nl.end(), 0);
    std::fill(sw.begin(), sw.end(), 0.0);
    std::fill(sw2.begin(), sw2.end(), 0.0);
    s_abs = 0.0;
    for (int64_t i = 0; i < n; ++i) {
      const int k = cls_of[el[i] * 16 + ((gr[i] + 1) & gmask)];
      const double w = occ[i];
      if (k < 0 || w == 0.0) {
        word[i] = kDropped;
      } else if (w == w0[k]) {
        word[i] = (uint32_t)k << 24 | (uint32_t)nu[k]++;
      } else if (round == 0 && w0[k] == 0.0) {
        w0[k] = w;
        word[i] = (uint32_t)k << 24 | (uint32_t)nu[k]++;
      } else {
        word[i] = (uint32_t)k << 24 | kLooseBit | (uint32_t)nl[k]++;
        sw[k] += w;
        sw2[k] += w * w;
        s_abs += std::fabs(w);
      }
    }
    bool again = false;
    for (int k = 0; k < TA; ++k) again = again || nl[k] > nu[k];
    if (!again || round == 1) break;
    std::vector<int64_t> votes(TA, 0);
    for (int64_t i = 0; i < n; ++i) {
      const int k = cls_of[el[i] * 16 + ((gr[i] + 1) & gmask)];
      const double w = occ[i];
      if (k < 0 || w == 0.0) continue;
      if (votes[k] == 0) w0[k] = w;
      votes[k] += w == w0[k] ? 1 : -1;
    }
  }
  // tiles: a class's loose atoms, then its counted ones
  std::vector<int> tile0(2 * (size_t)T, 0);
  auto tiles = [&](HistRange& R, int64_t m, double w) {
    R.t0 = (int)X.tile_cnt.size();
    R.n = (int)((m + kTile - 1) / kTile);
    R.atoms = m;
    R.w = w;
    for (int64_t at = 0; at < m; at += kTile) X.tile_cnt.push_back((int)std::min<int64_t>(kTile, m - at));
    return R.t0;
  };
  int64_t points = g.m;
  for (int k = 0; k < T; ++k) {
    const bool site = k == TA;
    tile0[2 * k + 1] = tiles(X.loose[k], site ? 0 : nl[k], 0.0);
    tile0[2 * k] = tiles(X.uni[k], site ? g.m : nu[k], site ? 1.0 : w0[k]);
    const double m = (double)X.uni[k].atoms, w = X.uni[k].w;
    sw[k] += m * w;
    sw2[k] += m * w * w;
    s_abs += m * std::fabs(w);
    if (!site) {
      points += count[k];
      X.any_loose = X.any_loose || nl[k] > 0;
    }
  }
  X.sum_abs_w = s_abs;
  // amplitudes, sums per type and tile starts travel with the plan's tables
  std::vector<ClassAmp> amp;
  for (int k = 0; k < T; ++k)
    amp.push_back(class_amp(k < TA ? cls[k] : AtomClass{-1, -1}, implicit, solvent ? solvent->shell_thickness : 0.0));
  if (grid || !solvent)
    for (ClassAmp& a : amp) a.shell = 0.0;  // no analytic shell
  amp.push_back(class_amp(AtomClass{CRAB_EL_H, -1}, false, 0.0));
  const size_t o_sums = (amp.size() * sizeof(ClassAmp) + 15) / 16 * 16, o_tile = o_sums + 2 * (size_t)T * sizeof(double);
  X.more.resize(o_tile + tile0.size() * sizeof(int));
  std::memcpy(X.more.data(), amp.data(), amp.size() * sizeof(ClassAmp));
  std::memcpy(X.more.data() + o_sums, sw2.data(), (size_t)T * sizeof(double));
  std::memcpy(X.more.data() + o_sums + (size_t)T * sizeof(double), sw.data(), (size_t)T * sizeof(double));
  std::memcpy(X.more.data() + o_tile, tile0.data(), tile0.size() * sizeof(int));

  HistPoolRelease hist_release{ctx};
  PairPlan P;
  P.pooled = true;
  P.shard = shard;
  P.n_shards = n_shards;
  P.nq = nq;
  P.q = qs;
  P.L.T = T;
  P.L.n = points;
  P.L.n_tiles = (int)X.tile_cnt.size();
  P.n_pairs = T * (T + 1) / 2;
  P.skip_last = grid;
  cudaStream_t s = ctx->stream;
  try {
    if (!hist_build(ctx, P, X, nullptr, nullptr)) return false;
  } catch (const Error& e) {  // no room on the device for its sums: the general path has less to hold
    if (e.code != CRAB_ENOMEM || n_shards > 1) throw;  // every shard takes the same path
    cudaGetLastError();
    return false;
  }
  HistPart& H = P.hist;
  const int terms = solvent ? 6 : 1;
  P.d_out = (double*)ctx->dev("pair.out", (size_t)P.n_pairs * nq * sizeof(double));
  // the result and the kernels' status come back together
  const size_t out_bytes = (size_t)terms * nq * sizeof(double);
  auto* d_res = (unsigned char*)ctx->dev("front.result", out_bytes + 2 * sizeof(int));
  P.d_status = (int*)(d_res + out_bytes);
  P.d_next = P.d_status + 1;
  auto* d_word = (uint32_t*)ctx->dev("front.word", (size_t)n * sizeof(uint32_t));
  copy_h2d(ctx, d_word, word, (size_t)n * sizeof(uint32_t), s);
  double* d_occ = nullptr;
  if (X.any_loose || keep) {
    d_occ = (double*)ctx->dev("front.occ", (size_t)n * sizeof(double));
    copy_h2d(ctx, d_occ, occ, (size_t)n * sizeof(double), s);
  }
  if (grid && shard == 0) {
    int64_t span[3];
    for (int d = 0; d < 3; ++d) span[d] = (int64_t)std::ceil((hi[d] - lo[d] + 2.0 * g.outer) / g.spacing) + 1;
    lattice_plan_init_device(ctx, P, g.d_cells, g.m, g.spacing, span);
  }
  const int* d_tile0 = (const int*)(H.d_more + o_tile);
  k_front_points<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_xyz, d_word, d_occ, d_tile0, n, c[0], c[1], c[2], H.d_pts,
                                                             H.d_weight);
  CRAB_CUDA_CHECK(cudaGetLastError());
  if (g.m) {
    int4* cells = P.lattice.active ? P.lattice.d_cells
                                   : (int4*)ctx->dev("pair.lattice_cells", (size_t)g.m * sizeof(int4));
    k_front_sites<<<(unsigned)((g.m + 255) / 256), 256, 0, s>>>(g.d_sites, g.d_cells, g.m, X.uni[TA].t0, c[0], c[1],
                                                                c[2], H.d_pts, H.d_weight, cells);
    CRAB_CUDA_CHECK(cudaGetLastError());
    ctx->launches += 1;
  }
  pair_plan_launch(ctx, P, s, true);
  TermsArg A;
  A.cls = (const ClassAmp*)H.d_more;
  A.sums = (const double*)(H.d_more + o_sums);
  A.raw = P.d_out;
  A.lattice = P.lattice.active ? P.lattice.d_out : nullptr;
  A.q = P.d_q;
  A.T = T;
  A.nq = (int)nq;
  A.terms = terms;
  A.shard = shard;
  A.density = solvent ? solvent->bulk_density : 0.0;
  A.site_volume = g.voxel_volume;
  // the attribute belongs to the function, whatever context sets it: always the same value
  constexpr size_t kTermsSmem = 3 * (size_t)kFrontClasses * kTQ * sizeof(double);
  CRAB_CUDA_CHECK(cudaFuncSetAttribute(k_debye_terms, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTermsSmem));
  const size_t smem = 3 * (size_t)T * kTQ * sizeof(double);
  k_debye_terms<<<(unsigned)((nq + kTQ - 1) / kTQ), dim3(kTQ, kTR), smem, s>>>(A, (double*)d_res);
  CRAB_CUDA_CHECK(cudaGetLastError());
  ctx->launches += 2;
  auto* h_res = (unsigned char*)ctx->host("front.result", out_bytes + 2 * sizeof(int));
  copy_d2h(ctx, h_res, d_res, out_bytes + sizeof(int), s);
  if (keep) {
    keep->d_xyz = d_xyz;
    keep->d_occ = d_occ;
    keep->d_word = d_word;
    keep->tile0 = tile0;
    keep->tile_type.assign(X.tile_cnt.size(), 0);
    for (int k = 0; k < T; ++k)
      for (const HistRange* R : {&X.loose[k], &X.uni[k]})
        std::fill_n(keep->tile_type.begin() + R->t0, R->n, k);
    std::copy(c, c + 3, keep->centre);
    keep->rmax = rmax;
    keep->meanwhile(cls);
  }
  CRAB_CUDA_CHECK(cudaStreamSynchronize(s));
  float ms = 0.0f;
  CRAB_CUDA_CHECK(cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
  ctx->last_pair_ms = ms;
  ctx->last_pair_q = 0.5 * (double)points * (double)(points - 1) * (double)nq;
  int status;
  std::memcpy(&status, h_res + out_bytes, sizeof(int));
  if (status) throw Error(status, "pair kernel: a bounded wait on a j-tile copy ran out");
  std::memcpy(out, h_res, out_bytes);
  return true;
}

}  // namespace crab
