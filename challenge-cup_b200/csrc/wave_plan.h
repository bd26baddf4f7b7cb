// How a multi-step launch (wave_kernel.cuh) is split over CTAs: the geometry
// of a CTA's part, its shared-memory layout, the choice of a split, and which
// cells belong to which CTA.  Plain C++ on the host side, so that splits can be
// checked without a device.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define WAVE_HD __host__ __device__
#else
#define WAVE_HD
#endif

namespace ertm {

constexpr int WAVE_NT = 512;     // threads of a CTA
constexpr int WAVE_HALO = 4;     // cells the 8th-order stencils read beyond their own
constexpr int WAVE_SMEM_MAX = 227 * 1024 - 2048;   // dynamic shared memory (the static part left out)

// Rows [i0, i0 + th) and column groups [g0, g0 + gw) of CTA c of a pz × px
// split with row cuts cut[0 … pz] and column-group cuts cut[pz + 1 …].
struct WaveTile {
  int i0, th, g0, gw, tr, tc;
};
WAVE_HD inline WaveTile wave_tile(const int16_t* cut, int pz, int px, int c) {
  WaveTile t;
  t.tr = c / px;
  t.tc = c - t.tr * px;
  t.i0 = cut[t.tr];
  t.th = cut[t.tr + 1] - t.i0;
  t.g0 = cut[pz + 1 + t.tc];
  t.gw = cut[pz + 2 + t.tc] - t.g0;
  return t;
}
constexpr int WAVE_MAX_CUTS = 160;   // pz + px + 2 of a split over up to 156 CTAs

// Strip columns / rows of [lo, hi) in ψ-array coordinates: first index and count.
WAVE_HD inline void wave_strip(int lo, int hi, int n, int a, int b, int& first, int& count) {
  // strip index of position q: q for q < a, a + q − (n − b) for q ≥ n − b
  const int l0 = lo < a ? lo : a, l1 = hi < a ? hi : a;
  const int r0 = lo > n - b ? lo : n - b, r1 = hi < n ? hi : n;
  const int nl = l1 > l0 ? l1 - l0 : 0, nr = r1 > r0 ? r1 - r0 : 0;
  first = nl > 0 ? l0 : a + (r0 - (n - b));
  count = nl + nr;
  if (count == 0) first = 0;
}

// Shared-memory layout of one CTA, in floats from the start of dynamic shared
// memory (every array a multiple of 16 bytes).
struct WaveLayout {
  int W, H, cw;          // halo-field pitch and rows, cell-array pitch
  int field, field_n;    // halo fields, floats per field
  int cell, cell_n;      // per-cell arrays, floats per array
  int qidx;              // viscoacoustic Q index bytes
  int epi;               // P (and S) of the last step for the epilogue
  int src;               // stored source fields of the last step
  int acc;               // imaging sums, two floats a cell each
  int psix, psix_n;      // x-strip memories (pitch nsx), floats per term
  int psiz, psiz_n;      // z-strip memories (pitch cw), floats per term
  int col, row;          // per column / row: profile a, b, strip index and flags
  int units, units_n;    // exchange tables (int4 per unit, two phases)
  int total;
};

WAVE_HD inline int wave_r4(int n) { return (n + 3) / 4 * 4; }

// pad: floats between the rows of a halo field beyond its own cells.  8 holds
// the halo; with 32 the rows' first cells continue the bank sequence of the
// cells before them, so a warp that spans rows has no bank conflicts.
WAVE_HD inline WaveLayout wave_layout(bool elastic, bool visco, int L, int pad, int th, int gw, int nsx,
                                      int nsz, int n_epi, int n_src, int n_acc) {
  WaveLayout y;
  const int nf = elastic ? 5 : 3, nx = elastic ? 2 : 1, n_psi = elastic ? 4 : 2;
  y.cw = 4 * gw;
  y.W = y.cw + pad;
  y.H = th + 2 * WAVE_HALO;
  int o = 0;
  y.field = o;
  y.field_n = y.W * y.H;
  o += nf * y.field_n;
  y.cell = o;
  y.cell_n = th * y.cw;
  o += (visco ? 4 + 2 * L : (elastic ? 5 : 3)) * y.cell_n;
  y.qidx = o;
  o += visco ? wave_r4(th * gw) : 0;   // one byte per cell
  y.epi = o;
  o += n_epi * y.cell_n;
  y.src = o;
  o += n_src * y.cell_n;
  y.acc = o;
  o += 2 * n_acc * y.cell_n;
  y.psix = o;
  y.psix_n = wave_r4(th * nsx);
  o += n_psi * y.psix_n;
  y.psiz = o;
  y.psiz_n = nsz * y.cw;
  o += n_psi * y.psiz_n;
  y.col = o;
  o += 4 * y.cw;
  y.row = o;
  o += 4 * th;
  y.units_n = 2 * nx * th + 2 * nx * 4 * gw;
  y.units = o;
  o += 2 * 4 * y.units_n;
  y.total = o;
  return y;
}

// What a split depends on: the padded grid, its CPML strips and the engine.
struct WaveGrid {
  bool elastic = false, visco = false;
  int L = 0;                    // viscoacoustic mechanisms
  int nzp = 0, nxp = 0;         // padded grid
  int npx_l = 0, npx_r = 0, npz_t = 0, npz_b = 0;
};

// How a propagator is split over at most `ncta` CTAs.
struct WavePlan {
  int px = 0, pz = 0;
  int cells = 1;      // neighbouring cells of a thread's block
  int thmax = 0, n_src = 0, n_acc = 0;
  std::vector<int16_t> cut;   // see wave_tile
  int pad = 8;        // halo-field row padding (wave_layout)
  int smem = 0;       // bytes
  int64_t half = 0;   // exchange units per CTA and phase
  bool ok() const { return px > 0; }
  int ctas() const { return px * pz; }
};

// What a work does besides stepping, for its shared memory: epilogue fields
// (P, S), stored source fields read, imaging sums that could be resident.
struct WaveNeeds {
  int n_epi = 0, n_src = 0, n_acc = 0;
};

// Largest shared-memory need of a split, in bytes.
inline int wave_smem(const WaveGrid& h, const WavePlan& p, const WaveNeeds& n) {
  int most = 0;
  for (int c = 0; c < p.px * p.pz; ++c) {
    const WaveTile t = wave_tile(p.cut.data(), p.pz, p.px, c);
    int f, nsx, nsz;
    wave_strip(4 * t.g0, std::min(4 * (t.g0 + t.gw), h.nxp), h.nxp, h.npx_l, h.npx_r, f, nsx);
    wave_strip(t.i0, t.i0 + t.th, h.nzp, h.npz_t, h.npz_b, f, nsz);
    const WaveLayout y = wave_layout(h.elastic, h.visco, h.L, p.pad, t.th, t.gw, nsx, nsz,
                                     n.n_epi, p.n_src, p.n_acc);
    most = std::max(most, y.total * 4);
  }
  return most;
}

// Cuts of n positions into k parts of about equal weight, each at least
// `least` long; position q weighs weight(q).
template <class F>
void wave_cuts(int n, int k, int least, F&& weight, int16_t* cut) {
  double total = 0.0;
  for (int q = 0; q < n; ++q) total += weight(q);
  double sum = 0.0;
  int at = 0, first = 0;
  cut[0] = 0;
  for (int c = 0; c < k; ++c) {
    const int last = n - least * (k - 1 - c);   // leave the later parts their least
    while (at < last && (at - first < least || c + 1 == k || sum + 0.5 * weight(at) < total * (c + 1) / k)) {
      sum += weight(at);
      ++at;
    }
    cut[c + 1] = (int16_t)at;
    first = at;
  }
}

// Split over at most `ncta` CTAs.  Measured over px = 5 … 24 and strip weights
// 0 … 2 on five grids: CTAs about 2.2 times as wide as tall are within 2 % of
// the best, and so is a weight of 1.6 for CPML strips (their cells take the
// general form and memory updates) with two cells a thread; with one cell a
// thread (small grids, one pass of 512) 0.4.  Elastic 401×601 (µs a step):
// 6.9 so, 7.9 with equal cuts, 11.6 the worst; acoustic 301×201 3.4 with one
// cell a thread, 4.6 with two.  Imaging sums that do not fit in shared memory
// cost about two round trips to L2 a step; a grid whose coefficients do not
// fit has no split.
inline WavePlan make_wave_plan(const WaveGrid& h, int ncta, const WaveNeeds& n) {
  WavePlan best;
  const int ng = (h.nxp + 3) / 4, nx = h.elastic ? 2 : 1;
  ncta = std::min(ncta, WAVE_MAX_CUTS - 4);
  const double ideal = std::sqrt((double)h.nxp * ncta / (2.2 * h.nzp));
  // cells per thread and pass; a split of one pass (WAVE_NT blocks a CTA at
  // most) is cut for that rather than by weight
  const double avg = (double)h.nzp * 4 * ng / (0.93 * WAVE_NT * ncta);
  const int cells = avg <= 1.0 ? 1 : 2;
  const bool single = avg <= 2.0;
  double cost = 0.0;
  for (const double strip : {single ? 0.4 : 1.6, 0.8, 0.0})
  for (int px = std::max(1, std::min(ng, (int)ideal) - 2); px <= std::min({ncta, ng, (int)ideal + 3}); ++px) {
    const int pz = std::min(ncta / px, h.nzp / WAVE_HALO);
    if (pz < 1) continue;
    auto row_w = [&](int i) { return i < h.npz_t || i >= h.nzp - h.npz_b ? 1.0 + strip : 1.0; };
    auto col_w = [&](int g) {
      int s = 0;
      for (int j = 4 * g; j < 4 * g + 4; ++j) s += j < h.npx_l || (j >= h.nxp - h.npx_r && j < h.nxp) ? 1 : 0;
      return 4.0 + strip * s;
    };
    WavePlan p;
    p.px = px;
    p.pz = pz;
    p.cells = cells;
    p.cut.resize(pz + px + 2);
    wave_cuts(h.nzp, pz, WAVE_HALO, row_w, p.cut.data());
    wave_cuts(ng, px, 1, col_w, p.cut.data() + pz + 1);
    int gw = 0, most = 0;
    for (int c = 0; c < p.ctas(); ++c) {
      const WaveTile t = wave_tile(p.cut.data(), pz, px, c);
      p.thmax = std::max(p.thmax, t.th);
      gw = std::max(gw, t.gw);
      most = std::max(most, t.th * t.gw * 4);
    }
    p.half = (int64_t)2 * nx * p.thmax + (int64_t)2 * nx * 4 * gw;
    // the most that fits: resident sums first, then conflict-free rows
    bool fits = false;
    for (int k = 0; k < 4 && !fits; ++k) {
      p.n_acc = (k & 2) == 0 ? n.n_acc : 0;
      p.n_src = p.n_acc ? n.n_src : 0;
      p.pad = (k & 1) == 0 ? 32 : 8;
      p.smem = wave_smem(h, p, n);
      fits = p.smem <= WAVE_SMEM_MAX;
    }
    if (!fits) continue;
    // relative cost of a step: SMs left idle, the shape, equal cuts (measured
    // 14 % with two cells a thread), a second pass of a few cells, sums that
    // do not fit
    const double c = (double)ncta / p.ctas() * (1.0 + 0.03 * std::fabs(px - ideal)) *
                     (single ? 1.0 + 0.05 * std::fabs(strip - 0.4) : 1.0 + 0.09 * (1.6 - strip)) *
                     (single && most > WAVE_NT * cells ? 1.3 : 1.0) * (p.n_acc < n.n_acc ? 1.25 : 1.0);
    if (!best.ok() || c < cost) {
      best = p;
      cost = c;
    }
  }
  return best;
}

// Shots of a batch or session run through multi-step launches, one shot after
// another, when their padded grids are small and at most a few small ones of an
// engine are in flight; else in ticks that all shots share.  A tick's launches
// cost much the same for one small shot as for several, a multi-step launch
// follows the shots.  Ticks over multi-step launches, times of 200 steps of
// batches on 256×256 to 440×440 grids:
//
//   shots           1          2          3          4          8         16         45
//   acoustic        1.7–2.0    1.2–1.6    1.07–1.12  0.96–1.13  0.86–0.93 0.76–0.89  0.78–0.91
//   elastic         1.5–1.9    1.2–1.4    0.97–1.04  0.88–0.99  0.76–0.82 0.70–0.74  0.73–0.75
//   viscoacoustic   1.4–1.8    1.02–1.2   0.82–0.95  0.80–0.98  0.67–0.72 0.63–0.74  0.64–0.75
//
// (a viscoacoustic tick's low-passes share their transforms' launches).  Above
// 200,000 cells two shots of an engine come out between 0.94 and 1.5; those
// keep the ticks.  The serving loop with 45 shots of 256×256 to 1024×512 in
// flight: 33.0 shots/s so, 32.7 all in ticks, 28.6 with every small shot in
// multi-step launches; the same jobs arriving at 6, 9, 12 and 16 a second, 99 %
// of the shots done within 0.29, 0.41, 0.57 and 0.61 s so, 0.34, 0.50, 0.57 s
// (6, 9, 12) all in ticks, 0.28, 0.38, 0.54 and 0.65 s with every small shot in
// multi-step launches.  Counting large shots too gave 0.45 s at 9 a second.
inline bool wave_small(int64_t cells) { return cells <= 200000; }
inline bool wave_few(bool visco, int together) { return together <= (visco ? 2 : 3); }

// Whether modelling `nt` steps takes multi-step launches: fewer than 8 cost
// more to set up than they save (step by step and so, ms: 301×201 acoustic 2
// steps 0.137 and 0.179, 5 steps 0.178 and 0.187, 8 steps 0.232 and 0.191;
// 401×601 elastic 0.184 and 0.240, 0.240 and 0.269, 0.307 and 0.282).
inline bool wave_long(int nt) { return nt >= 8; }

// Whether `corners` receiver corner values a step, at most `most` of them in
// one CTA, are few enough: the CTA writes its own, 512 at a time, while the
// others wait, and the host groups all of them once per call.  200 steps, step
// by step and so, ms: 16,000 receivers in a row on 301×201 acoustic (64,000
// corners, 7,700 in a CTA) 5.2 and 3.7, two components of as many on 401×601
// elastic (21,800 in a CTA) 7.6 and 8.6; 60,000 all over 301×201 (240,000
// corners, 1,600 in a CTA) 14.9 and 15.3.
inline bool wave_samples(int64_t corners, int64_t most) { return corners <= 131072 && most <= 8192; }

// Whether an injection that adds at most `most` record values to one cell is
// spread thin enough: a thread adds them one after the other between two
// steps.  Migrations of 200 steps with receivers in a row, step by step and so,
// ms: 401×601 elastic 20 values a cell 12.8 and 9.3, 80 values 15.6 and 20.1;
// 801×601 acoustic 40 values 14.0 and 12.0, 150 values 19.0 and 36.1.
inline bool wave_injects(int most) { return most <= 48; }

// CTA of each padded cell's row and column group.
struct WaveOwner {
  std::vector<int> tr, tc;
  int px;
  WaveOwner(const WaveGrid& h, const WavePlan& p) : tr(h.nzp), tc((h.nxp + 3) / 4), px(p.px) {
    for (int c = 0; c < p.pz; ++c)
      for (int i = p.cut[c]; i < p.cut[c + 1]; ++i) tr[i] = c;
    for (int c = 0; c < p.px; ++c)
      for (int g = p.cut[p.pz + 1 + c]; g < p.cut[p.pz + 2 + c]; ++g) tc[g] = c;
  }
  int of(int i, int j) const { return tr[i] * px + tc[j / 4]; }
};

// Points of the padded grid grouped by the CTAs of a split: CTA c owns
// order[first[c]] … order[first[c + 1] − 1].
struct WaveGroups {
  std::vector<int32_t> first, order;
};
template <class F>
WaveGroups wave_groups(const WaveGrid& h, const WavePlan& p, int n, F&& row_col) {   // row_col(k): {row, column}
  const WaveOwner own(h, p);
  WaveGroups g;
  std::vector<int> cta(n);
  g.first.assign(p.ctas() + 1, 0);
  for (int k = 0; k < n; ++k) {
    const auto [i, j] = row_col(k);
    cta[k] = own.of(i, j);
    ++g.first[cta[k] + 1];
  }
  for (int c = 0; c < p.ctas(); ++c) g.first[c + 1] += g.first[c];
  std::vector<int32_t> pos(g.first.begin(), g.first.end() - 1);
  g.order.resize(n);
  for (int k = 0; k < n; ++k) g.order[pos[cta[k]]++] = k;
  return g;
}

// Tables grouped for one split of a grid serve another when the keys are equal.
// The key is the whole split: the strip weight behind the cuts depends on what
// the work keeps in shared memory, so equal px × pz do not mean equal cuts.
using WaveKey = std::vector<int16_t>;
inline WaveKey wave_key(const WavePlan& p) {
  WaveKey k{(int16_t)p.px, (int16_t)p.pz};
  k.insert(k.end(), p.cut.begin(), p.cut.end());
  return k;
}

}  // namespace ertm
