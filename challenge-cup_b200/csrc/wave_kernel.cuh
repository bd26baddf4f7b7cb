// Many time steps of one or several propagators in one cooperative launch.
//
// The tile kernels of step_kernels.cuh are two launches per time step.  On the
// grids of single shots (0.06–1 M cells) such a step is not bound by memory
// or arithmetic but by the latency of each launch: descriptor loads, staging,
// one pass of arithmetic, drain (4–9 µs a kernel, 14–21 µs a step with the
// receiver or injection kernel).  Here every propagator is split over CTAs
// (one per SM) that keep their part of the wavefield in shared memory for all
// steps of a launch and exchange only the four-cell edges the 8th-order
// stencils read:
//
//  * a CTA owns a rectangle of rows × 4-column groups of the padded grid.  The
//    fields a stencil reads live in shared memory with a four-cell halo, and so
//    do the per-cell coefficients (those that meet dt as a product already
//    multiplied by it), the CPML memories and the viscoacoustic ε and r_l: a
//    step touches global memory only for edges, images and samples.
//  * edges travel through L2 as units of four values, each value in one
//    64-bit word with the exchange's number (epoch): a reader polls the words
//    themselves, so an exchange needs no fence and no flag, and a word of an
//    earlier exchange is never taken for a new one.  A step is two exchanges
//    (stresses before the velocity phase, velocities before the stress
//    phase).  A slot is rewritten only after its reader has published the
//    opposite phase, which it does after it consumed the slot.
//  * imaging sums, stored source fields and receiver samples are written
//    between publishing an edge and waiting for the neighbours'; checkpoints
//    at the end of their step.
//
// What bounds a step now is the chain publish → neighbour's poll → sync (about
// 1700 cycles, twice) plus the two phases of the slowest CTA; a phase is a
// pass of 512 blocks of one or two cells at 750 (straight-line form) to 2200
// cycles (general form) of latency plus 0.8–2 cycles a cell of issue and
// shared-memory bandwidth.  So an edge CTA runs the straight-line form where
// it can, cuts weigh CPML strips, and imaging sums stay in shared memory for
// the launch where they fit (1000 elastic steps of 401×601: 7.9 → 6.7 ms,
// an 800-step PP/PS migration 27.1 → 24.5 ms).  512 threads (up to 128
// registers; the viscoacoustic two-cell form spills 108 bytes, the others none)
// beat 640, 768 and 1024 (64 registers): 1500 acoustic steps of 301×201 with
// 151 receivers 4.6 ms against 5.2, 5.4 and 5.7 ms; 2 × 2 cells a thread were
// no faster than 2 × 1.  Against two or three launches a step: that run
// 24.9 → 4.6 ms, the elastic one 20.9 → 6.7 ms, a 1500-step acoustic migration
// 63.3 → 13.7 ms, the PP/PS migration 50.7 → 24.5 ms.
//
// Every wait is bounded: when a wait runs out the CTA sets STATUS_STALLED and
// leaves; its neighbours' waits then run out too, and later launches on the
// propagator return at once until its status is cleared.  Co-residency is the
// cooperative launch's guarantee.
//
// Arithmetic: expression for expression that of the tile kernels, so fields,
// records and images are the same bit for bit.
#pragma once

#include <type_traits>

#include "step_kernels.cuh"
#include "wave_plan.h"

namespace ertm {

constexpr int WAVE_MAX_WORKS = 2;     // a shot's replay beside its backward pass
constexpr int WAVE_SPIN_LIMIT = 1 << 20;   // polls of one packet (about a second)

// One exchange unit: four cells of one field on one side of a CTA.  It sends
// own cells `src` and receives into halo cells `dst` (offsets from own cell
// (0, 0) of field `slot`); packets `put` of this CTA and `get` of CTA `nb`
// (−1: no neighbour there).  Phase 0 carries the stresses, 1 the velocities.
struct WaveUnit {
  int slot, src, dst, put, get, nb;
};
__host__ __device__ inline WaveUnit wave_unit(bool elastic, int phase, int u, const WaveTile& T, int px, int pz,
                                              int thmax, int W) {
  const int nx = elastic ? 2 : 1, th = T.th, gw = T.gw, cw = 4 * gw;
  const int nxu = nx * th, nzu = nx * 4 * gw;   // units of a left/right side, of an upper/lower side
  const int cta = T.tr * px + T.tc;
  WaveUnit q;
  if (u < 2 * nxu) {
    const int side = u / nxu, v = u - side * nxu, f = v / th, r = v - f * th;
    q.slot = elastic ? (phase == 0 ? (f == 0 ? E_SXX : E_SXZ) : (f == 0 ? E_VX : E_VZ)) : (phase == 0 ? A_P : A_VX);
    q.src = r * W + (side == 0 ? 0 : cw - 4);
    q.dst = r * W + (side == 0 ? -4 : cw);
    q.nb = side == 0 ? (T.tc > 0 ? cta - 1 : -1) : (T.tc + 1 < px ? cta + 1 : -1);
    q.put = u;
    q.get = (1 - side) * nxu + v;
  } else {
    const int u2 = u - 2 * nxu, side = u2 / nzu, v = u2 - side * nzu;
    const int f = v / (4 * gw), v2 = v - f * 4 * gw, k = v2 / gw, c4 = 4 * (v2 - k * gw);
    q.slot = elastic ? (phase == 0 ? (f == 0 ? E_SXZ : E_SZZ) : (f == 0 ? E_VX : E_VZ)) : (phase == 0 ? A_P : A_VZ);
    q.src = (side == 0 ? k : th - 4 + k) * W + c4;
    q.dst = (side == 0 ? k - 4 : th + k) * W + c4;
    q.nb = side == 0 ? (T.tr > 0 ? cta - px : -1) : (T.tr + 1 < pz ? cta + px : -1);
    q.put = 2 * nx * thmax + u2;
    q.get = 2 * nx * thmax + (1 - side) * nzu + v;
  }
  return q;
}

// Blocks (C neighbouring cells) of a CTA whose cells are all physical, clear of
// strips and of the free surface: rows [b0, b1) × block columns [v0, v1) of
// nb × nv.  A CTA of one pass takes one form for all its blocks: two passes
// would cost more than the general form does.
struct WaveInner {
  int nb, nv, b0, b1, v0, v1;
  __host__ __device__ int inner() const { return (b1 - b0) * (v1 - v0); }
  __host__ __device__ int frame() const { return nb * nv - inner(); }
};
template <class GEO>
__host__ __device__ inline WaveInner wave_inner(const GEO& G, const WaveTile& T, int C) {
  auto lo = [](int a, int b) { return a < b ? a : b; };
  auto hi = [](int a, int b) { return a > b ? a : b; };
  const int i0 = T.i0, j0 = 4 * T.g0, cw = 4 * T.gw;
  const int lo_i = hi(hi(G.pad, G.npz_t), G.free_surface ? G.pad + 1 : 0) - i0;
  const int hi_i = lo(G.pad + G.nz, G.nzp - G.npz_b) - i0;
  const int lo_j = hi(G.pad, G.npx_l) - j0, hi_j = lo(G.pad + G.nx, G.nxp - G.npx_r) - j0;
  WaveInner I;
  I.nb = T.th;
  I.nv = cw / C;
  I.b0 = lo(hi(lo_i, 0), I.nb);
  I.b1 = hi(I.b0, lo(hi(hi_i, 0), T.th));
  I.v0 = lo((hi(lo_j, 0) + C - 1) / C, I.nv);
  I.v1 = hi(I.v0, lo(hi(hi_j, 0), cw) / C);
  if (I.b0 == I.b1 || I.v0 == I.v1 || (I.frame() > 0 && I.nb * I.nv <= WAVE_NT)) I.b0 = I.b1 = I.v0 = I.v1 = 0;
  return I;
}

constexpr int WAVE_STAB = 1;        // compensated viscoacoustic amplitude cap inside the launch
constexpr int WAVE_SKIP_LAST = 2;   // the last step's epilogue runs after the launch (a low-pass comes first)

// Time-reversed injection, cells grouped by CTA.
struct WaveInject {
  const int32_t* cta;       // [ncta + 1] into the cell arrays; nullptr: no injection
  const int32_t* slot;      // field slot per cell
  const int32_t* ij;        // padded row << 16 | column per cell
  const int32_t* start;     // [cells + 1] into the contributions
  const int32_t* src;       // record offset per contribution
  const double* wa;
  const double* wb;
  const float* record;
  int64_t nrec;             // floats between time samples
};

// Receiver sampling: every CTA writes the corner cells it owns.
struct WaveSample {
  const int32_t* cta;       // [ncta + 1]; nullptr: no sampling
  const int32_t* slot;      // field slot, −1: ½(σxx + σzz)
  const int32_t* ij;
  const int32_t* out;       // position in a step's row of corner values
  float* buf;               // row k: the corner values after step k
  int64_t stride;
};

struct WaveWork {
  const DevProp* prop;
  int32_t cta0, px, pz, thmax;       // thmax: the tallest CTA
  int16_t cut[WAVE_MAX_CUTS];        // see wave_tile
  int32_t n_steps, t0, sign;         // time index of step k: t0 + sign·k
  int32_t flags, pad;                // WAVE_* bits; halo-field row padding (wave_layout)
  int32_t n_src, n_acc;              // stored source fields staged and imaging sums kept in shared memory
  uint32_t epoch;                    // epochs epoch + 1 … epoch + 2·n_steps
  int32_t start_step;                // cross-correlate from this time on
  const float* wavelet;              // nullptr: no source
  const float* load;                 // state block to start from (nullptr: the propagator's own)
  float* ck;                         // checkpoint block of time ck_t, then one each ck_every steps (or nullptr)
  int32_t ck_every;
  int32_t slot_t;                    // replay slot 0's time
  int64_t ck_floats, slot_floats;    // floats per checkpoint and per replay slot
  double cap;                        // amplitude cap
  StabState* stab;
  int64_t step_index;                // of the first step (stabilisation)
  Epilogue epi;                      // out[]/src[] of replay slot 0
  WaveInject inj;
  WaveSample smp;
};

struct WaveSet {
  int32_t n, drop;                   // works; drop: edges go unread (tests)
  uint64_t* xbuf;                    // exchange buffer: per CTA 2 phases × half units × 2 words, in two planes
  int64_t half;                      // units per CTA and phase
  int64_t plane;                     // words per plane
  uint64_t* peaks;                   // [2][gridDim] stabilisation words
  WaveWork w[WAVE_MAX_WORKS];
};

// Publish / collect one unit: values 0 and 1 in the first plane of 16-byte
// words, 2 and 3 in the second (`plane` words further on), so that a warp's
// accesses are contiguous.
__device__ __forceinline__ void wave_put(uint64_t* p, int64_t plane, const float4& v, uint32_t e) {
  const uint64_t h = (uint64_t)e << 32;
  const uint64_t a = h | __float_as_uint(v.x), b = h | __float_as_uint(v.y), c = h | __float_as_uint(v.z),
                 d = h | __float_as_uint(v.w);
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n" ::"l"(p), "l"(a), "l"(b) : "memory");
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n" ::"l"(p + plane), "l"(c), "l"(d) : "memory");
}
__device__ __forceinline__ bool wave_get(const uint64_t* p, int64_t plane, uint32_t e, float4& v) {
#pragma unroll 1
  for (int it = 0; it < WAVE_SPIN_LIMIT; ++it) {
    uint64_t a, b, c, d;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(c), "=l"(d) : "l"(p + plane) : "memory");
    if ((uint32_t)(a >> 32) == e && (uint32_t)(b >> 32) == e && (uint32_t)(c >> 32) == e &&
        (uint32_t)(d >> 32) == e) {
      v = make_float4(__uint_as_float((uint32_t)a), __uint_as_float((uint32_t)b), __uint_as_float((uint32_t)c),
                      __uint_as_float((uint32_t)d));
      return true;
    }
  }
  return false;
}

// C neighbouring cells of a row: loads, stores, and the windows a stencil reads.
template <int C>
__device__ __forceinline__ void ldv(const float* p, float (&v)[C]) {
  if constexpr (C == 2) {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x;
    v[1] = q.y;
  } else {
    v[0] = *p;
  }
}
template <int C>
__device__ __forceinline__ void stv(float* p, const float (&v)[C]) {
  if constexpr (C == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else *p = v[0];
}
// columns −4 … C + 3 around the first cell; cell c sits at index 4 + c
template <int C>
__device__ __forceinline__ void xwin(const float* p, float (&v)[8 + C]) {
  if constexpr (C == 2) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float2 q = *reinterpret_cast<const float2*>(p - 4 + 2 * k);
      v[2 * k] = q.x;
      v[2 * k + 1] = q.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = p[k - 4];
  }
}
// rows −4 … 4; row 0 at index 4 (rows no stencil uses are not loaded)
template <int C>
__device__ __forceinline__ void zwin(const float* p, int W, float (&z)[C][9]) {
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    float q[C];
    ldv<C>(p + (k - 4) * W, q);
#pragma unroll
    for (int c = 0; c < C; ++c) z[c][k] = q[c];
  }
}
// The 8th-order numerators with the coefficients as constants (sum_plus and
// sum_minus of the tile kernels, term for term).
__device__ __forceinline__ float wave_plus(const float* f, int o) {
  constexpr float c1 = (float)(1225.0 / 1024.0), c2 = (float)(-245.0 / 3072.0), c3 = (float)(49.0 / 5120.0),
                  c4 = (float)(-5.0 / 7168.0);
  float a = fmul(c1, fsub(f[o + 1], f[o]));
  a = fadd(a, fmul(c2, fsub(f[o + 2], f[o - 1])));
  a = fadd(a, fmul(c3, fsub(f[o + 3], f[o - 2])));
  return fadd(a, fmul(c4, fsub(f[o + 4], f[o - 3])));
}
__device__ __forceinline__ float wave_minus(const float* f, int o) { return wave_plus(f, o - 1); }

__device__ __forceinline__ bool nonfinite(float v) { return !(fabsf(v) <= 3.402823466e38f); }

// C neighbouring cells through the work's epilogue at time t (run_epilogue's
// arithmetic), except the imaging condition with float64 sums.
template <int C>
__device__ __forceinline__ void wave_epilogue(const WaveWork& w, int t, ptrdiff_t c0, const bool (&ok)[C],
                                              size_t npix, const float (&pv)[C], const float (&sv)[C]) {
  const Epilogue& E = w.epi;
  const ptrdiff_t at = c0 + (ptrdiff_t)(t - w.slot_t) * w.slot_floats;   // in the replay slots
  if (E.kind == EPI_STORE) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (!ok[c]) continue;
      if (E.out[0]) E.out[0][at + c] = pv[c];
      if (E.out[1]) E.out[1][at + c] = sv[c];
    }
  } else if (E.kind == EPI_IMAGE) {
    const bool cross = t >= w.start_step;
    float s[2][C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      s[0][c] = (ok[c] && E.src[0]) ? E.src[0][at + c] : 0.f;
      s[1][c] = (ok[c] && E.src[1]) ? E.src[1][at + c] : 0.f;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (!ok[c]) continue;
#pragma unroll 1
      for (int k = 0; k < E.n_images; ++k) {
        const float a = E.src_slot[k] ? s[1][c] : s[0][c];
        const float r = E.rcv_wave[k] ? sv[c] : pv[c];
        if (E.illum && E.ill[k]) acc_term(E.ill[k], 1, c0 + c, npix, fmul(a, a));
        if (E.rillum && E.ril[k]) acc_term(E.ril[k], 1, c0 + c, npix, fmul(r, r));
        if (cross) acc_term(E.num[k], 1, c0 + c, npix, fmul(a, r));
      }
    }
  } else if (E.kind == EPI_EXC_TRACK) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (!ok[c]) continue;
      const float a = fabsf(pv[c]);
      if (a > E.running[c0 + c]) {
        E.running[c0 + c] = a;
        E.peak_step[c0 + c] = t;
      }
    }
  } else if (E.kind == EPI_EXC_IMAGE) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (!ok[c] || E.peak_step[c0 + c] != t) continue;
      const double a = (double)E.running[c0 + c];
#pragma unroll 1
      for (int k = 0; k < E.n_images; ++k) {
        const float r = E.rcv_wave[k] ? sv[c] : pv[c];
        E.num[k][c0 + c] = dadd(E.num[k][c0 + c], dmul(a, (double)r));
        if (E.ril[k]) E.ril[k][c0 + c] = dadd(E.ril[k][c0 + c], (double)fmul(r, r));
      }
    }
  }
}

// The imaging condition with float64 sums in global memory for U pieces of C
// cells: two sums of every piece are loaded together before any is stored,
// so a step waits for one or two round trips to L2 instead of one per piece
// and sum.
template <int U, int C>
struct WavePieces {
  ptrdiff_t at[U];       // physical offset of the first cell
  unsigned ok;           // bit u·C + c: the cell is physical
  float pv[U][C], sv[U][C];
};
template <int U, int C>
__device__ __forceinline__ void wave_image_global(const WaveWork& w, int t, const WavePieces<U, C>& K) {
  const Epilogue& E = w.epi;
  const bool cross = t >= w.start_step;
  const ptrdiff_t slot = (ptrdiff_t)(t - w.slot_t) * w.slot_floats;
  float s[2][U][C];
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < C; ++c)
        s[n][u][c] = (E.src[n] && (K.ok >> (u * C + c) & 1)) ? E.src[n][slot + K.at[u] + c] : 0.f;
  // term kinds: 0 S², 1 R², 2 S·R
  auto term = [&](int kind, int k, int u, int c) {
    const float a = E.src_slot[k] ? s[1][u][c] : s[0][u][c];
    const float r = E.rcv_wave[k] ? K.sv[u][c] : K.pv[u][c];
    return (double)(kind == 0 ? fmul(a, a) : (kind == 1 ? fmul(r, r) : fmul(a, r)));
  };
  double* p0 = nullptr;
  int kind0 = 0, k0 = 0;
  auto run = [&](double* p, int kind, int k) {   // pairs up the sums
    if (!p0) {
      p0 = p;
      kind0 = kind;
      k0 = k;
      return;
    }
    double v0[U][C], v1[U][C];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (K.ok >> (u * C + c) & 1) {
          v0[u][c] = p0[K.at[u] + c];
          if (p) v1[u][c] = p[K.at[u] + c];
        }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (K.ok >> (u * C + c) & 1) {
          p0[K.at[u] + c] = dadd(v0[u][c], term(kind0, k0, u, c));
          if (p) p[K.at[u] + c] = dadd(v1[u][c], term(kind, k, u, c));
        }
    p0 = nullptr;
  };
#pragma unroll 1
  for (int k = 0; k < E.n_images; ++k) {
#pragma unroll 1
    for (int kind = 0; kind < 3; ++kind) {
      double* const p = kind == 0 ? (E.illum ? E.ill[k] : nullptr) : (kind == 1 ? (E.rillum ? E.ril[k] : nullptr)
                                                                                : (cross ? E.num[k] : nullptr));
      if (p) run(p, kind, k);
    }
  }
  if (p0) run(nullptr, 0, 0);
}

// The imaging condition with the sums resident (see wave_epilogue): sums of
// the thread's cells at offset o of the tile, source values staged.
template <int C>
__device__ __forceinline__ void wave_image_resident(const Epilogue& E, bool cross, float* acc, const float* src, int CN,
                                                    int o, const float (&pv)[C], const float (&sv)[C]) {
  float s[2][C] = {};
  int q = 0;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (E.src[k]) ldv<C>(src + (q++) * CN + o, s[k]);
  auto add = [&](bool live, const float (&term)[C]) {
    if (live) {
      if (!E.kahan) {
        double* const a = reinterpret_cast<double*>(acc) + o;
#pragma unroll
        for (int c = 0; c < C; ++c) a[c] = dadd(a[c], (double)term[c]);
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const float y = fsub(term[c], acc[CN + o + c]), v = acc[o + c], t = fadd(v, y);
          acc[CN + o + c] = fsub(fsub(t, v), y);
          acc[o + c] = t;
        }
      }
    }
    acc += 2 * CN;
  };
#pragma unroll 1
  for (int k = 0; k < E.n_images; ++k) {
    float a[C], r[C], t[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      a[c] = E.src_slot[k] ? s[1][c] : s[0][c];
      r[c] = E.rcv_wave[k] ? sv[c] : pv[c];
    }
    if (E.illum && E.ill[k]) {
#pragma unroll
      for (int c = 0; c < C; ++c) t[c] = fmul(a[c], a[c]);
      add(true, t);
    }
    if (E.rillum && E.ril[k]) {
#pragma unroll
      for (int c = 0; c < C; ++c) t[c] = fmul(r[c], r[c]);
      add(true, t);
    }
#pragma unroll
    for (int c = 0; c < C; ++c) t[c] = fmul(a[c], r[c]);
    add(cross, t);
  }
}

// The work's imaging sums in the order wave_image_resident walks them.
template <class F>
__device__ __forceinline__ void wave_each_sum(const Epilogue& E, F&& f) {
  int q = 0;
#pragma unroll 1
  for (int k = 0; k < E.n_images; ++k) {
    if (E.illum && E.ill[k]) f(q++, E.ill[k]);
    if (E.rillum && E.ril[k]) f(q++, E.ril[k]);
    f(q++, E.num[k]);
  }
}

__device__ __forceinline__ void cp_async4(float* smem, const float* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}

// Column and row table entries: profile values, strip index (−1: none) with
// flags.
constexpr int WAVE_IN = 1;        // the derivative across this axis is inside the stencil's range
constexpr int WAVE_OK = 2;        // column of the padded grid (not row padding)
constexpr int WAVE_SURFACE = 4;   // the free-surface row
__device__ __forceinline__ int wave_strip_of(const float4& t) { return __float_as_int(t.z); }
__device__ __forceinline__ int wave_flags_of(const float4& t) { return __float_as_int(t.w); }

// ENG: Engine; C: neighbouring cells a thread updates together.
template <int ENG, int C>
__global__ void __launch_bounds__(WAVE_NT, 1) k_wave(const __grid_constant__ WaveSet S) {
  constexpr int M = 4;
  static_assert(C == 1 || C == 2, "one or two cells per thread");
  constexpr int NT = WAVE_NT;
  constexpr bool EL = ENG == ENGINE_ELASTIC, VISCO = ENG == ENGINE_VISCO;
  constexpr int NF = EL ? 5 : 3;         // fields with halos
  constexpr int NX = EL ? 2 : 1;         // fields exchanged per side and phase
  constexpr int NPSI = EL ? 4 : 2;
  extern __shared__ __align__(128) float sm[];
  __shared__ int s_abort;
  __shared__ float s_red[NT / 32 + 1];
  const int tid = threadIdx.x;
  int wi = 0;
#pragma unroll 1
  while (wi + 1 < S.n && (int)blockIdx.x >= S.w[wi + 1].cta0) ++wi;
  // the work and its propagator's descriptor in shared memory (the parameter
  // block is too large for the constant cache to keep)
  __shared__ WaveWork w;
  __shared__ DevProp P;
  {
    static_assert(sizeof(WaveWork) % 4 == 0 && sizeof(DevProp) % 4 == 0, "copied by words");
    const int* const a = reinterpret_cast<const int*>(&S.w[wi]);
    const int* const b = reinterpret_cast<const int*>(S.w[wi].prop);
#pragma unroll 1
    for (int k = tid; k < (int)(sizeof(WaveWork) / 4); k += NT) reinterpret_cast<int*>(&w)[k] = a[k];
#pragma unroll 1
    for (int k = tid; k < (int)(sizeof(DevProp) / 4); k += NT) reinterpret_cast<int*>(&P)[k] = b[k];
    __syncthreads();
  }
  const Geo G(P);
  const int nL = VISCO ? P.L : 0;
  const int cta = (int)blockIdx.x - w.cta0;
  const WaveTile T = wave_tile(w.cut, w.pz, w.px, cta);
  const int i0 = T.i0, th = T.th, gw = T.gw, j0 = 4 * T.g0;
  int sx0, nsx, sz0, nsz;
  wave_strip(j0, min(j0 + 4 * gw, G.nxp), G.nxp, G.npx_l, G.npx_r, sx0, nsx);
  wave_strip(i0, i0 + th, G.nzp, G.npz_t, G.npz_b, sz0, nsz);
  const int ekind = w.epi.kind;
  const int n_epi = (!EL || ekind == EPI_NONE) ? 0 : (w.epi.need_s ? 2 : 1);   // P and S kept beside the fields
  const WaveLayout Y = wave_layout(EL, VISCO, nL, w.pad, th, gw, nsx, nsz, n_epi, w.n_src, w.n_acc);
  const int W = Y.W, cw = Y.cw;
  float* const own = sm + Y.field + WAVE_HALO * W + WAVE_HALO;   // own cell (0, 0) of field 0
  const int FN = Y.field_n;
  float* const cells = sm + Y.cell;
  const int CN = Y.cell_n;
  unsigned char* const qsm = reinterpret_cast<unsigned char*>(sm + Y.qidx);
  float* const e_p = sm + Y.epi;
  float* const e_s = e_p + CN;
  float* const e_src = sm + Y.src;
  float* const accs = sm + Y.acc;
  const float4* const coltab = reinterpret_cast<const float4*>(sm + Y.col);
  const float4* const rowtab = reinterpret_cast<const float4*>(sm + Y.row);
  // ψ of x term t at (row r, strip column s): psx(t)[r·nsx + s]; of z term t
  // at (strip row s, tile column c): psz(t)[s·cw + c]
  auto psx = [&](int t) -> float* { return sm + Y.psix + t * Y.psix_n - sx0; };
  auto psz = [&](int t) -> float* { return sm + Y.psiz + t * Y.psiz_n - sz0 * cw; };
  // cell arrays: acoustic dt·κ dt·irx dt·irz; elastic λ λ+2μ dt·μ dt·irx dt·irz;
  // viscoacoustic K_R dt·irx dt·irz b_l ε r_l
  // ------------------------------------------------------------------ load
  if (tid == 0) s_abort = (*static_cast<volatile uint32_t*>(P.status) & STATUS_STALLED) ? 1 : 0;
#pragma unroll 1
  for (int k = tid; k < NF * FN / 4; k += NT) st4(sm + Y.field + 4 * k, make_float4(0.f, 0.f, 0.f, 0.f));
#pragma unroll 1
  for (int k = tid; k < (Y.psix - Y.cell) / 4; k += NT) st4(sm + Y.cell + 4 * k, make_float4(0.f, 0.f, 0.f, 0.f));
  __syncthreads();
  if (s_abort) return;   // an earlier launch of the run stalled: nothing to go on from
  const ptrdiff_t ld_delta = w.load ? w.load - P.f[0] : 0;
#pragma unroll 1
  for (int k = tid; k < th * gw; k += NT) {
    const int r = k / gw, c4 = 4 * (k - r * gw);
    const size_t g = (size_t)(i0 + r) * G.ld + j0 + c4;
#pragma unroll
    for (int f = 0; f < NF; ++f) st4(own + f * FN + r * W + c4, ld4(P.f[f] + ld_delta + g));
    const int o = r * cw + c4;
    auto scaled = [&](int a, const float* src) {
      const float4 v = ldg4(src + g);
      st4(cells + a * CN + o, make_float4(fmul(G.dt, v.x), fmul(G.dt, v.y), fmul(G.dt, v.z), fmul(G.dt, v.w)));
    };
    if constexpr (EL) {
      st4(cells + 0 * CN + o, ldg4(P.coef[CE_LAM] + g));
      st4(cells + 1 * CN + o, ldg4(P.coef[CE_L2M] + g));
      scaled(2, P.coef[CE_MUXZ]);
      scaled(3, P.coef[CE_IRX]);
      scaled(4, P.coef[CE_IRZ]);
    } else if constexpr (VISCO) {
      st4(cells + 0 * CN + o, ldg4(P.coef[CV_KR] + g));
      scaled(1, P.coef[CV_IRX]);
      scaled(2, P.coef[CV_IRZ]);
#pragma unroll 1
      for (int l = 0; l < nL; ++l) st4(cells + (3 + l) * CN + o, ldg4(P.coef[CV_B0 + l] + g));
#pragma unroll 1
      for (int l = 0; l <= nL; ++l) st4(cells + (3 + nL + l) * CN + o, ld4(P.f[V_EPS + l] + ld_delta + g));
      *reinterpret_cast<uchar4*>(qsm + o) = *reinterpret_cast<const uchar4*>(P.qidx + g);
    } else {
      scaled(0, P.coef[CA_KAPPA]);
      scaled(1, P.coef[CA_IRX]);
      scaled(2, P.coef[CA_IRZ]);
    }
  }
#pragma unroll
  for (int t = 0; t < NPSI; ++t) {
#pragma unroll 1
    for (int k = tid; k < th * nsx; k += NT) {
      const int r = k / nsx, s = k - r * nsx;
      psx(t)[r * nsx + sx0 + s] = (P.psix[t] + ld_delta)[(size_t)(i0 + r) * G.wx + sx0 + s];
    }
#pragma unroll 1
    for (int k = tid; k < nsz * gw; k += NT) {
      const int s = k / gw, c4 = 4 * (k - s * gw);
      st4(psz(t) + (sz0 + s) * cw + c4, ld4(P.psiz[t] + ld_delta + (size_t)(sz0 + s) * G.ld + j0 + c4));
    }
  }
#pragma unroll 1
  for (int k = tid; k < cw; k += NT) {
    const int j = j0 + k, jc = min(j, G.nxp - 1), s = j < G.nxp ? G.sx(j) : -1;
    const int f = (j >= M && j < G.nxp - M ? WAVE_IN : 0) | (j < G.nxp ? WAVE_OK : 0);
    st4(sm + Y.col + 4 * k, make_float4(P.ax[jc], P.bx[jc], __int_as_float(s), __int_as_float(f)));
  }
#pragma unroll 1
  for (int k = tid; k < th; k += NT) {
    const int i = i0 + k;
    const int f = (i >= M && i < G.nzp - M ? WAVE_IN : 0) |
                  (G.free_surface && i == G.pad ? WAVE_SURFACE : 0);
    st4(sm + Y.row + 4 * k, make_float4(P.az[i], P.bz[i], __int_as_float(G.sz(i)), __int_as_float(f)));
  }
  // exchange tables: per unit (one float4 of one field on one side) the
  // shared-memory source and destination and the packet positions
  const int nu = Y.units_n;
  {
    int4* const tab = reinterpret_cast<int4*>(sm + Y.units);
#pragma unroll 1
    for (int k = tid; k < 2 * nu; k += NT) {
      const WaveUnit q = wave_unit(EL, k / nu, k % nu, T, w.px, w.pz, w.thmax, W);
      const int64_t at = ((int64_t)blockIdx.x * 2 + k / nu) * S.half;
      // dropped edges: the CTA waits at its own word of the other phase, which
      // never holds the number it waits for
      const int64_t from = S.drop ? ((int64_t)blockIdx.x * 2 + 1 - k / nu) * S.half
                                  : ((int64_t)(w.cta0 + q.nb) * 2 + k / nu) * S.half;
      tab[k] = make_int4(q.slot * FN + q.src, q.slot * FN + q.dst, (int)(at + q.put), q.nb < 0 ? -1 : (int)(from + q.get));
    }
  }
  __syncthreads();
  const int4* const tab0 = reinterpret_cast<const int4*>(sm + Y.units);
  const size_t npix = (size_t)G.nz * G.nx;
  const bool want_curl = EL && ekind != EPI_NONE && w.epi.sep == 1 && w.epi.need_s;
  const int esep = w.epi.sep;
  const int inj_a = w.inj.cta ? w.inj.cta[cta] : 0, inj_b = w.inj.cta ? w.inj.cta[cta + 1] : 0;
  const int smp_a = w.smp.cta ? w.smp.cta[cta] : 0, smp_b = w.smp.cta ? w.smp.cta[cta + 1] : 0;
  double ref_amp = (VISCO && (w.flags & WAVE_STAB)) ? w.stab->ref_amp : 0.0;
  // the thread's first sampled corner: offset in the halo fields (−2 − offset:
  // the pressure there), −1 none
  int smp_off = -1, smp_out = 0;
  if (smp_a + tid < smp_b) {
    const int ij = w.smp.ij[smp_a + tid], s = w.smp.slot[smp_a + tid];
    const int o = ((ij >> 16) - i0) * W + (ij & 0xffff) - j0;
    smp_off = s >= 0 ? s * FN + o : -2 - o;
    smp_out = w.smp.out[smp_a + tid];
  }
  int clipped = 0;
  float last_peak = 0.f;
  bool bad = false;
  const int mech = P.mech;
  // the thread's cells: blocks of C cells tid, tid + NT, … in row-major
  // order; body(first row, first column)
  const int nv = cw / C;
  const int row0 = tid / nv, col0 = (tid - row0 * nv) * C;
  const int drow = NT / nv, dcol = (NT - drow * nv) * C;
  auto each = [&](auto&& body) {
    int r = row0, c = col0;
#pragma unroll 1
    while (r < th) {
      body(r, c);
      r += drow;
      c += dcol;
      if (c >= cw) {
        c -= cw;
        ++r;
      }
    }
  };

  // the CTA's straight-line rectangle; the frame around it takes the general
  // form of the updates
  const WaveInner I = wave_inner(G, T, C);
  const int nb = I.nb, b0 = I.b0, b1 = I.b1, v0 = I.v0, v1 = I.v1;
  const int n_inner = (b1 - b0) * (v1 - v0), n_frame = nb * nv - n_inner;
  auto frame_block = [&](int k, int& r, int& c) {   // rows above, rows below, then the sides
    const int above = b0 * nv, below = (nb - b1) * nv;
    int b, v;
    if (k < above) {
      b = k / nv;
      v = k - b * nv;
    } else if (k < above + below) {
      k -= above;
      b = k / nv;
      v = k - b * nv;
      b += b1;
    } else {
      k -= above + below;
      const int side = nv - (v1 - v0);
      b = k / side;
      v = k - b * side;
      b += b0;
      if (v >= v0) v += v1 - v0;
    }
    r = b;
    c = v * C;
  };
  const int wi_ = max(v1 - v0, 1);
  const int in_r = b0 + tid / wi_, in_c = (v0 + tid % wi_) * C;   // the thread's first inner block
  const int in_dr = NT / wi_, in_dc = NT % wi_ * C;
  int fr_r = 0, fr_c = 0;                                               // and its first frame block
  if (tid < n_frame) frame_block(tid, fr_r, fr_c);
  auto update = [&](auto&& body) {
#pragma unroll 1
    for (int k = tid, r = in_r, c = in_c; k < n_inner; k += NT) {
      body(std::false_type{}, r, c);
      r += in_dr;
      c += in_dc;
      if (c >= v1 * C) {
        c -= (v1 - v0) * C;
        ++r;
      }
    }
#pragma unroll 1
    for (int k = tid, r = fr_r, c = fr_c; k < n_frame;) {
      body(std::true_type{}, r, c);
      k += NT;
      if (k < n_frame) frame_block(k, r, c);
    }
  };
  // the source: its cell's owner adds the amplitude after its update
  const bool src_here = w.wavelet && G.src_iz >= i0 && G.src_iz < i0 + th && G.src_ix >= j0 && G.src_ix < j0 + cw &&
                        G.src_ix < G.nxp;
  const int src_o = src_here ? (G.src_iz - i0) * W + G.src_ix - j0 : 0;
  const int src_e = src_here ? (G.src_iz - i0) * cw + G.src_ix - j0 : 0;
  int src_tid = -1;   // the thread that updates the source's block (frame_block and the inner walk inverted)
  if (src_here) {
    const int b = G.src_iz - i0, v = (G.src_ix - j0) / C, side = nv - (v1 - v0);
    int k;
    if (b >= b0 && b < b1 && v >= v0 && v < v1) k = (b - b0) * (v1 - v0) + v - v0;
    else if (b < b0) k = b * nv + v;
    else if (b >= b1) k = b0 * nv + (b - b1) * nv + v;
    else k = (b0 + nb - b1) * nv + (b - b0) * side + (v < v0 ? v : v - (v1 - v0));
    src_tid = k % NT;
  }

  // injection: the thread's first cell and its first contribution
  auto inject_cell = [&](int q) -> float* {
    const int ij = w.inj.ij[q], s = w.inj.slot[q], i = ij >> 16, j = ij & 0xffff;
    if (VISCO && s >= V_EPS)
      return cells + (3 + nL) * CN + (i - i0) * cw + j - j0;
    return own + s * FN + (i - i0) * W + j - j0;
  };
  float* inj_cell = nullptr;
  int inj_c0 = 0, inj_c1 = 0;
  double inj_wa = 0.0, inj_wb = 0.0;
  // (threads without a contribution follow the record's rows at column 0, so
  // the look-ahead below is an unconditional load inside the record)
  const float* inj_p = w.inj.cta ? w.inj.record + (int64_t)w.t0 * w.inj.nrec : nullptr;
  float inj_v = 0.f;
  if (inj_a + tid < inj_b) {
    const int q = inj_a + tid;
    inj_cell = inject_cell(q);
    inj_c0 = w.inj.start[q];
    inj_c1 = w.inj.start[q + 1];
    if (inj_c0 < inj_c1) {
      inj_p += w.inj.src[inj_c0];
      inj_wa = w.inj.wa[inj_c0];
      inj_wb = w.inj.wb[inj_c0];
      inj_v = *inj_p;
    }
  }

  // hot scalars of the work in registers (it lies in shared memory), and what
  // this CTA does between steps: nothing for most CTAs of a forward run
  const int n_steps = w.n_steps, sign = w.sign, flags = w.flags, n_acc = w.n_acc;
  const bool between = ekind != EPI_NONE || smp_b > smp_a || inj_b > inj_a || n_acc;
  const bool has_ck = w.ck != nullptr;
  uint64_t* const xbuf = S.xbuf;
  const int64_t plane = S.plane;

  // Publish this phase's edges; the caller may do other work, then collects.
  auto publish = [&](int ph, uint32_t e) {
#pragma unroll 1
    for (int u = tid; u < nu; u += NT) {
      const int4 q = tab0[ph * nu + u];
      if (q.w >= 0) wave_put(xbuf + 2 * (size_t)q.z, plane, ld4(own + q.x), e);
    }
  };
  auto collect = [&](int ph, uint32_t e) {
#pragma unroll 1
    for (int u = tid; u < nu; u += NT) {
      const int4 q = tab0[ph * nu + u];
      if (q.w < 0) continue;
      float4 v;
      if (wave_get(xbuf + 2 * (size_t)q.w, plane, e, v)) st4(own + q.y, v);
      else s_abort = 1;
    }
  };
  // What a finished step leaves behind: imaging or stored fields, samples.
  auto finish = [&](int k) {
    const int t = w.t0 + w.sign * k;
    bool run = ekind != EPI_NONE && !((w.flags & WAVE_SKIP_LAST) && k + 1 == w.n_steps);
    if (t < w.start_step && (ekind == EPI_EXC_IMAGE || (ekind == EPI_IMAGE && !w.epi.illum && !w.epi.rillum)))
      run = false;
    if (run && w.n_acc) cp_async_wait_all();   // each thread staged its own cells
    if (run && !w.n_acc && ekind == EPI_IMAGE && !w.epi.kahan) {
      // two blocks of the thread at a time
      constexpr int U = 2;
      int r = row0, c0 = col0;
#pragma unroll 1
      while (r < th) {
        WavePieces<U, C> K;
        K.ok = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int ii = i0 + r - G.pad, jj = j0 + c0 - G.pad;
          K.at[u] = (ptrdiff_t)ii * G.nx + jj;
          if (r < th && ii >= 0 && ii < G.nz) {
#pragma unroll
            for (int c = 0; c < C; ++c)
              if (jj + c >= 0 && jj + c < G.nx) K.ok |= 1u << (u * C + c);
            if constexpr (EL) ldv<C>(e_p + r * cw + c0, K.pv[u]);
            else ldv<C>(own + A_P * FN + r * W + c0, K.pv[u]);
            if (n_epi == 2) ldv<C>(e_s + r * cw + c0, K.sv[u]);
          }
          r += drow;
          c0 += dcol;
          if (c0 >= cw) {
            c0 -= cw;
            ++r;
          }
        }
        wave_image_global<U, C>(w, t, K);
      }
    } else if (run) {
      each([&](int r, int c0) {
        const int ii = i0 + r - G.pad, jj = j0 + c0 - G.pad;
        if (ii < 0 || ii >= G.nz) return;
        float pv[C], sv[C] = {};
        if constexpr (EL) ldv<C>(e_p + r * cw + c0, pv);
        else ldv<C>(own + A_P * FN + r * W + c0, pv);
        if (n_epi == 2) ldv<C>(e_s + r * cw + c0, sv);
        if (n_acc) {   // cells outside the physical grid sum into slots nobody reads
          wave_image_resident<C>(w.epi, t >= w.start_step, accs, e_src, CN, r * cw + c0, pv, sv);
        } else {
          bool ok[C];
#pragma unroll
          for (int c = 0; c < C; ++c) ok[c] = jj + c >= 0 && jj + c < G.nx;
          wave_epilogue<C>(w, t, (ptrdiff_t)ii * G.nx + jj, ok, npix, pv, sv);
        }
      });
    }
    if (smp_off != -1) {
      // the thread's first corner cell; further ones from the list
      float* const row = w.smp.buf + (int64_t)k * w.smp.stride;
      row[smp_out] = smp_off >= 0 ? own[smp_off] : fmul(0.5f, fadd(own[E_SXX * FN - smp_off - 2], own[E_SZZ * FN - smp_off - 2]));
#pragma unroll 1
      for (int q = smp_a + tid + NT; q < smp_b; q += NT) {
        const int ij = w.smp.ij[q], s = w.smp.slot[q];
        const int o = ((ij >> 16) - i0) * W + (ij & 0xffff) - j0;
        row[w.smp.out[q]] = s >= 0 ? own[s * FN + o] : fmul(0.5f, fadd(own[E_SXX * FN + o], own[E_SZZ * FN + o]));
      }
    }
  };
  // Stage the source fields of time t for finish(): each thread its own cells.
  auto stage_sources = [&](int t) {
    const ptrdiff_t s = (ptrdiff_t)(t - w.slot_t) * w.slot_floats;
    each([&](int r, int c0) {
      const int ii = i0 + r - G.pad, jj = j0 + c0 - G.pad;
      if (ii < 0 || ii >= G.nz) return;
      int n = 0;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (!w.epi.src[k]) continue;
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (jj + c >= 0 && jj + c < G.nx)
            cp_async4(e_src + n * CN + r * cw + c0 + c, w.epi.src[k] + s + (ptrdiff_t)ii * G.nx + jj + c);
        ++n;
      }
    });
    cp_async_commit();
  };
  // Imaging sums between global memory and their resident copies.
  auto move_sums = [&](bool in) {
#pragma unroll 1
    for (int k = tid; k < th * cw; k += NT) {
      const int r = k / cw, c = k - r * cw, ii = i0 + r - G.pad, jj = j0 + c - G.pad;
      if (ii < 0 || ii >= G.nz || jj < 0 || jj >= G.nx) continue;
      const size_t p = (size_t)ii * G.nx + jj;
      wave_each_sum(w.epi, [&](int q, double* g) {
        float* const a = accs + 2 * q * CN;
        if (!w.epi.kahan) {
          double* const d = reinterpret_cast<double*>(a) + k;
          if (in) *d = g[p];
          else g[p] = *d;
        } else {
          float* const f = reinterpret_cast<float*>(g);
          if (in) {
            a[k] = f[p];
            a[CN + k] = f[npix + p];
          } else {
            f[p] = a[k];
            f[npix + p] = a[CN + k];
          }
        }
      });
    }
  };
  // Write the CTA's part of the state into a state block (own or checkpoint).
  auto store_state = [&](ptrdiff_t delta) {
#pragma unroll 1
    for (int k = tid; k < th * gw; k += NT) {
      const int r = k / gw, c4 = 4 * (k - r * gw);
      const size_t g = (size_t)(i0 + r) * G.ld + j0 + c4;
#pragma unroll
      for (int f = 0; f < NF; ++f) st4(P.f[f] + delta + g, ld4(own + f * FN + r * W + c4));
      if constexpr (VISCO) {
#pragma unroll 1
        for (int l = 0; l <= nL; ++l)
          st4(P.f[V_EPS + l] + delta + g, ld4(cells + (3 + nL + l) * CN + r * cw + c4));
      }
    }
#pragma unroll
    for (int t = 0; t < NPSI; ++t) {
#pragma unroll 1
      for (int k = tid; k < th * nsx; k += NT) {
        const int r = k / nsx, s = k - r * nsx;
        (P.psix[t] + delta)[(size_t)(i0 + r) * G.wx + sx0 + s] = psx(t)[r * nsx + sx0 + s];
      }
#pragma unroll 1
      for (int k = tid; k < nsz * gw; k += NT) {
        const int s = k / gw, c4 = 4 * (k - s * gw);
        st4(P.psiz[t] + delta + (size_t)(sz0 + s) * G.ld + j0 + c4, ld4(psz(t) + (sz0 + s) * cw + c4));
      }
    }
  };

  // cell array `a` (per-cell coefficients) of the thread's cells
  auto coef = [&](int a, int r, int c0, float (&v)[C]) { ldv<C>(cells + a * CN + r * cw + c0, v); };
  // CPML memories of the thread's cells (edge CTAs): N terms at once, all
  // loaded before any is stored; d[n][c] ← corrected derivative
  auto strips_x = [&](auto first, auto& d, int r, const float4 (&ct)[C]) {
    constexpr int N = sizeof(d) / sizeof(d[0]);
    float q[N][C];
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int c = 0; c < C; ++c)
        q[n][c] = wave_strip_of(ct[c]) >= 0 ? psx(first + n)[r * nsx + wave_strip_of(ct[c])] : 0.f;
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (wave_strip_of(ct[c]) >= 0) {
          (*d[n])[c] = cpml((*d[n])[c], q[n][c], ct[c].x, ct[c].y);
          psx(first + n)[r * nsx + wave_strip_of(ct[c])] = q[n][c];
        }
  };
  auto strips_z = [&](auto first, auto& d, int c0, const float4& rt, const float4 (&ct)[C]) {
    constexpr int N = sizeof(d) / sizeof(d[0]);
    float q[N][C];
#pragma unroll
    for (int n = 0; n < N; ++n) ldv<C>(psz(first + n) + wave_strip_of(rt) * cw + c0, q[n]);
#pragma unroll
    for (int n = 0; n < N; ++n) {
#pragma unroll
      for (int c = 0; c < C; ++c)
        if (wave_flags_of(ct[c]) & WAVE_OK) (*d[n])[c] = cpml((*d[n])[c], q[n][c], rt.x, rt.y);
      stv<C>(psz(first + n) + wave_strip_of(rt) * cw + c0, q[n]);
    }
  };

  // pressure engines image p itself, so a CTA that injects finishes a step
  // before the next one's injection, every other CTA after publishing
  const bool early = !EL && inj_b > inj_a;
  int t = w.t0;
  uint32_t e = w.epoch + 1;
#pragma unroll 1
  for (int k = 0;; ++k, t += sign, e += 2) {
    if (between) {
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {   // one copy of finish()
        if (k > 0 && (pass == 0) == early) {
          finish(k - 1);
          if (early) __syncthreads();
        }
        if (pass == 0 && k < n_steps) {
          if (inj_b > inj_a) {
            const int64_t off = (int64_t)t * w.inj.nrec;
#pragma unroll 1
            for (int q = inj_a + tid; q < inj_b; q += NT) {
              const bool mine = q == inj_a + tid;   // the thread's first cell: its list entry is in registers
              const int c1 = mine ? inj_c1 : w.inj.start[q + 1];
              int c = mine ? inj_c0 : w.inj.start[q];
              float* f = mine ? inj_cell : inject_cell(q);
              float acc = *f;
              if (mine && c < c1) {
                acc = __double2float_rn(dadd((double)acc, dmul(dmul((double)inj_v, inj_wa), inj_wb)));
                ++c;
              }
#pragma unroll 1
              for (; c < c1; ++c) {
                const double v = (double)w.inj.record[w.inj.src[c] + off];
                acc = __double2float_rn(dadd((double)acc, dmul(dmul(v, w.inj.wa[c]), w.inj.wb[c])));
              }
              *f = acc;
            }
            __syncthreads();
            // the next step's sample of the first contribution, in flight until then
            if (k + 1 < n_steps) inj_p += sign * w.inj.nrec;
            inj_v = *inj_p;
          }
          publish(0, e);
        }
      }
      // the sums come in before the first step's imaging and go out after the
      // last's
      if (n_acc && (k == 0 || k == n_steps)) {
        __syncthreads();
        move_sums(k == 0);
        __syncthreads();
      }
    } else if (k < n_steps) {
      publish(0, e);
    }
    if (k > 0 && (has_ck || k == n_steps)) {   // states go out after their step
#pragma unroll 1
      for (int out = 0; out < 2; ++out) {
        const int done = t - sign;   // time of the last finished step
        if (out == 0 ? (has_ck && done % w.ck_every == 0) : k == n_steps)
          store_state(out == 0 ? (w.ck - P.f[0]) + (ptrdiff_t)(done / w.ck_every) * w.ck_floats : 0);
      }
    }
    if (k == n_steps) break;
    if (n_acc) stage_sources(t);
    collect(0, e);
    __syncthreads();
    if (s_abort) break;
    // -------------------------------------------------------------- velocity
    // EDGE: the CTA touches strips, the rim, the free surface or the source
    auto velocity = [&](auto edge, int r, int c0) {
      constexpr bool EDGE = decltype(edge)::value;
      float* const at = own + r * W + c0;
      float4 ct[C];
      if constexpr (EDGE) {
#pragma unroll
        for (int c = 0; c < C; ++c) ct[c] = coltab[c0 + c];
      }
      float z1[C][9], z2[EL ? C : 1][9];
      zwin<C>(at + (EL ? E_SXZ : A_P) * FN, W, z1);
      if constexpr (EL) zwin<C>(at + E_SZZ * FN, W, z2);
      float4 rt;
      if constexpr (EDGE) rt = rowtab[r];
      const bool zin = !EDGE || (wave_flags_of(rt) & WAVE_IN);
      float ax[C], az[C], bx[C], bz[C];   // x and z terms of vx, then of vz
      float v[8 + C];
      if constexpr (!EL) {
        xwin<C>(at + A_P * FN, v);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool xin = !EDGE || (wave_flags_of(ct[c]) & WAVE_IN);
          ax[c] = xin ? G.dxf(wave_plus(v, 4 + c)) : 0.f;
          bz[c] = zin ? G.dzf(wave_plus(z1[c], 4)) : 0.f;
        }
      } else {
        xwin<C>(at + E_SXX * FN, v);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool xin = !EDGE || (wave_flags_of(ct[c]) & WAVE_IN);
          ax[c] = xin ? G.dxf(wave_plus(v, 4 + c)) : 0.f;
          az[c] = zin ? G.dzf(wave_minus(z1[c], 4)) : 0.f;
        }
        xwin<C>(at + E_SXZ * FN, v);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool xin = !EDGE || (wave_flags_of(ct[c]) & WAVE_IN);
          bx[c] = xin ? G.dxf(wave_minus(v, 4 + c)) : 0.f;
          bz[c] = zin ? G.dzf(wave_plus(z2[c], 4)) : 0.f;
        }
      }
      if constexpr (EDGE) {
        if constexpr (EL) {
          float(*const dx[2])[C] = {&ax, &bx};
          float(*const dz[2])[C] = {&az, &bz};
          if (nsx) strips_x(0, dx, r, ct);
          if (nsz && wave_strip_of(rt) >= 0) strips_z(0, dz, c0, rt, ct);
        } else {
          float(*const dx[1])[C] = {&ax};
          float(*const dz[1])[C] = {&bz};
          if (nsx) strips_x(0, dx, r, ct);
          if (nsz && wave_strip_of(rt) >= 0) strips_z(0, dz, c0, rt, ct);
        }
      }
      float* const pvx = at + (EL ? E_VX : A_VX) * FN;
      float* const pvz = at + (EL ? E_VZ : A_VZ) * FN;
      float ox[C], oz[C], kx[C], kz[C];
      ldv<C>(pvx, ox);
      ldv<C>(pvz, oz);
      coef(EL ? 3 : 1, r, c0, kx);
      coef(EL ? 4 : 2, r, c0, kz);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if (EDGE && !(wave_flags_of(ct[c]) & WAVE_OK)) continue;
        ox[c] = fadd(ox[c], fmul(kx[c], EL ? fadd(ax[c], az[c]) : ax[c]));
        oz[c] = fadd(oz[c], fmul(kz[c], EL ? fadd(bx[c], bz[c]) : bz[c]));
      }
      stv<C>(pvx, ox);
      stv<C>(pvz, oz);
    };
    update(velocity);
    __syncthreads();
    publish(1, e + 1);
    float amp = 0.f, amp_eps = 0.f;
    if (src_here) {
      amp = w.wavelet[t];
      if (VISCO && amp != 0.f)
        amp_eps = __double2float_rn(
            __ddiv_rn((double)amp, (double)P.coef[CV_KR][(size_t)G.src_iz * G.ld + G.src_ix]));
    }
    collect(1, e + 1);
    __syncthreads();
    if (s_abort) break;
    // ---------------------------------------------------------------- stress
    float peak = 0.f;
    auto stress = [&](auto edge, int r, int c0) {
      constexpr bool EDGE = decltype(edge)::value;
      float* const at = own + r * W + c0;
      float z1[C][9], z2[EL ? C : 1][9];
      zwin<C>(at + (EL ? E_VZ : A_VZ) * FN, W, z1);
      if constexpr (EL) zwin<C>(at + E_VX * FN, W, z2);
      float4 ct[C], rt;
      bool live[C];   // column of the grid
      if constexpr (EDGE) rt = rowtab[r];
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if constexpr (EDGE) ct[c] = coltab[c0 + c];
        live[c] = !EDGE || (wave_flags_of(ct[c]) & WAVE_OK);
      }
      const bool zin = !EDGE || (wave_flags_of(rt) & WAVE_IN);
      const bool zstrip = EDGE && nsz && wave_strip_of(rt) >= 0;
      const bool surface = EDGE && (wave_flags_of(rt) & WAVE_SURFACE);
      float dx[C], dz[C];
      if constexpr (!EL) {
        float v[8 + C];
        xwin<C>(at + A_VX * FN, v);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool xin = !EDGE || (wave_flags_of(ct[c]) & WAVE_IN);
          dx[c] = xin ? G.dxf(wave_minus(v, 4 + c)) : 0.f;
          dz[c] = zin ? G.dzf(wave_minus(z1[c], 4)) : 0.f;
        }
        if constexpr (EDGE) {
          float(*const ex[1])[C] = {&dx};
          float(*const ez[1])[C] = {&dz};
          if (nsx) strips_x(1, ex, r, ct);
          if (zstrip) strips_z(1, ez, c0, rt, ct);
        }
        float* const pp = at + A_P * FN;
        float out[C], kk[C];
        ldv<C>(pp, out);
        if constexpr (!VISCO) {
          coef(0, r, c0, kk);
#pragma unroll
          for (int c = 0; c < C; ++c) {
            if (!live[c]) continue;
            out[c] = fadd(out[c], fmul(kk[c], fadd(dx[c], dz[c])));
            if (surface) out[c] = 0.f;
          }
        } else {
          const int o = r * cw + c0;
          float* const pe = cells + (3 + nL) * CN + o;
          float* const pr = cells + (4 + nL) * CN + o;
          const float* const pb = cells + 3 * CN + o;
          const unsigned char* const pq = qsm + o;
          float ev[C], rl[kRelaxUnroll][C], bl[kRelaxUnroll][C], tot[C];
          int q[C];
          ldv<C>(pe, ev);
          coef(0, r, c0, kk);
          // every mechanism's memory and coefficient before any is stored
#pragma unroll
          for (int c = 0; c < C; ++c) q[c] = pq[c] * nL;
#pragma unroll
          for (int l = 0; l < kRelaxUnroll; ++l)
            if (l < nL) {
              ldv<C>(pr + l * CN, rl[l]);
              ldv<C>(pb + l * CN, bl[l]);
            }
          float inc[C];
#pragma unroll
          for (int c = 0; c < C; ++c) {
            inc[c] = fmul(G.dt, fadd(dx[c], dz[c]));
            tot[c] = 0.f;
          }
#pragma unroll
          for (int l = 0; l < kRelaxUnroll; ++l)
            if (l < nL) {
#pragma unroll
              for (int c = 0; c < C; ++c) {
                const float rv = fadd(fmul(rl[l][c], __ldg(P.relax_a + q[c] + l)), fmul(bl[l][c], inc[c]));
                if (live[c]) rl[l][c] = rv;
                tot[c] = l == 0 ? rv : fadd(tot[c], rv);
              }
              stv<C>(pr + l * CN, rl[l]);
            }
#pragma unroll
          for (int c = 0; c < C; ++c) {
            if (!live[c]) continue;
            float ee = fadd(ev[c], inc[c]);
            float pv = fadd(fmul(kk[c], ee), tot[c]);
            ev[c] = ee;
            out[c] = pv;
            peak = fmaxf(peak, fabsf(pv));
          }
          stv<C>(pe, ev);
        }
        stv<C>(pp, out);
#pragma unroll
        for (int c = 0; c < C; ++c) bad |= nonfinite(out[c]);
      } else {
        float gx[C], gz[C], pv[C], sv[C] = {};   // ∂x vz and ∂z vx of σxz; P and S of the epilogue
        float v[8 + C];
        xwin<C>(at + E_VX * FN, v);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool xin = !EDGE || (wave_flags_of(ct[c]) & WAVE_IN);
          dx[c] = xin ? G.dxf(wave_minus(v, 4 + c)) : 0.f;
          dz[c] = zin ? G.dzf(wave_minus(z1[c], 4)) : 0.f;
          pv[c] = fadd(dx[c], dz[c]);
        }
        xwin<C>(at + E_VZ * FN, v);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const bool xin = !EDGE || (wave_flags_of(ct[c]) & WAVE_IN);
          gx[c] = xin ? G.dxf(wave_plus(v, 4 + c)) : 0.f;
          gz[c] = zin ? G.dzf(wave_plus(z2[c], 4)) : 0.f;
          if (want_curl) sv[c] = fsub(G.dzf(wave_minus(z2[c], 4)), G.dxf(wave_minus(v, 4 + c)));
        }
        if constexpr (EDGE) {
          float(*const ex[2])[C] = {&dx, &gx};
          float(*const ez[2])[C] = {&dz, &gz};
          if (nsx) strips_x(2, ex, r, ct);
          if (zstrip) strips_z(2, ez, c0, rt, ct);
        }
        float* const pxx = at + E_SXX * FN;
        float* const pzz = at + E_SZZ * FN;
        float* const pxz = at + E_SXZ * FN;
        float oxx[C], ozz[C], oxz[C], lam[C], l2m[C], dmu[C];
        ldv<C>(pxx, oxx);
        ldv<C>(pzz, ozz);
        ldv<C>(pxz, oxz);
        coef(0, r, c0, lam);
        coef(1, r, c0, l2m);
        coef(2, r, c0, dmu);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (!live[c]) continue;
          oxx[c] = fadd(oxx[c], fmul(G.dt, fadd(fmul(l2m[c], dx[c]), fmul(lam[c], dz[c]))));
          ozz[c] = fadd(ozz[c], fmul(G.dt, fadd(fmul(lam[c], dx[c]), fmul(l2m[c], dz[c]))));
          oxz[c] = fadd(oxz[c], fmul(dmu[c], fadd(gz[c], gx[c])));
          if (surface) {
            ozz[c] = 0.f;
            oxz[c] = 0.f;
          }
        }
        stv<C>(pxx, oxx);
        stv<C>(pzz, ozz);
        stv<C>(pxz, oxz);
#pragma unroll
        for (int c = 0; c < C; ++c) bad |= nonfinite(oxx[c]) || nonfinite(ozz[c]) || nonfinite(oxz[c]);
        if (n_epi) {
          if (esep == 0) {
#pragma unroll
            for (int c = 0; c < C; ++c) {
              pv[c] = fmul(0.5f, fadd(oxx[c], ozz[c]));
              sv[c] = oxz[c];
            }
          }
          stv<C>(e_p + r * cw + c0, pv);
          if (n_epi == 2) stv<C>(e_s + r * cw + c0, sv);
        }
      }
    };
    update(stress);
    // the source, by the thread that has just updated its cell
    if (tid == src_tid && amp != 0.f) {
      auto add = [&](float* f, float a) {
        *f = fadd(*f, a);
        bad |= nonfinite(*f);
      };
      const bool surface = G.free_surface && G.src_iz == G.pad;   // the surface zeroes p, σzz and σxz after it
      if constexpr (EL) {
        if (mech == MECH_SHEAR) {
          if (!surface) add(own + E_SXZ * FN + src_o, amp);
        } else if (mech == MECH_EXPLOSIVE) {
          add(own + E_SXX * FN + src_o, amp);
          if (!surface) add(own + E_SZZ * FN + src_o, amp);
        }
        if (n_epi && esep == 0) {
          e_p[src_e] = fmul(0.5f, fadd(own[E_SXX * FN + src_o], own[E_SZZ * FN + src_o]));
          if (n_epi == 2) e_s[src_e] = own[E_SXZ * FN + src_o];
        }
      } else if (!surface) {
        add(own + A_P * FN + src_o, amp);
        if constexpr (VISCO) add(cells + (3 + nL) * CN + src_e, amp_eps);
      }
    }
    __syncthreads();
    if (EL && mech == MECH_FORCE_Z && src_here && amp != 0.f) {
      // a vertical force lands on vz once every thread has read it
      if (tid == src_tid) own[E_VZ * FN + src_o] = fadd(own[E_VZ * FN + src_o], amp);
      __syncthreads();
    }
    // -------------------------------------------- compensated amplitude cap
    if (VISCO && (flags & WAVE_STAB)) {
      const int ncta = w.px * w.pz;
#pragma unroll 1
      for (int o = 16; o > 0; o >>= 1) peak = fmaxf(peak, __shfl_xor_sync(0xffffffffu, peak, o));
      if ((tid & 31) == 0) s_red[tid >> 5] = peak;
      __syncthreads();
      uint64_t* const words = S.peaks + (size_t)(k & 1) * gridDim.x + w.cta0;
      if (tid == 0) {
        float m = s_red[0];
#pragma unroll 1
        for (int q = 1; q < NT / 32; ++q) m = fmaxf(m, s_red[q]);
        const uint64_t word = ((uint64_t)e << 32) | __float_as_uint(m);
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(words + cta), "l"(word) : "memory");
      }
      __syncthreads();
      float m = 0.f;
#pragma unroll 1
      for (int q = tid; q < ncta; q += NT) {
        uint64_t word = 0;
        int it = 0;
#pragma unroll 1
        for (; it < WAVE_SPIN_LIMIT; ++it) {
          asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(word) : "l"(words + q) : "memory");
          if ((uint32_t)(word >> 32) == e) break;
        }
        if (it == WAVE_SPIN_LIMIT) s_abort = 1;
        m = fmaxf(m, __uint_as_float((uint32_t)word));
      }
#pragma unroll 1
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((tid & 31) == 0) s_red[tid >> 5] = m;
      __syncthreads();
      if (s_abort) break;
      m = s_red[0];
#pragma unroll 1
      for (int q = 1; q < NT / 32; ++q) m = fmaxf(m, s_red[q]);
      last_peak = m;
      const double pk = (double)m;
      if (w.step_index + k < 30) {
        ref_amp = ref_amp > pk ? ref_amp : pk;
      } else {
        const double limit = w.cap * (ref_amp > 1e-30 ? ref_amp : 1e-30);
        if (pk > limit) {
          const float s = __double2float_rn(__ddiv_rn(limit, pk));
          ++clipped;
          auto scale4 = [&](float* f) {
            const float4 v = ld4(f);
            st4(f, make_float4(fmul(v.x, s), fmul(v.y, s), fmul(v.z, s), fmul(v.w, s)));
          };
#pragma unroll 1
          for (int q = tid; q < th * gw; q += NT) {
            const int r = q / gw, c4 = 4 * (q - r * gw);
#pragma unroll
            for (int f = 0; f < NF; ++f) scale4(own + f * FN + r * W + c4);
#pragma unroll 1
            for (int l = 0; l <= nL; ++l)
              scale4(cells + (3 + nL + l) * CN + r * cw + c4);
          }
        }
      }
      __syncthreads();
    }
  }
  cp_async_wait_all();   // never leave with copies into shared memory in flight
  __syncthreads();
  if (bad) atomicOr(P.status, STATUS_NONFINITE);
  if (s_abort) {
    if (tid == 0) atomicOr(P.status, STATUS_STALLED);
    return;
  }
  if (w.n_steps > 0) {
    if (VISCO && (w.flags & WAVE_STAB) && cta == 0 && tid == 0) {
      w.stab->ref_amp = ref_amp;
      w.stab->clipped += clipped;
      *P.peak = last_peak;
    }
  }
}

// Launch k_wave for an engine: `grid` CTAs (at most one per SM), `smem` bytes
// of dynamic shared memory (wave.cu).
cudaError_t wave_launch(int engine, int cells, const WaveSet& S, int grid, int smem, int smem_max, cudaStream_t st);

}  // namespace ertm
