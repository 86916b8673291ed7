// Neighbour loops of the per-particle passes.
//
// One thread per cell-sorted slot (several in small scenes).  Only ~15 % of a particle's 27-cell grid
// candidates (the reference's hash_grid_query set) lie inside the support,
// and every pass of a substep after the first reuses the same grid.  The
// first pass over a grid therefore scans the candidates (scan_visit) and
// records each particle's in-support ones (plus a skin when positions will
// move) as a list in the reference's visiting order; later passes iterate
// those ~35-60 entries instead of ~216 candidates, with all lanes of a warp
// busy on pair terms.
#pragma once

#include "fs_internal.cuh"

namespace fs {

// Neighbour kernels are compiled for blocks of up to kNbBlockMax threads;
// the launch size (64, 128 or 256) and the particles per thread come from
// the context's tuning (fs_context_set_tuning, chosen by the autotuner).
constexpr int kNbBlockMax = 256;
#define FS_NB_BOUNDS __launch_bounds__(kNbBlockMax)

// support test margin: FMA-evaluated r^2 may differ from the individually
// rounded r^2 by about one ulp; anything the reference counts (r <= h) passes
constexpr float kSupportMargin = 1.000002f;

// ---------------------------------------------------- fast kernel math --
// Division-free forms; every pair term stays within a few ulp of the
// reference expression (the passes are checked at 1e-5 relative).
struct Cubic {        // cubic spline, support h (solver_wcsph.py:21-51)
  float inv_h, k, g_in, g_out;  // g_in = 6 k / h^2, g_out = -6 k / h
  FS_DEV explicit Cubic(float h) {
    inv_h = 1.0f / h;
    k = 8.0f / (kPi * (h * h * h));
    g_in = 6.0f * k * inv_h * inv_h;
    g_out = -6.0f * k * inv_h;
  }
  FS_DEV float w_of_q(float q) const {
    if (q > 1.f) return 0.f;
    if (q <= 0.5f) return k * fmaf(6.f * q, q * q, fmaf(-6.f, q * q, 1.f));
    const float t = 1.f - q;
    return 2.f * k * (t * t * t);
  }
  FS_DEV float w(float r) const { return w_of_q(r * inv_h); }
  // grad W(d) = s * d for |d| = r; rinv = 1 / r
  FS_DEV float grad_scale(float r, float rinv) const {
    const float q = r * inv_h;
    if (!(r > 1.0e-5f) || q > 1.f) return 0.f;
    if (q <= 0.5f) return g_in * fmaf(3.f, q, -2.f);
    const float t = 1.f - q;
    return g_out * t * t * rinv;
  }
};

struct Poly6Spiky {   // PBF kernels (solver_pbf.py:24-45)
  float h, h2, kw, kg;
  FS_DEV explicit Poly6Spiky(float h_) : h(h_), h2(h_ * h_) {
    const float c = h_ * h_ * h_;
    kw = 315.0f / (64.0f * kPi * (c * c * c));
    kg = -45.0f / (kPi * (c * c));
  }
  FS_DEV float w_r2(float r2) const {  // poly6 from r^2
    if (!(r2 < h2)) return 0.f;
    const float d = h2 - r2;
    return kw * (d * d * d);
  }
  FS_DEV float grad_scale(float r, float rinv) const {  // spiky
    if (!(r > 1.0e-6f) || !(r < h)) return 0.f;
    const float d = h - r;
    return kg * d * d * rinv;
  }
};

// r and 1/r from r^2 (r2 == 0 gives r = 0, 1/r = 0)
FS_DEV void r_and_inv(float r2, float& r, float& rinv) {
  rinv = r2 > 0.f ? rsqrtf(r2) : 0.f;
  r = r2 * rinv;
}

// `r < h` with r = sqrt(r^2) rounded as in a strict FP32 evaluation, from
// an r^2 the caller already has (any rounding within a few ulp, e.g. FMA
// contracted): only the few pairs within 2e-6 of the support boundary
// recompute r^2 with individually rounded operations and take the exact
// square root.
FS_DEV bool exact_lt_h(float r2_any, float dx, float dy, float dz, float h, float h2) {
  if (r2_any < h2 * 0.999998f) return true;
  if (r2_any > h2 * 1.000002f) return false;
  return sqrtf(dist2_rn(dx, dy, dz)) < h;
}


// ======================================================= neighbour lists ==
// The first pass over a set of positions scans the grid and records, per
// particle, its candidates within the support (in the reference's visiting
// order); the following passes at the same positions iterate those entries.
//   idx[k * stride + s]  k-th entry (cell-sorted slot) of slot s  -- a warp
//                        reads one row k with consecutive addresses
//   cnt[s]               entries of s; kNbMax + 1 marks an overflow (s rescans)
// A list is exact for a later pass at unchanged positions: the grid, the
// positions and hence the candidate set and every distance are the ones
// recorded.  Each new grid build invalidates the lists (ListCtl.valid).
// 192 entries: about 5x the ~35 neighbours of fluid at rest.  DFSPH's
// iteration caps let the dam break compress well past that where the column
// hits the wall (0.2 % of the particles above 96 entries after 300 substeps,
// 1.1 % after 500), and each overflowing particle rescans the grid in every
// pass at those positions, its whole warp with it.
constexpr int kNbMax = 192;

// The mass that the pair terms read for each neighbour.  Particles of one
// fluid mostly share one: the gather notes whether they do (ListCtl), and then
// no pair loads it.  The list passes are held by the L1's data cycles (a
// gather of 16 bytes takes a warp about 12, of 4 bytes 4), so that a load
// saved counts: with the records of a pass (the position and one value) the
// gathers of a pair went from 32 to 24 bytes in the DFSPH rate, from 24 to 16
// in its correction and PBF's delta, 40 to 32 in PBF's non-pressure pass.
// B200, 401,856 particles, us a launch: rate 71 -> 65, correction 50 -> 46,
// delta 51 -> 46, non-pressure 85 -> 73, lambda 115 -> 110.  (Not so the WCSPH
// force, 40 -> 32 bytes: 1 % for what its density pass then writes.)  With
// several lanes per particle the latency of the note itself would count: the
// mass is always loaded.
template <int G>
struct Masses {
  const float* p;
  float first = 0.f;
  bool mixed = true;
  FS_DEV Masses(const float* p_, const ListCtl* ctl) : p(p_) {
    if (G > 1) return;
    mixed = ctl->mixed_mass != 0;
    // no thread index orders this load behind grid_begin(): it stays where it is written
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(first) : "l"(p_) : "memory");
  }
  FS_DEV float operator()(int t) const { return mixed ? __ldg(p + t) : first; }
};

// The coordinates of the cell-order particles for the grid scans: groups of
// four slots, x[4], y[4], z[4] (48 bytes, 16-byte aligned); an inactive
// particle lies outside any support (kScanInactive).
struct ScanXyz {
  const float* g;
};

struct NbrList {
  int32_t* idx;
  int32_t* cnt;
  int64_t stride;
  ListCtl* ctl;
};

// ------------------------------------------------------------ grid scan --
// A scan tests ~216 candidates per particle for ~35 hits, so it is bound by
// the instructions and the L1 data cycles (128 bytes a cycle and SM, with
// 16-byte records 4 cycles per warp and candidate) of one candidate.  It
// therefore reads a separate copy of the cell-order coordinates (ScanXyz:
// 12 bytes a candidate, three 16-byte loads for four), forms r^2 - h2 for two candidates at a time with packed f32x2 operations,
// and shifts the sign bits into one 32-bit word: 5-6 instructions a candidate
// where a test with a predicated store and a counter took about 14.  The
// non-empty words of a particle (9-12) wait in shared memory; its hits are
// then taken from them in visiting order, so every lane of a warp does pair
// math in every step, and the list entries of step k leave the warp as one
// coalesced row (a store at each hit cost one 32-byte sector a hit).
// B200, against the recorder that tested and stored candidate by candidate:
// WCSPH density at 4,194,304 particles 1.63 -> 1.00 ms, DFSPH density + factor
// at 401,856 0.158 -> 0.121, PBF density 0.140 -> 0.106, lambda (mean of one
// reusing and three scanning launches) 0.136 -> 0.114.  What bounds it now:
// the L1's data cycles and the latency of its misses (a third of the time is
// the word loop at about 55 % of the L1's data rate with 28 resident warps).
// 10 or 16 words instead of 12: density +2 %.
constexpr int kWords = 12;                 // words per thread between two visits
constexpr float kScanSlack = 1.000004f;    // the scan takes a few more (never fewer) than the visit's test

using f32x2 = unsigned long long;
FS_DEV f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
FS_DEV f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
FS_DEV f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Where a particle's scan stands: the next row (z, y), segment j of the row,
// and the next candidate t of that segment (negative: its first).
struct ScanPos {
  int z, y, j, t;
};

// Writes the slot ranges of the query of slot s, in visiting order
// (for_each_range's ranges) and cut into pieces of at most 32 candidates
// (counted from the 16-byte group that holds the first), to words[k * nthr]
// as (first, end), from pos on until CAP pieces are written or the query
// is exhausted (live = false); returns their number.  COUNT adds the
// candidates other than s (no distance test, inactive ones too) to ncand.
template <bool COUNT, int CAP>
FS_DEV int scan_pieces(const GridDev& g, int s, float4 xi, float h, uint2* words, int nthr, ScanPos& pos, bool& live,
                       int& ncand) {
  const WorldDev* W = g.worlds ? g.worlds + world_index(world_of(xi), g.nworlds) : nullptr;
  const QueryBox b = W ? query_box_world(g, *W, xi.x, xi.y, xi.z, h) : query_box_hash(g, xi.x, xi.y, xi.z, h);
  const int nx = b.x1 - b.x0 + 1;
  int c0 = b.x0, len1 = nx, nseg = 1;
  bool slow = false;  // far outside the shifted range: cells clamp, one segment per cell
  if (!W) {
    const int xa = b.x0 + (1 << 20);
    slow = xa < 0;
    c0 = slow ? 0 : (g.mask_x >= 0 ? (xa & g.mask_x) : xa % g.dim_x);
    len1 = min(nx, g.dim_x - c0);
    nseg = slow ? nx : (nx > len1 ? 2 : 1);  // a run that wraps modulo dim_x splits in two
  }
  int nw = 0;
  auto count = [&](int a, int e) { ncand += (e - a) - ((s >= a && s < e) ? 1 : 0); };
  const int ny = b.y1 - b.y0 + 1, nz = b.z1 - b.z0 + 1;
  if (pos.z == INT32_MIN) {
    pos.z = b.z0, pos.y = b.y0;
    // The usual query: up to 3 x 3 rows of one segment each, in a world's box
    // or a hash grid of power-of-two dims.  All their offsets load at once
    // (one row at a time spent a latency a row and a fifth of the scan).
    const bool plain = W ? true : (g.mask_y | g.mask_z) >= 0 && nseg == 1 && !slow && min(b.y0, b.z0) >= -(1 << 20);
    if (plain && nx > 0 && ny <= 3 && nz <= 3) {
      const int shift = W ? 0 : 1 << 20;
      const int my = W ? INT32_MAX : g.mask_y, mz = W ? INT32_MAX : g.mask_z;
      const int sy = W ? W->dims[0] : g.dim_x, sz = sy * (W ? W->dims[1] : g.dim_y);
      const int32_t* const o = g.off + c0 + (W ? W->base : 0);
      int a[9], e[9];
#pragma unroll
      for (int z = 0; z < 3; ++z)
#pragma unroll
        for (int y = 0; y < 3; ++y) {
          const int row = ((b.z0 + z + shift) & mz) * sz + ((b.y0 + y + shift) & my) * sy;
          const bool in = z < nz && y < ny;
          a[z * 3 + y] = in ? __ldg(o + row) : 0;
          e[z * 3 + y] = in ? __ldg(o + row + nx) : 0;
        }
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        if (COUNT) count(a[k], e[k]);
        for (int f = a[k]; f < e[k];) {
          const int stop = min(e[k], (f & ~3) + 32);
          if (nw == CAP) {
            pos.z = b.z0 + k / 3, pos.y = b.y0 + k % 3, pos.t = f;
            return nw;
          }
          words[nw * nthr] = make_uint2((uint32_t)f, (uint32_t)stop);
          ++nw;
          f = stop;
        }
      }
      live = false;
      return nw;
    }
  }
  if (nx <= 0 || b.y0 > b.y1) pos.z = b.z1 + 1;
  auto load = [&](int z, int y, int j, int& a, int& e) {
    const int row = W ? W->base + (z * W->dims[1] + y) * W->dims[0]
                      : (wrap_axis(z, g.dim_z, g.mask_z) * g.dim_y + wrap_axis(y, g.dim_y, g.mask_y)) * g.dim_x;
    int first = c0, len = len1;
    if (j) first = 0, len = nx - len1;
    if (slow) first = wrap_axis(b.x0 + j, g.dim_x, g.mask_x), len = 1;
    a = __ldg(g.off + row + first);
    e = __ldg(g.off + row + first + len);
  };
  int a = 0, e = 0;
  if (pos.z <= b.z1) load(pos.z, pos.y, pos.j, a, e);
  while (pos.z <= b.z1) {
    // the next range's offsets load while this one is cut
    int z = pos.z, y = pos.y, j = pos.j + 1, an = 0, en = 0;
    if (j == nseg) {
      j = 0;
      if (++y > b.y1) y = b.y0, ++z;
    }
    if (z <= b.z1) load(z, y, j, an, en);
    int f = pos.t;
    if (f < 0) {
      f = a;
      if (COUNT) count(a, e);
    }
    while (f < e) {
      if (nw == CAP) {
        pos.t = f;
        return nw;
      }
      const int stop = min(e, (f & ~3) + 32);
      words[nw * nthr] = make_uint2((uint32_t)f, (uint32_t)stop);
      ++nw;
      f = stop;
    }
    pos = ScanPos{z, y, j, -1};
    a = an, e = en;
  }
  live = false;
  return nw;
}

// A particle's position and squared radius (negative), doubled for the packed
// operations of the scan.
struct ScanQuery {
  f32x2 nx, ny, nz, nh;
  FS_DEV ScanQuery(float4 xi, float h2)
      : nx(pack2(-xi.x, -xi.x)), ny(pack2(-xi.y, -xi.y)), nz(pack2(-xi.z, -xi.z)), nh(pack2(-h2, -h2)) {}
};

// The hit word of the piece [first, end), not empty, at most 32 slots from the
// group of four that holds the first: bit b set = slot last - b is within.
// INACTIVE: ninactive is the number of inactive particles in the piece, three
// more operations a candidate (DFSPH's density pass, whose candidates are
// counted; with their flags read one by one it took 152 us at 401,856
// particles, one of them inactive, for 107 with none; now 109, at 10 % 153 -> 107).
template <bool INACTIVE = false>
FS_DEV uint32_t scan_word(const ScanXyz& q, const ScanQuery& o, uint32_t first, uint32_t end, uint32_t& last,
                          int* ninactive = nullptr) {
  const uint32_t g0 = first >> 2, g1 = (end + 3) >> 2;
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(q.g) + (size_t)g0 * 3;
  uint32_t m = 0, far = 0;
#pragma unroll 2  // two groups of loads in flight (density time with 1: +1 to 3 %, with 4: up to +7 %)
  for (uint32_t i = g0; i < g1; ++i, p += 3) {
    const ulonglong2 x2 = __ldg(p), y2 = __ldg(p + 1), z2 = __ldg(p + 2);
    const f32x2 dx0 = add2(x2.x, o.nx), dx1 = add2(x2.y, o.nx);
    const f32x2 dy0 = add2(y2.x, o.ny), dy1 = add2(y2.y, o.ny);
    const f32x2 dz0 = add2(z2.x, o.nz), dz1 = add2(z2.y, o.nz);
    const f32x2 r0 = fma2(dx0, dx0, fma2(dy0, dy0, fma2(dz0, dz0, o.nh)));
    const f32x2 r1 = fma2(dx1, dx1, fma2(dy1, dy1, fma2(dz1, dz1, o.nh)));
    m = __funnelshift_l((uint32_t)r0, m, 1);  // the sign bit of r^2 - h2: set = within
    m = __funnelshift_l((uint32_t)(r0 >> 32), m, 1);
    m = __funnelshift_l((uint32_t)r1, m, 1);
    m = __funnelshift_l((uint32_t)(r1 >> 32), m, 1);
    if (INACTIVE) {
      // x = +inf (kScanInactive, no active particle's): the sum's sign bit is
      // set for it and for negative x
      auto mark = [&](uint32_t x) { far = __funnelshift_l((x + 0x00800000u) & ~x, far, 1); };
      mark((uint32_t)x2.x), mark((uint32_t)(x2.x >> 32)), mark((uint32_t)x2.y), mark((uint32_t)(x2.y >> 32));
    }
  }
  // without the slots of the groups outside the piece: before its first, after its last
  const uint32_t in = (0xffffffffu >> (32 - 4 * (g1 - g0) + (first & 3))) & (0xffffffffu << (4 * g1 - end));
  if (INACTIVE) *ninactive = __popc(far & in);
  last = 4 * g1 - 1;
  return m & in;
}

// Replaces the pieces in `words` by their non-empty hit words (mask, last);
// INACTIVE takes the inactive candidates from ncand.
template <bool INACTIVE>
FS_DEV int scan_words(const ScanXyz& q, float4 xi, float h2, uint2* words, int nthr, int np, int& ncand) {
  const ScanQuery o(xi, h2);
  int nw = 0;
  for (int k = 0; k < np; ++k) {
    const uint2 piece = words[k * nthr];
    uint32_t last;
    int ninactive = 0;
    const uint32_t m = scan_word<INACTIVE>(q, o, piece.x, piece.y, last, &ninactive);
    if (INACTIVE) ncand -= ninactive;
    if (m) {
      words[nw * nthr] = make_uint2(m, last);
      ++nw;
    }
  }
  return nw;
}

// Records the list of slot s (candidates within the radius whose square is
// h2rec, in visiting order; LIST says which) and calls pair(t, xj, payload) for
// those that pass visit_with's test at h2m, in the same order; load(t) is
// issued together with the position gather.  Returns the DFSPH candidate
// count when COUNT.  More than kNbMax entries mark the list overflowed; the
// pairs are still all visited here.  REUSE: a particle with reuse >= 0 visits
// the `reuse` entries its list already holds instead of scanning (in the same
// loop: lanes that scan and lanes that reuse share the warp's pair math).
// LIST: what the list holds beside the pairs within h2rec.  kAll: the particle
// itself too, and the few candidates that the scan takes past the radius;
// kOthers: not itself; kExact: neither, only what passes the test at h2m, so
// that its readers gather nothing in vain and test nothing again.  Which is
// best depends on the readers, since the stores of kExact wait for the
// positions (at 401,856 particles and, WCSPH, 4M):
//                       kAll              kOthers           kExact
//   DFSPH density       118.2 us          117.8             118.2
//     17 rate, correct  64.8, 43.6        63.2, 42.6        60.4, 41.5
//   WCSPH density       999 us            1015              1024
//     force             708               695               669
//   PBF lambda          109.9 us          109.1             113.5
//     delta             44.0              42.4              39.4
// The PBF density's list is visited again with the particle itself: kAll.
// The bound on a list counts the particle in any case.
enum ListOf { kAll, kOthers, kExact };

template <bool WITH_SELF, bool COUNT, bool REUSE, ListOf LIST, class Load, class Pair>
FS_DEV int scan_visit(const GridDev& g, const ScanXyz& q, const float4* __restrict__ xs, int s, float4 xi, float h,
                      float h2rec, float h2m, const NbrList& L, uint2* smem, Load&& load, Pair&& pair,
                      int reuse = -1) {
  const int nthr = blockDim.x;
  uint2* const words = smem + threadIdx.x;
  const bool inactive = COUNT && L.ctl->inactive;
  ScanPos pos{INT32_MIN, 0, 0, -1};
  bool live = true;
  int n = 0, ncand = 0;
  int32_t* const col = L.idx + s;
  auto within = [&](float4 xj) {
    const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    return fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, xj.w))) <= h2m;
  };
  auto one = [&](int t, float4 xj, const auto& p) {
    if (within(xj) && (WITH_SELF || t != s)) pair(t, xj, p);
  };
  static_assert(!REUSE || LIST != kExact, "a list that is visited again holds more");
  const bool scan = !REUSE || reuse < 0;
  while (live) {
    int nw = 0;
    if (scan) {
      const int np = scan_pieces<COUNT, kWords>(g, s, xi, h, words, nthr, pos, live, ncand);
      nw = COUNT && inactive ? scan_words<COUNT>(q, xi, h2rec * kScanSlack, words, nthr, np, ncand)
                             : scan_words<false>(q, xi, h2rec * kScanSlack, words, nthr, np, ncand);
    } else {
      live = false;
    }
    int w = 0;
    uint32_t m = 0, last = 0;
    auto pop = [&](bool& ok) {
      if (!m && w < nw) {
        const uint2 v = words[w * nthr];
        m = v.x, last = v.y;
        ++w;
      }
      ok = m != 0;
      const uint32_t hi = 31 - __clz(m);  // ok: the first slot of the word that is left
      m &= ~(1u << (hi & 31));
      return ok ? (int)(last - hi) : s;
    };
    while (scan ? (m || w < nw) : n < reuse) {
      bool k0, k1, k2, k3;
      int t0, t1, t2, t3;
      if (scan) {
        t0 = pop(k0), t1 = pop(k1), t2 = pop(k2), t3 = pop(k3);
      } else {
        const int32_t* const o = col + (int64_t)n * L.stride;
        k0 = true, k1 = n + 1 < reuse, k2 = n + 2 < reuse, k3 = n + 3 < reuse;
        t0 = o[0];
        t1 = k1 ? o[L.stride] : s;
        t2 = k2 ? o[2 * L.stride] : s;
        t3 = k3 ? o[3 * L.stride] : s;
      }
      const float4 x0 = __ldg(xs + t0), x1 = __ldg(xs + t1), x2 = __ldg(xs + t2), x3 = __ldg(xs + t3);
      const auto p0 = load(t0), p1 = load(t1), p2 = load(t2), p3 = load(t3);
      if constexpr (LIST == kExact) {
        k0 = within(x0), k1 = k1 && within(x1), k2 = k2 && within(x2), k3 = k3 && within(x3);
        const int tt[4] = {t0, t1, t2, t3};
        const bool rr[4] = {k0 && t0 != s, k1 && t1 != s, k2 && t2 != s, k3 && t3 != s};
        int32_t* o = col + (int64_t)n * L.stride;
        if (n + 4 <= kNbMax) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (rr[e]) *o = tt[e], o += L.stride;
          n += (int)rr[0] + (int)rr[1] + (int)rr[2] + (int)rr[3];
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (rr[e]) {
              if (n < kNbMax) col[(int64_t)n * L.stride] = tt[e];
              ++n;
            }
        }
        if (k0 && (WITH_SELF || t0 != s)) pair(t0, x0, p0);
        if (k1 && (WITH_SELF || t1 != s)) pair(t1, x1, p1);
        if (k2 && (WITH_SELF || t2 != s)) pair(t2, x2, p2);
        if (k3 && (WITH_SELF || t3 != s)) pair(t3, x3, p3);
      } else {
        if (LIST == kOthers && scan) {
          const bool r0 = t0 != s, r1 = t1 != s, r2 = t2 != s, r3 = t3 != s;  // a slot that was not popped is s
          int32_t* o = col + (int64_t)n * L.stride;
          if (n + 4 <= kNbMax) {
            *o = t0;
            if (r0) o += L.stride;
            if (r1) *o = t1, o += L.stride;
            if (r2) *o = t2, o += L.stride;
            if (r3) *o = t3;
            n += (int)r0 + (int)r1 + (int)r2 + (int)r3;
          } else {
            const int tt[4] = {t0, t1, t2, t3};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (tt[e] != s) {
                if (n < kNbMax) col[(int64_t)n * L.stride] = tt[e];
                ++n;
              }
          }
        } else if (!scan) {
        } else if (n + 4 <= kNbMax) {
          int32_t* const o = col + (int64_t)n * L.stride;
          o[0] = t0;
          if (k1) o[L.stride] = t1;
          if (k2) o[2 * L.stride] = t2;
          if (k3) o[3 * L.stride] = t3;
        } else {
          const int tt[4] = {t0, t1, t2, t3};
          const bool kk[4] = {k0, k1, k2, k3};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (kk[e] && n + e < kNbMax) col[(int64_t)(n + e) * L.stride] = tt[e];
        }
        if (LIST == kAll || !scan) n += (int)k0 + (int)k1 + (int)k2 + (int)k3;
        one(t0, x0, p0);
        if (k1) one(t1, x1, p1);
        if (k2) one(t2, x2, p2);
        if (k3) one(t3, x3, p3);
      }
    }
  }
  if (scan) L.cnt[s] = n + (LIST != kAll) <= kNbMax ? n : kNbMax + 1;
  return ncand;
}

// Grid scan that calls pair(t, xj) directly (no usable list for this particle).
template <bool WITH_SELF, class Pair>
FS_DEV void scan_grid(const GridDev& g, const float4* __restrict__ xs, int s, float4 xi, float h, float h2m,
                      Pair&& pair) {
  for_each_candidate(g, world_of(xi), xi.x, xi.y, xi.z, h, [&](int t) {
    const float4 xj = __ldg(xs + t);
    const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    if (fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, xj.w))) <= h2m && (WITH_SELF || t != s)) pair(t, xj);
  });
}

// The same for lists that overflowed and passes that run by themselves, without
// lists: pair(t, rec[t]), by RESCAN
//   kPositions  scan_grid (the record is the position: rec = xs)
//   kGrid       scan_grid, then the record
//   kRecords    the positions from the records that the pairs gather anyway; a
//               hit's flag is read only where some particle is inactive
//   kAhead      and the next record loads while one is tested
// DFSPH substep with lists that all overflow (four spacings to the support,
// about 250 neighbours), in ms at 61,740 and 401,856 particles: kGrid 15.9,
// 34.3; kRecords 14.4, 31.1; kAhead 13.2, 33.2; kAhead but in the correction,
// which is short of registers there, 13.4, 31.0.  Passes by themselves at 401,856:
// PBF's delta 221 us with kGrid, 178 with kAhead, DFSPH's correction 200, 175.
// kPositions and kGrid where the others cost the path with lists: WCSPH's force
// 1 %, PBF's passes 0.4 % of a substep of 100,003 particles, several lanes per
// particle 0.4 % at 4,079.
enum Rescan { kPositions, kGrid, kRecords, kAhead };

template <bool WITH_SELF, Rescan RESCAN, class Pair>
FS_DEV void rescan(const GridDev& g, const float4* __restrict__ xs, const float4* __restrict__ rec, int s, float4 xi,
                   float h, float h2m, const NbrList& L, Pair&& pair) {
  if constexpr (RESCAN == kPositions) {
    scan_grid<WITH_SELF>(g, xs, s, xi, h, h2m, pair);
  } else if constexpr (RESCAN == kGrid) {
    scan_grid<WITH_SELF>(g, xs, s, xi, h, h2m, [&](int t, float4) { pair(t, __ldg(rec + t)); });
  } else {
    const bool inactive = L.ctl->inactive != 0;
    for_each_range(g, world_of(xi), xi.x, xi.y, xi.z, h, [&](int a, int e) {
      if (a >= e) return;
      float4 next = __ldg(rec + a);
      for (int t = a; t < e; ++t) {
        const float4 xj = RESCAN == kAhead ? next : __ldg(rec + t);
        if (RESCAN == kAhead && t + 1 < e) next = __ldg(rec + t + 1);
        const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= h2m && (WITH_SELF || t != s) &&
            (!inactive || (pf_of(__ldg(xs + t)) & PF_ACTIVE)))
          pair(t, xj);
      }
    });
  }
}

// One entry of a list, past L1, which the neighbours' data fill (the lists
// stay in L2): DFSPH rate 63.1 -> 62.2 us, correct 42.7 -> 42.1 at 401,856
// particles.
FS_DEV int32_t ld_list(const int32_t* p) {
  int32_t v;
  asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Visits the neighbours of slot s within h2m through its recorded list when
// lists_ok and the list did not overflow, else by rescanning the grid.
// rec: the record gathered with each neighbour, its position and one value
// (xs itself, or a pass's own); pair(t, rec[t]).  EXACT: a kExact list, whose
// entries need no test (with one: rate 62.2 instead of 60.4 us, WCSPH force
// 695 instead of 669).
template <bool WITH_SELF, bool EXACT, Rescan RESCAN, class Pair>
FS_DEV void visit(const GridDev& g, const float4* __restrict__ xs, const float4* __restrict__ rec, int s, float4 xi,
                  float h, float h2m, const NbrList& L, bool lists_ok, Pair&& pair) {
  const int n = lists_ok ? __ldg(L.cnt + s) : kNbMax + 1;
  const bool use = n <= kNbMax;
  if (use) {
    const int32_t* col = L.idx + s;
    auto entry = [&](int k) { return __ldg(col + (int64_t)k * L.stride); };
    auto one = [&](int t, float4 xj) {
      const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
      if (EXACT || (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= h2m && (WITH_SELF || t != s))) pair(t, xj);
    };
    int k = 0;
    for (; k + 3 < n; k += 4) {  // four independent gathers in flight
      const int t0 = entry(k), t1 = entry(k + 1), t2 = entry(k + 2), t3 = entry(k + 3);
      const float4 x0 = __ldg(rec + t0), x1 = __ldg(rec + t1), x2 = __ldg(rec + t2), x3 = __ldg(rec + t3);
      one(t0, x0);
      one(t1, x1);
      one(t2, x2);
      one(t3, x3);
    }
    // the last one to three together: one after the other each waited a latency
    // (DFSPH rate 66.1 -> 64.8 us, PBF delta 45.8 -> 44.0 at 401,856 particles,
    // WCSPH force 719 -> 708 at 4M)
    if (k < n) {
      const bool k1 = k + 1 < n, k2 = k + 2 < n;
      const int t0 = entry(k), t1 = k1 ? entry(k + 1) : s, t2 = k2 ? entry(k + 2) : s;
      const float4 x0 = __ldg(rec + t0), x1 = __ldg(rec + t1), x2 = __ldg(rec + t2);
      one(t0, x0);
      if (k1) one(t1, x1);
      if (k2) one(t2, x2);
    }
  } else {
    rescan<WITH_SELF, RESCAN>(g, xs, rec, s, xi, h, h2m, L, pair);
  }
}

// visit() for pair terms that read a second per-neighbour record (velocity,
// kappa ratio, lambda ...): load(t) is issued together with the position
// gather of each group of four list entries, so the two gathers of a
// neighbour overlap instead of the second waiting for the distance test.
// pair(t, xj, payload) is called in the same order and for the same entries
// as visit() calls pair(t, xj).  Only for lists recorded at the current
// positions (every entry within h2m except the particle itself), where the
// early load fetches nothing that visit() would not.
// EVICT_FIRST: entries are loaded evict-first (ld.global.cs), leaving the
// caches to the neighbours' data.  Measured faster for the PBF passes whose
// lists at most one later pass reads again (delta, non-pressure, XSPH:
// 1.304 -> 1.287 ms per substep at 401,856 particles); the DFSPH iteration
// passes, which read the same lists 34 times a substep, were slower with it.
template <bool WITH_SELF, bool EVICT_FIRST, bool EXACT, Rescan RESCAN, class Load, class Pair>
FS_DEV void visit_with(const GridDev& g, const float4* __restrict__ xs, const float4* __restrict__ rec, int s,
                       float4 xi, float h, float h2m, const NbrList& L, bool lists_ok, Load&& load, Pair&& pair) {
  const int n = lists_ok ? __ldg(L.cnt + s) : kNbMax + 1;
  const bool use = n <= kNbMax;
  auto one = [&](int t, float4 xj, const auto& p) {
    const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    if (EXACT || (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= h2m && (WITH_SELF || t != s))) pair(t, xj, p);
  };
  if (use) {
    const int32_t* col = L.idx + s;
    auto entry = [&](int k) {
      return EVICT_FIRST ? __ldcs(col + (int64_t)k * L.stride) : ld_list(col + (int64_t)k * L.stride);
    };
    int k = 0;
    for (; k + 3 < n; k += 4) {
      const int t0 = entry(k), t1 = entry(k + 1), t2 = entry(k + 2), t3 = entry(k + 3);
      const float4 x0 = __ldg(rec + t0), x1 = __ldg(rec + t1), x2 = __ldg(rec + t2), x3 = __ldg(rec + t3);
      const auto p0 = load(t0), p1 = load(t1), p2 = load(t2), p3 = load(t3);
      one(t0, x0, p0);
      one(t1, x1, p1);
      one(t2, x2, p2);
      one(t3, x3, p3);
    }
    if (k < n) {
      const bool k1 = k + 1 < n, k2 = k + 2 < n;
      const int t0 = entry(k), t1 = k1 ? entry(k + 1) : s, t2 = k2 ? entry(k + 2) : s;
      const float4 x0 = __ldg(rec + t0), x1 = __ldg(rec + t1), x2 = __ldg(rec + t2);
      const auto p0 = load(t0), p1 = load(t1), p2 = load(t2);
      one(t0, x0, p0);
      if (k1) one(t1, x1, p1);
      if (k2) one(t2, x2, p2);
    }
  } else {
    rescan<WITH_SELF, RESCAN>(g, xs, rec, s, xi, h, h2m, L, [&](int t, float4 xj) { pair(t, xj, load(t)); });
  }
}

// ------------------------------------------------------ lanes in a group --
// A small scene leaves most of the GPU idle with one thread per particle, and
// each thread then walks its candidates and neighbours alone, one memory
// latency after the other: at 4,079 particles a lambda pass took 28 us with
// 128 warps for 148 SMs.  G lanes (4, 8 or 16) share a
// particle instead: each scans every G-th group of four candidates, the hits
// are compacted in visiting order, each lane evaluates every G-th pair term,
// and the terms are then added up in visiting order by broadcasting them one
// after the other, so every sum has the bits of the one-thread form (a lane
// without a term broadcasts zeros, which change no sum).  What bounds a pass
// at these sizes is the chain of dependent steps of one warp (load, scan,
// compact, gather, add up).  nb_group() holds the rule for G.
//
// With G > 1 a particle's list is a row (entry k of slot s at
// idx[s * kNbMax + k], read by its lanes side by side) instead of a column.
// Every kernel of a context and particle count takes the same G.
constexpr int kGroupList = 128;  // hits of a particle held in shared memory between two visits

constexpr int kGroupRows = 9;    // rows of a usual query, each scanned by one lane

// Shared memory of a recording launch: one thread per particle keeps kWords
// words at stride `threads`, a group kGroupRows pieces and kGroupList hits.
inline size_t scan_smem(int threads, int group) {
  return group == 1 ? sizeof(uint2) * kWords * threads
                    : (sizeof(uint2) * kGroupRows + sizeof(int32_t) * kGroupList) * (threads / group);
}

// K floats a pair contributes; the zero value changes no sum.  K = 0: the
// term adds itself to its lane's own sums, which the caller adds up
// afterwards (sums without a prescribed order).
template <int K>
struct Terms {
  float v[K] = {};
};
template <>
struct Terms<0> {};

template <int G, int K>
FS_DEV Terms<K> group_bcast(const Terms<K>& u, int j) {
  Terms<K> o;
#pragma unroll
  for (int k = 0; k < K; ++k) o.v[k] = __shfl_sync(0xffffffffu, u.v[k], j, G);
  return o;
}

template <int G, class V>
FS_DEV V group_sum(V v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, G);
  return v;
}

// acc(term) in order for the n entries of the group's particle (n is the same
// in all its lanes; 0: nothing), entry(k) being the k-th slot.  All lanes of
// the warp call it together.
template <int G, bool WITH_SELF, int K, class Entry, class Load, class Term, class Acc>
FS_DEV void group_visit(const float4* __restrict__ rec, int s, float4 xi, float h2m, int n, Entry&& entry, Load&& load,
                        Term&& term, Acc&& acc) {
  const int lane = threadIdx.x & (G - 1);
  const int nmax = __reduce_max_sync(0xffffffffu, n);
  // the gathers of the next round are issued before this round's sums
  int t = lane < n ? entry(lane) : s;
  float4 xj = __ldg(rec + t);
  auto p = load(t);
  for (int k0 = 0; k0 < nmax; k0 += G) {
    const bool mine = k0 + lane < n;
    const int t0 = t;
    const float4 x0 = xj;
    const auto p0 = p;
    if (k0 + G + lane < n) {
      t = entry(k0 + G + lane);
      xj = __ldg(rec + t);
      p = load(t);
    }
    Terms<K> u;
    if (mine) {
      const float dx = xi.x - x0.x, dy = xi.y - x0.y, dz = xi.z - x0.z;
      if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= h2m && (WITH_SELF || t0 != s)) u = term(t0, x0, p0);
    }
    if constexpr (K > 0) {
      const int lim = min(G, nmax - k0);
      for (int j = 0; j < lim; j += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) acc(group_bcast<G>(u, j + i));
      }
    }
  }
}

// The rows of a usual query (up to 3 x 3 rows of one slot range each, at most
// two pieces a row): lane l of the group gets rows l, l + G, ... as [f, e),
// empty where there is none.  False where the query is none of the usual ones;
// f and e are then not to be used.
template <int G, int N>
FS_DEV bool group_rows(const GridDev& g, float4 xi, float h, int (&f)[N], int (&e)[N]) {
  const WorldDev* W = g.worlds ? g.worlds + world_index(world_of(xi), g.nworlds) : nullptr;
  const QueryBox b = W ? query_box_world(g, *W, xi.x, xi.y, xi.z, h) : query_box_hash(g, xi.x, xi.y, xi.z, h);
  const int nx = b.x1 - b.x0 + 1, ny = b.y1 - b.y0 + 1, nz = b.z1 - b.z0 + 1;
  int c0 = b.x0;
  bool plain = nx > 0 && ny <= 3 && nz <= 3;
  if (!W) {
    const int xa = b.x0 + (1 << 20);
    c0 = g.mask_x >= 0 ? (xa & g.mask_x) : xa % g.dim_x;
    plain = plain && xa >= 0 && c0 + nx <= g.dim_x && min(b.y0, b.z0) >= -(1 << 20);
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int r = (int)(threadIdx.x & (G - 1)) + k * G, z = (r * 11) >> 5, y = r - 3 * z;
    f[k] = e[k] = 0;
    if (plain && r < kGroupRows && z < nz && y < ny) {
      const int row = W ? W->base + ((b.z0 + z) * W->dims[1] + b.y0 + y) * W->dims[0]
                        : (wrap_axis(b.z0 + z, g.dim_z, g.mask_z) * g.dim_y + wrap_axis(b.y0 + y, g.dim_y, g.mask_y)) *
                              g.dim_x;
      f[k] = __ldg(g.off + row + c0);
      e[k] = __ldg(g.off + row + c0 + nx);
    }
  }
#pragma unroll
  for (int k = 0; k < N; ++k) plain = plain && e[k] - (f[k] & ~3) <= 64;
  return plain;
}

// scan_visit by the G lanes of a group (`on` and `reuse` are the same in all
// of them; `on` = false: the particle takes no part).  All lanes of the warp
// call it together.  Each lane scans whole rows (other queries: pieces cut by
// scan_pieces), the hits get their places in visiting order from a scan of
// the lanes' counts, and group_visit takes them from shared memory.
template <int G, bool WITH_SELF, bool COUNT, bool REUSE, int K, class Load, class Term, class Acc>
FS_DEV int group_scan(const GridDev& g, const ScanXyz& q, const float4* __restrict__ xs, int s, float4 xi, float h,
                      float h2rec, float h2m, const NbrList& L, void* smem, bool on, int reuse, Load&& load,
                      Term&& term, Acc&& acc) {
  constexpr int N = (kGroupRows + G - 1) / G;  // rows per lane
  const int lane = threadIdx.x & (G - 1), grp = threadIdx.x / G;
  uint2* const pieces = (uint2*)smem + grp * kGroupRows;
  int32_t* const list = (int32_t*)((uint2*)smem + (blockDim.x / G) * kGroupRows) + grp * kGroupList;
  int32_t* const row = L.idx + (int64_t)s * kNbMax;
  const bool inactive = COUNT && L.ctl->inactive;
  const ScanQuery o(xi, h2rec * kScanSlack);
  const bool scan = on && (!REUSE || reuse < 0);
  int f[N], e[N];
  const bool usual = group_rows<G>(g, xi, h, f, e);
  // the whole group takes the usual way, or none of it
  const unsigned votes = __ballot_sync(0xffffffffu, usual) >> (threadIdx.x & (32 - G));
  const bool plain = (votes & (unsigned)((1ull << G) - 1)) == (unsigned)((1ull << G) - 1);
  ScanPos pos{INT32_MIN, 0, 0, -1};
  bool live = on;
  int n = 0, ncand = 0;
  while (__any_sync(0xffffffffu, live)) {
    const bool now = live && scan, again = REUSE && live && !scan;  // (other groups of the warp may go on)
    if (now && !plain) {
      int nc = 0;
      const int np = scan_pieces<COUNT, kGroupRows>(g, s, xi, h, pieces, 1, pos, live, nc);
      if (lane == 0) ncand += nc;
      // every lane has written the same pieces
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const bool in = lane + k * G < np;
        f[k] = in ? (int)pieces[lane + k * G].x : 0;
        e[k] = in ? (int)pieces[lane + k * G].y : 0;
      }
    } else {
      live = false;
    }
    static_assert(N <= 3, "hits of the rounds, ten bits each");
    uint32_t w[N][2], last[N][2], cnt = 0;  // hit words; hits of the rounds
#pragma unroll
    for (int k = 0; k < N; ++k) {
      if (COUNT && now && plain) ncand += (e[k] - f[k]) - ((s >= f[k] && s < e[k]) ? 1 : 0);
      const int mid = min(e[k], (f[k] & ~3) + 32);
      w[k][0] = w[k][1] = last[k][0] = last[k][1] = 0;
      auto word = [&](int first, int end, uint32_t& at) {
        if (!(COUNT && inactive)) return scan_word(q, o, first, end, at);
        int ninactive;
        const uint32_t m = scan_word<true>(q, o, first, end, at, &ninactive);
        ncand -= ninactive;
        return m;
      };
      if (now && f[k] < mid) w[k][0] = word(f[k], mid, last[k][0]);
      if (now && mid < e[k]) w[k][1] = word(mid, e[k], last[k][1]);
      cnt |= (uint32_t)(__popc(w[k][0]) + __popc(w[k][1])) << (10 * k);
    }
    // hits before this lane's in each round, and in all lanes (at most 9 rows of 64: ten bits)
    const uint32_t own = cnt;
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, cnt, d, G);
      if (lane >= d) cnt += v;
    }
    const uint32_t tot = __shfl_sync(0xffffffffu, cnt, G - 1, G);
    cnt -= own;
    int nb = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) nb += (int)((tot >> (10 * k)) & 1023);
    if (again) nb = reuse;
    const int nbmax = __reduce_max_sync(0xffffffffu, nb);
    for (int w0 = 0; w0 < nbmax; w0 += kGroupList) {
      if (again) {
        for (int k = lane; k < kGroupList && w0 + k < nb; k += G) list[k] = row[w0 + k];
      } else {
        int base = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) {
          int p = base + (int)((cnt >> (10 * k)) & 1023);
          base += (int)((tot >> (10 * k)) & 1023);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            for (uint32_t m = w[k][u]; m; ++p) {
              const uint32_t hi = 31 - __clz(m);
              m ^= 1u << hi;
              const int t = (int)(last[k][u] - hi);
              if (p >= w0 && p < w0 + kGroupList) {
                list[p - w0] = t;
                if (n + p < kNbMax) row[n + p] = t;
              }
            }
          }
        }
      }
      __syncwarp();
      group_visit<G, WITH_SELF, K>(xs, s, xi, h2m, min(max(nb - w0, 0), kGroupList), [&](int k) { return list[k]; },
                                   load, term, acc);
      __syncwarp();
    }
    n += nb;
  }
  if (scan && lane == 0) L.cnt[s] = n <= kNbMax ? n : kNbMax + 1;
  return COUNT ? group_sum<G>(ncand) : 0;
}

// The two neighbour sums of the passes, for one thread (G = 1) or a group of
// lanes per particle: acc(term(t, xj, load(t))) in visiting order.
//   scan_sum  scans the grid and records the list (scan_visit, group_scan)
//   list_sum  iterates the recorded list (visit, visit_with, group_visit),
//             or rescans where there is none; LAZY: load(t) only after the
//             distance test (G = 1), where the early load costs registers;
//             RESCAN with one thread per particle (several: kGrid)
// A particle with on = false takes no part.
template <int G, bool WITH_SELF, bool COUNT, bool REUSE, ListOf LIST, int K, class Load, class Term, class Acc>
FS_DEV int scan_sum(const GridDev& g, const ScanXyz& q, const float4* __restrict__ xs, int s, float4 xi, float h,
                    float h2rec, float h2m, const NbrList& L, void* smem, bool on, int reuse, Load&& load, Term&& term,
                    Acc&& acc) {
  if constexpr (G == 1) {
    if (!on) return 0;
    return scan_visit<WITH_SELF, COUNT, REUSE, LIST>(
        g, q, xs, s, xi, h, h2rec, h2m, L, (uint2*)smem, load,
        [&](int t, float4 xj, const auto& p) { acc(term(t, xj, p)); }, reuse);
  } else {
    return group_scan<G, WITH_SELF, COUNT, REUSE, K>(g, q, xs, s, xi, h, h2rec, h2m, L, smem, on, reuse, load, term,
                                                     acc);
  }
}

template <int G, bool WITH_SELF, bool EVICT_FIRST, bool LAZY, bool EXACT, int K, Rescan RESCAN, class Load,
          class Term, class Acc>
FS_DEV void list_sum(const GridDev& g, const float4* __restrict__ xs, const float4* __restrict__ rec, int s, float4 xi,
                     float h, float h2m, const NbrList& L, bool lists_ok, bool on, Load&& load, Term&& term,
                     Acc&& acc) {
  if constexpr (G == 1) {
    if (!on) return;
    if constexpr (LAZY)
      visit<WITH_SELF, EXACT, RESCAN>(g, xs, rec, s, xi, h, h2m, L, lists_ok, [&](int t, float4 xj) { acc(term(t, xj, load(t))); });
    else
      visit_with<WITH_SELF, EVICT_FIRST, EXACT, RESCAN>(g, xs, rec, s, xi, h, h2m, L, lists_ok, load,
                                         [&](int t, float4 xj, const auto& p) { acc(term(t, xj, p)); });
  } else {
    const int n = !on ? 0 : (lists_ok ? __ldg(L.cnt + s) : kNbMax + 1);
    const bool over = n > kNbMax;
    const int32_t* const row = L.idx + (int64_t)s * kNbMax;
    group_visit<G, WITH_SELF, K>(rec, s, xi, h2m, over ? 0 : n, [&](int k) { return __ldg(row + k); }, load, term, acc);
    if (over && (K > 0 || (threadIdx.x & (G - 1)) == 0))  // each lane adds up the whole sum (K = 0: the first)
      rescan<WITH_SELF, kGrid>(g, xs, rec, s, xi, h, h2m, L, [&](int t, float4 xj) { acc(term(t, xj, load(t))); });
  }
}

// f(s, live, lead) for the slots of this launch: G = 1 as for_slots; else each
// group of G lanes takes one slot, every lane of the warp calls f (live =
// false past the last slot) and lead marks the lane that writes.
template <int G, class F>
FS_DEV void for_groups(int64_t n, F&& f) {
  if constexpr (G == 1) {
    for_slots(n, [&](int64_t s) { f(s, true, true); });
  } else {
    const int64_t s = thread_id() / G;
    const bool live = s < n;
    f(live ? s : n - 1, live, live && (threadIdx.x & (G - 1)) == 0);
  }
}

// Lanes per particle of the neighbour kernels for n particles.
int nb_group(int64_t n);

// Launches KERNEL<G>(args) for n particles at the context's block size.
#define FS_NB_CASE(KERNEL, G, SMEM, ...)                                                                      \
  launch(KERNEL<G>, (unsigned)((n_ * G + c_->nb_block - 1) / c_->nb_block), c_->nb_block,                     \
         (SMEM) ? scan_smem(c_->nb_block, G) : 0, st_, __VA_ARGS__)
#define FS_NB_LAUNCH(KERNEL, c, n, group, st, SMEM, ...)                                                      \
  do {                                                                                                        \
    const fs_context* c_ = (c);                                                                               \
    const int64_t n_ = (n);                                                                                   \
    cudaStream_t st_ = (st);                                                                                  \
    switch (group) {                                                                                          \
      case 4: FS_NB_CASE(KERNEL, 4, SMEM, __VA_ARGS__); break;                                                \
      case 8: FS_NB_CASE(KERNEL, 8, SMEM, __VA_ARGS__); break;                                                \
      case 16: FS_NB_CASE(KERNEL, 16, SMEM, __VA_ARGS__); break;                                              \
      default:                                                                                                \
        launch(KERNEL<1>, nb_blocks(c_, n_), c_->nb_block, (SMEM) ? scan_smem(c_->nb_block, 1) : 0, st_,      \
               __VA_ARGS__);                                                                                 \
    }                                                                                                         \
  } while (0)

// Whether lists recorded for the current grid and positions exist.
FS_DEV bool lists_usable(const NbrList& L) { return L.ctl->valid != 0; }

NbrList nbr_list(const fs_context* c);
ScanXyz scan_xyz(const fs_context* c);

// Marks freshly recorded lists valid (first thread of the recording kernel);
// a grid build resets the mark.
FS_DEV void lists_recorded(const NbrList& L) {
  if (blockIdx.x == 0 && threadIdx.x == 0) L.ctl->valid = 1;
}

}  // namespace fs
