// legal_par.cu -- the greedy legaliser of electro_place/mod.rs:206-255 on the
// whole GPU, with results identical to the reference's exhaustive scan
// (common.rs:294-374): cells in order (macros first, an extension), each onto
// the free anchor of minimum (bx - x)^2 + (by - y)^2 in FP64, ties to the
// lowest tile.
//
// The greedy is sequential as written, but its result does not need the
// sequence.  own[s] holds the lowest order index that claims site s; a site
// is open to cell q while own[s] > q (or own[s] == q, its own claim).
//
// Unit cells: the greedy is a serial dictatorship, which is the stable
// matching in which every site prefers the lower order index, and a stable
// matching with strict preferences is reached by deferred acceptance whatever
// the order of the proposals.  A CTA takes a cell q, finds the open site of
// least (cost, tile) and claims it with atomicMin(own, q).  If the site was
// held by a later cell, the CTA goes on with the cell it displaced; if an
// earlier cell got there first, it looks again.  own[s] only ever falls, so
// a site once closed to q stays closed: no waiting, no rounds, and every
// lost or won claim lowers some own[s], so it ends.  (Where many unit cells have
// one target they are placed in windows instead: lists against the map as it
// stands, then each takes what the cells before it leave.  See k_lp_lists.)
//
// Macros (several sites per claim, and a macro that moves opens sites again)
// reach their fixed point in rounds over a window of the next kLpWindow
// macros: each macro of the window takes the best anchor given the claims of
// the earlier ones as they stand, if anything that could matter to it changed
// in the last round (its block is under an earlier claim, or an earlier macro
// gave up a block next to an anchor no worse than its own).  The macros
// before the first one that changed in a round are final: each has the best
// anchor given earlier ones that did not move.  The lowest macro of the window
// does not change twice, so the window advances at least every second round.
// 9,980 macros of a 200k-cell checkpoint take about 55 rounds.
//
// The displacement is the sequential FP64 sum of the costs, formed in
// parallel: while the running total stays within one binade, adding a cost
// adds a whole number of units in the last place that depends on the total
// only through its lowest bit (round half to even), so the additions compose
// as maps of that bit and are scanned.
//
// A 200k-cell checkpoint (5 % macros, half of the cells in six piles): 150 to
// 200 ms as rounds of candidate lists, disturbance passes and one CTA's serial
// pass over the cells whose lists interact (a hundred rounds and more of 20
// launches), 7.4 ms in this form (macros 2.3 ms in 54 rounds, units 4.7, the
// displacement's sum 0.33).  The checkpoint at the end of such a run, cells
// spread: 1.3 to 3 ms (macros 0.6, units 0.2 to 2.1 by the design, sum 0.26).
#include <cuda_runtime.h>

#include <cstdint>

#include "legal_par.cuh"

namespace eplace {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int32_t kNone = 0x7fffffff;  // own[] of a site nobody claims
constexpr int kInfHi = 0x7ff00000;     // high word of +infinity
constexpr int kLpWarps = 16;           // warps per CTA of the macro kernels (a power of two)

__device__ __forceinline__ double sq(double d) { return __dmul_rn(d, d); }

// own[] and seg[] change under the readers: L2 loads, never kept in L1.  A
// segment's two words change in an order that its readers rely on, so where
// they are read while they change, every access is of the 64-bit pair: those to
// one location keep their order.
__device__ __forceinline__ int32_t ld_own(const int32_t *p) {
  int32_t v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_seg(const uint2 *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return make_uint2((unsigned)v, (unsigned)(v >> 32));
}
// Clears a bit of the first word and raises the second, as a signed number, to
// q, in one; s: what the pair was at some time.  (Bits only go, so one that is
// clear in s has gone; ends, since a pair that changed under it has fewer bits
// or a higher second word.)
__device__ __forceinline__ void take_bit(uint2 *p, uint2 s, unsigned bit, int32_t q) {
  while (s.x & bit) {
    const unsigned y = (unsigned)max((int32_t)s.y, q);
    const unsigned long long was = ((unsigned long long)s.y << 32) | s.x;
    const unsigned long long is = atomicCAS(reinterpret_cast<unsigned long long *>(p), was,
                                            ((unsigned long long)y << 32) | (s.x & ~bit));
    if (is == was) break;
    s = make_uint2((unsigned)is, (unsigned)(is >> 32));
  }
}
// Bit b set: site b of the segment has a claim of q or later, or none; only
// the groups of four sites with a bit in `ask` are looked at.
__device__ __forceinline__ unsigned open_sites(const int32_t *own32, unsigned ask, int32_t q) {
  unsigned m = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    if (!((ask >> (4 * u)) & 15u)) continue;
    int4 v;
    asm volatile("ld.relaxed.gpu.global.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(own32 + 4 * u)
                 : "memory");
    m |= ((v.x >= q ? 1u : 0u) | (v.y >= q ? 2u : 0u) | (v.z >= q ? 4u : 0u) | (v.w >= q ? 8u : 0u)) << (4 * u);
  }
  return m;
}
__device__ __forceinline__ int32_t *own_at(const LpArgs &a, int x, int y) {
  return a.own + (size_t)y * (32 * a.SW) + x;
}
__device__ __forceinline__ uint2 *seg_at(const LpArgs &a, int x, int y) { return a.seg + (size_t)y * a.SW + (x >> 5); }

struct Cell {
  double tx, ty;  // target (the continuous position)
  double ox, oy;  // anchor -> block centre offset, (w - 1) / 2
  int w, h;
  int AW, AH;     // anchor grid
  int cx, cy;     // the anchor nearest to the target
  int fx;         // the last anchor column at or left of the target, -1: none
  bool inside;    // the target lies on the anchor grid
};

__device__ __forceinline__ int nearest_in(double v, int n) {  // n >= 1
  return (int)fmin(fmax(rint(v), 0.0), (double)(n - 1));
}

__device__ __forceinline__ Cell make_cell(const LpArgs &a, float2 p, uchar2 s) {
  Cell c;
  c.tx = (double)p.x;
  c.ty = (double)p.y;
  c.w = s.x;
  c.h = s.y;
  c.ox = 0.5 * (double)(c.w - 1);
  c.oy = 0.5 * (double)(c.h - 1);
  c.AW = a.W - c.w + 1;
  c.AH = a.H - c.h + 1;
  const double ux = __dsub_rn(c.tx, c.ox), uy = __dsub_rn(c.ty, c.oy);
  c.cx = nearest_in(ux, c.AW);
  c.cy = nearest_in(uy, c.AH);
  c.fx = (int)fmin(fmax(floor(ux), -1.0), (double)(c.AW - 1));
  c.inside = ux >= 0.0 && ux <= (double)(c.AW - 1) && uy >= 0.0 && uy <= (double)(c.AH - 1);
  return c;
}
__device__ __forceinline__ Cell load_cell(const LpArgs &a, uint32_t q, bool unit) {
  const uint32_t cell = a.order[q];
  return make_cell(a, a.pos[cell], unit ? make_uchar2(1, 1) : a.fsize[cell]);
}

// Cost of anchor (ax, ay), formed as the host legaliser forms it.
__device__ __forceinline__ double axis2(double at, double off, double target) {
  return sq(__dsub_rn(__dadd_rn(at, off), target));
}
__device__ __forceinline__ double col_dx2(const Cell &c, int ax) { return axis2((double)ax, c.ox, c.tx); }
__device__ __forceinline__ double row_dy2(const Cell &c, int ay) { return axis2((double)ay, c.oy, c.ty); }

// A cell whose target is no number, infinite, or more than 2^24 sites from its
// nearest anchor finds no site.  Up to there the costs of two sites in a row on
// the same side of the target differ in FP64 (whole sites apart, an ulp of
// 2^-5), and FP32 bounds on them stay far from overflow; from 2^26.5 on sites
// of one row tie, and past 2^64 a cost in FP32 is infinite.
constexpr double kFarCost = 281474976710656.0;  // (2^24)^2
__device__ __forceinline__ bool placeable(const Cell &c) {
  return c.AW > 0 && c.AH > 0 && __dadd_rn(col_dx2(c, c.cx), row_dy2(c, c.cy)) <= kFarCost;
}

// The least (cost, tile) seen; tile kNone: none.  Costs are >= 0, so the
// words of a cost order like the cost.
struct Best {
  double cost;
  int tile;
  __device__ __forceinline__ void take(double c, int t) {
    if (c < cost || (c == cost && t < tile)) {
      cost = c;
      tile = t;
    }
  }
  __device__ __forceinline__ Best warp_min() const {
    const unsigned hi = (unsigned)__double2hiint(cost), lo = (unsigned)__double2loint(cost);
    const unsigned mh = __reduce_min_sync(kFull, hi);
    const unsigned ml = __reduce_min_sync(kFull, hi == mh ? lo : ~0u);
    const int t = (int)__reduce_min_sync(kFull, (unsigned)(hi == mh && lo == ml ? tile : kNone));
    return Best{__hiloint2double((int)mh, (int)ml), t};
  }
};
__device__ __forceinline__ Best no_best() { return Best{__hiloint2double(kInfHi, 0), kNone}; }

// FP32 costs, to rule rows, segments and most sites out: coordinates are whole
// or FP32 numbers (halves, for a block's centre), so such a cost is within
// 2^-21 of the exact one; kOver and kUnder cover twice that.
constexpr float kOver = 1.000002f, kUnder = 0.999998f;
constexpr float kInf = __builtin_huge_valf();

__device__ __forceinline__ float fast_sqrt(float v) {  // within 2^-22
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// Hints.  When cell k has its place, every anchor cheaper than its own was
// closed to it, and what is closed to k is closed to every later cell of the
// same or a larger footprint.  Entry (size class, 16 x 16 sites) keeps the
// largest such radius seen from the middle of those sites, with its k: a
// later cell with a target near by starts its search on that circle instead
// of at its target.  A pile of some hundred sites is walked through once for
// each 16 x 16 of targets instead of once for each cell.
__device__ __forceinline__ float2 hint_middle(int cx, int cy) {
  return make_float2((float)((cx & ~15) + 8), (float)((cy & ~15) + 8));
}
__device__ __forceinline__ float hint_dist(const Cell &c) {  // target to the middle, rounding allowed for
  const float2 m = hint_middle(c.cx, c.cy);
  const float dx = (float)(c.tx - c.ox) - m.x, dy = (float)(c.ty - c.oy) - m.y;
  return sqrtf(dx * dx + dy * dy) + 0.01f;
}
__device__ __forceinline__ unsigned long long *hint_at(const LpArgs &a, const Cell &c, int size) {
  const size_t tw = (a.W + 15) / 16, tiles = tw * ((a.H + 15) / 16);
  return a.hint + (size - 1) * tiles + (c.cy >> 4) * tw + (c.cx >> 4);
}
__device__ __forceinline__ void put_hint(const LpArgs &a, int32_t q, const Cell &c, double cost) {
  const int size = max(c.w, c.h);
  if (!c.inside || size > kLpHintClasses || !(cost > 64.0)) return;
  const float r = sqrtf((float)cost) * 0.9999f - hint_dist(c);
  if (r > 4.0f) atomicMax(hint_at(a, c, size), ((unsigned long long)__float_as_uint(r) << 32) | (unsigned)q);
}
// A cost below which no anchor is open to q.
__device__ __forceinline__ double get_hint(const LpArgs &a, int32_t q, const Cell &c) {
  if (!c.inside) return 0.0;
  float r = 0.0f;
  unsigned long long e[kLpHintClasses];  // what was closed to a smaller footprint is closed to this one
#pragma unroll
  for (int k = 0; k < kLpHintClasses; ++k) e[k] = k < min(c.w, c.h) ? __ldcg(hint_at(a, c, k + 1)) : 0ull;
#pragma unroll
  for (int k = 0; k < kLpHintClasses; ++k)
    if ((int32_t)(unsigned)e[k] < q) r = fmaxf(r, __uint_as_float((unsigned)(e[k] >> 32)));
  r = (r - hint_dist(c)) * 0.9999f;
  return r > 0.0f ? (double)r * (double)r : 0.0;
}

// ---------------------------------------------------------------------------
// Macros
// ---------------------------------------------------------------------------

// seg[] while the macros are placed: x has a bit for each site without a
// final claim (of a macro before the window, or a fixed cell), y for each site
// with a claim of the window.  Sites with both bits are open to some macros of
// the window only; their own[] tells.
__device__ __forceinline__ unsigned open_word(const LpArgs &a, int32_t q, int y, int g, uint2 s) {
  const unsigned ask = s.x & s.y;
  return ask ? (s.x & (~s.y | open_sites(own_at(a, 32 * g, y), ask, q))) : s.x;
}

// The open anchor of least (cost, tile) for macro q of at most 32 x 16 sites,
// none of cost below c0 being open, by the CTA: bands of 33 - h anchor rows
// outward from the target, a lane per site row, in a band the segments outward
// from the circle of cost c0, to the right and to the left by different warps,
// each segment tested as bit words (a run of w open sites along the row, then
// h such rows), stopped by the least cost so far (*least, shared, FP32).
// Latency bound (a word per lane and segment from L2, four segments in flight,
// and own[] of the words that need it).  Returns this lane's best.
__device__ Best search_block(const LpArgs &a, int32_t q, const Cell &c, double c0, int warp, int lane,
                             unsigned *least) {
  Best b = no_best();
  const int nb = 33 - c.h;
  const float tx = (float)c.tx, ty = (float)c.ty, ox = (float)c.ox, oy = (float)c.oy;
  float most = kInf;
  auto d2 = [](float at, float off, float t) {
    const float d = at + off - t;
    return d * d;
  };
  // anchors of segment g whose block is open: wc, wn the words of segments g, g + 1
  auto eval = [&](int g, int a0, unsigned wc, unsigned wn) {
    most = __uint_as_float(*(volatile unsigned *)least);
    if (!__any_sync(kFull, wc != 0)) return;
    uint64_t t = (uint64_t)wc | ((uint64_t)wn << 32);
    for (int s = 1; s < c.w;) {
      const int d = min(s, c.w - s);
      t &= t >> d;
      s += d;
    }
    unsigned v = (unsigned)t;
    for (int s = 1; s < c.h;) {
      const int d = min(s, c.h - s);
      v &= __shfl_down_sync(kFull, v, d);
      s += d;
    }
    if (lane >= nb) v = 0;  // its rows below the band are not here
    float mine = kInf;
    if (v) {
      // (split at the target, not at the nearest column: two columns half a
      // site away on either side are a tie for the lower one)
      const int ay = a0 + lane, f = c.fx - 32 * g;
      const float dy2 = d2((float)ay, oy, ty);
      const unsigned left = f < 0 ? 0u : (f >= 31 ? ~0u : (2u << f) - 1u);
      const unsigned vl = v & left, vr = v & ~left;
      const int xl = 32 * g + 31 - __clz(vl), xr = 32 * g + __ffs(vr) - 1;
      const float cl = vl ? d2((float)xl, ox, tx) + dy2 : kInf, cr = vr ? d2((float)xr, ox, tx) + dy2 : kInf;
      mine = fminf(cl, cr);
      const float bound = fminf(most, mine * kOver) * kOver;
      if (vl && cl <= bound) b.take(__dadd_rn(col_dx2(c, xl), row_dy2(c, ay)), ay * a.W + xl);
      if (vr && cr <= bound) b.take(__dadd_rn(col_dx2(c, xr), row_dy2(c, ay)), ay * a.W + xr);
    }
    const unsigned all = __reduce_min_sync(kFull, __float_as_uint(mine * kOver));
    if (lane == 0 && all < __float_as_uint(most)) atomicMin(least, all);
    most = fminf(most, __uint_as_float(all));
  };
  const int base0 = c.cy - nb / 2;
  for (int k = 0;; ++k) {
    bool any = false;
    most = __uint_as_float(*(volatile unsigned *)least);
    for (int side = 0; side < (k ? 2 : 1); ++side) {
      const int a0 = base0 + (side ? -k * nb : k * nb);
      const int r0 = max(a0, 0), r1 = min(a0 + nb, c.AH) - 1;
      if (r0 > r1) continue;
      const float dmin = d2((float)min(max(c.cy, r0), r1), oy, ty);
      if (dmin > most) continue;
      any = true;
      const int part = (2 * (2 * k + side) - warp) & (kLpWarps - 1);  // 0: right, 1: left is this warp's
      const bool right = part == 0, left = ((part + 1) & (kLpWarps - 1)) == 0;
      if (!right && !left) continue;
      const int y = a0 + lane;
      const bool row = y >= 0 && y < a.H;
      auto raw = [&](int g) {
        return row && g >= 0 && g < a.SW ? ld_seg(a.seg + (size_t)y * a.SW + g) : make_uint2(0u, 0u);
      };
      // Columns nearer than `skip` cost less than c0 in every row of the band.
      const double far = fmax(row_dy2(c, r0), row_dy2(c, r1));
      const int skip = c0 > far ? max((int)sqrtf((float)__dsub_rn(c0, far)) - 2, 0) : 0;
      const int gr = min(max(c.fx + skip, 0), c.AW - 1) >> 5, gl = max(c.fx - skip, 0) >> 5;
      uint2 p[5];
      if (right) {
#pragma unroll
        for (int u = 0; u < 5; ++u) p[u] = raw(gr + u);
        unsigned cur = open_word(a, q, y, gr, p[0]);
        for (int g = gr;; g += 4) {
          bool done = false;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int at = g + u;
            done = done || 32 * at >= c.AW || (at > gr && d2((float)(32 * at), ox, tx) + dmin > most);
            if (!done) {
              const unsigned nxt = open_word(a, q, y, at + 1, p[u + 1]);
              eval(at, a0, cur, nxt);
              cur = nxt;
            }
          }
          if (done) break;
#pragma unroll
          for (int u = 1; u < 5; ++u) p[u] = raw(g + 4 + u);
        }
      } else {
        const int g0 = gl == gr ? gl - 1 : gl;  // the other warp has the segment they share
        if (g0 < 0) continue;
        p[4] = raw(g0 + 1);
        unsigned nxt = 0, cur;
        for (int g = g0; g >= 0; g -= 4) {
#pragma unroll
          for (int u = 0; u < 4; ++u) p[u] = raw(g - u);
          if (g == g0) nxt = open_word(a, q, y, g0 + 1, p[4]);
          bool done = false;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int at = g - u;
            done = done || at < 0 || (at < (c.cx >> 5) && d2((float)(32 * at + 31), ox, tx) + dmin > most);
            if (!done) {
              cur = open_word(a, q, y, at, p[u]);
              eval(at, a0, cur, nxt);
              nxt = cur;
            }
          }
          if (done) break;
        }
      }
    }
    if (!any) break;  // outside the chip or too far on both sides, and the next bands too
  }
  return b;
}

// The same for any footprint (wider or higher ones): a warp per anchor row, the
// rows outward from the target, a lane per site row of the block (32 at a time),
// whose words tell 32 anchors at once: a run of w open sites is one of 32 and
// those behind it, the last shifted.  (A lane per anchor that looked at each
// site of its block, by one warp: 15 macros of 40 x 40 among 20k cells, all in a
// pile, 468 ms -> 5.1 (61 as rounds of lists); 20 of 90 to 130 x 70 to 110 among
// 100k, spread, 631 -> 3.3 ms (41).)
__device__ Best search_large(const LpArgs &a, int32_t q, const Cell &c, double c0, int warp, int lane,
                             unsigned *least) {
  Best b = no_best();
  const float tx = (float)c.tx, ty = (float)c.ty, ox = (float)c.ox, oy = (float)c.oy;
  const int one = min(c.w, 32), rows = max(c.cy, c.AH - 1 - c.cy);
  auto d2 = [](float at, float off, float t) {
    const float d = at + off - t;
    return d * d;
  };
  // bit k: sites 32 g + k .. + one - 1 of row y are open
  auto run = [&](int y, int g) -> unsigned {
    const uint2 *seg = a.seg + (size_t)y * a.SW;
    const uint2 s0 = g < a.SW ? ld_seg(seg + g) : make_uint2(0u, 0u);
    const uint2 s1 = g + 1 < a.SW ? ld_seg(seg + g + 1) : make_uint2(0u, 0u);
    uint64_t t = (uint64_t)open_word(a, q, y, g, s0) | (uint64_t)open_word(a, q, y, g + 1, s1) << 32;
    for (int s = 1; s < one;) {
      const int d = min(s, one - s);
      t &= t >> d;
      s += d;
    }
    return (unsigned)t;
  };
  auto anchors = [&](int ay, int g) -> unsigned {
    unsigned v = ~0u;
    for (int y0 = 0; y0 < c.h && v; y0 += 32) {
      unsigned r = ~0u;
      if (y0 + lane < c.h) {
        const int y = ay + y0 + lane;
        r = run(y, g);
        for (int k = 1; 32 * (k + 1) <= c.w && r; ++k) r &= run(y, g + k);
        const int rest = c.w & 31, k = c.w >> 5;
        if (c.w > 32 && rest && r) r &= (run(y, g + k - 1) >> rest) | (run(y, g + k) << (32 - rest));
      }
      v &= __reduce_and_sync(kFull, r);
    }
    return v;
  };
  float most = kInf;
  auto found = [&](int x, int ay) {
    b.take(__dadd_rn(col_dx2(c, x), row_dy2(c, ay)), ay * a.W + x);
    const unsigned mine = __float_as_uint((d2((float)x, ox, tx) + d2((float)ay, oy, ty)) * kOver);
    if (lane == 0) atomicMin(least, mine);
  };
  for (int k = warp; k <= 2 * rows; k += kLpWarps) {
    most = __uint_as_float(*(volatile unsigned *)least);
    const float away = (float)((k + 1) >> 1) - 0.5f;
    if (k && away * away > most) break;
    const int ay = c.cy + ((k & 1) ? -(k + 1) / 2 : k / 2);
    if (ay < 0 || ay >= c.AH) continue;
    const float dy2 = d2((float)ay, oy, ty);
    if (dy2 > most) continue;
    const double far = row_dy2(c, ay);
    const int skip = c0 > far ? max((int)sqrtf((float)__dsub_rn(c0, far)) - 2, 0) : 0;
    const int gr = min(max(c.fx + skip, 0), c.AW - 1) >> 5, gl = max(c.fx - skip, 0) >> 5;
    for (int g = gr; 32 * g < c.AW; ++g) {
      most = __uint_as_float(*(volatile unsigned *)least);
      if (g > gr && d2((float)(32 * g), ox, tx) + dy2 > most) break;
      const int f = c.fx - 32 * g;
      const unsigned v = anchors(ay, g) & (f < 0 ? ~0u : f >= 31 ? 0u : ~0u << (f + 1));
      if (v) {
        found(32 * g + __ffs(v) - 1, ay);
        break;
      }
    }
    for (int g = gl; g >= 0; --g) {
      most = __uint_as_float(*(volatile unsigned *)least);
      if (g < gl && d2((float)(32 * g + 31), ox, tx) + dy2 > most) break;
      const int f = c.fx - 32 * g;
      const unsigned v = anchors(ay, g) & (f < 0 ? 0u : f >= 31 ? ~0u : (2u << f) - 1u);
      if (v) {
        found(32 * g + 31 - __clz(v), ay);
        break;
      }
    }
  }
  return b;
}

// Targets in the same square of 1 / tie_scale sites have one key.
constexpr unsigned long long kNoTie = 1ull << 63;  // none: the column of no target within 2^25 sites
__device__ __forceinline__ unsigned long long tie_key(const LpArgs &a, float2 p) {
  constexpr float kMost = 33554432.0f;  // 2^25 (farther ones find no site)
  if (!(fabsf(p.x) < kMost && fabsf(p.y) < kMost)) return kNoTie;
  return ((unsigned long long)(unsigned)(int)floorf(p.x * a.tie_scale) << 32) |
         (unsigned)(int)floorf(p.y * a.tie_scale);
}

// Few unit cells: whether enough of them share targets, by a CTA, from 512 of them
// at even distances (all of fewer).  Ties are cells whose target a 32nd of these
// have (or what 32 of all are, of few); enough is a tenth.
constexpr uint32_t kTieSample = 512;
__device__ void sample_ties(const LpArgs &a) {
  constexpr uint32_t kMask = 2 * kTieSample - 1;
  __shared__ unsigned long long key[kMask + 1];
  __shared__ uint32_t count[kMask + 1], ties;
  const uint32_t tid = threadIdx.x, units = a.n - a.n_mac, m = units < kTieSample ? units : kTieSample;
  for (uint32_t h = tid; h <= kMask; h += blockDim.x) {
    key[h] = kNoTie;
    count[h] = 0u;
  }
  if (tid == 0) ties = 0u;
  __syncthreads();
  for (uint32_t k = tid; k < m; k += blockDim.x) {
    const uint32_t i = (uint32_t)((uint64_t)k * units / m);
    const unsigned long long t = tie_key(a, a.pos[a.order[a.n_mac + i]]);
    if (t == kNoTie) continue;
    uint32_t h = (uint32_t)((t * 0x9e3779b97f4a7c15ull) >> 32) & kMask;
    while (true) {  // (half of the table stays empty)
      const unsigned long long was = atomicCAS(&key[h], kNoTie, t);
      if (was == kNoTie || was == t) break;
      h = (h + 1) & kMask;
    }
    atomicAdd(&count[h], 1u);
  }
  __syncthreads();
  const uint32_t few = 32u * m / units, least = few > m / 32 ? few : m / 32;
  for (uint32_t h = tid; h <= kMask; h += blockDim.x)
    if (count[h] >= least) atomicAdd(&ties, count[h]);
  __syncthreads();
  if (tid != 0 || ties < least || 10u * ties < m) return;
  a.st->tied = 1u;
  if (a.tie_loop) cudaGraphSetConditional(a.windows, 1u);
  else atomicMax(&a.st->status, kLpTied);
}

__global__ void __launch_bounds__(256) k_lp_init(const LpArgs a) {
  const int lane = threadIdx.x & 31;
  const int nseg = a.SW * a.H;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nseg; i += (gridDim.x * blockDim.x) >> 5) {
    const int y = i / a.SW, x = 32 * (i - y * a.SW) + lane;
    const bool open = x < a.W && ((a.free0[(size_t)y * a.WR + (x >> 6)] >> (x & 63)) & 1u);
    *own_at(a, x, y) = open ? kNone : -1;
    const unsigned m = __ballot_sync(kFull, open);
    if (lane == 0) a.seg[i] = make_uint2(m, 0u);
  }
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < a.n_mac; q += gridDim.x * blockDim.x) {
    a.choice[q] = -1;
    const bool in = q < kLpWindow;  // the first round's
    a.queued[q] = in ? 1u : 0u;
    if (in) a.work[q] = q;
  }
  const uint32_t hints = kLpHintClasses * (uint32_t)((a.W + 15) / 16) * (uint32_t)((a.H + 15) / 16);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < hints; i += gridDim.x * blockDim.x) a.hint[i] = 0ull;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n - a.n_mac; i += gridDim.x * blockDim.x)
    a.cand[(size_t)kLpCand * i] = -1;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; !a.tie_few && i <= a.tie_mask; i += gridDim.x * blockDim.x) {
    a.tie_key[i] = kNoTie;
    a.tie_count[i] = 0u;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    *a.st = LpState{0u, 0u, (uint32_t)kNone, 0u, 0u, {min(a.n_mac, kLpWindow), 0u}, 0u, 0u, 0u, 0u, 0u, 0};
  if (a.tie_few && blockIdx.x == 0) {
    __syncthreads();  // the state is written
    sample_ties(a);
  }
}

// A round, first half: each macro of the work list (whose choice may have
// become wrong) chooses again; the blocks given up are entered in the round's
// list and leave own[].  (A macro that reads own[] while another leaves it
// sees some sites of the old block open and some not; the block is in the
// list, so it is looked at again in the next round if that could matter to it.)
// A CTA per macro: a round lasts as long as its longest search.
__global__ void __launch_bounds__(kLpWarps * 32) k_lp_choose(const LpArgs a) {
  __shared__ Best sbest[kLpWarps];
  __shared__ unsigned least;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  LpState *st = a.st;
  const uint32_t par = st->rounds & 1u, nwork = st->nwork[par];
  for (uint32_t item = blockIdx.x; item < nwork; item += gridDim.x) {
    const uint32_t qi = a.work[par * kLpWindow + item];
    const int32_t q = (int32_t)qi;
    const Cell c = load_cell(a, qi, false);
    const int32_t old = a.choice[q];
    // nothing of a lower cost than its own is open when only its own block was lost
    double c0 = old >= 0 && !(a.queued[q] & 2) && c.inside ? a.mcost[q] : 0.0;
    c0 = fmax(c0, get_hint(a, q, c));
    if (tid == 0) least = __float_as_uint(kInf);
    __syncthreads();
    Best b = no_best();
    if (placeable(c)) {
      if (c.w <= 32 && c.h <= 16) b = search_block(a, q, c, c0, warp, lane, &least);
      else b = search_large(a, q, c, c0, warp, lane, &least);
    }
    b = b.warp_min();
    if (lane == 0) sbest[warp] = b;
    __syncthreads();
    if (warp == 0) {
      b = (lane < kLpWarps ? sbest[lane] : no_best()).warp_min();
      const int32_t now = b.tile == kNone ? -2 : b.tile;
      if (lane == 0) a.queued[q] = 0;
      if (now != old) {
        if (old >= 0) {
          const int oldx = old % a.W, oldy = old / a.W;
          for (int s = lane; s < c.w * c.h; s += 32) {
            const int x = oldx + s % c.w, y = oldy + s / c.w;
            int32_t *o = own_at(a, x, y);
            if (ld_own(o) == q) {  // nobody else writes a site that q holds
              *o = kNone;
              atomicAnd(reinterpret_cast<unsigned long long *>(seg_at(a, x, y)), ~(1ull << (32 + (x & 31))));
            }
          }
        }
        if (lane == 0) {
          atomicMin(&st->first, qi);
          if (old >= 0) a.freed[atomicAdd(&st->nfreed, 1u)] = LpFreed{q, old, c.w, c.h};
          a.choice[q] = now;
          a.mcost[q] = b.cost;
        }
      }
    }
    __syncthreads();  // sbest and least are free again
  }
}

// Enters macro q in the next round's work list, once; why: 1: its block was
// lost, 2: something was given up that may be better.
__device__ __forceinline__ void queue_macro(const LpArgs &a, uint32_t q, unsigned why) {
  if (atomicOr(&a.queued[q], why) != 0u) return;
  const uint32_t par = (a.st->rounds + 1) & 1u;
  a.work[par * kLpWindow + atomicAdd(&a.st->nwork[par], 1u)] = q;
}

// Second half, a warp per macro of the window: every macro enters its claim
// again (a macro that left may have covered a later one's); who finds an
// earlier claim on its block, or loses a site to one here, and who could gain
// from a block given up in this round, chooses again in the next.  The last
// CTA moves the window to the first macro that changed; those that enter it
// choose for the first time.
__global__ void __launch_bounds__(kLpWarps * 32) k_lp_claim(const LpArgs a) {
  __shared__ bool last;
  const int lane = threadIdx.x & 31;
  LpState *st = a.st;
  const uint32_t base = st->base, end = min(base + kLpWindow, a.n_mac);
  const uint32_t stop = min(__ldcg(&st->first), end);
  const uint32_t q = base + blockIdx.x * kLpWarps + (threadIdx.x >> 5);
  if (q < end) {
    const int32_t t = a.choice[q];
    const Cell c = load_cell(a, q, false);
    if (t >= 0) {
      const int ax = t % a.W, ay = t / a.W;
      bool lost = false;
      for (int k = lane; k < c.w * c.h; k += 32) {
        const int x = ax + k % c.w, y = ay + k / c.w;
        int32_t *o = own_at(a, x, y);
        int32_t was = ld_own(o);
        if (was > (int32_t)q) {
          was = atomicMin(o, (int32_t)q);
          atomicOr(&seg_at(a, x, y)->y, 1u << (x & 31));
          if (was > (int32_t)q && was < (int32_t)end) queue_macro(a, (uint32_t)was, 1u);
        }
        lost |= was < (int32_t)q;
        if (q < stop) atomicAnd(&seg_at(a, x, y)->x, ~(1u << (x & 31)));  // final
      }
      if (__any_sync(kFull, lost) && lane == 0) queue_macro(a, q, 1u);
      if (q < stop && lane == 0) put_hint(a, (int32_t)q, c, a.mcost[q]);
    } else if (q < stop && lane == 0) {
      atomicMax(&st->status, 1);  // final, and no anchor was open
    }
    if (q >= stop) {
      const double mine = t >= 0 ? a.mcost[q] : __hiloint2double(kInfHi, 0);
      bool gain = false;
      const uint32_t nf = __ldcg(&st->nfreed);
      for (uint32_t e = lane; e < nf; e += 32) {
        const LpFreed f = a.freed[e];
        if (f.q >= (int32_t)q) continue;
        // the least cost of an anchor whose block meets the freed one
        const int fx = f.tile % a.W, fy = f.tile / a.W;
        const int x0 = max(fx - c.w + 1, 0), x1 = min(fx + f.w - 1, c.AW - 1);
        const int y0 = max(fy - c.h + 1, 0), y1 = min(fy + f.h - 1, c.AH - 1);
        if (x0 > x1 || y0 > y1) continue;
        gain |= __dadd_rn(col_dx2(c, min(max(c.cx, x0), x1)), row_dy2(c, min(max(c.cy, y0), y1))) <= mine;
      }
      if (__any_sync(kFull, gain) && lane == 0) queue_macro(a, q, 2u);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (uint32_t i = end + threadIdx.x; i < min(stop + kLpWindow, a.n_mac); i += blockDim.x) queue_macro(a, i, 1u);
  __syncthreads();
  if (threadIdx.x != 0) return;
  st->base = stop;
  st->first = (uint32_t)kNone;
  st->nfreed = 0;
  st->nwork[st->rounds & 1u] = 0;
  st->rounds += 1;
  st->ticket = 0;
  if (stop < a.n_mac && st->rounds >= a.max_rounds) atomicMax(&st->status, 2);
  if (ld_own(a.cancel)) atomicMax(&st->status, 4);
  if (stop >= a.n_mac || atomicAdd(&st->status, 0) != 0) cudaGraphSetConditional(a.handle, 0u);
}

// ---------------------------------------------------------------------------
// Unit cells
// ---------------------------------------------------------------------------

// seg[] while the unit cells are placed: x has a bit for each site that
// nobody has claimed yet (cleared after the claim, so a bit may be late), y
// the largest order index that cleared one of them.  A segment with x == 0 and y < q has
// no site open to q; with y < q the bits of x are the open sites.
//
// Counts a unit cell that k_lp_near left over under its key (the table has twice
// as many entries as cells or more; a warp adds those of one key together), and
// the cells of the keys that have tie_least or more.
__device__ void count_tie(const LpArgs &a, uint32_t i, bool in) {  // a warp; in: unit cell i counts
  const unsigned long long key = in ? tie_key(a, a.pos[a.order[a.n_mac + i]]) : kNoTie;
  const unsigned same = __match_any_sync(kFull, key);
  if (key == kNoTie || (int)(threadIdx.x & 31) != __ffs(same) - 1) return;
  uint32_t h = (uint32_t)((key * 0x9e3779b97f4a7c15ull) >> 32) & a.tie_mask;
  for (uint32_t k = 0; k <= a.tie_mask; ++k, h = (h + 1) & a.tie_mask) {
    const unsigned long long was = atomicCAS(a.tie_key + h, kNoTie, key);
    if (was != kNoTie && was != key) continue;
    const uint32_t n = (uint32_t)__popc(same), had = atomicAdd(a.tie_count + h, n);
    if (had + n >= a.tie_least) atomicAdd(&a.st->ties, had >= a.tie_least ? n : had + n);
    return;
  }
}

__global__ void __launch_bounds__(256) k_lp_segments(const LpArgs a) {
  const int lane = threadIdx.x & 31;
  const int nseg = a.SW * a.H;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nseg; i += (gridDim.x * blockDim.x) >> 5) {
    const unsigned m = __ballot_sync(kFull, a.own[(size_t)32 * i + lane] == kNone);
    if (lane == 0) a.seg[i] = make_uint2(m, ~0u);
  }
}

// Search of the sites around unit cell q's target by one warp: the 5 x 5 sites
// around the nearest one, a lane each.  A site outside costs at least 2.5^2,
// so a cheaper one inside is the answer.  seen: the answer's segment, if asked for.
__device__ __forceinline__ Best search_near(const LpArgs &a, int32_t q, const Cell &c, int lane, uint2 *seen) {
  Best b = no_best();
  const int x = c.cx - 2 + lane % 5, y = c.cy - 2 + lane / 5;
  uint2 s = make_uint2(0u, 0u);
  if (lane < 25 && x >= 0 && x < a.W && y >= 0 && y < a.H) {
    const int32_t held = ld_own(own_at(a, x, y));
    if (seen) s = ld_seg(seg_at(a, x, y));
    if (held > q) b.take(__dadd_rn(col_dx2(c, x), row_dy2(c, y)), y * a.W + x);
  }
  const Best all = b.warp_min();
  if (seen) {
    const int l = __ffs(__ballot_sync(kFull, b.tile == all.tile)) - 1;  // (any lane where there is none)
    *seen = make_uint2(__shfl_sync(kFull, s.x, l), __shfl_sync(kFull, s.y, l));
  }
  return all;
}

// Claims site (x, y) for q (one thread): kNone: it was free; a later cell: q
// has it now, and that cell has lost it; an earlier cell: q did not get it.
// The first to claim it takes its bit, or whoever meets a bit that is late;
// the site's holder is never later than the one that took the bit.  (The two
// atomics are under way together: whichever is first, the claim will stand.)
// seen: the segment as it was at some time; nullptr while nobody reads any.
__device__ __forceinline__ int32_t claim_site(const LpArgs &a, int32_t q, int x, int y, const uint2 *seen) {
  uint2 *s = seg_at(a, x, y);
  const unsigned bit = 1u << (x & 31);
  const int32_t held = atomicMin(own_at(a, x, y), q);
  if (seen) {
    take_bit(s, *seen, bit, q);
  } else if (held == kNone || held < q) {
    atomicMax(reinterpret_cast<int32_t *>(&s->y), q);
    atomicAnd(&s->x, ~bit);
  }
  return held;
}

// The same by a warp, whose lanes read the displaced cell's list next: its
// writer's fence and claim are paired with a fence here (claims are relaxed).
__device__ __forceinline__ int32_t claim_and_acquire(const LpArgs &a, int32_t q, int x, int y, uint2 seen, int lane) {
  int32_t held = 0;
  if (lane == 0) {
    held = claim_site(a, q, x, y, &seen);
    if (held > q && held != kNone) asm volatile("fence.acq_rel.gpu;" ::: "memory");
  }
  __syncwarp();
  return __shfl_sync(kFull, held, 0);
}

// First all unit cells at once, a warp each: the best open site near the
// target, claimed.  A cell that finds none, or is displaced by an earlier one
// that was under way at the same time, is left over: the answer doesn't depend
// on the order of the proposals.  But the work does, where many cells want the
// same sites: a claim made too early is displaced again.  So with more than one
// cell in kLeftMost left over, the claims are undone (0.1 ms for 200k cells) and
// k_lp_units takes all cells, nearly in order.
// Units of a 200k-cell checkpoint at the end of a run, 0.65 % left over: 1.74 ->
// 0.22 ms; of 30k cells, 4.8 % left over: 0.30 -> 0.20.  Half of the cells in
// six piles, 41 % left over: 70 ms, against 4.9 in order; trying it first costs
// 0.04 of 7.6 ms there.  Below kNearFrom cells the attempt costs about what it
// saves (3k cells in piles 0.15 -> 0.18 ms, 10k with macros 0.75 -> 0.81).
constexpr uint32_t kLeftMost = 12, kNearFrom = 16384;
__device__ __forceinline__ bool few_left(const LpArgs &a) { return kLeftMost * (uint64_t)a.st->npend <= a.n - a.n_mac; }

constexpr int kNearTries = 4;
__global__ void __launch_bounds__(256) k_lp_near(const LpArgs a) {
  if (a.st->status != 0) return;
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= a.n - a.n_mac) return;
  const int lane = threadIdx.x & 31;
  const int32_t q = (int32_t)(a.n_mac + i);
  const Cell c = load_cell(a, (uint32_t)q, true);
  int32_t site = -1;
  for (int k = 0; k < kNearTries && placeable(c); ++k) {
    const Best b = search_near(a, q, c, lane, nullptr);
    if (!(b.cost < 6.25)) break;
    int32_t held = 0;
    if (lane == 0) held = claim_site(a, q, b.tile % a.W, b.tile / a.W, nullptr);
    held = __shfl_sync(kFull, held, 0);
    if (held > q) {  // (kNone too)
      site = b.tile;
      break;
    }
  }
  if (lane == 0) a.near[i] = site;
}

// Whether unit cell i has not kept a site.
__device__ __forceinline__ bool left_over(const LpArgs &a, uint32_t i) {
  if (i >= a.n - a.n_mac) return false;
  const int32_t t = a.near[i];
  return t < 0 || *own_at(a, t % a.W, t / a.W) != (int32_t)(a.n_mac + i);
}

// The cells left over, in order: counted by a CTA for each kLpChunk of them,
// then listed behind those of the chunks before.
// (Nothing was taken, and near[] is not written, where the macros failed or
// the result is no longer wanted; the status doesn't change in between.)
__global__ void __launch_bounds__(kLpChunk) k_lp_count(const LpArgs a) {
  if (a.st->status != 0) return;
  const uint32_t i = blockIdx.x * kLpChunk + threadIdx.x;
  const bool left = left_over(a, i);
  if (__any_sync(kFull, left)) count_tie(a, i, left);
  const int n = __syncthreads_count(left);
  if (threadIdx.x == 0) a.left[blockIdx.x] = (uint32_t)n;
}
__global__ void __launch_bounds__(kLpChunk) k_lp_pending(const LpArgs a) {
  __shared__ uint32_t part[kLpChunk / 32];
  if (a.st->status != 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto block_sum = [&](uint32_t v) {
    v = __reduce_add_sync(kFull, v);
    if (lane == 0) part[warp] = v;
    __syncthreads();
    v = __reduce_add_sync(kFull, part[lane]);
    __syncthreads();
    return v;
  };
  uint32_t v = 0;
  for (uint32_t j = threadIdx.x; j < blockIdx.x; j += kLpChunk) v += a.left[j];
  const uint32_t before = block_sum(v);
  const uint32_t i = blockIdx.x * kLpChunk + threadIdx.x;
  const bool left = left_over(a, i);
  const unsigned m = __ballot_sync(kFull, left);
  if (lane == 0) part[warp] = __popc(m);
  __syncthreads();
  const uint32_t mine = __reduce_add_sync(kFull, lane < warp ? part[lane] : 0u);
  if (left) a.pend[before + mine + __popc(m & ((1u << lane) - 1u))] = a.n_mac + i;
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kLpChunk - 1) {
    const uint32_t npend = before + mine + __popc(m), ties = a.st->ties, units = a.n - a.n_mac;
    a.st->npend = npend;
    const bool tied = 64ull * ties >= units && 5ull * ties >= npend;  // (the rule: at k_lp_lists)
    if (tied) a.st->tied = 1u;
    if (tied || !few_left(a)) cudaGraphSetConditional(a.many, 1u);
  }
}

// Undoes the claims of the unit cells when too many are left over.
__global__ void __launch_bounds__(256) k_lp_undo(const LpArgs a) {
  const int lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0 && a.st->tied) cudaGraphSetConditional(a.windows, 1u);
  const int nseg = a.SW * a.H;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nseg; i += (gridDim.x * blockDim.x) >> 5) {
    const bool open = a.own[(size_t)32 * i + lane] >= (int32_t)a.n_mac;  // (kNone too)
    if (open) a.own[(size_t)32 * i + lane] = kNone;
    const unsigned m = __ballot_sync(kFull, open);
    if (lane == 0) a.seg[i] = make_uint2(m, ~0u);
  }
}

// The search over the whole chip by the CTA, none of cost below c0 being
// open: rows outward from the target, sixteen per warp and pass, two lanes a
// row, one for each direction, from the circle of cost c0 on.  A lane first
// walks the segments away from the target to the first site that nobody holds
// (their bits alone); the least of these bounds the cost for the whole CTA
// (*least).  Then it looks for a site held by a later cell that is cheaper
// still, in the segments where there can be one, within the bound.  Bounds
// are FP32 costs; the few sites within them are costed in FP64.  Bound by the latency of a pass (a few
// hundred instructions, two or three loads from L2).  Returns this lane's best.
constexpr int kUnitWarps = 16;
__device__ Best search_rows(const LpArgs &a, int32_t q, const Cell &c, double c0, int warp, int lane,
                            unsigned *least) {
  Best b = no_best();
  const bool right = lane & 1;
  const int dir = right ? 1 : -1;
  const float tx = (float)c.tx, ty = (float)c.ty, low = (float)c0 * kUnder;
  const int rows = max(c.cy, a.H - 1 - c.cy);  // rows on the longer side
  // a pass covers the rows at distance p0 .. p0 + 8 kUnitWarps - 1; every
  // row from there on is at least p0 - 1/2 away
  float most = __uint_as_float(*(volatile unsigned *)least);
  for (int p0 = 0; p0 <= rows; p0 += 8 * kUnitWarps) {
    // (most is the same in every thread here: read between the pass's barriers)
    if (p0 && ((float)p0 - 0.5f) * ((float)p0 - 0.5f) > most) break;
    // rows m0, -(m0 + 1), m0 + 1, -(m0 + 2), ... of cy, and cy itself once
    const int k = (lane >> 1) + 2 * (p0 + 8 * warp);
    const int y = c.cy + ((k & 1) ? -(k + 1) / 2 : k / 2);
    const float dy = (float)y - ty, dy2 = dy * dy;
    int x = right ? c.fx + 1 : c.fx;
    if (low > dy2) {
      const float d = fast_sqrt(low - dy2) - 0.01f;
      x = right ? max(x, (int)ceilf(tx + d)) : min(x, (int)floorf(tx - d));
    }
    float dx = (float)x - tx;
    const bool in = y >= 0 && y < a.H && x >= 0 && x < a.W && dx * dx + dy2 <= most;
    const unsigned side0 = right ? ~0u << (x & 31) : ~0u >> (31 - (x & 31));  // of the first segment
    const int g0 = x >> 5;
    const uint2 *row = a.seg + (size_t)y * a.SW;
    // Sites that nobody holds; late: bit u: the u-th segment of the walk has
    // a claim of a later cell, bit 31: one from the 31st on has.
    const bool in1 = in && g0 + dir >= 0 && g0 + dir < a.SW;
    const uint2 s0 = in ? ld_seg(row + g0) : make_uint2(0u, ~0u);
    const uint2 s1 = in1 ? ld_seg(row + g0 + dir) : make_uint2(0u, ~0u);
    unsigned m = s0.x & side0;
    unsigned late = ((int32_t)s0.y > q ? 1u : 0u) | (!m && (int32_t)s1.y > q ? 2u : 0u);
    int g = g0;
    if (!m) {
      m = s1.x;
      g += dir;
    }
    bool go = in1 && !m;
    auto site_cost = [&] {  // of the site found, if any
      x = right ? 32 * g + __ffs(m) - 1 : 32 * g + 31 - __clz(m);
      dx = (float)x - tx;
      return m ? dx * dx + dy2 : kInf;
    };
    auto bound = [&](float cost) {
      const unsigned all = __reduce_min_sync(kFull, __float_as_uint(cost * kOver));
      if (lane == 0 && all < __float_as_uint(most)) atomicMin(least, all);
    };
    if (__any_sync(kFull, go)) bound(site_cost());
    for (int i = 2; __any_sync(kFull, go); ++i) {
      most = __uint_as_float(*(volatile unsigned *)least);
      if (go) {
        g += dir;
        dx = (float)(right ? 32 * g : 32 * g + 31) - tx;  // the segment's nearest site
        go = g >= 0 && g < a.SW && dx * dx + dy2 <= most;
        if (go) {
          const uint2 s = ld_seg(row + g);
          if ((int32_t)s.y > q) late |= 1u << min(i, 31);
          m = s.x;
          go = !m;
        }
      }
    }
    const float cost = site_cost();
    bound(cost);
    __syncthreads();
    most = __uint_as_float(*(volatile unsigned *)least);
    if (cost * kUnder <= most && m) b.take(__dadd_rn(col_dx2(c, x), row_dy2(c, y)), y * a.W + x);
    // Sites held by later cells, nearest segment first, columns within the bound.
    const float left = most - dy2;
    go = in && late && left >= 0.0f;
    if (__any_sync(kFull, go)) {
      const float reach = fast_sqrt(fmaxf(left, 0.0f)) + 0.01f;
      const int last = right ? (int)fminf(floorf(tx + reach), (float)(32 * a.SW - 1))
                             : (int)fmaxf(ceilf(tx - reach), 0.0f);
      while (go) {
        const int i = __ffs(late) - 1;
        late &= late - 1;
        for (int j = i; go; ++j) {  // one segment, or all from the 31st on
          const int at = g0 + j * dir, end = last - 32 * at;  // the bound's column in the segment
          go = at >= 0 && at < a.SW && (right ? end >= 0 : end <= 31);
          if (!go) break;
          const unsigned within = right ? ~0u >> (31 - min(end, 31)) : ~0u << max(end, 0);
          const unsigned ask = j ? within : within & side0;
          const unsigned n = ask ? open_sites(own_at(a, 32 * at, y), ask, q) & ask : 0u;
          if (n) {
            const int ox = right ? 32 * at + __ffs(n) - 1 : 32 * at + 31 - __clz(n);
            b.take(__dadd_rn(col_dx2(c, ox), row_dy2(c, y)), y * a.W + ox);
            go = false;
          }
          if (i < 31) break;
        }
        go = go && late;
      }
      // what was found bounds the next passes
      const unsigned now = __reduce_min_sync(kFull, __float_as_uint(__double2float_ru(b.cost) * kOver));
      if (lane == 0 && now < __float_as_uint(most)) atomicMin(least, now);
    }
    __syncthreads();
    most = __uint_as_float(*(volatile unsigned *)least);
    __syncthreads();  // read before the next pass lowers it
  }
  return b;
}

// The open sites of cost `best` (the least) to best + ring_of, by the whole CTA,
// unsorted: the next answers of this cell, should it be displaced.  Sites
// cheaper than `best` are closed, so only the few columns of each row between
// the two circles are looked at.  *count may exceed kLpRingMax: too many to
// keep.
// Wide enough for some ten to thirty sites: a cell at the rim of a pile of
// radius r has open sites on one side only, in a ring of 1 to 2 sites' width.
__device__ __forceinline__ float ring_of(double best) { return 60.0f + 2.4f * fast_sqrt((float)best); }

__device__ void list_ring(const LpArgs &a, int32_t q, const Cell &c, double best, float ring, int warp, int lane,
                          Best *list, int *count) {
  const bool right = lane & 1;
  const int dir = right ? 1 : -1;
  const float tx = (float)c.tx, ty = (float)c.ty, low = (float)best * kUnder;
  const float most = (float)best * kOver + ring;
  const int rows = max(c.cy, a.H - 1 - c.cy);
  for (int p0 = 0; p0 <= rows; p0 += 8 * kUnitWarps) {
    if (p0 && ((float)p0 - 0.5f) * ((float)p0 - 0.5f) > most) break;
    const int k = (lane >> 1) + 2 * (p0 + 8 * warp);
    const int y = c.cy + ((k & 1) ? -(k + 1) / 2 : k / 2);
    const float dy = (float)y - ty, dy2 = dy * dy, left = most - dy2;
    if (y < 0 || y >= a.H || left < 0.0f) continue;
    int x = right ? c.fx + 1 : c.fx;
    if (low > dy2) {
      const float d = fast_sqrt(low - dy2) - 0.01f;
      x = right ? max(x, (int)ceilf(tx + d)) : min(x, (int)floorf(tx - d));
    }
    const float reach = fast_sqrt(left) + 0.01f;
    const int last = right ? (int)fminf(floorf(tx + reach), (float)(a.W - 1)) : (int)fmaxf(ceilf(tx - reach), 0.0f);
    if (right ? x > last || x >= a.W : x < last || x < 0) continue;
    for (int g = x >> 5; right ? g <= last >> 5 : g >= last >> 5; g += dir) {
      const int lo = max((right ? x : last) - 32 * g, 0), hi = min((right ? last : x) - 32 * g, 31);
      const unsigned ask = (~0u << lo) & (~0u >> (31 - hi));
      const uint2 s = ld_seg(a.seg + (size_t)y * a.SW + g);
      unsigned m = ((int32_t)s.y > q ? open_sites(own_at(a, 32 * g, y), ask, q) : s.x) & ask;
      while (m) {
        const int at = 32 * g + __ffs(m) - 1;
        m &= m - 1;
        const double cost = __dadd_rn(col_dx2(c, at), row_dy2(c, y));
        if (cost > best + (double)ring) continue;
        const int n = atomicAdd(count, 1);
        if (n < kLpRingMax) list[n] = Best{cost, y * a.W + at};
      }
    }
  }
}

// Sorts the (at most 32) entries, one per lane; lane l then has the l-th.
__device__ __forceinline__ Best warp_sorted(Best b) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      Best o;
      o.cost = __shfl_xor_sync(kFull, b.cost, j);
      o.tile = __shfl_xor_sync(kFull, b.tile, j);
      const bool less = o.cost < b.cost || (o.cost == b.cost && o.tile < b.tile);
      const bool low = ((lane & j) == 0) == ((lane & k) == 0);  // this lane keeps the smaller one
      if (less == low) b = o;
    }
  return b;
}

// A CTA per unit cell (kAll: each CTA has one; else those left over, taken up
// in order), and the cells that its claim displaces one after the other.  What
// takes the time is the chain of cells that each take a site from the next
// (about a thousand cells at the rims of a 200k-cell design's piles), so one
// answer is made short: one warp, with no barrier, finds an answer near the
// target, and that of a displaced cell in the list its search left (closed
// sites stay closed, so the first one still open is the best); any other
// search takes all 16 warps, and lists the sites next in cost for a later
// displacement.  CTAs start in about the order of the cells, so a claim is
// displaced only by a cell that was under way at the same time; several cells
// per CTA, or a warp for each, put more cells under way and displace more
// claims.  Units of a 200k-cell checkpoint, half of the cells in six piles:
// 4.9 ms and 117k searches of the whole CTA; without the lists 7.5 ms and 283k;
// without them and with 2 / 4 / 8 cells per CTA 13.4 / 20 / 30 ms, with a warp
// per cell 27 to 70 ms.
struct UnitShared {
  Best best[kUnitWarps], list[kLpRingMax];
  unsigned least;
  int count;
  // the cell under way: index, target, cost below which no site is open
  int32_t q;
  float2 pos;
  double c0;
};

// Nothing to do for a legalisation that failed or is not wanted (a warp).
__device__ __forceinline__ bool wanted(const LpArgs &a, int lane) {
  const bool off = ld_own(a.cancel) != 0;
  if (off && lane == 0) atomicMax(&a.st->status, 4);
  return !off && ld_own(&a.st->status) == 0;
}

// Warp 0: cell q and the cells that its claims displace, one after the other,
// while one warp can tell; listed: q has lost site (px, py) and may have a
// list.  Returns -1 when all have a site, else the cell that needs a search of
// the whole CTA (its target and c0 are entered).
__device__ __forceinline__ int32_t settle(const LpArgs &a, UnitShared &sh, int32_t q, bool &listed, int &px, int &py,
                                          int lane) {
  while (q >= 0) {
    double c0 = 0.0;
    float2 p;
    if (listed) {
      const int32_t *l = a.cand + (size_t)kLpCand * (q - (int32_t)a.n_mac);
      const int32_t t = lane < kLpCand ? ld_own(l + lane) : -1;
      const unsigned ends = __ballot_sync(kFull, t < 0);  // the list ends at its first -1
      const int len = __ffs(ends) - 1;
      const int x = t % a.W, y = t / a.W;
      const int32_t on = lane < len ? ld_own(own_at(a, x, y)) : -1;
      const uint2 s = lane < len ? ld_seg(seg_at(a, x, y)) : make_uint2(0u, 0u);
      const unsigned open = __ballot_sync(kFull, on > q);
      if (open) {
        const int l0 = __ffs(open) - 1;
        px = __shfl_sync(kFull, x, l0);
        py = __shfl_sync(kFull, y, l0);
        const uint2 seen = make_uint2(__shfl_sync(kFull, s.x, l0), __shfl_sync(kFull, s.y, l0));
        const int32_t held = claim_and_acquire(a, q, px, py, seen, lane);
        if (held == kNone) q = -1;
        else if (held > q) q = held;
        continue;  // (an earlier cell was faster: the list again)
      }
      p = a.pos[a.order[q]];
      const Cell c = make_cell(a, p, make_uchar2(1, 1));
      if (len > 0) {  // all of it closed, as everything cheaper
        px = __shfl_sync(kFull, x, len - 1);
        py = __shfl_sync(kFull, y, len - 1);
      }
      if (c.inside) c0 = __dadd_rn(col_dx2(c, px), row_dy2(c, py));
    } else {
      p = a.pos[a.order[q]];
      c0 = get_hint(a, q, make_cell(a, p, make_uchar2(1, 1)));
    }
    listed = false;
    const Cell c = make_cell(a, p, make_uchar2(1, 1));
    if (c0 < 6.25 && placeable(c)) {
      uint2 seen;
      const Best b = search_near(a, q, c, lane, &seen);
      if (b.cost < 6.25) {
        px = b.tile % a.W;
        py = b.tile / a.W;
        const int32_t held = claim_and_acquire(a, q, px, py, seen, lane);
        if (held == kNone) {
          q = -1;
        } else if (held > q) {
          q = held;
          listed = true;
        }
        continue;
      }
    }
    if (lane == 0) {
      sh.pos = p;
      sh.c0 = c0;
      sh.least = __float_as_uint(kInf);
      sh.count = 0;
    }
    break;
  }
  return q;
}

// The search for cell q by the whole CTA, and the sites next in cost listed.
__device__ __forceinline__ Best search_cta(const LpArgs &a, UnitShared &sh, int32_t q, const Cell &c, float &ring,
                                           int warp, int lane) {
  Best b = no_best();
  if (placeable(c)) b = search_rows(a, q, c, sh.c0, warp, lane, &sh.least);
  b = b.warp_min();
  if (lane == 0) sh.best[warp] = b;
  __syncthreads();
  b = (lane < kUnitWarps ? sh.best[lane] : no_best()).warp_min();
  if (ring == 0.0f) ring = ring_of(b.cost);
  if (b.tile != kNone) list_ring(a, q, c, b.cost, ring, warp, lane, sh.list, &sh.count);
  __syncthreads();
  return b;
}

// Warp 0: leaves the cheapest 32 or fewer entries of the list, the ring (below
// 2^26) halved until they are.  Returns how many; -1: no list.
__device__ __forceinline__ int shrink_list(UnitShared &sh, const Best &b, int lane, double &ring) {
  const int n = sh.count;
  Best e0 = lane < n ? sh.list[lane] : no_best(), e1 = lane + 32 < n ? sh.list[lane + 32] : no_best();
  unsigned m0 = 0, m1 = 0;
  for (int k = 0; k < 37; ++k) {
    m0 = __ballot_sync(kFull, e0.cost <= b.cost + ring);
    m1 = __ballot_sync(kFull, e1.cost <= b.cost + ring);
    if (__popc(m0) + __popc(m1) <= 32 || ring < 1e-3) break;
    ring *= 0.5;
  }
  const unsigned below = (1u << lane) - 1;
  const int i0 = __popc(m0 & below), i1 = __popc(m0) + __popc(m1 & below);
  __syncwarp();
  if ((m0 >> lane & 1) && i0 < 32) sh.list[i0] = e0;
  if ((m1 >> lane & 1) && i1 < 32) sh.list[i1] = e1;
  __syncwarp();
  const int m = __popc(m0) + __popc(m1);
  return n <= kLpRingMax && m <= 32 ? m : -1;
}

// Warp 0: q's list and claim of its best site b.  Returns the cell to go on
// with (displaced, or q itself where an earlier cell was faster), -1: none.
__device__ __forceinline__ int32_t list_and_claim(const LpArgs &a, UnitShared &sh, int32_t q, const Cell &c,
                                                  const Best &b, double ring, int &px, int &py, int lane) {
  px = b.tile % a.W;
  py = b.tile / a.W;
  const uint2 seen = ld_seg(seg_at(a, px, py));
  const int m = shrink_list(sh, b, lane, ring);
  const Best e = m >= 0 ? warp_sorted(lane < m ? sh.list[lane] : no_best()) : no_best();
  if (lane < kLpCand)
    a.cand[(size_t)kLpCand * (q - (int32_t)a.n_mac) + lane] =
        m >= 0 && e.tile != kNone ? e.tile : lane == 0 && m < 0 ? b.tile : -1;
  __syncwarp();
  if (lane == 0) {
    put_hint(a, q, c, b.cost);
    __threadfence();  // the list before the claim: who displaces q reads it
  }
  const int32_t held = claim_and_acquire(a, q, px, py, seen, lane);
  return held == kNone ? -1 : held > q ? held : q;
}

template <bool kAll>
__global__ void __launch_bounds__(kUnitWarps * 32, 32 / kUnitWarps) k_lp_units(const LpArgs a) {
  __shared__ UnitShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int32_t next = -1;    // warp 0: the cell to place, -1: none
  bool listed = false;  // it may have a list
  int px = 0, py = 0;   // a displaced cell: the site it lost
  if (a.st->tied || (!kAll && !few_left(a))) return;
  bool fresh = true;  // no cell under way
  if (kAll && warp == 0 && wanted(a, lane)) next = (int32_t)(a.n_mac + blockIdx.x);
  while (true) {
    if (!kAll && warp == 0 && fresh) {
      uint32_t item = 0;
      if (lane == 0) item = atomicAdd(&a.st->taken, 1u);
      item = __shfl_sync(kFull, item, 0);
      next = item < a.st->npend && wanted(a, lane) ? (int32_t)a.pend[item] : -1;
      listed = false;
    }
    if (warp == 0) {
      const int32_t q = settle(a, sh, next, listed, px, py, lane);
      // (-1: done; -2: there may be others to take up)
      if (lane == 0) sh.q = q >= 0 || kAll || (fresh && next < 0) ? q : -2;
    }
    __syncthreads();
    const int32_t q = sh.q;
    if (kAll ? q < 0 : q == -1) return;
    if (!kAll) {
      fresh = q < 0;
      if (fresh) {
        __syncthreads();  // read before it changes
        continue;
      }
    }
    const Cell c = make_cell(a, sh.pos, make_uchar2(1, 1));
    float ring = 0.0f;
    const Best b = search_cta(a, sh, q, c, ring, warp, lane);
    if (b.tile == kNone) {  // no site is open to it
      if (tid == 0) atomicMax(&a.st->status, 1);
      return;
    }
    if (warp == 0) {
      next = list_and_claim(a, sh, q, c, b, ring, px, py, lane);
      listed = true;
    }
  }
}

// Cells on one target.  Above, those under way want the same site: all but the
// first lose it and search again, and so does who is displaced from it (13 us
// each).  So where many share a target (positions clamped into a corner of the
// chip, as the reference's field leaves them), the unit cells are placed in
// windows of the next ones in order instead, whose searches see a map that does
// not change: first each cell's list, then each takes of its list what the
// cells before it leave.  A window ends early at the first cell whose list is
// used up: after some 50 cells of one target.
// ms, in order without windows -> with (in brackets as rounds of lists and a
// serial pass, before deferred acceptance), unit cells alone: all on one spot 1k 11.0
// -> 0.9 (2.2), 30k 419 -> 27 (87), 200k 3697 -> 192 (1173); 40 % in a corner,
// the others spread: 5k 17 -> 2.1 (6.5), 60k 308 -> 24 (84).  Runs with the
// reference's field, 5k cells, 300 iterations 1297 -> 31 (48), 30k with macros,
// 100 iterations, 4568 -> 290 (285).  Bound by the list kernel: two dependent
// passes over the rows, 20 us a window, and two launches.
// The rule (k_lp_pending): ties (cells of a target that has 1/64 of all or more)
// are at least 1/64 of the unit cells and 1/5 of those left over by k_lp_near; or,
// where that isn't tried, 1/10 of a sample (sample_ties).  The line lies
// where both ways take about as long: 200k cells, 2 % in a corner 29 -> 18 ms,
// 30k 2.8 -> 2.6; 16 spots of 30k cells 23 -> 3.4; but a wide pile of 30k cells
// of which 10 % are on one spot would take 14 -> 70 (40 %: 86 -> 64): its other
// cells use up their lists too.  A loop that is not entered costs some 12 us, so
// it stands inside the if node where there is one, and few cells have a second
// graph for it (a run's first such checkpoint, and each call, is launched twice).

// A CTA per cell of the window: the open sites of least cost, in order.
__global__ void __launch_bounds__(kUnitWarps * 32, 32 / kUnitWarps) k_lp_lists(const LpArgs a) {
  __shared__ UnitShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t i = a.st->wbase + blockIdx.x;
  if (i >= a.n - a.n_mac || a.st->status != 0) return;
  const int32_t q = (int32_t)(a.n_mac + i);
  const Cell c = load_cell(a, (uint32_t)q, true);
  if (tid == 0) {
    sh.c0 = get_hint(a, q, c);
    sh.least = __float_as_uint(kInf);
    sh.count = 0;
  }
  __syncthreads();
  // A ring of cost w round the best site holds about pi w open sites, half or a
  // quarter of that at an edge or in a corner: another width where too few or
  // too many are found.
  float ring = 16.0f;
  const Best b = search_cta(a, sh, q, c, ring, warp, lane);
  int n = sh.count;
  for (int k = 0; k < 3 && b.tile != kNone && (n > kLpRingMax || n < 24); ++k) {
    __syncthreads();
    if (tid == 0) sh.count = 0;
    __syncthreads();
    ring *= 44.0f / (float)max(n, 1);
    list_ring(a, q, c, b.cost, ring, warp, lane, sh.list, &sh.count);
    __syncthreads();
    n = sh.count;
  }
  if (n > kLpRingMax) {  // too many sites tie
    __syncthreads();
    if (tid == 0) sh.list[0] = b;
    __syncthreads();
    n = 1;
  }
  if (b.tile == kNone) n = 0;
  if (tid < n) {
    const Best e = sh.list[tid];
    int k = 0;
    for (int t = 0; t < n; ++t) {
      const Best o = sh.list[t];
      k += o.cost < e.cost || (o.cost == e.cost && o.tile < e.tile) ? 1 : 0;
    }
    a.list[kLpRingMax * blockIdx.x + k] = e.tile;
  }
  if (tid == 0) a.list_len[blockIdx.x] = n;
}

// One CTA, a thread per cell of the window: each onto the first entry of its
// list that no earlier cell of the window takes (everything cheaper was closed,
// everything off the list costs more), again by deferred acceptance: who has
// lost its site to an earlier cell goes on to its next entry.  The cells before
// the first whose entries are all lost are final; the next window begins there.
constexpr int kTakenBits = kUnitWindowBits + 2;  // table of the sites proposed to (each is held by some cell)
__global__ void __launch_bounds__(kUnitWindow) k_lp_take(const LpArgs a) {
  extern __shared__ int32_t list[];  // [kUnitWindow][kLpRingMax + 1]: no two cells' entries in one bank
  __shared__ int32_t site[1 << kTakenBits], holder[1 << kTakenBits];
  __shared__ int done;
  LpState *st = a.st;
  const int tid = threadIdx.x;
  const uint32_t units = a.n - a.n_mac, base = st->wbase;
  const int count = (int)min(kUnitWindow, units - base);
  if (st->status == 0) {
    for (int k = tid; k < 1 << kTakenBits; k += kUnitWindow) {
      site[k] = -1;
      holder[k] = kNone;
    }
    for (int k = tid; k < count * kLpRingMax; k += kUnitWindow)
      list[k + k / kLpRingMax] = a.list[k];
    if (tid == 0) done = count;
    const int len = tid < count ? a.list_len[tid] : 0;
    __syncthreads();
    int at = 0;          // entry of the list
    int32_t where = -1;  // its place in the table
    bool propose = tid < count;
    while (true) {
      if (propose && at < len) {
        const int32_t t = list[tid * (kLpRingMax + 1) + at];
        uint32_t h = ((uint32_t)t * 2654435761u) >> (32 - kTakenBits);
        while (true) {
          const int32_t was = atomicCAS(&site[h], -1, t);
          if (was == -1 || was == t) break;
          h = (h + 1) & ((1u << kTakenBits) - 1u);
        }
        where = (int32_t)h;
        atomicMin(&holder[h], tid);
      }
      __syncthreads();
      propose = tid < count && at < len && holder[where] != tid;
      if (propose) ++at;
      if (!__syncthreads_or(propose)) break;
    }
    if (tid < count && at >= len) atomicMin(&done, tid);
    __syncthreads();
    if (tid < done) {
      const int32_t q = (int32_t)(a.n_mac + base) + tid, t = site[where];
      const int x = t % a.W, y = t / a.W;
      const Cell c = load_cell(a, (uint32_t)q, true);
      *own_at(a, x, y) = q;
      atomicAnd(&seg_at(a, x, y)->x, ~(1u << (x & 31)));
      put_hint(a, q, c, __dadd_rn(col_dx2(c, x), row_dy2(c, y)));
    }
    if (tid == 0) {
      st->wbase = base + (uint32_t)done;
      if (done == 0) atomicMax(&st->status, 1);  // the first cell's list is empty: no site is open to it
    }
  }
  __syncthreads();
  if (tid != 0) return;
  if (ld_own(a.cancel)) atomicMax(&st->status, 4);
  if (st->wbase >= units || atomicAdd(&st->status, 0) != 0) cudaGraphSetConditional(a.windows, 0u);
}

// ---------------------------------------------------------------------------
// Results
// ---------------------------------------------------------------------------
__device__ __forceinline__ void put_result(const LpArgs &a, uint32_t q, int t, bool unit) {
  const Cell c = load_cell(a, q, unit);
  const int ax = t % a.W, ay = t / a.W;
  const uint32_t cell = a.order[q];
  a.sites[cell] = make_int2(ax, ay);
  if (a.loc) a.loc[cell] = make_int2(ax + (c.w - 1) / 2, ay + (c.h - 1) / 2);
  a.cost[q] = __dadd_rn(col_dx2(c, ax), row_dy2(c, ay));
}

__global__ void __launch_bounds__(256) k_lp_result(const LpArgs a) {
  if (a.st->status != 0) return;
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, ts = gridDim.x * blockDim.x;
  for (uint32_t q = t0; q < a.n_mac; q += ts) put_result(a, q, a.choice[q], false);
  const uint32_t pitch = 32u * (uint32_t)a.SW, sites = pitch * (uint32_t)a.H;
  for (uint32_t s = t0; s < sites; s += ts) {
    const int32_t q = a.own[s];
    if (q < (int32_t)a.n_mac || q == kNone) continue;
    const uint32_t y = s / pitch;
    put_result(a, (uint32_t)q, (int)(y * (uint32_t)a.W + (s - y * pitch)), true);
  }
}

// A run of additions to a total of t units in the last place: the units added
// when t is even and when it is odd.  Counts saturate above 2^53, where the
// total would leave its binade.
struct AddRun {
  unsigned long long even, odd;
};
constexpr unsigned long long kTop = 1ull << 53;
__device__ __forceinline__ unsigned long long sat(unsigned long long v) { return v < kTop ? v : kTop; }
__device__ __forceinline__ AddRun then(const AddRun &f, const AddRun &g) {  // f first
  return AddRun{sat(f.even + ((f.even & 1) ? g.odd : g.even)), sat(f.odd + ((f.odd & 1) ? g.even : g.odd))};
}
// v >= 0 added to a total whose unit in the last place is 1 / scale:
// v in units is v * scale, exact (a power of two).
__device__ __forceinline__ AddRun add_one(double v, double scale) {
  const double u = __dmul_rn(v, scale);
  if (!(u < 9007199254740992.0)) return AddRun{kTop, kTop};
  const double fl = floor(u), fr = __dsub_rn(u, fl);
  const unsigned long long n = (unsigned long long)fl;
  if (fr < 0.5) return AddRun{n, n};
  if (fr > 0.5) return AddRun{n + 1, n + 1};
  return (n & 1) ? AddRun{n + 1, n} : AddRun{n, n + 1};  // half way: to the even total
}

constexpr int kSumThreads = 1024, kSumEach = 8;

// The displacement, one CTA: the first costs one after the other (the total
// soon leaves its binade there), then 8192 a step.  The first addition that
// leaves the binade (or the first cost that is not zero, while the total is)
// is made as it stands and the next step starts after it: nine or ten times in
// 200k costs.  0.4 ms with every cost in steps.
constexpr uint32_t kSumFirst = 512;
__global__ void __launch_bounds__(kSumThreads) k_lp_finish(const LpArgs a) {
  __shared__ AddRun wrun[32];
  __shared__ double total;
  __shared__ uint32_t stop;  // first cost of the step that has to be added by itself
  __shared__ double next;    // the total after it, or after the whole step
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool ok = a.st->status == 0;
  uint32_t at = min(a.n, kSumFirst);
  if (w == 0) {
    double t = 0.0;
    for (uint32_t i = 0; ok && i < at; i += 32) {
      const double v = i + lane < at ? __ldcg(a.cost + i + lane) : 0.0;  // + 0.0 leaves the total
#pragma unroll
      for (int l = 0; l < 32; ++l) t = __dadd_rn(t, __shfl_sync(kFull, v, l));
    }
    if (lane == 0) total = t;
  }
  __syncthreads();
  while (ok && at < a.n) {
    const double t0 = total;
    if (tid == 0) stop = 0xffffffffu;
    double v[kSumEach];
    const uint32_t i0 = at + (uint32_t)tid * kSumEach;
#pragma unroll
    for (int k = 0; k < kSumEach; ++k) v[k] = i0 + k < a.n ? __ldcg(a.cost + i0 + k) : 0.0;
    __syncthreads();  // total read, stop set
    if (t0 == 0.0) {
#pragma unroll
      for (int k = kSumEach - 1; k >= 0; --k)
        if (v[k] != 0.0) atomicMin(&stop, i0 + k);
      __syncthreads();
      if (stop != 0xffffffffu && stop - i0 < kSumEach) {
#pragma unroll
        for (int k = 0; k < kSumEach; ++k)
          if (i0 + k == stop) total = v[k];
      }
    } else {
      // unit in the last place of t0: 2^(e - 52) for 2^e <= t0 < 2^(e + 1)
      const int e = ilogb(t0);
      const double unit = scalbn(1.0, e - 52), scale = scalbn(1.0, 52 - e);
      AddRun f[kSumEach];
      AddRun mine{0, 0};
#pragma unroll
      for (int k = 0; k < kSumEach; ++k) {
        f[k] = add_one(v[k], scale);
        mine = then(mine, f[k]);
      }
      // exclusive scan over the threads, in order
      AddRun inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        AddRun p;
        p.even = __shfl_up_sync(kFull, inc.even, o);
        p.odd = __shfl_up_sync(kFull, inc.odd, o);
        if (lane >= o) inc = then(p, inc);
      }
      AddRun ex;
      ex.even = __shfl_up_sync(kFull, inc.even, 1);
      ex.odd = __shfl_up_sync(kFull, inc.odd, 1);
      if (lane == 0) ex = AddRun{0, 0};
      if (lane == 31) wrun[w] = inc;
      __syncthreads();
      if (w == 0) {
        AddRun x = wrun[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          AddRun p;
          p.even = __shfl_up_sync(kFull, x.even, o);
          p.odd = __shfl_up_sync(kFull, x.odd, o);
          if (lane >= o) x = then(p, x);
        }
        wrun[lane] = x;
      }
      __syncthreads();
      if (w) ex = then(wrun[w - 1], ex);
      const unsigned long long base = (unsigned long long)__dmul_rn(t0, scale);  // 2^52 .. 2^53 - 1
      unsigned long long t = base + ((base & 1) ? ex.odd : ex.even);
      unsigned long long before = t;
      int out = -1;
#pragma unroll
      for (int k = 0; k < kSumEach; ++k) {
        if (out >= 0) continue;
        before = t;
        t += (t & 1) ? f[k].odd : f[k].even;
        if (t >= kTop) out = k;
      }
      if (out >= 0) atomicMin(&stop, i0 + out);
      __syncthreads();
      if (out >= 0 && i0 + out == stop) {
        double add = 0.0;
#pragma unroll
        for (int k = 0; k < kSumEach; ++k)
          if (k == out) add = v[k];
        next = __dadd_rn(__dmul_rn((double)before, unit), add);
      }
      if (stop == 0xffffffffu && tid == kSumThreads - 1) next = __dmul_rn((double)t, unit);
      __syncthreads();
      if (tid == 0) total = next;
    }
    __syncthreads();
    at = stop != 0xffffffffu ? stop + 1 : at + kSumThreads * kSumEach;
    __syncthreads();  // stop read before it is set again
  }
  if (tid == 0) {
    *a.disp = total;
    *a.status = a.st->status;
  }
}

}  // namespace

void LpGraph::clear() {
  if (exec) cudaGraphExecDestroy(exec);
  if (graph) cudaGraphDestroy(graph);
  exec = nullptr;
  graph = nullptr;
}

cudaError_t lp_build_graph(LpArgs a, LpGraph &g, bool windows) {
  g.clear();
  cudaError_t e;
  cudaGraph_t graph = nullptr;
  if ((e = cudaGraphCreate(&graph, 0)) != cudaSuccess) return e;
  g.graph = graph;
  // Nodes of a graph, one after the other.
  struct Chain {
    cudaGraph_t graph;
    cudaGraphNode_t tail = nullptr;
  };
  auto add = [&](Chain &c, void (*func)(LpArgs), unsigned grid, unsigned block, unsigned shared = 0) -> cudaError_t {
    void *args[] = {&a};
    cudaKernelNodeParams kp = {};
    kp.func = reinterpret_cast<void *>(func);
    kp.gridDim = dim3(grid);
    kp.blockDim = dim3(block);
    kp.sharedMemBytes = shared;
    kp.kernelParams = args;
    cudaGraphNode_t node;
    const cudaError_t r = cudaGraphAddKernelNode(&node, c.graph, c.tail ? &c.tail : nullptr, c.tail ? 1 : 0, &kp);
    c.tail = node;
    return r;
  };
  auto add_cond = [&](Chain &c, cudaGraphConditionalHandle handle, cudaGraphConditionalNodeType type, Chain *body) {
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = type;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    const cudaError_t r = cudaGraphAddNode(&node, c.graph, c.tail ? &c.tail : nullptr, c.tail ? 1 : 0, &cp);
    c.tail = node;
    if (r == cudaSuccess) body->graph = cp.conditional.phGraph_out[0];
    return r;
  };
  auto handle = [](cudaGraphConditionalHandle *h, const Chain &c, unsigned value) {
    return cudaGraphConditionalHandleCreate(h, c.graph, value, cudaGraphCondAssignDefault);
  };
  // (grids of 8, 4 and 2 CTAs for each of this chip's 148 SMs: what is resident;
  // the kernels loop, so any other number gives the same)
  const size_t sites = (size_t)a.W * a.H;
  const unsigned site_grid = (unsigned)((sites + 255) / 256 < 1184 ? (sites + 255) / 256 : 1184);
  const uint32_t units = a.n - a.n_mac;
  constexpr unsigned kTakeShared = (unsigned)(sizeof(int32_t) * kUnitWindow * (kLpRingMax + 1));
  if ((e = cudaFuncSetAttribute(k_lp_take, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTakeShared)) !=
      cudaSuccess)
    return e;
  const bool at_once = units >= kNearFrom;
  // Few cells: targets that differ by less than a tenth of a site crowd like equal
  // ones (5k in a pile of sigma 0.1: 13.7 -> 7.0 ms, but 60k 135 -> 230).
  a.tie_scale = at_once ? 64.0f : 16.0f;
  a.tie_least = units / 64;
  a.tie_few = units && !at_once;
  a.tie_loop = at_once || windows;
  Chain top{graph};
  // The loop over the windows of unit cells, entered when some kernel of the
  // chain before it has set its handle.
  auto add_windows = [&](Chain &c) -> cudaError_t {
    Chain body{};
    cudaError_t r;
    if ((r = add_cond(c, a.windows, cudaGraphCondTypeWhile, &body)) != cudaSuccess) return r;
    if ((r = add(body, k_lp_lists, units < kUnitWindow ? units : kUnitWindow, kUnitWarps * 32)) != cudaSuccess) return r;
    return add(body, k_lp_take, 1, kUnitWindow, kTakeShared);
  };
  if (a.n_mac && (e = handle(&a.handle, top, 1)) != cudaSuccess) return e;
  if (at_once && (e = handle(&a.many, top, 0)) != cudaSuccess) return e;
  if (units && !at_once && windows && (e = handle(&a.windows, top, 0)) != cudaSuccess) return e;
  if ((e = add(top, k_lp_init, site_grid, 256)) != cudaSuccess) return e;
  if (a.n_mac) {
    Chain body{};
    if ((e = add_cond(top, a.handle, cudaGraphCondTypeWhile, &body)) != cudaSuccess) return e;
    const uint32_t most = a.n_mac < kLpWindow ? a.n_mac : kLpWindow;
    if ((e = add(body, k_lp_choose, most < 592 ? most : 592, kLpWarps * 32)) != cudaSuccess) return e;
    if ((e = add(body, k_lp_claim, (most + kLpWarps - 1) / kLpWarps, kLpWarps * 32)) != cudaSuccess) return e;
  }
  if ((e = add(top, k_lp_segments, site_grid, 256)) != cudaSuccess) return e;
  if (units && !at_once) {
    if ((e = add(top, k_lp_units<true>, units, kUnitWarps * 32)) != cudaSuccess) return e;
    if (windows && (e = add_windows(top)) != cudaSuccess) return e;
  } else if (units) {
    const uint32_t chunks = (uint32_t)lp_chunks(units);
    if ((e = add(top, k_lp_near, (units + 7) / 8, 256)) != cudaSuccess) return e;
    if ((e = add(top, k_lp_count, chunks, kLpChunk)) != cudaSuccess) return e;
    if ((e = add(top, k_lp_pending, chunks, kLpChunk)) != cudaSuccess) return e;
    // too many left over, or ties: all of them again, in order or in windows
    Chain body{};
    if ((e = add_cond(top, a.many, cudaGraphCondTypeIf, &body)) != cudaSuccess) return e;
    if ((e = handle(&a.windows, body, 0)) != cudaSuccess) return e;
    if ((e = add(body, k_lp_undo, site_grid, 256)) != cudaSuccess) return e;
    if ((e = add(body, k_lp_units<true>, units, kUnitWarps * 32)) != cudaSuccess) return e;
    if ((e = add_windows(body)) != cudaSuccess) return e;
    if ((e = add(top, k_lp_units<false>, 296, kUnitWarps * 32)) != cudaSuccess) return e;
  }
  if ((e = add(top, k_lp_result, site_grid, 256)) != cudaSuccess) return e;
  if ((e = add(top, k_lp_finish, 1, kSumThreads)) != cudaSuccess) return e;
  return cudaGraphInstantiate(&g.exec, graph, 0);
}

}  // namespace eplace
