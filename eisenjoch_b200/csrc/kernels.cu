// kernels.cu -- sm_100a kernels of the ElectroPlace iteration.
//
//   k_wa            WA wirelength gradient (placer/common.rs:205-291,
//                   solver/wa.rs:51-101): nets grouped by degree class, a
//                   fixed lane-group width per class (one thread per net up
//                   to a warp per net), deterministic fixed-point scatter.
//   k_scatter       cell -> bin overlap areas (electro_place/density.rs:54-76),
//                   fixed-point atomics (order independent, bit-reproducible).
//   k_density_final sums for the overlap (density.rs:79-86), FP32 charge map
//                   for the transform, resets the accumulator.
//   k_sgemm, k_sgemm_panel
//                   FP32 DCT-matrix GEMMs (density.rs:96-166), spectral
//                   Poisson scaling fused into the second GEMM's epilogue.
//   k_step          field gather + penalty + preconditioner + Barzilai-
//                   Borwein + FISTA + clamp + next look-ahead and its scatter in one
//                   cooperative kernel (density.rs:171-206,
//                   electro_place/mod.rs:131-173, solver/nesterov.rs:41-101,
//                   :199-218).
//   k_hpwl          integer HPWL (metrics/wirelength.rs:10-51).
#include <cooperative_groups.h>

#include "kernels.cuh"

namespace eplace {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr float kLog2e = 1.4426950408889634f;
// Bound on any spin wait: ~2 s at the B200's clock (clock64 counts SM cycles).
constexpr long long kSpinCycles = 4000000000ll;

__device__ __forceinline__ unsigned long long to_fix(float v) {
  return (unsigned long long)__float2ll_rn(v * 4294967296.0f);
}
__device__ __forceinline__ double from_fix(unsigned long long v) {
  return (double)(long long)v * (1.0 / 4294967296.0);
}

struct OpMax {
  __device__ float operator()(float a, float b) const { return fmaxf(a, b); }
};
struct OpMin {
  __device__ float operator()(float a, float b) const { return fminf(a, b); }
};
struct OpAdd {
  __device__ float operator()(float a, float b) const { return a + b; }
};

template <typename Op>
__device__ __forceinline__ float warp_allreduce(float v, Op op) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Deterministic block sum of a double (fixed tree for a fixed block size),
// valid in thread 0.
__device__ __forceinline__ double block_sum_d(double v, double *smem /* [32] */) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum_d(v);
  if (lane == 0) smem[wid] = v;
  __syncthreads();
  return wid == 0 ? warp_sum_d(lane < nw ? smem[lane] : 0.0) : 0.0;
}

// Per-axis WA terms with max/min shifts.  The reference shifts by the pin
// mean (wa.rs:58); shifting the positive exponentials by the maximum and the
// negative ones by the minimum leaves value and gradient unchanged and keeps
// every exponential in (0, 1], so FP32 cannot overflow.
//   d_max_i = e+_i/S+ (1 + g (u_i - A+/S+)),  u = x - max
//   d_min_i = e-_i/S- (1 - g (v_i - A-/S-)),  v = x - min
// iSp / iSm are 1/S+ and 1/S- (one reciprocal per segment).
__device__ __forceinline__ float wa_pin_grad(float u, float v, float ep, float em, float iSp, float Ap,
                                             float iSm, float Am, float gamma) {
  const float dmax = ep * iSp * (1.0f + gamma * (u - Ap * iSp));
  const float dmin = em * iSm * (1.0f - gamma * (v - Am * iSm));
  return dmax - dmin;
}

// 2^x for x <= 0 (MUFU.EX2; subnormal results flush to zero, harmless here).
__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Reduction over the g lanes of an aligned lane group (g a power of two,
// the same on all lanes of the warp); every lane takes part.  Each xor step
// adds a pair in both orders, and FP32 addition commutes, so all lanes of a
// group get the same bits.
template <typename Op>
__device__ __forceinline__ float group_allreduce(float v, int g, Op op) {
  for (int o = g >> 1; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// Nets of one degree class: g lanes per net (32 / g nets per warp), lane l
// of a group holding pins l, l + g, ..., l + (np - 1) g of its net in
// registers (pin ids and positions gathered once; np <= P, uniform over the
// warp).  Max/min and the eight exponential sums are reduced over the group;
// the exponentials are kept for the gradient when P <= 4 and recomputed
// otherwise (register budget).  Nets with fewer than two pins contribute
// nothing (wa.rs:58).
template <int P>
__device__ __forceinline__ void wa_group(const WaArgs &a, const WaClass &cl, int g, int pp, int wi, int lane) {
  constexpr bool kKeep = P <= 4;
  const float kg = a.gamma * kLog2e;
  const int gl = lane & (g - 1);
  const int idx = wi * (32 / g) + lane / g;
  const bool valid = idx < cl.nets;
  // The lane's pp (<= P) pin slots in one vector load: no CSR offsets.
  uint32_t cc[P];
#pragma unroll
  for (int k = 0; k < P; ++k) cc[k] = 0xffffffffu;
  if (valid) {
    const uint32_t *sp = a.slots + cl.slot_base + (long long)idx * (g * pp) + gl * pp;
    if (pp == 2) {
      const uint2 v = *reinterpret_cast<const uint2 *>(sp);
      cc[0] = v.x;
      cc[1] = v.y;
    } else if (pp == 4 || P < 8) {
      const uint4 v = *reinterpret_cast<const uint4 *>(sp);
      cc[0] = v.x;
      cc[1] = v.y;
      cc[P > 2 ? 2 : 0] = P > 2 ? v.z : cc[0];
      cc[P > 3 ? 3 : 0] = P > 3 ? v.w : cc[0];
    } else {
      const uint4 v0 = *reinterpret_cast<const uint4 *>(sp), v1 = *reinterpret_cast<const uint4 *>(sp + 4);
      cc[0] = v0.x;
      cc[1] = v0.y;
      cc[P > 2 ? 2 : 0] = P > 2 ? v0.z : cc[0];
      cc[P > 3 ? 3 : 0] = P > 3 ? v0.w : cc[0];
      cc[P > 4 ? 4 : 0] = P > 4 ? v1.x : cc[0];
      cc[P > 5 ? 5 : 0] = P > 5 ? v1.y : cc[0];
      cc[P > 6 ? 6 : 0] = P > 6 ? v1.z : cc[0];
      cc[P > 7 ? 7 : 0] = P > 7 ? v1.w : cc[0];
    }
  }
  float px[P], py[P];
  float mx = -INFINITY, mn = INFINITY, my = -INFINITY, ny = INFINITY;
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const float2 p = (cc[k] != 0xffffffffu) ? a.pos[cc[k]] : make_float2(0.f, 0.f);
    px[k] = p.x;
    py[k] = p.y;
    if (cc[k] != 0xffffffffu) {
      mx = fmaxf(mx, p.x);
      mn = fminf(mn, p.x);
      my = fmaxf(my, p.y);
      ny = fminf(ny, p.y);
    }
  }
  mx = group_allreduce(mx, g, OpMax());
  mn = group_allreduce(mn, g, OpMin());
  my = group_allreduce(my, g, OpMax());
  ny = group_allreduce(ny, g, OpMin());
  float e[kKeep ? P : 1][4];
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < P; ++k) {
    if (cc[k] == 0xffffffffu) continue;
    const float ux = px[k] - mx, vx = px[k] - mn, uy = py[k] - my, vy = py[k] - ny;
    const float epx = ex2(kg * ux), emx = ex2(-kg * vx);
    const float epy = ex2(kg * uy), emy = ex2(-kg * vy);
    if (kKeep) {
      e[kKeep ? k : 0][0] = epx;
      e[kKeep ? k : 0][1] = emx;
      e[kKeep ? k : 0][2] = epy;
      e[kKeep ? k : 0][3] = emy;
    }
    s[0] += epx; s[1] += ux * epx; s[2] += emx; s[3] += vx * emx;
    s[4] += epy; s[5] += uy * epy; s[6] += emy; s[7] += vy * emy;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s[k] = group_allreduce(s[k], g, OpAdd());
  if (!valid) return;  // every net of a class has two pins or more
  const float ipx = 1.0f / s[0], imx = 1.0f / s[2], ipy = 1.0f / s[4], imy = 1.0f / s[6];
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const uint32_t c = cc[k];
    if (c >= a.N) continue;  // fixed cells and empty slots
    const float ux = px[k] - mx, vx = px[k] - mn, uy = py[k] - my, vy = py[k] - ny;
    float epx, emx, epy, emy;
    if (kKeep) {
      epx = e[kKeep ? k : 0][0];
      emx = e[kKeep ? k : 0][1];
      epy = e[kKeep ? k : 0][2];
      emy = e[kKeep ? k : 0][3];
    } else {
      epx = ex2(kg * ux);
      emx = ex2(-kg * vx);
      epy = ex2(kg * uy);
      emy = ex2(-kg * vy);
    }
    const float gx = wa_pin_grad(ux, vx, epx, emx, ipx, s[1], imx, s[3], a.gamma);
    const float gy = wa_pin_grad(uy, vy, epy, emy, ipy, s[5], imy, s[7], a.gamma);
    atomicAdd(&a.acc[c], pack_grad(__float2ll_rn(gx * a.grad_scale), __float2ll_rn(gy * a.grad_scale)));
  }
}

// A net of more than 224 pins on one warp, three passes over its pins.
__device__ void wa_big_net(const WaArgs &a, int pb, int pe, int lane) {
  const float kg = a.gamma * kLog2e;
  float mx = -INFINITY, mn = INFINITY, my = -INFINITY, ny = INFINITY;
  for (int q = pb + lane; q < pe; q += 32) {
    const float2 p = a.pos[a.pin_cell[q]];
    mx = fmaxf(mx, p.x);
    mn = fminf(mn, p.x);
    my = fmaxf(my, p.y);
    ny = fminf(ny, p.y);
  }
  mx = warp_allreduce(mx, OpMax());
  mn = warp_allreduce(mn, OpMin());
  my = warp_allreduce(my, OpMax());
  ny = warp_allreduce(ny, OpMin());
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int q = pb + lane; q < pe; q += 32) {
    const float2 p = a.pos[a.pin_cell[q]];
    const float ux = p.x - mx, vx = p.x - mn, uy = p.y - my, vy = p.y - ny;
    const float epx = ex2(kg * ux), emx = ex2(-kg * vx);
    const float epy = ex2(kg * uy), emy = ex2(-kg * vy);
    s[0] += epx; s[1] += ux * epx; s[2] += emx; s[3] += vx * emx;
    s[4] += epy; s[5] += uy * epy; s[6] += emy; s[7] += vy * emy;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) s[k] = warp_allreduce(s[k], OpAdd());
  const float ipx = 1.0f / s[0], imx = 1.0f / s[2], ipy = 1.0f / s[4], imy = 1.0f / s[6];
  for (int q = pb + lane; q < pe; q += 32) {
    const uint32_t c = a.pin_cell[q];
    if (c >= a.N) continue;
    const float2 p = a.pos[c];
    const float ux = p.x - mx, vx = p.x - mn, uy = p.y - my, vy = p.y - ny;
    const float gx = wa_pin_grad(ux, vx, ex2(kg * ux), ex2(-kg * vx), ipx, s[1], imx, s[3], a.gamma);
    const float gy = wa_pin_grad(uy, vy, ex2(kg * uy), ex2(-kg * vy), ipy, s[5], imy, s[7], a.gamma);
    atomicAdd(&a.acc[c], pack_grad(__float2ll_rn(gx * a.grad_scale), __float2ll_rn(gy * a.grad_scale)));
  }
}

// Nets are ordered by degree and split into degree classes (WaClass): each
// warp takes 32 / G nets of one class, so the reductions run over a fixed
// group width with no per-lane segment logic.  Warps are visited from the
// heaviest class down.
__global__ void __launch_bounds__(kWaBlock) k_wa(const WaArgs a) {
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int t = gw; t < a.nwarps; t += nw) {
    const int w = a.nwarps - 1 - t;
    int j = 0;
#pragma unroll
    for (int k = 1; k < kWaClasses; ++k) j += (w >= a.cls[k].first_warp) ? 1 : 0;
    const WaClass &cl = a.cls[j];
    const int wi = w - cl.first_warp;
    switch (j) {
      case 0: case 1: case 2: case 3: case 4: {  // up to 32 pins: 1..8 lanes per net, <= 4 pins per lane
        const int g = j <= 1 ? 1 : (1 << (j - 1));   // kWaGroup
        wa_group<4>(a, cl, g, j == 0 ? 2 : 4, wi, lane);  // kWaSlots
        break;
      }
      case 5: case 6: case 7:  // 33..224 pins: a warp per net, <= 8 slots per lane
        wa_group<8>(a, cl, 32, j == 5 ? 2 : (j == 6 ? 4 : 8), wi, lane);
        break;
      default: {
        const uint32_t n = cl.first_net + wi;
        wa_big_net(a, a.net_off[n], a.net_off[n + 1], lane);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Footprint helpers shared by the scatter and the gather.  Footprint
// [x - w/2, x + w/2] x [y - h/2, y + h/2] in sites; bin b covers
// [b*s, (b+1)*s) (s sites per bin, an integer).  With w = h = s = 1 this is
// cell_bin_overlap / bin_overlap_area (density.rs:20-48).
// The arithmetic is exact in FP32 up to the final product of the two 1-D
// overlaps: a coordinate is split into its integer part i and fraction f
// (both exact), every edge difference is formed as (integer - f), and the
// bin range comes from integer floor / ceiling divisions.  Forming x + w/2
// directly would round once the sum crosses a power of two (at 1024 sites
// the FP32 spacing doubles to 1.2e-4), which shows up as area lost from one
// bin.
// ---------------------------------------------------------------------------
struct Foot {
  float fx, fy;   // fractional parts of the centre, in [0, 1)
  float hw, hh;   // half extents
  int ix, iy;     // integer parts of the centre
  int bx0, bx1, by0, by1;
};

// floor(a / s) for s > 0; a shift when s is a power of two (arithmetic
// shifts floor negative values too), which is the usual bin size.
__device__ __forceinline__ int floor_div(int a, int s) {
  if ((s & (s - 1)) == 0) return a >> (__ffs(s) - 1);
  return a >= 0 ? a / s : -((s - 1 - a) / s);
}
__device__ __forceinline__ int ceil_div(int a, int s) { return -floor_div(-a, s); }

__device__ __forceinline__ Foot make_foot(float2 p, float hw, float hh, int BX, int BY, int sx, int sy) {
  Foot f;
  const float flx = floorf(p.x), fly = floorf(p.y);
  f.ix = (int)flx;
  f.iy = (int)fly;
  f.fx = p.x - flx;
  f.fy = p.y - fly;
  f.hw = hw;
  f.hh = hh;
  // floor(x - hw) = ix + floor(fx - hw), ceil(x + hw) = ix + ceil(fx + hw)
  f.bx0 = max(0, floor_div(f.ix + (int)floorf(f.fx - hw), sx));
  f.bx1 = min(BX, max(0, ceil_div(f.ix + (int)ceilf(f.fx + hw), sx)));
  f.by0 = max(0, floor_div(f.iy + (int)floorf(f.fy - hh), sy));
  f.by1 = min(BY, max(0, ceil_div(f.iy + (int)ceilf(f.fy + hh), sy)));
  return f;
}

// Length of [c - h, c + h] inside [b*s, (b+1)*s), c = i + fr:
// min(h, (b+1)s - c) - max(-h, b s - c), each difference formed exactly.
__device__ __forceinline__ float overlap_1d(int i, float fr, float h, int b, int s) {
  const int k0 = b * s - i;
  const float hi = fminf(h, (float)(k0 + s) - fr);
  const float lo = fmaxf(-h, (float)k0 - fr);
  return fmaxf(hi - lo, 0.0f);
}
__device__ __forceinline__ float overlap_x(const Foot &f, int bx, int s) { return overlap_1d(f.ix, f.fx, f.hw, bx, s); }
__device__ __forceinline__ float overlap_y(const Foot &f, int by, int s) { return overlap_1d(f.iy, f.fy, f.hh, by, s); }

// Adds a footprint's part in a bin to the map.
__device__ __forceinline__ void add_bin(unsigned long long *dens, const Foot &f, int bx, int by, int BX, int isx,
                                        int isy) {
  const float ar = overlap_x(f, bx, isx) * overlap_y(f, by, isy);
  if (ar > 0.0f) atomicAdd(&dens[(size_t)by * BX + bx], to_fix(ar));
}

// One cell per lane of the warp (p, hf: centre and half extents; `in`: the
// lane has one).  A footprint of at most 2 x 2 bins (every unit cell) is
// unrolled.  A few larger ones are shared out over the warp, a bin per lane, so
// that 31 lanes don't wait for one macro's bins; where most lanes have one, each
// adds its own (1M cells of 2 x 2 to 3 x 3 bins 151 -> 52 us).  The passes of both ways
// are counted, handing a cell round as two.
__device__ __forceinline__ void scatter_warp(const ScatterArgs &a, unsigned long long *dens, float2 p, float2 hf,
                                             bool in) {
  const Foot f = make_foot(p, hf.x, hf.y, a.BX, a.BY, a.isx, a.isy);
  const bool wide = in && (f.bx1 - f.bx0 > 2 || f.by1 - f.by0 > 2);
  if (in && !wide) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int by = f.by0 + (k >> 1), bx = f.bx0 + (k & 1);
      if (by < f.by1 && bx < f.bx1) add_bin(dens, f, bx, by, a.BX, a.isx, a.isy);
    }
  }
  unsigned m = __ballot_sync(kFull, wide);
  if (!m) return;
  const unsigned own = wide ? (unsigned)max((f.bx1 - f.bx0) * (f.by1 - f.by0), 0) : 0u;
  if (__reduce_max_sync(kFull, own) <= __reduce_add_sync(kFull, wide ? (own + 31) / 32 + 2 : 0u)) {
    if (wide)
      for (int by = f.by0; by < f.by1; ++by)
        for (int bx = f.bx0; bx < f.bx1; ++bx) add_bin(dens, f, bx, by, a.BX, a.isx, a.isy);
    return;
  }
  while (m) {
    const int l = __ffs(m) - 1;
    m &= m - 1;
    const float2 q = make_float2(__shfl_sync(kFull, p.x, l), __shfl_sync(kFull, p.y, l));
    const float2 h = make_float2(__shfl_sync(kFull, hf.x, l), __shfl_sync(kFull, hf.y, l));
    const Foot g = make_foot(q, h.x, h.y, a.BX, a.BY, a.isx, a.isy);
    const int nx = g.bx1 - g.bx0, bins = nx * (g.by1 - g.by0);
    for (int k = threadIdx.x & 31; k < bins; k += 32) {
      const int r = k / nx;
      add_bin(dens, g, g.bx0 + k - r * nx, g.by0 + r, a.BX, a.isx, a.isy);
    }
  }
}

// Every cell by such warps: 32 cells from `first` on, then `step` further on.
__device__ __forceinline__ void scatter_all(const ScatterArgs &a, unsigned long long *dens, uint32_t first,
                                            uint32_t step) {
  for (uint32_t i0 = first & ~31u; i0 < a.N; i0 += step) {
    const uint32_t i = i0 + (threadIdx.x & 31);
    const bool in = i < a.N;
    scatter_warp(a, dens, in ? a.pos[i] : make_float2(0.f, 0.f),
                 in && a.half ? a.half[i] : make_float2(0.5f, 0.5f), in);
  }
}

// Unit cells first (a 1x1 footprint covers at most 2 x 2 bins: unrolled, no
// footprint load), then the macros from their own list, so a warp of unit
// cells never waits for one macro's loop.  Fixed-point atomics make the
// order irrelevant.  Without a macro list but with footprints, every cell
// takes the general form.
__global__ void __launch_bounds__(kScatterBlock) k_scatter(const ScatterArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, ts = gridDim.x * blockDim.x;
  if (a.sums) {
    if (t0 < kOverlapWords) a.sums[t0] = 0ull;
    if (t0 == 0) *a.ticket = 0u;
  }
  if (a.half && !a.mflag) {
    scatter_all(a, a.dens, t0, ts);
    return;
  }
  for (uint32_t i = t0; i < a.N; i += ts) {
    if (a.mflag && a.mflag[i]) continue;
    const Foot f = make_foot(a.pos[i], 0.5f, 0.5f, a.BX, a.BY, a.isx, a.isy);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int by = f.by0 + (k >> 1), bx = f.bx0 + (k & 1);
      if (by < f.by1 && bx < f.bx1) add_bin(a.dens, f, bx, by, a.BX, a.isx, a.isy);
    }
  }
  for (uint32_t k = t0; k < a.n_mac; k += ts) {
    const uint32_t i = a.mac_idx[k];
    const float2 hf = a.half[i];
    const Foot f = make_foot(a.pos[i], hf.x, hf.y, a.BX, a.BY, a.isx, a.isy);
    for (int by = f.by0; by < f.by1; ++by)
      for (int bx = f.bx0; bx < f.bx1; ++bx) add_bin(a.dens, f, bx, by, a.BX, a.isx, a.isy);
  }
}

// Streams the map once (8 bytes read and zeroed, the outputs written), four
// bins per thread and step, 16-byte accesses where the buffers allow it.  The
// overlap's sums are whole numbers, so each CTA adds its own with atomics and
// the last one forms the quotient (FP64 partial sums, which the last CTA read
// back and added in a fixed order, held the kernel up after its last bin).
// The launch overlaps the end of the scatter before it (launch_density_final,
// after).  Scatter and finalise of the allocation-free entry, which also made
// three clears and a copy, back to back: 64^2 bins, 2k unit cells 14.3 -> 5.1
// us; 512^2 bins, 200k cells with macros 21.8 -> 10 us (5.3 MB at least: 0.8).
// A single CTA with the map in its shared memory was slower from 1,000 cells
// on (2k cells 6.2 us, 8k 14 us).
__global__ void __launch_bounds__(kFinalBlock) k_density_final(const FinalArgs a) {
  __shared__ long long sm[kOverlapWords * kFinalBlock / 32];
  long long v[kOverlapWords] = {};
  // Groups of four consecutive bins per thread and step: 16-byte loads and
  // stores (when every pointer is aligned for them; a ragged tail, or
  // unaligned caller buffers, take the scalar loop below).
  const int ng = a.vec4 ? (a.nb >> 2) : 0;
  const int nblocks = (int)gridDim.x - (a.norms.part2 ? 1 : 0);  // the last one adds the norms up
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x, ts = nblocks * blockDim.x;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if ((int)blockIdx.x == nblocks) {
    if (threadIdx.x < 32) finish_norms(a.norms);
    return;
  }
  for (int gi = t0; gi < ng; gi += ts) {
    ulonglong2 *dp = reinterpret_cast<ulonglong2 *>(a.dens) + 2 * gi;
    const ulonglong2 q0 = dp[0], q1 = dp[1];
    dp[0] = make_ulonglong2(0ull, 0ull);
    dp[1] = make_ulonglong2(0ull, 0ull);
    const unsigned long long q[4] = {q0.x, q0.y, q1.x, q1.y};
    const double d[4] = {from_fix(q0.x), from_fix(q0.y), from_fix(q1.x), from_fix(q1.y)};
    float r[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      r[k] = (float)(d[k] - a.c0);
      count_bin(q[k], a.cap, v);
    }
    if (a.rho) reinterpret_cast<float4 *>(a.rho)[gi] = make_float4(r[0], r[1], r[2], r[3]);
    if (a.rho_hi) {
      __nv_bfloat16 h[4], l[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        h[k] = __float2bfloat16_rn(r[k]);
        l[k] = __float2bfloat16_rn(r[k] - __bfloat162float(h[k]));
      }
      uint2 hv, lv;
      hv.x = (uint32_t)__bfloat16_as_ushort(h[0]) | ((uint32_t)__bfloat16_as_ushort(h[1]) << 16);
      hv.y = (uint32_t)__bfloat16_as_ushort(h[2]) | ((uint32_t)__bfloat16_as_ushort(h[3]) << 16);
      lv.x = (uint32_t)__bfloat16_as_ushort(l[0]) | ((uint32_t)__bfloat16_as_ushort(l[1]) << 16);
      lv.y = (uint32_t)__bfloat16_as_ushort(l[2]) | ((uint32_t)__bfloat16_as_ushort(l[3]) << 16);
      reinterpret_cast<uint2 *>(a.rho_hi)[gi] = hv;
      reinterpret_cast<uint2 *>(a.rho_lo)[gi] = lv;
    }
    if (a.dens_out) {
      reinterpret_cast<double2 *>(a.dens_out)[2 * gi] = make_double2(d[0], d[1]);
      reinterpret_cast<double2 *>(a.dens_out)[2 * gi + 1] = make_double2(d[2], d[3]);
    }
  }
  for (int i = 4 * ng + t0; i < a.nb; i += ts) {
    const unsigned long long q = a.dens[i];
    const double d = from_fix(q);
    a.dens[i] = 0ull;
    const float r = (float)(d - a.c0);
    if (a.rho) a.rho[i] = r;
    if (a.rho_hi) {
      const __nv_bfloat16 h = __float2bfloat16_rn(r);
      a.rho_hi[i] = h;
      a.rho_lo[i] = __float2bfloat16_rn(r - __bfloat162float(h));
    }
    if (a.dens_out) a.dens_out[i] = d;
    count_bin(q, a.cap, v);
  }
  const int lane = threadIdx.x & 31;
  const long long c = warp_sum_words(v);
  if ((lane & 7) == 0) sm[kOverlapWords * (threadIdx.x >> 5) + (lane >> 3)] = c;
  __syncthreads();
  if (threadIdx.x >= kOverlapWords) return;
  long long t = 0;
#pragma unroll
  for (int w = 0; w < kFinalBlock / 32; ++w) t += sm[kOverlapWords * w + threadIdx.x];
  if (t) atomicAdd(&a.sums[threadIdx.x], (unsigned long long)t);
  __threadfence();
  __syncwarp((1u << kOverlapWords) - 1u);
  if (threadIdx.x != 0 || atomicAdd(a.ticket, 1u) != (unsigned)nblocks - 1) return;
  __threadfence();
  const double ov = take_overlap(a.sums);
  if (a.overlap) {
    *a.overlap = ov;
  } else {
    a.sc->overlap = ov;
    a.log[a.sc->iter].overlap = ov;
  }
  *a.ticket = 0u;
}

// ---------------------------------------------------------------------------
// FP32 SIMT GEMM: TM x TN CTA tile (64 x 64 with 256 threads, or 32 x 32 with
// 64 threads when the large tile leaves SMs idle), BK = 16, 4 x 4 outputs per
// thread, double-buffered shared memory.  Bounds are checked on every load
// and store, so any M, N, K works; multiples of 4 take the float4 path.
// Every output sums k = 0 .. K-1 in order whatever the tile, so both tile
// sizes give the same bits.
// ---------------------------------------------------------------------------
constexpr int GK = 16;

// S > 1: split K over a cluster of S CTAs (cluster dims 1 x 1 x S along z).
// CTA rank r sums k in [r K/S, (r+1) K/S) in order, parks its partial tile in
// its shared memory, and after a cluster barrier adds the S partials of a
// TM/S-row slice of the tile in rank order ((p0 + p1) + p2) + ... through
// distributed shared memory, then runs the epilogue on that slice.  The
// order is the same for both tile sizes, so they still give the same bits.
// One output of a SIMT GEMM.  With SPECTRAL: density.rs:114-153, scale
// 4/(WH), x1/2 on the kx = 0 and ky = 0 lines, phi = a / (2(1-cos wx) +
// 2(1-cos wy)), E = phi * w, at the frequencies (ky, kx) the op's layout
// gives the output (row, column); phi is written at its natural place.
template <bool SPECTRAL>
__device__ __forceinline__ void gemm_store(const GemmOp &op, const SpectralArgs &sp, int r, int c, int N, float v) {
  const size_t o = (size_t)r * op.ldc + c;
  if (SPECTRAL) {
    const int ky = op.row_par < 0 ? r : 2 * r + op.row_par;
    const int kx = op.col_split ? (c < N / 2 ? 2 * c : 2 * (c - N / 2) + 1) : c;
    float s = sp.scale;
    if (kx == 0) s *= 0.5f;
    if (ky == 0) s *= 0.5f;
    const float den = sp.gx2[kx] + sp.gy2[ky];
    float phi = 0.0f, ex = 0.0f, ey = 0.0f;
    if (!(den < 1e-30f)) {
      phi = v * s / den;
      ex = phi * sp.wx[kx];
      ey = phi * sp.wy[ky];
    }
    op.C[o] = ex;
    op.C2[o] = ey;
    if (sp.phi) sp.phi[(size_t)ky * N + kx] = phi;
  } else {
    op.C[o] = v;
  }
}

// a + m b, m = +-1
__device__ __forceinline__ float4 fold4(float4 a, float m, float4 b) {
  return make_float4(a.x + m * b.x, a.y + m * b.y, a.z + m * b.z, a.w + m * b.w);
}

template <bool SPECTRAL, int TM, int TN, int S>
__global__ void __launch_bounds__((TM / 4) * (TN / 4)) k_sgemm(const GemmOp *ops, int M, int N, int K,
                                                               SpectralArgs sp) {
  constexpr int T = (TM / 4) * (TN / 4);
  constexpr int LA = TM * GK / (4 * T), LB = GK * TN / (4 * T);  // float4 loads per thread
  static_assert(S == 1 || (TM % S == 0 && (TM / S) * (TN / 4) == T), "one float4 per thread in the split reduction");
  const GemmOp op = ops[blockIdx.z / S];
  __shared__ __align__(16) float smem[2 * GK * (TM + 4) + 2 * GK * (TN + 4)];
  static_assert(S == 1 || TM * TN <= 2 * GK * (TM + 4) + 2 * GK * (TN + 4), "partial tile fits the staging buffers");
  auto As = reinterpret_cast<float(*)[GK][TM + 4]>(smem);
  auto Bs = reinterpret_cast<float(*)[GK][TN + 4]>(smem + 2 * GK * (TM + 4));
  const int tid = threadIdx.x, tx = tid % (TN / 4), ty = tid / (TN / 4);
  const int bm = blockIdx.y * TM, bn = blockIdx.x * TN;
  const bool vec = ((K & 3) == 0) && ((N & 3) == 0) && ((op.lda & 3) == 0) && ((op.ldb & 3) == 0) &&
                   ((op.a_full & 3) == 0);
  const float mir = (float)(op.a_mir ? op.a_mir : op.b_mir);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // Loads of a step are all in flight together: what a folded operand adds
  // (u: one operand of a product is folded, and folded grids take the float4
  // path) is added when the step is stored.
  float4 ra[LA], rb[LB], u[LA > LB ? LA : LB];
  auto load = [&](int k0) {
#pragma unroll
    for (int l = 0; l < LA; ++l) {
      const int f = tid + l * T;
      const int gr = bm + f / (GK / 4), gk = k0 + (f % (GK / 4)) * 4;
      const float *p = op.A + (size_t)gr * op.lda + gk;
      if (vec) ra[l] = gr < M && gk < K ? *reinterpret_cast<const float4 *>(p) : zero;
      else
        ra[l] = make_float4(gr < M && gk < K ? p[0] : 0.f, gr < M && gk + 1 < K ? p[1] : 0.f,
                            gr < M && gk + 2 < K ? p[2] : 0.f, gr < M && gk + 3 < K ? p[3] : 0.f);
    }
#pragma unroll
    for (int l = 0; l < LB; ++l) {
      const int f = tid + l * T;
      const int gk = k0 + f / (TN / 4), gc = bn + (f % (TN / 4)) * 4;
      const float *p = op.B + (size_t)gk * op.ldb + gc;
      if (vec) rb[l] = gk < K && gc < N ? *reinterpret_cast<const float4 *>(p) : zero;
      else
        rb[l] = make_float4(gk < K && gc < N ? p[0] : 0.f, gk < K && gc + 1 < N ? p[1] : 0.f,
                            gk < K && gc + 2 < N ? p[2] : 0.f, gk < K && gc + 3 < N ? p[3] : 0.f);
    }
    if (op.a_mir) {
#pragma unroll
      for (int l = 0; l < LA; ++l) {  // columns a_full-1-gk-j, j = 0..3: the block below, reversed
        const int f = tid + l * T;
        const int gr = bm + f / (GK / 4), gk = k0 + (f % (GK / 4)) * 4;
        u[l] = gr < M && gk < K
                   ? *reinterpret_cast<const float4 *>(op.A + (size_t)gr * op.lda + (op.a_full - 4 - gk)) : zero;
      }
    } else if (op.b_mir) {
#pragma unroll
      for (int l = 0; l < LB; ++l) {
        const int f = tid + l * T;
        const int gk = k0 + f / (TN / 4), gc = bn + (f % (TN / 4)) * 4;
        u[l] = gk < K && gc < N
                   ? *reinterpret_cast<const float4 *>(op.B + (size_t)(op.b_full - 1 - gk) * op.ldb + gc) : zero;
      }
    }
  };
  auto store = [&](int buf) {
    if (op.a_mir) {
#pragma unroll
      for (int l = 0; l < LA; ++l) ra[l] = fold4(ra[l], mir, make_float4(u[l].w, u[l].z, u[l].y, u[l].x));
    } else if (op.b_mir) {
#pragma unroll
      for (int l = 0; l < LB; ++l) rb[l] = fold4(rb[l], mir, u[l]);
    }
#pragma unroll
    for (int l = 0; l < LA; ++l) {
      const int f = tid + l * T;
      const int r = f / (GK / 4), k = (f % (GK / 4)) * 4;
      As[buf][k][r] = ra[l].x;
      As[buf][k + 1][r] = ra[l].y;
      As[buf][k + 2][r] = ra[l].z;
      As[buf][k + 3][r] = ra[l].w;
    }
#pragma unroll
    for (int l = 0; l < LB; ++l) {
      const int f = tid + l * T;
      *reinterpret_cast<float4 *>(&Bs[buf][f / (TN / 4)][(f % (TN / 4)) * 4]) = rb[l];
    }
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  // This CTA's k range (all of K when S == 1; the launcher splits only when
  // S * GK divides K).
  const int kpart = (S == 1) ? K : K / S;
  const int kbeg = (S == 1) ? 0 : (int)(blockIdx.z % S) * kpart;
  const int nk = (kpart + GK - 1) / GK;
  load(kbeg);
  store(0);
  __syncthreads();
  for (int kt = 0; kt < nk; ++kt) {
    const int cur = kt & 1;
    if (kt + 1 < nk) load(kbeg + (kt + 1) * GK);
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4 *>(&As[cur][kk][ty * 4]);
      const float4 b4 = *reinterpret_cast<const float4 *>(&Bs[cur][kk][tx * 4]);
      const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (kt + 1 < nk) {
      store(cur ^ 1);
      __syncthreads();
    }
  }
  if constexpr (S > 1) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __syncthreads();  // the staging buffers become the partial tile
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4 *>(&smem[(ty * 4 + i) * TN + tx * 4]) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    cluster.sync();
    const int rank = (int)cluster.block_rank();
    const int lr = rank * (TM / S) + tid / (TN / 4), lc = (tid % (TN / 4)) * 4;
    float4 v = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(&smem[lr * TN + lc], 0));
#pragma unroll
    for (int q = 1; q < S; ++q) {
      const float4 w = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(&smem[lr * TN + lc], q));
      v.x += w.x;
      v.y += w.y;
      v.z += w.z;
      v.w += w.w;
    }
    const float vv[4] = {v.x, v.y, v.z, v.w};
    const int r = bm + lr;
    if (r < M) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int cidx = bn + lc + j;
        if (cidx >= N) continue;
        gemm_store<SPECTRAL>(op, sp, r, cidx, N, vv[j]);
      }
    }
    cluster.sync();  // no CTA leaves while another reads its partial tile
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = bm + ty * 4 + i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cidx = bn + tx * 4 + j;
      if (cidx >= N) continue;
      gemm_store<SPECTRAL>(op, sp, r, cidx, N, acc[i][j]);
    }
  }
}

// ---------------------------------------------------------------------------
// k_sgemm_panel: the same products where K has no split in four (the side, half
// of it when folded, is not a multiple of 64).
//
// Bound by latency: such a product is a few hundred kFMA to some MFMA, and
// tiles of 64 x 64 leave most SMs without one and go through K in steps of 16
// with a barrier and an L2 round trip each.  Here a tile is 16 or 32 x 32, a
// step is 64 of K, loaded by 128 threads while the step before is multiplied,
// and a thread has 2 x 2 or 2 x 4 outputs.  With PAIR a CTA has both halves E
// and O of a folded transform, 128 threads each, and writes the butterfly
// E + O, sig (E - O) itself (cols: about the middle column, else about the
// middle row): E and O never go to memory and the butterfly's launch goes.
// Each output sums k = 0 .. K-1 in order as in k_sgemm: the same bits.
// The four products (with butterflies) of a square grid back to back, before
// -> now: side 69 36.9 -> 15.0 us, 72 34.8 -> 10.2, 133 59.5 -> 21.6, 200
// 54.9 -> 23.1, 269 106 -> 55, 533 223 -> 131; an iteration of 1k cells on 69^2
// bins 53.3 -> 26.7 us, of 10k on 133^2 80.7 -> 37.3, of 200k on 533^2 312 -> 196.
// ---------------------------------------------------------------------------
constexpr int PN = 32, PK = 64;

template <bool SPECTRAL, bool PAIR, int PM>
__global__ void __launch_bounds__(PAIR ? 256 : 128)
    k_sgemm_panel(const GemmOp *ops, const FlyOp *fly, int cols, int M, int N, int K, SpectralArgs sp) {
  constexpr int TC = PM / 8;  // columns of a thread; it has two rows
  constexpr int LA = PM * PK / 128, LB = PK * PN / 128;
  __shared__ __align__(16) float as_[PAIR ? 2 : 1][PM][PK + 4];
  __shared__ __align__(16) float bs_[PAIR ? 2 : 1][PK][PN];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int half = PAIR ? (int)threadIdx.x >> 7 : 0, tid = threadIdx.x & 127;
  const GemmOp op = ops[PAIR ? 2 * blockIdx.z + half : blockIdx.z];
  auto As = as_[half];
  auto Bs = bs_[half];
  const int tx = tid % (PN / TC), ty = tid / (PN / TC);
  const int bm = blockIdx.y * PM, bn = blockIdx.x * PN;
  const bool vec = ((K & 3) == 0) && ((N & 3) == 0) && ((op.lda & 3) == 0) && ((op.ldb & 3) == 0) &&
                   ((op.a_full & 3) == 0);
  const float mir = (float)(op.a_mir ? op.a_mir : op.b_mir);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // float4 l of a thread: elements 4 (tid + 128 l) .. + 3 (vec), or elements
  // tid + 512 l + 128 j, j = 0 .. 3.  u as in k_sgemm.
  float4 ra[LA / 4], rb[LB / 4], u[LB / 4];
  auto load = [&](int k0) {
    if (vec) {
#pragma unroll
      for (int l = 0; l < LA / 4; ++l) {
        const int f = tid + 128 * l, gr = bm + f / (PK / 4), gk = k0 + (f % (PK / 4)) * 4;
        ra[l] = gr < M && gk < K ? *reinterpret_cast<const float4 *>(op.A + (size_t)gr * op.lda + gk) : zero;
      }
#pragma unroll
      for (int l = 0; l < LB / 4; ++l) {
        const int f = tid + 128 * l, gk = k0 + f / (PN / 4), gc = bn + (f % (PN / 4)) * 4;
        rb[l] = gk < K && gc < N ? *reinterpret_cast<const float4 *>(op.B + (size_t)gk * op.ldb + gc) : zero;
      }
      if (op.a_mir) {
#pragma unroll
        for (int l = 0; l < LA / 4; ++l) {  // columns a_full-1-gk-j, j = 0..3: the block below, reversed
          const int f = tid + 128 * l, gr = bm + f / (PK / 4), gk = k0 + (f % (PK / 4)) * 4;
          u[l] = gr < M && gk < K
                     ? *reinterpret_cast<const float4 *>(op.A + (size_t)gr * op.lda + (op.a_full - 4 - gk)) : zero;
        }
      } else if (op.b_mir) {
#pragma unroll
        for (int l = 0; l < LB / 4; ++l) {
          const int f = tid + 128 * l, gk = k0 + f / (PN / 4), gc = bn + (f % (PN / 4)) * 4;
          u[l] = gk < K && gc < N
                     ? *reinterpret_cast<const float4 *>(op.B + (size_t)(op.b_full - 1 - gk) * op.ldb + gc) : zero;
        }
      }
    } else {
      const int ak = k0 + tid % PK, ar = bm + tid / PK, bk = k0 + tid / PN, bc = bn + tid % PN;
      const float *pa = op.A + (size_t)ar * op.lda + ak, *pb = op.B + (size_t)bk * op.ldb + bc;
      constexpr int SA = 128 / PK, SB = 128 / PN;  // rows between a thread's elements
      auto ea = [&](int i) { return ak < K && ar + SA * i < M ? pa[(size_t)(SA * i) * op.lda] : 0.f; };
      auto eb = [&](int i) { return bc < N && bk + SB * i < K ? pb[(size_t)(SB * i) * op.ldb] : 0.f; };
#pragma unroll
      for (int l = 0; l < LA / 4; ++l) ra[l] = make_float4(ea(4 * l), ea(4 * l + 1), ea(4 * l + 2), ea(4 * l + 3));
#pragma unroll
      for (int l = 0; l < LB / 4; ++l) rb[l] = make_float4(eb(4 * l), eb(4 * l + 1), eb(4 * l + 2), eb(4 * l + 3));
    }
  };
  auto store = [&]() {
    float *af = &As[tid / PK][tid % PK], *bf = &Bs[tid / PN][tid % PN];
    if (vec) {
      if (op.a_mir) {
#pragma unroll
        for (int l = 0; l < LA / 4; ++l) ra[l] = fold4(ra[l], mir, make_float4(u[l].w, u[l].z, u[l].y, u[l].x));
      } else if (op.b_mir) {
#pragma unroll
        for (int l = 0; l < LB / 4; ++l) rb[l] = fold4(rb[l], mir, u[l]);
      }
#pragma unroll
      for (int l = 0; l < LA / 4; ++l) {
        const int f = tid + 128 * l;
        *reinterpret_cast<float4 *>(&As[f / (PK / 4)][(f % (PK / 4)) * 4]) = ra[l];
      }
#pragma unroll
      for (int l = 0; l < LB / 4; ++l) {
        const int f = tid + 128 * l;
        *reinterpret_cast<float4 *>(&Bs[f / (PN / 4)][(f % (PN / 4)) * 4]) = rb[l];
      }
    } else {
      constexpr int SA = 128 / PK * (PK + 4), SB = 128;
#pragma unroll
      for (int l = 0; l < LA / 4; ++l) {
        af[4 * l * SA] = ra[l].x;
        af[(4 * l + 1) * SA] = ra[l].y;
        af[(4 * l + 2) * SA] = ra[l].z;
        af[(4 * l + 3) * SA] = ra[l].w;
      }
#pragma unroll
      for (int l = 0; l < LB / 4; ++l) {
        bf[4 * l * SB] = rb[l].x;
        bf[(4 * l + 1) * SB] = rb[l].y;
        bf[(4 * l + 2) * SB] = rb[l].z;
        bf[(4 * l + 3) * SB] = rb[l].w;
      }
    }
  };
  asm volatile("griddepcontrol.wait;" ::: "memory");
  float acc[2][TC] = {};
  load(0);
  for (int k0 = 0; k0 < K; k0 += PK) {
    store();
    __syncthreads();
    if (k0 + PK < K) load(k0 + PK);
    const int kn = min(PK, (K - k0 + 3) & ~3);  // the rest of the step is zeros
#pragma unroll 4
    for (int k = 0; k < kn; k += 4) {
      const float4 a0 = *reinterpret_cast<const float4 *>(&As[2 * ty][k]);
      const float4 a1 = *reinterpret_cast<const float4 *>(&As[2 * ty + 1][k]);
      const float av[2][4] = {{a0.x, a0.y, a0.z, a0.w}, {a1.x, a1.y, a1.z, a1.w}};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float b[TC];
        if constexpr (TC == 2) {
          const float2 t = *reinterpret_cast<const float2 *>(&Bs[k + j][2 * tx]);
          b[0] = t.x, b[1] = t.y;
        } else {
          const float4 t = *reinterpret_cast<const float4 *>(&Bs[k + j][4 * tx]);
          b[0] = t.x, b[1] = t.y, b[2] = t.z, b[3] = t.w;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int c = 0; c < TC; ++c) acc[i][c] = fmaf(av[i][j], b[c], acc[i][c]);
      }
    }
    __syncthreads();
  }
  if constexpr (PAIR) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int c = 0; c < TC; ++c) Bs[2 * ty + i][TC * tx + c] = acc[i][c];
    __syncthreads();
    const FlyOp f = fly[blockIdx.z];
    const int W = cols ? 2 * N : N;
    for (int q = tid; q < PM * PN; q += 128) {
      const int lr = q / PN, lc = q % PN, r = bm + lr, c = bn + lc;
      if (r >= M || c >= N) continue;
      const float e = bs_[0][lr][lc], o = bs_[1][lr][lc];
      if (half == 0) f.out[(size_t)r * W + c] = e + o;
      else f.out[(size_t)(cols ? r : 2 * M - 1 - r) * W + (cols ? W - 1 - c : c)] = f.sig * (e - o);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = bm + 2 * ty + i;
#pragma unroll
      for (int j = 0; j < TC; ++j) {
        const int c = bn + TC * tx + j;
        if (r < M && c < N) gemm_store<SPECTRAL>(op, sp, r, c, N, acc[i][j]);
      }
    }
  }
}

// SMs of the current device (cached per device).
int device_sms() {
  static int sms[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!sms[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    sms[dev] = v;
  }
  return sms[dev];
}

// Split K: the small tile when the 64 x 64 grid would leave more than half the
// SMs without a CTA (measured: 64 CTAs of 512^3 gain from the small tile, 128
// CTAs do not).
bool sgemm_small_tile(int M, int N, int nb) {
  return 2L * ((N + 63) / 64) * ((M + 63) / 64) * nb * 4 < device_sms();
}

// ---------------------------------------------------------------------------
// The step: field gather, penalty, preconditioner, Barzilai-Borwein step,
// FISTA, clamp, next look-ahead, and the next iteration's density scatter.
//
// Bound by latency: 200k cells are 15.7 MB of L2-resident state (2.4 us at the
// HBM rate), but the loads of a cell depend on one another (look-ahead ->
// field), and the step length needs a sum over all cells in between.  So:
//  * a thread keeps its cells over the whole step: nothing but the block sums
//    crosses blocks, and the state that the second half needs is loaded while
//    the block waits for the others;
//  * a macro (25 bins and more) is gathered by eight lanes, a column of bins
//    each, four macros a warp, spread over all blocks (MANY: a thread each, see
//    step_kernel).  The bins are summed in
//    the row-major order of one thread, so the bits are the same; one thread
//    per macro walked its rows one memory latency at a time, and held the
//    barrier up for 8 us at 200k cells (10k macros);
//  * the block sums are formed with six FP64 shuffles a warp for four sums;
//  * the next look-ahead is scattered into the density map while it is in
//    registers (a launch, and a read of the positions, less);
//  * the step norms, which only the log needs, are left as block sums for a
//    kernel of the next iteration (finish_norms) instead of a last block;
//  * there is one copy of the code of a cell in each half, in a loop over the
//    thread's cells with the next one's loads under way: two cells side by side
//    doubled the instructions, and a block runs them once, so that waiting for
//    their fetch was its longest stall.
// Inside one launch (5k / 200k / 800k cells), first half done 3 / 9 / 33 us,
// sums known 5 / 12 / 36, end 8 / 20 / 67 (with the scatter; before, without
// it: 200k 14, 20, 25).  Whole iterations with the FFT transform, reference
// field, mean of 100: 5k cells 30.9 -> 20.6 us, 30k 52.7 -> 35.5, 200k 111.6 ->
// 58.5, 800k 229 -> 200 (the last three with the cells of a bin added once).
// ---------------------------------------------------------------------------

// The four sums v over the block; lane k < 4 of warp 0 gets sum k in v[0].
// sm: [4 * 16].  One barrier; sm must not be in use before it.
__device__ __forceinline__ double block_sum4(const double (&v)[4], double *sm) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // each exchange halves the sums a lane carries: 4 -> 2 -> 1, then three adds
  const bool up = lane & 16, up2 = lane & 8;
  double a = up ? v[2] : v[0], b = up ? v[3] : v[1];
  a += __shfl_xor_sync(kFull, up ? v[0] : v[2], 16);
  b += __shfl_xor_sync(kFull, up ? v[1] : v[3], 16);
  double c = up2 ? b : a;
  c += __shfl_xor_sync(kFull, up2 ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
  // lanes 8 k .. 8 k + 7 carry sum k
  if ((lane & 7) == 0) sm[4 * w + (lane >> 3)] = c;
  __syncthreads();
  double t = 0.0;
  if (w == 0) {  // lane: sum lane & 3 of warps lane / 4 and lane / 4 + 8
    const int k = lane & 3, i = lane >> 2;
    t = (i < nw ? sm[4 * i + k] : 0.0) + (i + 8 < nw ? sm[4 * (i + 8) + k] : 0.0);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) t += __shfl_xor_sync(kFull, t, o);
  }
  return t;
}

// The block sums part[4 b + k] of all blocks, by the whole block: every
// thread gets the four totals (in a fixed order).  sm: [4 * 16], tot: [4].
__device__ __forceinline__ void total_of(const double *part, unsigned nblocks, double (&out)[4], double *sm,
                                         double *tot) {
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (unsigned b = threadIdx.x; b < nblocks; b += blockDim.x) {
    const double2 p = __ldcg(reinterpret_cast<const double2 *>(part) + 2 * b);
    const double2 q = __ldcg(reinterpret_cast<const double2 *>(part) + 2 * b + 1);
    v[0] += p.x;
    v[1] += p.y;
    v[2] += q.x;
    v[3] += q.y;
  }
  const double t = block_sum4(v, sm);
  if (threadIdx.x < 4) tot[threadIdx.x] = t;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) out[k] = tot[k];
}

// Grid barrier of the cooperative step, once the block's sums (lane k < 4 of
// warp 0: sum t) are in part[].  Every wait is bounded: on timeout the block
// records the error in sc->err and leaves the kernel, so the kernel always
// terminates, no block computes on partial data, and the host reports
// EPLACE_ERR_TIMEOUT (the next run resets the device state).
// bar[0..1] is one 64-bit arrival count that is never reset inside a run:
// every launch on it has the same grid and passes whole barriers, so a launch
// starts at a multiple of gridDim.x, and barrier k of the run is complete when
// the count reaches (k + 1) * gridDim.x.  The last block's own add releases
// the others.  The host zeroes the count at every load and run start.
__device__ __forceinline__ bool publish_and_wait(double *part, double t, unsigned *bar, DevScalars *sc, int *gave_up) {
  if (threadIdx.x < 32) {
    if (threadIdx.x < 4) __stcg(part + 4 * blockIdx.x + threadIdx.x, t);
    __syncwarp();
    if (threadIdx.x == 0) {
      *gave_up = 0;
      unsigned long long *cnt = reinterpret_cast<unsigned long long *>(bar);
      const long long limit = sc->spin_cycles > 0 ? sc->spin_cycles : kSpinCycles;
      __threadfence();  // the sums before the arrival
      const unsigned long long old = atomicAdd(cnt, 1ull);
      // (a run's arrivals stay far below 2^32: a 64-bit remainder is slow)
      const unsigned long long target =
          old < 0xffffffffull ? old - (unsigned)old % gridDim.x + gridDim.x : old - old % gridDim.x + gridDim.x;
      const long long t0 = clock64();
      while (true) {
        unsigned long long v;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(cnt) : "memory");
        if (v >= target) break;
        if (clock64() - t0 > limit) {
          atomicExch(&sc->err, 1);
          *gave_up = 1;
          break;
        }
      }
      __threadfence();
    }
  }
  __syncthreads();
  return !*gave_up;
}

// The at most 2 x 2 bins of a 1x1 footprint (bins are >= 1 site wide): the
// lower left one and the lengths along x and y, 0 outside the chip.
struct UnitFoot {
  int at;           // bin (bx0, by0); bins bx0 + 1, by0 + 1 only where ox[1], oy[1] > 0
  float ox[2], oy[2];
};
__device__ __forceinline__ UnitFoot unit_foot(int BX, int BY, int isx, int isy, float2 p) {
  const Foot f = make_foot(p, 0.5f, 0.5f, BX, BY, isx, isy);
  UnitFoot u;
  u.at = f.by0 * BX + f.bx0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    u.ox[k] = f.bx0 + k < f.bx1 ? overlap_x(f, f.bx0 + k, isx) : 0.0f;
    u.oy[k] = f.by0 + k < f.by1 ? overlap_y(f, f.by0 + k, isy) : 0.0f;
  }
  return u;
}
__device__ __forceinline__ UnitFoot unit_foot(const StepArgs &a, float2 p) {
  return unit_foot(a.BX, a.BY, a.isx, a.isy, p);
}

// Field gather of a 1x1 footprint: all field loads at once, summed in the
// row-major order of the general form.
__device__ __forceinline__ float2 gather_unit(const StepArgs &a, float2 p) {
  const UnitFoot u = unit_foot(a, p);
  float w[4], e[4], h[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    w[k] = u.ox[k & 1] * u.oy[k >> 1];
    const int at = u.at + (k >> 1) * a.BX + (k & 1);
    e[k] = w[k] > 0.0f ? a.Ex[at] : 0.0f;
    h[k] = w[k] > 0.0f ? a.Ey[at] : 0.0f;
  }
  float fx = 0.f, fy = 0.f, wt = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (w[k] > 0.0f) {
      fx = fmaf(w[k], e[k], fx);
      fy = fmaf(w[k], h[k], fy);
      wt += w[k];
    }
  float2 g = make_float2(0.f, 0.f);
  if (wt > 1e-10f) {
    g.x = fx / wt;
    g.y = fy / wt;
  }
  return g;
}

// A warp's eight-lane groups, one macro each.
struct Macro {
  uint32_t i;   // cell
  bool in;      // the group has one
  int col;      // this lane's column of the group, 0 .. 7
  float2 hf;
  float area;
};

// Weighted-mean field gather of the groups' macros at p, scaled by the area
// (compute_density_gradient, density.rs:171-206): each lane loads its column
// of the footprint's bins, eight columns and up to kRows rows in flight, and
// every lane of the group sums the bins in row-major order.  All lanes of the
// warp call it; every lane of a group gets the result.
__device__ __forceinline__ float2 gather_macro(const StepArgs &a, const Macro &m, float2 p) {
  constexpr int kRows = 5;
  const Foot f = make_foot(p, m.hf.x, m.hf.y, a.BX, a.BY, a.isx, a.isy);
  const int nx = max(f.bx1 - f.bx0, 0), parts = (nx + 7) >> 3;  // eight-bin parts of a row
  const int n = m.in ? parts * max(f.by1 - f.by0, 0) : 0;
  const int most = (int)__reduce_max_sync(kFull, (unsigned)n);
  const int cols = (int)__reduce_max_sync(kFull, (unsigned)min(nx, 8));
  const int lead = threadIdx.x & 24;
  float fx = 0.f, fy = 0.f, wt = 0.f;
  int by = f.by0, part = 0;
  for (int r0 = 0; r0 < most; r0 += kRows) {
    float w[kRows], e[kRows], h[kRows];
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int bx = f.bx0 + 8 * part + m.col;
      w[u] = (r0 + u < n && bx < f.bx1) ? overlap_x(f, bx, a.isx) * overlap_y(f, by, a.isy) : 0.0f;
      const int at = by * a.BX + bx;
      e[u] = w[u] > 0.0f ? a.Ex[at] : 0.0f;
      h[u] = w[u] > 0.0f ? a.Ey[at] : 0.0f;
      if (++part == parts) {
        part = 0;
        ++by;
      }
    }
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
#pragma unroll 1
      for (int k = 0; k < cols; ++k) {
        const float wk = __shfl_sync(kFull, w[u], lead + k);
        const float ek = __shfl_sync(kFull, e[u], lead + k), hk = __shfl_sync(kFull, h[u], lead + k);
        if (wk > 0.0f) {
          fx = fmaf(wk, ek, fx);
          fy = fmaf(wk, hk, fy);
          wt += wk;
        }
      }
    }
  }
  float2 g = make_float2(0.f, 0.f);
  if (wt > 1e-10f) {
    g.x = m.area * (fx / wt);
    g.y = m.area * (fy / wt);
  }
  return g;
}

// The same by one thread, four bins of a row in flight, summed in the same
// order: for designs with so many macros that eight lanes each would be work for
// more warps than there are.
__device__ __forceinline__ float2 gather_wide(const StepArgs &a, float2 p, float2 hf, float area) {
  const Foot f = make_foot(p, hf.x, hf.y, a.BX, a.BY, a.isx, a.isy);
  float fx = 0.f, fy = 0.f, wt = 0.f;
#pragma unroll 1
  for (int by = f.by0; by < f.by1; ++by) {
    const float oy = overlap_y(f, by, a.isy);
#pragma unroll 1
    for (int b0 = f.bx0; b0 < f.bx1; b0 += 4) {
      float w[4], e[4], h[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        w[k] = b0 + k < f.bx1 ? overlap_x(f, b0 + k, a.isx) * oy : 0.0f;
        const int at = by * a.BX + b0 + k;
        e[k] = w[k] > 0.0f ? a.Ex[at] : 0.0f;
        h[k] = w[k] > 0.0f ? a.Ey[at] : 0.0f;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (w[k] > 0.0f) {
          fx = fmaf(w[k], e[k], fx);
          fy = fmaf(w[k], h[k], fy);
          wt += w[k];
        }
    }
  }
  float2 g = make_float2(0.f, 0.f);
  if (wt > 1e-10f) {
    g.x = area * (fx / wt);
    g.y = area * (fy / wt);
  }
  return g;
}

// g = (g_wl + lam g_den) / max(1, pw + lam area)   (mod.rs:145-156)
__device__ __forceinline__ float2 combine(float2 gw, float2 gd, double lam, float pw, float area) {
  const double ipc = 1.0 / fmax((double)pw + lam * (double)area, 1.0);
  return make_float2((float)(((double)gw.x + lam * (double)gd.x) * ipc),
                     (float)(((double)gw.y + lam * (double)gd.y) * ipc));
}

// What the first half of the step knows of a cell before the gather.
struct CellIn {
  float2 look, x, xp, gp;
  unsigned long long acc;
  float pw;
};

__device__ __forceinline__ CellIn load_in(const StepArgs &a, uint32_t i, bool was_init) {
  CellIn c;
  c.look = a.look[i];
  c.acc = a.acc[i];
  c.pw = a.pw[i];
  if (was_init) {
    c.x = a.x[i];
    c.xp = a.xp[i];
    c.gp = a.gprev[i];
  }
  return c;
}

__device__ __forceinline__ void bb_terms(double (&v)[4], float2 x, float2 xp, float2 g, float2 gp) {
  const double dx = (double)x.x - xp.x, dy = (double)x.y - xp.y;
  v[0] += dx * dx;
  v[1] += dx * ((double)g.x - gp.x);
  v[2] += dy * dy;
  v[3] += dy * ((double)g.y - gp.y);
}

// The rest of the first half: combined gradient and the terms of the sums
// (before the first penalty: the two gradients and their norms).
__device__ __forceinline__ void first_half(const StepArgs &a, uint32_t i, const CellIn &c, float2 gd, float area,
                                           bool was_init, double lam, double (&v)[4]) {
  long long sx, sy;
  unpack_grad(c.acc, &sx, &sy);
  const float2 gw = make_float2((float)((double)sx * a.grad_inv), (float)((double)sy * a.grad_inv));
  a.acc[i] = 0ull;
  if (was_init) {
    const float2 g = combine(gw, gd, lam, c.pw, area);
    a.g[i] = g;
    bb_terms(v, c.x, c.xp, g, c.gp);
    return;
  }
  a.tmp_wl[i] = gw;
  a.tmp_den[i] = gd;
  v[0] += (double)gw.x * gw.x + (double)gw.y * gw.y;
  v[1] += (double)gd.x * gd.x + (double)gd.y * gd.y;
}

// FISTA step (nesterov.rs:41-64), clamp (:67-72), next look-ahead (:95-101)
// clamped to the chip (common.rs:410-415), for one cell; returns the latter.
__device__ __forceinline__ float2 fista_cell(const StepArgs &a, uint32_t i, float2 x, float2 xp, float2 g, double m,
                                             double mn, const double (&alpha)[2], double (&nrm)[4]) {
  const double yx = (double)x.x + m * ((double)x.x - xp.x);
  const double yy = (double)x.y + m * ((double)x.y - xp.y);
  const double nx = yx - alpha[0] * g.x, ny = yy - alpha[1] * g.y;
  nrm[0] += (nx - x.x) * (nx - x.x);
  nrm[1] += (ny - x.y) * (ny - x.y);
  const float cx = fminf(fmaxf((float)nx, 0.0f), a.maxx);
  const float cy = fminf(fmaxf((float)ny, 0.0f), a.maxy);
  const float px = fminf(fmaxf(x.x, 0.0f), a.maxx);
  const float py = fminf(fmaxf(x.y, 0.0f), a.maxy);
  a.x[i] = make_float2(cx, cy);
  a.xp[i] = make_float2(px, py);
  a.gprev[i] = g;
  const double lx = (double)cx + mn * ((double)cx - px);
  const double ly = (double)cy + mn * ((double)cy - py);
  const float2 look = make_float2(fminf(fmaxf((float)lx, 0.0f), a.maxx), fminf(fmaxf((float)ly, 0.0f), a.maxy));
  a.look[i] = look;
  return look;
}

// The next iteration's density scatter of the warp's unit cells (p, where
// `in`), and of the groups' macros.  Additions to one bin go one after the
// other in L2 (0.6 ns each), and cells do pile up in one: the reference's field
// drives most of them against the chip's edges into a corner's bin (156k of
// 200k by iteration 300).  So where lanes lie on an edge, those that share the
// warp's most common bin add once.  Whole numbers: the same sums.  Mean of the
// first 300 iterations with that field, before -> now: 5k cells 21.2 -> 20.3 us,
// 30k 49.3 -> 35.2, 200k 139 -> 58, 800k 367 -> 208; fields that spread the
// cells (no lanes on an edge) +0.3 us at 5k, else the same.  From 4 lanes on:
// 6 and 10 gain less (200k without macros 55.3 and 57.2 us against 54.9).
constexpr unsigned kShared = 4;  // lanes from which the warp's sum is cheaper
__device__ __forceinline__ void scatter_shared(unsigned long long *dens, int BX, int BY, int isx, int isy, float2 p,
                                            bool in) {
  const UnitFoot u = unit_foot(BX, BY, isx, isy, p);
  const unsigned lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(kFull, in ? (unsigned)u.at : 0x80000000u | lane);
  const unsigned most = __reduce_max_sync(kFull, (unsigned)__popc(same) << 5 | lane);
  const bool shared = most >> 5 >= kShared;
  const bool member = shared && (__shfl_sync(kFull, same, most & 31) >> lane & 1);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float ar = u.ox[k & 1] * u.oy[k >> 1];
    unsigned long long q = in && ar > 0.0f ? to_fix(ar) : 0ull;
    if (shared) {  // q <= 2^32: the sums of its two parts fit
      const unsigned lo = __reduce_add_sync(kFull, member ? (unsigned)q & 0xffffu : 0u);
      const unsigned hi = __reduce_add_sync(kFull, member ? (unsigned)(q >> 16) : 0u);
      if (member) q = lane == (most & 31) ? lo + ((unsigned long long)hi << 16) : 0ull;
    }
    if (q) atomicAdd(&dens[u.at + (k >> 1) * BX + (k & 1)], q);
  }
}
__device__ __forceinline__ void scatter_units(const StepArgs &a, float2 p, bool in) {
  const bool edge = in && (p.x <= 0.0f || p.y <= 0.0f || p.x >= a.maxx || p.y >= a.maxy);
  if (__popc(__ballot_sync(kFull, edge)) >= (int)kShared) {
    scatter_shared(a.dens, a.BX, a.BY, a.isx, a.isy, p, in);
    return;
  }
  const UnitFoot u = unit_foot(a, p);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float ar = u.ox[k & 1] * u.oy[k >> 1];
    if (in && ar > 0.0f) atomicAdd(&a.dens[u.at + (k >> 1) * a.BX + (k & 1)], to_fix(ar));
  }
}
__device__ __forceinline__ void scatter_macro(const StepArgs &a, const Macro &m, float2 p) {
  if (!m.in) return;
  const Foot f = make_foot(p, m.hf.x, m.hf.y, a.BX, a.BY, a.isx, a.isy);
  for (int by = f.by0; by < f.by1; ++by)
    for (int bx = f.bx0 + m.col; bx < f.bx1; bx += 8) add_bin(a.dens, f, bx, by, a.BX, a.isx, a.isy);
}

// How a block's warps share the cells: the last `macro` warps take macros, the
// first `unit` warps unit cells.  Four macros make a task; with few enough
// tasks they get warps of their own (a macro costs a warp about as long as two
// passes of unit cells, and a warp with both held the block's sum up), else
// every warp takes both.
struct Shares {
  int unit, macro;
};
template <bool MANY>
__device__ __forceinline__ Shares shares(const StepArgs &a) {
  if (MANY) return Shares{(int)(blockDim.x >> 5), 0};
  const int nwb = blockDim.x >> 5;
  const uint32_t per = ((a.n_mac + 3) / 4 + gridDim.x - 1) / gridDim.x;  // tasks of a block, at most
  if (per == 0 || per > (uint32_t)(3 * nwb / 4)) return Shares{nwb, nwb};
  return Shares{nwb - (int)per, (int)per};
}

// The macros of this warp, four at a time: fn(Macro) with all lanes.
template <typename F>
__device__ __forceinline__ void each_macro(const StepArgs &a, const Shares &sh, F fn) {
  const int k0 = (int)(blockDim.x >> 5) - 1 - (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k0 >= sh.macro) return;
  const uint32_t tasks = (a.n_mac + 3) / 4;
#pragma unroll 1
  for (uint32_t t = blockIdx.x + gridDim.x * (uint32_t)k0; t < tasks; t += gridDim.x * (uint32_t)sh.macro) {
    Macro m;
    const uint32_t k = 4 * t + (lane >> 3);
    m.in = k < a.n_mac;
    m.i = a.mac_idx[m.in ? k : 0];
    m.col = lane & 7;
    m.hf = a.half[m.i];
    m.area = a.area[m.i];
    fn(m);
  }
}

// With MANY, a thread per macro instead: fn(cell), from the grid's last thread
// on, where the unit cells' passes are shortest.
template <typename F>
__device__ __forceinline__ void each_macro_alone(const StepArgs &a, F fn) {
  const uint32_t threads = gridDim.x * blockDim.x;
#pragma unroll 1
  for (uint32_t k = threads - 1 - (blockIdx.x * blockDim.x + threadIdx.x); k < a.n_mac; k += threads) fn(a.mac_idx[k]);
}

// Modes: 0: the whole step in one cooperative launch (grid barriers between
// its halves); 1: gather only (tmp_den <- density gradient); 2, 3, 4: first
// half, penalty-initialisation pass and second half as three ordinary launches
// of the same grid (launch order replaces the barriers, so no block ever waits
// for another).
template <bool MANY>
__global__ void __launch_bounds__(kStepBlock, 2) k_step(const StepArgs a) {
  __shared__ __align__(16) double sm[64], sm2[64], tot[4];
  __shared__ int gave_up;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // this thread's unit cells: tid0, tid0 + gstride, ...
  const Shares sh = shares<MANY>(a);
  const bool units = (int)(threadIdx.x >> 5) < sh.unit;
  const uint32_t gstride = gridDim.x * (uint32_t)sh.unit * 32;
  const uint32_t tid0 = units ? blockIdx.x * (uint32_t)sh.unit * 32 + threadIdx.x : a.N;
  const int it = a.sc->iter;
  const bool was_init = a.sc->lam_init != 0;
  double alpha[2] = {a.sc->step[0], a.sc->step[1]};
  double lam = a.sc->lam;
  bool lam_init = was_init;
  if (was_init) lam = (lam < 50.0) ? lam * 1.025 : lam + 1.0;  // mod.rs:139-143
  // A bounded wait already gave up in an earlier launch: every block sees the
  // same flag here and leaves before any barrier, so the rest of the
  // interval drains quickly and the host reports EPLACE_ERR_TIMEOUT.
  if (a.sc->err) return;

  if (a.mode == 1) {  // gather only: no barrier is reached
    if constexpr (MANY) {
      each_macro_alone(a, [&](uint32_t i) { a.tmp_den[i] = gather_wide(a, a.look[i], a.half[i], a.area[i]); });
    } else {
      each_macro(a, sh, [&](const Macro &m) {
        const float2 g = gather_macro(a, m, a.look[m.i]);
        if (m.in && m.col == 0) a.tmp_den[m.i] = g;
      });
    }
    for (uint32_t i = tid0; i < a.N; i += gstride)
      if (!a.mflag || !a.mflag[i]) a.tmp_den[i] = gather_unit(a, a.look[i]);
    return;
  }
  const bool coop = a.mode == 0;
  // The state that the second half needs of this thread's first cell, loaded
  // while the block waits for the others.
  struct State {
    float2 x, xp, g;
  };
  auto unit_at = [&](uint32_t i) { return i < a.N && (!a.mflag || !a.mflag[i]); };
  auto state_of = [&](uint32_t i) {
    State c{};
    if (i < a.N) c = State{a.x[i], a.xp[i], a.g[i]};
    return c;
  };
  State s0{};
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  if (coop || a.mode == 2) {
    if constexpr (MANY) {
      each_macro_alone(a, [&](uint32_t i) {
        const CellIn c = load_in(a, i, was_init);
        const float area = a.area[i];
        first_half(a, i, c, gather_wide(a, c.look, a.half[i], area), area, was_init, lam, v);
      });
    } else {
      each_macro(a, sh, [&](const Macro &m) {
        CellIn c;
        c.look = a.look[m.i];
        if (m.col == 0) c = load_in(a, m.i, was_init);
        const float2 gd = gather_macro(a, m, c.look);
        if (m.in && m.col == 0) first_half(a, m.i, c, gd, m.area, was_init, lam, v);
      });
    }
    // One cell at a time, the next one's state on the way (a macro's is loaded
    // for nothing: its flag arrives with it).
    CellIn c{};
    if (tid0 < a.N) c = load_in(a, tid0, was_init);
#pragma unroll 1
    for (uint32_t i = tid0; i < a.N; i += gstride) {
      const bool unit = !a.mflag || !a.mflag[i];
      CellIn next = c;
      if (i + gstride < a.N) next = load_in(a, i + gstride, was_init);
      const float2 gd = gather_unit(a, c.look);
      if (unit) first_half(a, i, c, gd, 1.0f, was_init, lam, v);
      c = next;
    }
    const double t = block_sum4(v, sm);
    if (a.mode == 2) {
      if (threadIdx.x < 4) a.part[4 * blockIdx.x + threadIdx.x] = t;
      return;
    }
    if (was_init) s0 = state_of(tid0);
    if (!publish_and_wait(a.part, t, a.bar, a.sc, &gave_up)) return;
  }

  if (!was_init) {
    // First penalty: 0.1 * |g_wl| / |g_den| when |g_den| > 1e-30 (mod.rs:132-138).
    double nr[4];
    total_of(a.part, gridDim.x, nr, sm2, tot);
    const double wl = sqrt(nr[0]);
    const double dn = sqrt(nr[1]);
    if (dn > 1e-30) {
      lam = 0.1 * wl / dn;
      lam_init = true;
    }
    if (coop || a.mode == 3) {
      for (int k = 0; k < 4; ++k) v[k] = 0.0;
      auto pass = [&](uint32_t i, float area) {
        const float2 g = combine(a.tmp_wl[i], a.tmp_den[i], lam, a.pw[i], area);
        a.g[i] = g;
        bb_terms(v, a.x[i], a.xp[i], g, a.gprev[i]);
      };
      if constexpr (MANY) {
        each_macro_alone(a, [&](uint32_t i) { pass(i, a.area[i]); });
      } else {
        each_macro(a, sh, [&](const Macro &m) {
          if (m.in && m.col == 0) pass(m.i, m.area);
        });
      }
      for (uint32_t i = tid0; i < a.N; i += gstride)
        if (!a.mflag || !a.mflag[i]) pass(i, 1.0f);
      const double t = block_sum4(v, sm);
      if (a.mode == 3) {
        if (threadIdx.x < 4) a.part_b[4 * blockIdx.x + threadIdx.x] = t;
        return;
      }
      s0 = state_of(tid0);
      if (!publish_and_wait(a.part_b, t, a.bar, a.sc, &gave_up)) return;
    }
  } else if (a.mode == 3) {
    return;
  }
  if (a.mode == 4) s0 = state_of(tid0);

  // Barzilai-Borwein per axis after the first iteration (mod.rs:158-166,
  // nesterov.rs:199-218): |dx.dx / dx.dg| clamped to [1e-4, 1], kept when
  // |dx.dg| < 1e-30.
  double t[4];
  total_of(was_init ? a.part : a.part_b, gridDim.x, t, sm2, tot);
  if (it > 0) {
    for (int ax = 0; ax < 2; ++ax) {
      const double dxdx = t[2 * ax], dxdg = t[2 * ax + 1];
      if (!(fabs(dxdg) < 1e-30)) alpha[ax] = fmin(fmax(fabs(dxdx / dxdg), 1e-4), 1.0);
    }
  }
  // Block 0 writes the scalars and the log entry once every block has read the
  // scalars: after a grid barrier, all have; in mode 4 the last block to get
  // here does it instead (its whole block is past its reads).
  bool writer = blockIdx.x == 0;
  if (!coop && threadIdx.x == 0) {
    __threadfence();
    writer = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
  }
  if (writer && threadIdx.x == 0) {
    IterLog &L = a.log[it];
    L.lam = lam;
    L.alpha[0] = alpha[0];
    L.alpha[1] = alpha[1];
    a.sc->lam = lam;
    a.sc->lam_init = lam_init ? 1 : 0;
    a.sc->step[0] = alpha[0];
    a.sc->step[1] = alpha[1];
    a.sc->iter = it + 1;
    *a.ticket = 0u;
  }
  // FISTA step (nesterov.rs:41-64), clamp (:67-72), next look-ahead
  // (:95-101) clamped to the chip (common.rs:410-415), and its density.
  const double m = a.mom[it], mn = a.mom[it + 1];
  double nrm[4] = {0.0, 0.0, 0.0, 0.0};
  if constexpr (MANY) {
    each_macro_alone(a, [&](uint32_t i) {
      const float2 p = fista_cell(a, i, a.x[i], a.xp[i], a.g[i], m, mn, alpha, nrm);
      if (!a.dens) return;
      const float2 hf = a.half[i];
      const Foot f = make_foot(p, hf.x, hf.y, a.BX, a.BY, a.isx, a.isy);
#pragma unroll 1
      for (int by = f.by0; by < f.by1; ++by)
#pragma unroll 1
        for (int bx = f.bx0; bx < f.bx1; ++bx) add_bin(a.dens, f, bx, by, a.BX, a.isx, a.isy);
    });
  } else {
    each_macro(a, sh, [&](const Macro &c) {
      float2 p = make_float2(0.f, 0.f);
      if (c.in && c.col == 0) p = fista_cell(a, c.i, a.x[c.i], a.xp[c.i], a.g[c.i], m, mn, alpha, nrm);
      if (a.dens) {
        const int lead = threadIdx.x & 24;
        p = make_float2(__shfl_sync(kFull, p.x, lead), __shfl_sync(kFull, p.y, lead));
        scatter_macro(a, c, p);
      }
    });
  }
#pragma unroll 1
  for (uint32_t i = tid0; units && (i & ~31u) < a.N; i += gstride) {  // a warp's 32 cells at a time
    const bool unit = unit_at(i);
    const State next = state_of(i + gstride);
    float2 look = make_float2(0.f, 0.f);
    if (unit) look = fista_cell(a, i, s0.x, s0.xp, s0.g, m, mn, alpha, nrm);
    if (a.dens) scatter_units(a, look, unit);
    s0 = next;
  }
  // The step norms stay block sums; the next iteration's first kernel adds them.
  const double s = block_sum4(nrm, sm);
  if (threadIdx.x < 2) a.part2[2 * blockIdx.x + threadIdx.x] = s;
}

// The end of an interval: the positions and scalars into a snapshot, and the
// last iteration's step norms into its log entry.
__global__ void __launch_bounds__(256) k_snapshot(const SnapArgs a) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) a.pos[i] = a.x[i];
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    finish_norms(a.norms);
    if (threadIdx.x == 0) *a.sc_out = *a.norms.sc;
  }
}

__global__ void __launch_bounds__(kHpwlBlock) k_hpwl(const HpwlArgs a) {
  __shared__ double sm[32];
  double v = 0.0;
  for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < a.NN; n += gridDim.x * blockDim.x) {
    const uint32_t b = a.net_off[n], e = a.net_off[n + 1];
    if ((a.has_driver && !a.has_driver[n]) || e - b < 2) continue;
    int x0 = INT_MAX, x1 = INT_MIN, y0 = INT_MAX, y1 = INT_MIN;
    for (uint32_t q = b; q < e; ++q) {
      const int2 l = a.loc[a.pin_cell[q]];
      x0 = min(x0, l.x);
      x1 = max(x1, l.x);
      y0 = min(y0, l.y);
      y1 = max(y1, l.y);
    }
    v += (double)((long long)(x1 - x0) + (long long)(y1 - y0));
  }
  // Per-thread partials are integers below 2^53, so the FP64 block sum is exact.
  v = block_sum_d(v, sm);
  if (threadIdx.x == 0) atomicAdd(a.total, (unsigned long long)(long long)v);
}

}  // namespace

cudaError_t launch_wa(const WaArgs &a, int grid, cudaStream_t s) {
  if (a.nwarps == 0) return cudaSuccess;
  k_wa<<<grid, kWaBlock, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_scatter(const ScatterArgs &a, int grid, cudaStream_t s) {
  if (a.N == 0) return cudaSuccess;
  k_scatter<<<grid, kScatterBlock, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_density_final(const FinalArgs &a_in, int grid, cudaStream_t s, bool after) {
  FinalArgs a = a_in;
  auto al = [](const void *p, uintptr_t m) { return ((uintptr_t)p & (m - 1)) == 0; };
  a.vec4 = al(a.dens, 16) && al(a.rho, 16) && al(a.rho_hi, 8) && al(a.rho_lo, 8) && al(a.dens_out, 16);
  Launch l(grid + (a.norms.part2 ? 1 : 0), kFinalBlock, s, after);
  return cudaLaunchKernelEx(&l.cfg, k_density_final, a);
}

// One SIMT GEMM launch.  K that is a multiple of 4 * GK (every transform of a
// power-of-two bin grid of at least 64) is split four ways over a cluster;
// which sums run in which order depends on K alone, never on the tile, so the
// tile stays a choice of time only.
constexpr int kSplitK = 4;

template <bool SPECTRAL, int TM, int TN>
cudaError_t sgemm_launch(const GemmOp *ops, int nb, int M, int N, int K, const SpectralArgs &sp, cudaStream_t s) {
  const dim3 tiles((N + TN - 1) / TN, (M + TM - 1) / TM, nb);
  constexpr int T = (TM / 4) * (TN / 4);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles.x, tiles.y, tiles.z * kSplitK);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = kSplitK;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_sgemm<SPECTRAL, TM, TN, kSplitK>, ops, M, N, K, sp);
}

// Rows of the panels that a product runs as, 0 for none.  Measured (us a
// product, rows 16 / rows 32 / 64 x 64 tiles; the folded third product of a
// square grid, in brackets the CTAs of the first and of the last form): side
// 264 6.9 / 9.8 / 14.4 (340, 60); 400 14.0 / 13.5 / 18.4 (700, 112); 600 35.1 /
// 28.9 / 34.8 (1520, 200); 808 70.6 / 60.8 / 56.9 (2652, 364).
int sgemm_panel(int M, int N, int nb, int K, int tile) {
  if (K % (kSplitK * GK) == 0) return 0;
  if (tile) return tile == 64 ? 0 : tile;
  const long ctas = (long)((N + PN - 1) / PN) * ((M + 15) / 16) * nb;
  const long large = (long)((N + 63) / 64) * ((M + 63) / 64) * nb;
  return ctas <= 5L * device_sms() ? 16 : 2 * large <= 3L * device_sms() ? 32 : 0;
}

template <bool SPECTRAL, bool PAIR>
cudaError_t panel_launch(const GemmOp *ops, const FlyOp *fly, bool cols, int nb, int M, int N, int K, int rows,
                         const SpectralArgs &sp, cudaStream_t s, bool after) {
  Launch l(1, PAIR ? 256 : 128, s, after);
  l.cfg.gridDim = dim3((N + PN - 1) / PN, (M + rows - 1) / rows, PAIR ? nb / 2 : nb);
  auto kernel = rows == 16 ? k_sgemm_panel<SPECTRAL, PAIR, 16> : k_sgemm_panel<SPECTRAL, PAIR, 32>;
  return cudaLaunchKernelEx(&l.cfg, kernel, ops, fly, (int)cols, M, N, K, sp);
}

template <bool SPECTRAL>
cudaError_t sgemm_any(const GemmOp *ops, int nb, int M, int N, int K, const SpectralArgs &sp, cudaStream_t s, int tile,
                      bool after) {
  if (const int rows = sgemm_panel(M, N, nb, K, tile))
    return panel_launch<SPECTRAL, false>(ops, nullptr, false, nb, M, N, K, rows, sp, s, after);
  if (K % (kSplitK * GK) != 0) {
    k_sgemm<SPECTRAL, 64, 64, 1><<<dim3((N + 63) / 64, (M + 63) / 64, nb), 256, 0, s>>>(ops, M, N, K, sp);
    return cudaGetLastError();
  }
  if (tile == 32 || (tile == 0 && sgemm_small_tile(M, N, nb)))
    return sgemm_launch<SPECTRAL, 32, 32>(ops, nb, M, N, K, sp, s);
  return sgemm_launch<SPECTRAL, 64, 64>(ops, nb, M, N, K, sp, s);
}

cudaError_t launch_sgemm(const GemmOp *ops, int nb, int M, int N, int K, cudaStream_t s, int tile, bool after) {
  return sgemm_any<false>(ops, nb, M, N, K, SpectralArgs{}, s, tile, after);
}

cudaError_t launch_sgemm_spectral(const GemmOp *ops, int nb, int M, int N, int K, const SpectralArgs &sp,
                                  cudaStream_t s, int tile, bool after) {
  return sgemm_any<true>(ops, nb, M, N, K, sp, s, tile, after);
}

namespace {
__global__ void k_fly_cols(const FlyOp *ops, int H, int W) {
  const FlyOp op = ops[blockIdx.z];
  const int hw = W / 2;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
  if (x >= hw || r >= H) return;
  const float e = op.E[(size_t)r * hw + x], o = op.O[(size_t)r * hw + x];
  op.out[(size_t)r * W + x] = e + o;
  op.out[(size_t)r * W + (W - 1 - x)] = op.sig * (e - o);
}
__global__ void k_fly_rows(const FlyOp *ops, int H, int W) {
  const FlyOp op = ops[blockIdx.z];
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= W || y >= H / 2) return;
  const float e = op.E[(size_t)y * W + x], o = op.O[(size_t)y * W + x];
  op.out[(size_t)y * W + x] = e + o;
  op.out[(size_t)(H - 1 - y) * W + x] = op.sig * (e - o);
}
}  // namespace

cudaError_t launch_sgemm_fly(const GemmOp *ops, const FlyOp *fly, int nb, int M, int N, int K, bool cols,
                             cudaStream_t s, int tile, bool after) {
  if (const int rows = sgemm_panel(M, N, nb, K, tile))
    return panel_launch<false, true>(ops, fly, cols, nb, M, N, K, rows, SpectralArgs{}, s, after);
  const cudaError_t e = launch_sgemm(ops, nb, M, N, K, s, tile, after);
  if (e != cudaSuccess) return e;
  if (cols) k_fly_cols<<<dim3((N + 127) / 128, M, nb / 2), 128, 0, s>>>(fly, M, 2 * N);
  else k_fly_rows<<<dim3((N + 127) / 128, M, nb / 2), 128, 0, s>>>(fly, 2 * M, N);
  return cudaGetLastError();
}

// Threads per block of the step: small designs spread over the SMs (one block
// of 512 threads takes four times as long for its instructions as one of 128
// on an SM of its own: 5k cells, ten blocks of 512 threads 15.9 us a step),
// large ones keep the barrier's arrivals few.
int step_block(int device, uint32_t cells) {
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) sms = 148;
  return cells <= 128u * (unsigned)sms ? 128 : cells <= 512u * (unsigned)sms ? 256 : kStepBlock;
}

// A thread per macro from three macros in ten cells on.  An iteration, eight
// lanes per macro / a thread each (before macros had lanes), us: macros of 2 x 2
// sites, all of 20k cells 55.5 / 29.7 (36.9), of 100k 85 / 49 (51), 40 % of 20k
// 41.6 / 30.6 (39.3); of 2 to 8 sites, 20 % of 100k cells 56 / 65 (58), 5 % of
// 20k 28.8 / 42.3 (42.2).
using StepKernel = void (*)(StepArgs);
StepKernel step_kernel(const StepArgs &a) { return 10ull * a.n_mac >= 3ull * a.N ? k_step<true> : k_step<false>; }

int step_max_grid(int device, int block) {
  int sms = 0, occ = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  int least = 1 << 30;
  for (StepKernel k : {k_step<false>, k_step<true>}) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, block, 0) != cudaSuccess) return 0;
    least = occ < least ? occ : least;
  }
  return sms * least;
}

cudaError_t launch_step(const StepArgs &a, int grid, int block, cudaStream_t s) {
  void *args[] = {const_cast<StepArgs *>(&a)};
  return cudaLaunchCooperativeKernel((const void *)step_kernel(a), dim3(grid), dim3(block), args, 0, s);
}
cudaError_t launch_step_split(const StepArgs &a, int grid, int block, cudaStream_t s) {
  for (int mode = 2; mode <= 4; ++mode) {
    StepArgs b = a;
    b.mode = mode;
    // the second and third may start while the one before ends (k_step waits)
    Launch l(grid, block, s, mode > 2);
    const cudaError_t e = cudaLaunchKernelEx(&l.cfg, step_kernel(a), b);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_snapshot(const SnapArgs &a, cudaStream_t s) {
  const unsigned g = (a.n + 255) / 256;  // up to 4 CTAs for each of the 148 SMs; the kernel loops
  k_snapshot<<<g < 1 ? 1 : g < 592 ? g : 592, 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_hpwl(const HpwlArgs &a, int grid, cudaStream_t s) {
  k_hpwl<<<grid, kHpwlBlock, 0, s>>>(a);
  return cudaGetLastError();
}

// The stage entries' inputs and outputs.  A thread moves four consecutive
// cells, so that a warp reads or writes 512 bytes of each host array in a row;
// the bus bounds these kernels.  They take the place of loops on the host that
// packed and unpacked pairs, converted the packed gradient and the density,
// and of copies from pageable memory.  Whole calls at 200k cells / 512^2 bins:
// wirelength gradient 919 -> 176 us, fused step 5.6 -> 1.5 ms, field 604 ->
// 203 us; mixed-precision field at 1024^2 bins 4.6 -> 0.67 ms.
namespace {
__global__ void __launch_bounds__(256) k_io_in(const IoArgs a) {
  const uint32_t i0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i0 >= a.n) return;
  float4 x[kIoPairs], y[kIoPairs];
#pragma unroll
  for (int k = 0; k < kIoPairs; ++k)
    if (k < a.pairs) {
      x[k] = *reinterpret_cast<const float4 *>(a.host + 2 * k * a.pitch + i0);
      y[k] = *reinterpret_cast<const float4 *>(a.host + (2 * k + 1) * a.pitch + i0);
    }
#pragma unroll
  for (int k = 0; k < kIoPairs; ++k)
    if (k < a.pairs) {
      const float vx[4] = {x[k].x, x[k].y, x[k].z, x[k].w}, vy[4] = {y[k].x, y[k].y, y[k].z, y[k].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i0 + j >= a.n) continue;
        if (k == 1 && a.scale != 0.0)
          a.acc[i0 + j] = pack_grad(__double2ll_rn((double)vx[j] * a.scale), __double2ll_rn((double)vy[j] * a.scale));
        else
          a.pair[k][i0 + j] = make_float2(vx[j], vy[j]);
      }
    }
  if (a.acc && a.scale == 0.0)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + j < a.n) a.acc[i0 + j] = 0ull;
}

__global__ void __launch_bounds__(256) k_io_out(const IoArgs a) {
  const uint32_t i0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i0 >= a.n) return;
#pragma unroll
  for (int k = 0; k < kIoPairs; ++k)
    if (k < a.pairs) {
      float vx[4] = {0.f, 0.f, 0.f, 0.f}, vy[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i0 + j >= a.n) continue;
        if (k == 0 && a.acc) {
          long long sx, sy;
          unpack_grad(a.acc[i0 + j], &sx, &sy);
          a.acc[i0 + j] = 0ull;
          vx[j] = (float)((double)sx * a.scale);
          vy[j] = (float)((double)sy * a.scale);
        } else {
          const float2 v = a.pair[k][i0 + j];
          vx[j] = v.x;
          vy[j] = v.y;
        }
      }
      *reinterpret_cast<float4 *>(a.host + 2 * k * a.pitch + i0) = make_float4(vx[0], vx[1], vx[2], vx[3]);
      *reinterpret_cast<float4 *>(a.host + (2 * k + 1) * a.pitch + i0) = make_float4(vy[0], vy[1], vy[2], vy[3]);
    }
}

__global__ void __launch_bounds__(256) k_io_rho(const double *d, size_t n, double c0, float *rho, __nv_bfloat16 *hi,
                                                __nv_bfloat16 *lo) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float r = (float)(d[i] - c0);
    if (rho) {
      rho[i] = r;
    } else {
      const __nv_bfloat16 h = __float2bfloat16_rn(r);
      hi[i] = h;
      lo[i] = __float2bfloat16_rn(r - __bfloat162float(h));
    }
  }
}
}  // namespace

cudaError_t launch_io_in(const IoArgs &a, cudaStream_t s) {
  if (a.n == 0) return cudaSuccess;
  k_io_in<<<(a.n + 1023) / 1024, 256, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_io_out(const IoArgs &a, cudaStream_t s) {
  if (a.n == 0) return cudaSuccess;
  k_io_out<<<(a.n + 1023) / 1024, 256, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_io_rho(const double *d, size_t n, double c0, float *rho, __nv_bfloat16 *hi, __nv_bfloat16 *lo,
                          cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const size_t g = (n + 255) / 256;
  k_io_rho<<<(unsigned)(g < 1184 ? g : 1184), 256, 0, s>>>(d, n, c0, rho, hi, lo);
  return cudaGetLastError();
}

}  // namespace eplace
