// kernels.cuh -- device-side state of one placement context and the launch
// wrappers of the hot-path kernels (defined in kernels.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace eplace {

// Scalars of the Nesterov loop kept on the device so a whole legalisation
// interval can be replayed as one CUDA graph without host round trips.
struct DevScalars {
  double lam;          // density_penalty (electro_place/mod.rs:100)
  double step[2];      // current step sizes (NesterovSolver::step_size)
  double overlap;      // overlap of the current iteration's density
  int32_t lam_init;    // density_initialized
  int32_t iter;        // index of the next iteration to execute
  int32_t err;         // non-zero: a bounded wait gave up
  int32_t pad_;
  int64_t spin_cycles; // bound of every grid-barrier wait in SM clock cycles (0: the default, ~2 s)
};

// One record per executed iteration (fields of the reference log line).
struct IterLog {
  double overlap;
  double lam;
  double step_norm[2];  // NesterovSolver::step return values
  double alpha[2];      // step sizes used by the FISTA step
};

// The step's block sums of the step norms, and where they go: the log entry
// of the iteration before sc->iter.
struct NormArgs {
  const double *part2;  // [2 * blocks], nullptr: none
  int blocks;
  const DevScalars *sc;
  IterLog *log;
};

#ifdef __CUDACC__
// One warp: adds the block sums up in a fixed order and writes the norms.
__device__ __forceinline__ void finish_norms(const NormArgs &a) {
  const int it = a.sc->iter - 1;
  if (it < 0 || a.sc->err) return;
  double x = 0.0, y = 0.0;
  for (int b = threadIdx.x & 31; b < a.blocks; b += 32) {
    const double2 p = reinterpret_cast<const double2 *>(a.part2)[b];
    x += p.x;
    y += p.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
  }
  if ((threadIdx.x & 31) == 0) {
    a.log[it].step_norm[0] = sqrt(x);
    a.log[it].step_norm[1] = sqrt(y);
  }
}
#endif

// The overlap (density.rs:79-86) from the fixed-point map: the sum of d and of
// max(d - cap, 0) over all bins, each in two 64-bit words, whole sites and
// 2^-32 sites: {sum, sum's fraction, over, over's fraction}.  A bin holds less
// than 2^31 sites, but all bins together may hold more, and one 64-bit word of
// 2^-32 sites wraps there.  Whole numbers: their order is free.
constexpr int kOverlapWords = 4;

// A bin's capacity in the map's unit; no bin reaches one of 2^31 sites and more.
inline long long fixed_capacity(long long sites) { return sites < (1ll << 31) ? sites << 32 : 0x7fffffffffffffffll; }

#ifdef __CUDACC__
__device__ __forceinline__ void count_bin(unsigned long long q, long long cap, long long (&v)[kOverlapWords]) {
  const long long d = (long long)q, over = d > cap ? d - cap : 0;
  v[0] += d >> 32;
  v[1] += (unsigned)d;
  v[2] += over >> 32;
  v[3] += (unsigned)over;
}

// The warp's four sums: lanes 8 k .. 8 k + 7 get sum k.  Each exchange halves
// the sums that a lane carries, 4 -> 2 -> 1.
__device__ __forceinline__ long long warp_sum_words(const long long (&v)[kOverlapWords]) {
  const bool up = threadIdx.x & 16, up2 = threadIdx.x & 8;
  long long a = up ? v[2] : v[0], b = up ? v[3] : v[1];
  a += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
  b += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
  long long c = up2 ? b : a;
  c += __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  return c;
}

// compute_overlap of the sums, which are zero again (one thread).
__device__ __forceinline__ double take_overlap(unsigned long long *sums) {
  long long w[kOverlapWords];
#pragma unroll
  for (int k = 0; k < kOverlapWords; ++k) w[k] = (long long)atomicExch(sums + k, 0ull);
  // carried first, so that each sum is rounded once
  const auto value = [](long long sites, long long frac) {
    return (double)(sites + (frac >> 32)) + (double)(frac & 0xffffffffll) * (1.0 / 4294967296.0);
  };
  const double sum = value(w[0], w[1]);
  return sum < 1e-30 ? 0.0 : value(w[2], w[3]) / sum;
}
#endif

// A launch that, with `after`, may start before the kernel ahead of it in the
// stream has ended (that kernel's griddepcontrol.wait keeps the order of the
// data: every kernel of such a chain executes it in every thread that reads
// or writes what the one before does).
struct Launch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  Launch(int grid, int block, cudaStream_t s, bool after, size_t smem = 0) {
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = after ? 1 : 0;
  }
  Launch(const Launch &) = delete;
  Launch &operator=(const Launch &) = delete;
};

// Degree classes of the WA kernel over the degree-sorted nets: class j holds
// the nets of degree (kWaDegHi[j-1], kWaDegHi[j]] (class 0 from degree 2;
// nets of fewer pins have no gradient) and runs kWaGroup[j] lanes per net,
// kWaSlots[j] pin slots per lane; the last class (more than 224 pins) runs a
// warp per net over its CSR pins in three passes.
constexpr int kWaClasses = 9;
constexpr int kWaDegHi[kWaClasses] = {2, 4, 8, 16, 32, 64, 128, 224, 0x7fffffff};
constexpr int kWaGroup[kWaClasses] = {1, 1, 2, 4, 8, 32, 32, 32, 32};
// Padded pin table: lane l of a net's group holds that net's pins l, l + G,
// l + 2G, ... in its kWaSlots[j] consecutive slots (one 8-, 16- or 32-byte
// load), unused slots 0xffffffff; a net takes G * kWaSlots[j] slots.
constexpr int kWaSlots[kWaClasses] = {2, 4, 4, 4, 4, 2, 4, 8, 0};

// The WA gradient of a cell is accumulated as one 64-bit integer per cell:
// x and y in fixed point (scale 2^k), packed as gx + 2^32 gy and summed with
// one 64-bit atomic per pin.  Two's-complement sums are exact modulo 2^64,
// so while |sum gx| and |sum gy| stay below 2^31 the low word is the x sum
// and the rest the y sum.  k is chosen per problem from the largest pin
// count of a cell (a pin's gradient is below 2 in magnitude; the bound used
// is 4 per pin), at most 24.
__host__ __device__ inline unsigned long long pack_grad(long long gx, long long gy) {
  return (unsigned long long)gx + ((unsigned long long)gy << 32);
}
__host__ __device__ inline void unpack_grad(unsigned long long v, long long *gx, long long *gy) {
  const int lo = (int)(unsigned)(v & 0xffffffffull);
  *gx = lo;
  *gy = (long long)(v - (unsigned long long)(long long)lo) >> 32;
}

struct WaClass {
  int first_net;        // index into the degree-sorted CSR
  int nets;
  int first_warp;       // warps of the classes before this one
  long long slot_base;  // first slot of the class in the padded pin table (multiple of 4)
};

struct WaArgs {
  WaClass cls[kWaClasses];
  int nwarps;
  const uint32_t *slots;    // padded pin table (kWaSlots)
  const uint32_t *net_off;
  const uint32_t *pin_cell;
  const float2 *pos;        // [N + F]: look-ahead positions, then fixed cells
  unsigned long long *acc;  // [N] packed fixed-point gradient (see pack_grad)
  uint32_t N;
  float gamma;
  float grad_scale;         // 2^k fixed-point scale of the packed gradient
};

struct ScatterArgs {
  const float2 *pos;
  const float2 *half;       // half extents, nullptr => unit cells
  const uint8_t *mflag;     // [N] 1 for a macro, nullptr: no macro list (general loop when half is set)
  const uint32_t *mac_idx;  // [n_mac] the macros' cell ids
  uint32_t n_mac;
  uint32_t N;
  int BX, BY;
  int isx, isy;              // sites per bin along x / y
  unsigned long long *dens; // [BY * BX] fixed point
  unsigned long long *sums = nullptr;  // of the finalise behind it: cleared here, with its ticket
  unsigned *ticket = nullptr;
};

struct FinalArgs {
  unsigned long long *dens;
  int nb;
  long long cap;            // capacity per bin (sites per bin), fixed_capacity
  double c0;                // constant removed before the transform
  float *rho;               // FP32 charge map (SIMT transform), or nullptr
  __nv_bfloat16 *rho_hi;    // BF16 hi/lo charge map (tensor-core transform), or nullptr
  __nv_bfloat16 *rho_lo;
  double *dens_out;         // optional FP64 copy (stage entry)
  int vec4;                 // set by launch_density_final: every pointer allows 16-byte groups
  unsigned long long *sums; // [kOverlapWords], zero between launches
  unsigned *ticket;
  double *overlap;          // where the overlap goes, or nullptr: into sc and the log
  DevScalars *sc;
  IterLog *log;
  NormArgs norms;           // with part2 set, one more CTA adds the step norms up
};

// C = A B with leading dimensions lda / ldb / ldc.  a_mir = +1 / -1 reads
// A(r, k) as A(r, k) +/- A(r, a_full - 1 - k) (columns folded about the
// middle of a_full); b_mir likewise folds B's rows about the middle of
// b_full.  The spectral epilogue takes output row r as frequency
// ky = 2 r + row_par (row_par < 0: ky = r) and, with col_split, column c as
// kx = 2 c (c < N/2) or 2 (c - N/2) + 1 (even frequencies first).
struct GemmOp {
  const float *A;
  const float *B;
  float *C;
  float *C2;
  int lda, ldb, ldc;
  int a_mir, a_full;
  int b_mir, b_full;
  int row_par, col_split;
};

struct SpectralArgs {
  const float *wx, *gx2;   // [BX]: pi kx / W, 2(1 - cos(pi kx / W))
  const float *wy, *gy2;   // [BY]
  float scale;             // 4 / (W H)
  float *phi;              // optional scaled potential spectrum
};

struct StepArgs {
  uint32_t N;
  int BX, BY;
  int isx, isy;              // sites per bin along x / y
  float maxx, maxy;
  float2 *look;             // [N] (fixed cells follow in the same buffer)
  const float2 *half;       // nullptr => unit cells
  const float *area;
  const uint8_t *mflag;     // [N] 1 for a macro (w*h > 1), nullptr when there are none
  const uint32_t *mac_idx;  // [n_mac] the macros' cell ids, ascending
  uint32_t n_mac;
  const float *pw;
  unsigned long long *acc;  // [N] packed WA accumulator, read then zeroed
  double grad_inv;          // 1 / WaArgs::grad_scale
  const float *Ex, *Ey;
  float2 *x, *xp, *g, *gprev;
  float2 *tmp_wl, *tmp_den; // [N] scratch for the penalty-initialisation phase
  const double *mom;        // momentum per iteration
  DevScalars *sc;
  IterLog *log;
  double *part;             // [4 * grid] block sums of the first half
  double *part2;            // [2 * grid] of the step norms
  double *part_b;           // [4 * grid] of the penalty-initialisation pass
  unsigned *bar;            // grid barrier: words 0-1 are one 64-bit arrival count
  unsigned *ticket;
  unsigned long long *dens; // density map that takes the next look-ahead, or nullptr
  int mode;                 // 0: full step (cooperative); 1: gather only (tmp_den <- density
                            // gradient); 2/3/4: first half / penalty-init pass / second half
};

struct SnapArgs {
  uint32_t n;
  const float2 *x;
  float2 *pos;         // [n] copy of the positions
  DevScalars *sc_out;  // copy of the scalars
  NormArgs norms;
};

struct HpwlArgs {
  const uint32_t *net_off;
  const uint32_t *pin_cell;
  const uint8_t *has_driver;
  const int2 *loc;          // [N + F] integer pin locations
  uint32_t NN;
  unsigned long long *total;
};

cudaError_t launch_wa(const WaArgs &a, int grid, cudaStream_t s);
cudaError_t launch_scatter(const ScatterArgs &a, int grid, cudaStream_t s);
// after: whether the launch may start before the kernel ahead of it in the
// stream has ended (it waits for that kernel's results itself).
cudaError_t launch_density_final(const FinalArgs &a, int grid, cudaStream_t s, bool after = false);
// C[b] = A[b] (M x K) * B[b] (K x N), row-major FP32; batches from ops[0..nb).
// tile: 64 (CTA tile edge), 32 (where 64 doesn't divide K: panels of 32 x 32)
// or, where 64 doesn't divide K, 16 (panels of 16 x 32), 0 = pick by grid size.  When 64 divides K the sum is
// split into four K quarters (a cluster of four CTAs per tile) added in
// quarter order; either way all tiles sum every output in the same order, so
// the tile never changes the bits.  after: the panels may launch while the
// kernel before them ends.
cudaError_t launch_sgemm(const GemmOp *ops_dev, int nb, int M, int N, int K, cudaStream_t s, int tile = 0,
                         bool after = false);
// As above with the spectral epilogue: C = Ex_hat, C2 = Ey_hat.
cudaError_t launch_sgemm_spectral(const GemmOp *ops_dev, int nb, int M, int N, int K,
                                  const SpectralArgs &sp, cudaStream_t s, int tile = 0, bool after = false);
// Products 2j and 2j+1 are the halves E and O (fly[j].E, fly[j].O: M x N) of a
// folded transform; as above, with the butterfly that completes it (see
// api.cu):
// cols: out[r][x] = E[r][x] + O[r][x], out[r][2N-1-x] = sig (E - O);
// rows: out[y][x] = E[y][x] + O[y][x], out[2M-1-y][x] = sig (E - O).
// The panels write the result alone, the other forms E and O too.
struct FlyOp {
  const float *E, *O;
  float *out;
  float sig;
};
cudaError_t launch_sgemm_fly(const GemmOp *ops_dev, const FlyOp *fly_dev, int nb, int M, int N, int K, bool cols,
                             cudaStream_t s, int tile = 0, bool after = false);
// Rows of the panels that a product runs as (one launch, with the butterfly),
// 0 for none.
int sgemm_panel(int M, int N, int nb, int K, int tile);
// block: step_block; grid: at most step_max_grid for the cooperative form.
cudaError_t launch_step(const StepArgs &a, int grid, int block, cudaStream_t s);
// The same step as three ordinary launches (modes 2, 3, 4): no grid barrier,
// safe beside long-running kernels of other streams.
cudaError_t launch_step_split(const StepArgs &a, int grid, int block, cudaStream_t s);
int step_block(int device, uint32_t cells);
int step_max_grid(int device, int block);
cudaError_t launch_snapshot(const SnapArgs &a, cudaStream_t s);
cudaError_t launch_hpwl(const HpwlArgs &a, int grid, cudaStream_t s);

// The stage entries' arrays: x and y apart in pinned host memory, which the
// kernels read and write over the bus, (x, y) pairs on the device.
constexpr int kIoPairs = 5;
struct IoArgs {
  uint32_t n;
  size_t pitch;                    // elements from one host array to the next (a multiple of 4)
  float *host;                     // [2 pairs][pitch]: x and y of pair 0, of pair 1, ...
  int pairs;
  float2 *pair[kIoPairs];
  unsigned long long *acc;         // packed WA gradient, or nullptr (see the launches)
  double scale;
};
// pair[k][i] = (host[2k][i], host[2k + 1][i]).  With acc and scale 0: acc
// zeroed; with acc and a scale: pair[1] is the WA gradient, packed into acc.
cudaError_t launch_io_in(const IoArgs &a, cudaStream_t s);
// The other way.  With acc: pair 0 comes from the packed gradient times scale
// and acc is zeroed.
cudaError_t launch_io_out(const IoArgs &a, cudaStream_t s);
// rho = d - c0 of n density values in pinned host memory, FP32 or as BF16
// hi / lo planes (rho == nullptr).
cudaError_t launch_io_rho(const double *d, size_t n, double c0, float *rho, __nv_bfloat16 *hi, __nv_bfloat16 *lo,
                          cudaStream_t s);

constexpr int kWaBlock = 256;
constexpr int kScatterBlock = 256;
constexpr int kFinalBlock = 256;
constexpr int kStepBlock = 512;
constexpr int kHpwlBlock = 256;

}  // namespace eplace
