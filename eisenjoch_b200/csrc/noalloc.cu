// noalloc.cu -- the density stage (cell -> bin overlap map and overlap
// metric) for callers that cannot allocate device memory.
//
// Some callers cannot call cudaMalloc: a real-time control loop that must
// not take the allocator's locks or stall on it, a host application whose
// device memory is handed out by another component (its own pool, a
// framework's caching allocator) and may not be grown behind its back, or
// code running under a fixed device-memory budget.  They own their inputs
// and outputs already; what they cannot do is give this library the working
// memory the density stage needs (the fixed-point accumulation map, the
// overlap's sums and the completion counter).  For them the scratch
// lives in one file-scope __device__ array, sized for at most
// kNoAllocMaxBins bins (512 x 512).  It is part of the library image: every
// GPU that loads libeplace.so holds it (about 2 MiB) until the process
// exits.
//
// The kernels are the library's own scatter and finalise kernels; only the
// scratch they are given differs.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <mutex>

#include "../../include/eplace.h"
#include "kernels.cuh"

namespace eplace {
namespace {

constexpr size_t kNoAllocMaxBins = 512 * 512;

// Layout of the scratch array (byte offsets, each 256-aligned):
//   [0, kMapBytes)                fixed-point bin map, must start at zero
//   [kSumOff, +256)               the overlap's sums, cleared by each call
//   [kTicketOff, +256)            completion counter, cleared by each call
constexpr size_t kMapBytes = kNoAllocMaxBins * sizeof(unsigned long long);
constexpr size_t kSumOff = kMapBytes;
constexpr size_t kTicketOff = kSumOff + 256;
constexpr size_t kScratchBytes = kTicketOff + 256;

static __device__ __align__(256) unsigned char g_density_scratch[kScratchBytes];

// Device address of g_density_scratch.  In host code the symbol is only a
// host-side stand-in, so its device address is looked up with the device
// current (cudaGetSymbolAddress) at set-up and cached per device.  The
// cache entry also records the unique id of the CUDA context it was looked
// up in: after cudaDeviceReset (or any other end of the primary context)
// the module is loaded again, possibly elsewhere, and the next call looks
// the address up again instead of using a stale one.  The driver calls are
// reached through the runtime's entry-point table, so the library does not
// link libcuda directly.
typedef CUresult (*CtxGetCurrentFn)(CUcontext *);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long *);

struct ScratchSlot {
  unsigned long long ctx_id = 0;
  void *addr = nullptr;
  int sms = 0;
  bool dirty = false;  // a call's launches did not all happen
};

std::mutex g_mu;
ScratchSlot g_slot[128];
CtxGetCurrentFn g_ctx_current = nullptr;
CtxGetIdFn g_ctx_id = nullptr;

// Id of the current context; 0 when no context is current yet.
eplace_status current_context_id(unsigned long long *id) {
  *id = 0;
  if (!g_ctx_current || !g_ctx_id) {
    void *f1 = nullptr, *f2 = nullptr;
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) != cudaSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) != cudaSuccess ||
        q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2)
      return EPLACE_ERR_CUDA;
    g_ctx_current = reinterpret_cast<CtxGetCurrentFn>(f1);
    g_ctx_id = reinterpret_cast<CtxGetIdFn>(f2);
  }
  CUcontext c = nullptr;
  if (g_ctx_current(&c) != CUDA_SUCCESS) return EPLACE_ERR_CUDA;
  if (!c) return EPLACE_OK;
  return g_ctx_id(c, id) == CUDA_SUCCESS ? EPLACE_OK : EPLACE_ERR_CUDA;
}

eplace_status scratch_for_current_device(void **out, bool *dirty, int *sms) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return EPLACE_ERR_NO_DEVICE;
  if (dev < 0 || dev >= 128) return EPLACE_ERR_NO_DEVICE;
  std::lock_guard<std::mutex> g(g_mu);
  unsigned long long id = 0;
  eplace_status st = current_context_id(&id);
  if (st != EPLACE_OK) return st;
  ScratchSlot &slot = g_slot[dev];
  if (id == 0 || !slot.addr || slot.ctx_id != id) {
    // Set-up: the symbol's device address in the current context (the
    // lookup also creates the device's primary context when none is current
    // yet, so the id is read again afterwards).
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_density_scratch) != cudaSuccess || !p) return EPLACE_ERR_CUDA;
    st = current_context_id(&id);
    if (st != EPLACE_OK) return st;
    if (id == 0) return EPLACE_ERR_CUDA;
    if (cudaDeviceGetAttribute(&slot.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return EPLACE_ERR_CUDA;
    slot.addr = p;
    slot.ctx_id = id;
    slot.dirty = false;  // a fresh image: all zero
  }
  *out = slot.addr;
  *dirty = slot.dirty;
  *sms = slot.sms;
  return EPLACE_OK;
}

// Whether the next call on the current device has to clear the scratch.
void scratch_state(bool dirty) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return;
  std::lock_guard<std::mutex> g(g_mu);
  g_slot[dev].dirty = dirty;
}

}  // namespace
}  // namespace eplace

using namespace eplace;

extern "C" eplace_status eplace_density_noalloc(const float *pos_xy, const float *half_wh, uint32_t num_cells,
                                                int32_t width, int32_t height, int32_t bins_x, int32_t bins_y,
                                                double *density, double *overlap, void *stream) {
  if (width <= 0 || height <= 0 || bins_x <= 0 || bins_y <= 0 || width % bins_x || height % bins_y)
    return EPLACE_ERR_INVALID;
  if ((size_t)bins_x * (size_t)bins_y > kNoAllocMaxBins) return EPLACE_ERR_INVALID;  // over the scratch size
  if (!density || !overlap || (num_cells && !pos_xy)) return EPLACE_ERR_INVALID;
  // The kernels read (x, y) and (w/2, h/2) as 8-byte pairs and write
  // doubles: a misaligned pointer would fault the caller's whole context.
  if (((uintptr_t)pos_xy | (uintptr_t)half_wh | (uintptr_t)density | (uintptr_t)overlap) & 7u)
    return EPLACE_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int nb = bins_x * bins_y, sx = width / bins_x, sy = height / bins_y;
  ScatterArgs a{reinterpret_cast<const float2 *>(pos_xy), reinterpret_cast<const float2 *>(half_wh), nullptr,
                nullptr, 0u, num_cells, bins_x, bins_y, sx, sy, nullptr};
  FinalArgs f{};
  f.nb = nb;
  f.cap = fixed_capacity((long long)sx * sy);
  f.dens_out = density;
  f.overlap = overlap;
  void *base = nullptr;
  bool dirty = false;
  int sms = 0;
  eplace_status st = scratch_for_current_device(&base, &dirty, &sms);
  if (st != EPLACE_OK) return st;
  unsigned char *b = static_cast<unsigned char *>(base);
  auto *map = reinterpret_cast<unsigned long long *>(b);
  a.dens = f.dens = map;
  f.sums = reinterpret_cast<unsigned long long *>(b + kSumOff);
  f.ticket = reinterpret_cast<unsigned *>(b + kTicketOff);
  // The scratch keeps the previous call's contents.  Its map starts at zero and
  // is zero again when every call has run (a call's finalise zeroes every bin
  // that its scatter may have added to); after a call whose second launch
  // failed it is cleared first.  Sums and counter are cleared by the scatter:
  // calls that overlapped by mistake may leave them anyhow.
  const bool clear = dirty;
  if (clear) {
    // a clear that is captured into a graph has not run yet: the mark stays
    cudaStreamCaptureStatus capture;
    if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) return EPLACE_ERR_CUDA;
    if (cudaMemsetAsync(base, 0, kScratchBytes, s) != cudaSuccess) return EPLACE_ERR_CUDA;
    dirty = capture != cudaStreamCaptureStatusNone;
  }
  if (!num_cells) {
    if (cudaMemsetAsync(f.sums, 0, kScratchBytes - kSumOff, s) != cudaSuccess) return EPLACE_ERR_CUDA;
  } else {
    a.sums = f.sums;
    a.ticket = f.ticket;
    long long g = ((long long)num_cells + kScatterBlock - 1) / kScatterBlock;
    if (g > (long long)sms * 16) g = (long long)sms * 16;
    if (launch_scatter(a, (int)g, s) != cudaSuccess) return EPLACE_ERR_CUDA;
  }
  long long fg = ((long long)nb / 4 + kFinalBlock - 1) / kFinalBlock;
  if (fg > (long long)sms * 4) fg = (long long)sms * 4;
  if (fg < 1) fg = 1;
  if (launch_density_final(f, (int)fg, s, num_cells != 0) != cudaSuccess) {
    scratch_state(true);
    return EPLACE_ERR_CUDA;
  }
  if (clear) scratch_state(dirty);
  return EPLACE_OK;
}
