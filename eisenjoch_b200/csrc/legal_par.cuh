// legal_par.cuh -- parallel exact greedy legaliser on the GPU (legal_par.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace eplace {

// Macros that a round works on at once.
constexpr uint32_t kLpWindow = 2048;

// Unit cells of a window (a power of two; with two CTAs per SM their searches
// run in one wave).
constexpr int kUnitWindowBits = 8;
constexpr uint32_t kUnitWindow = 1u << kUnitWindowBits;

// Sites that a search lists at most.
constexpr int kLpRingMax = 64;

// Sites kept of a unit cell's search.
constexpr int kLpCand = 16;

// Status of a graph without windows whose unit cells need them.
constexpr int32_t kLpTied = 3;

// State of one legalisation in flight, in device memory.
struct LpState {
  uint32_t base;       // macros [0, base) have their final anchors
  uint32_t rounds;     // macro rounds run
  uint32_t first;      // lowest macro whose choice changed in this round
  uint32_t ticket;     // CTAs of the claim kernel that have finished
  uint32_t nfreed;     // blocks given up in this round
  uint32_t nwork[2];   // macros to choose in this and in the next round
  uint32_t npend;      // unit cells left to k_lp_units
  uint32_t taken;      // of them, those that a CTA has taken up
  uint32_t ties;       // unit cells that share a target with tie_least or more
  uint32_t tied;       // too many do: the unit cells are placed in windows
  uint32_t wbase;      // unit cells [0, wbase) have been placed in windows
  int32_t status;      // 0 ok, 1 no free site for some cell, 2 round cap, kLpTied, 4 cancelled
};

// A block that a macro gave up in a round.
struct LpFreed {
  int32_t q, tile, w, h;
};

struct LpArgs {
  const float2 *pos;       // [N] continuous positions (the checkpoint)
  const uint32_t *order;   // [n] legalisation order: macros first, then unit cells, solver order within each
  const uchar2 *fsize;     // [N] footprint (w, h) per cell id, or nullptr when every cell is 1x1
  uint32_t n;              // cells to place
  uint32_t n_mac;          // macros among them (the first of the order)
  int W, H, WR;            // chip sites, 64-bit words per row
  int SW;                  // 32-site segments per row
  const uint64_t *free0;   // [H * WR] free map with the fixed cells bound (bit set = free)
  int32_t *own;            // [H][32 SW] lowest order index that claims the site; -1: never free, or no site
  uint2 *seg;              // [H][SW] what is known of each 32-site segment (see legal_par.cu)
  int32_t *choice;         // [n_mac] anchor (tile = y * W + x) of each macro; -1: none yet, -2: none free
  double *mcost;           // [n_mac] its cost
  LpFreed *freed;          // [kLpWindow] blocks given up in this round
  uint32_t *work;          // [2][kLpWindow] macros to choose in this and in the next round
  uint32_t *queued;        // [n_mac] why a macro is in the next list: 1: block lost or none yet, 2: may gain
  int32_t *cand;           // [n - n_mac][kLpCand] next best sites of a unit cell, best first; -1: no more
  unsigned long long *hint;  // [lp_hint_count] radii without an open anchor (see legal_par.cu)
  int32_t *near;           // [n - n_mac] site a unit cell took near its target, -1: none
  uint32_t *pend;          // [n - n_mac] order indices of the cells left to k_lp_units, ascending
  uint32_t *left;          // [lp_chunks] how many of them in each kLpChunk unit cells
  unsigned long long *tie_key;  // [tie_mask + 1] table of the unit cells' targets
  uint32_t *tie_count;     // [tie_mask + 1] how many have each
  uint32_t tie_mask;       // lp_tie_entries - 1
  float tie_scale;         // filled in by lp_build_graph, like the next two: squares per site that tell targets apart
  uint32_t tie_least;      // cells of one target from which they count as ties
  bool tie_few;            // decided before the first pass, from a sample, without the table
  bool tie_loop;           // the graph has the loop over them (else the status says that they are needed)
  int32_t *list;           // [kUnitWindow][kLpRingMax] sites of least cost of the window's cells
  int32_t *list_len;       // [kUnitWindow] how many
  LpState *st;
  int2 *sites;             // [N] anchor of every cell (out)
  int2 *loc;               // [N] pin location anchor + (size - 1) / 2 (out), or nullptr
  double *cost;            // [n] cost of each placement, by order index (out)
  double *disp;            // [1] total displacement, summed in order (out)
  int32_t *status;         // [1] 0 ok, 1 no free site, else an internal limit (out)
  const int32_t *cancel;   // [1] set by the host: the result is no longer wanted, and what there is is not one
  uint32_t max_rounds;
  cudaGraphConditionalHandle handle;  // of the loop over the macro rounds
  cudaGraphConditionalHandle many;    // of the pass over all unit cells in order
  cudaGraphConditionalHandle windows; // of the loop over the windows
};

// The hints: one entry per size class (1 .. 8 sites) and 16 x 16 sites.
constexpr int kLpHintClasses = 8;
inline size_t lp_hint_count(int W, int H) { return (size_t)kLpHintClasses * ((W + 15) / 16) * ((H + 15) / 16); }

// Entries of the table of the unit cells' targets.
inline size_t lp_tie_entries(size_t units) {
  size_t n = 64;
  while (n < 2 * units) n *= 2;
  return n;
}

// Unit cells that a CTA looks through for ones that are left.
constexpr uint32_t kLpChunk = 1024;
inline size_t lp_chunks(size_t units) { return (units + kLpChunk - 1) / kLpChunk; }

// Chips the device legaliser takes (tile ids and per-site claims sized by
// W x H): up to 4096 x 4096 sites.
inline bool legalize_supported(int W, int H) { return W > 0 && H > 0 && W <= 4096 && H <= 4096; }

// A legalisation as one CUDA graph: initialisation, a device-side while
// loop over the macro rounds (when there are macros), the unit cells (all at
// once and the few left over, or, where too many are, all in order or, where
// many share a target, in windows: an if node with a while node in it; few
// cells all in order, or in windows), the displacement sum.  Built once per slot and problem load; launched per
// checkpoint.
struct LpGraph {
  cudaGraphExec_t exec = nullptr;
  cudaGraph_t graph = nullptr;
  void clear();
  ~LpGraph() { clear(); }
};

// Builds the graph for args `a` (the handles are filled in).
// windows: also where that costs a conditional node of its own (few cells).
cudaError_t lp_build_graph(LpArgs a, LpGraph &g, bool windows);

}  // namespace eplace
