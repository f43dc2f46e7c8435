// tri_step_launch.h -- host side of the step kernels: what one domain's
// step needs (device pointers and sizes) and the launch functions.  The
// kernels are instantiated in two translation units: tri_step_f64.cu (IEEE,
// no contraction: bit-exact with the reference) and tri_step_f32.cu (FP32
// precision form, approximate division and square root).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "tri_types.cuh"

namespace tri {

constexpr int kStripCols = 30;   // interior columns per warp tile of the flux kernel
constexpr int kFluxVariants = 5; // register budgets (FluxBudget)
constexpr int kWetCols = 128;    // columns per block of the staged wet-dry/dt pass (single-launch batches)
// Blocks of 128 threads per SM that the flux kernel's register-budget
// variants are compiled for (__launch_bounds__ minimum), at most 128, 96, 80,
// 72 and 64 registers a thread in FP64 (from 96 down they spill to L1), 96, 80,
// 64, 48 and 40 in FP32.  flux_shape's comment has the default and what the
// others measured; the autotuner times all on a domain's own state.
template <typename T>
struct FluxBudget;
template <>
struct FluxBudget<double> {
  static constexpr int v0 = 4, v1 = 5, v2 = 6, v3 = 7, v4 = 8;
};
template <>
struct FluxBudget<float> {
  static constexpr int v0 = 5, v1 = 6, v2 = 8, v3 = 10, v4 = 12;
};

// Default launch shape of the flux kernel: register budget and tile height.
// tiles(rb): warp tiles of height rb in all; share: the part of them that is
// computed in a step (the others are dry and skipped).  What decides is how
// many tiles there are for `slots` = 16 resident warps per SM:
//  - few (a small grid): a launch lasts as long as one tile, whose rows are a
//    serial chain (about 2.5 us each), so the lowest height whose tiles are
//    resident at once (rain on 256^2, FP64: 16 us with 1 row, 27 with 8; 512^2:
//    26 with 4, 33 with 8);
//  - many: the tallest that leaves a warp about four tiles, since a tile
//    repeats one row of faces above it (rain on 2048^2, FP64: 199 us with 12
//    rows, 214 with 4; FP32 4096^2: 442 with 32, 468 with 6) and the last
//    round of tiles idles half the warps.
// FP64 takes the largest register budget (few spills; more warps are not
// faster: bowl 2048^2 97.4 us at 4 blocks per SM, 100.0 at 5, 112 at 6).  FP32
// is bound by issue and takes 8 blocks per SM (rain 2048^2 129 us, 137 at 5),
// but where one round holds all tiles the largest budget (bowl 256^2 12.6 us,
// 14.0).  A batch, which reads its context from shared memory and spills more,
// takes 6 while its tiles are short (members, cells in all, height: 11, 1.0 M, 8
// rows 58.9 us a step, 61.2 at 8 blocks; 9, 1.2 M, 8 rows 67.1 and 68.6; 24, 2.6
// M, 8 rows 123.9 and 124.2), 8 from 12 rows on (16, 4.0 M 172.0 us at 6 and
// 171.7 at 8; 24, 6.0 M 233.1 and 230.7; 24, 9.6 M 350.6 and 342.8; 48, 16.3 M
// 558 and 548; 256, 263 M 8369 and 8168).
struct FluxShape {
  int variant, rb;
};
template <typename F>
FluxShape flux_shape(bool fp64, bool batch, double share, F tiles) {
  constexpr double slots = 148 * 16;
  for (int rb = 1; rb <= 4; rb++)
    if (share * (double)tiles(rb) <= slots) return {0, rb};
  int best = 4;
  for (int rb : {6, 8, 12, 16, 24, 32})
    if (share * (double)tiles(rb) >= 4 * slots) best = rb;
  return {fp64 ? 0 : (batch && best < 12 ? 1 : 2), best};
}
// What the autotuners time: every budget at heights 1 to 32, and the default
// shape where its height is another.
inline std::vector<FluxShape> tuning_shapes(FluxShape def) {
  std::vector<FluxShape> v;
  bool listed = false;
  for (int variant = 0; variant < kFluxVariants; variant++)
    for (int rb : {1, 2, 4, 8, 16, 32}) {
      v.push_back({variant, rb});
      listed |= variant == def.variant && rb == def.rb;
    }
  if (!listed) v.push_back(def);
  return v;
}
// Blocks of 128 threads per SM that the post kernels are compiled for: a stream
// with two rows of loads in flight per warp, so as many as its registers allow
// without spills (the batched one reads its parameters from memory and needs
// more).  FP64 at 8, 6 and 5: bowl 2048^2 33.2, 29.9 and 33.1 us with 4 us of
// timing, a 10-member ensemble step 110, 107.5 and 103.5 us; FP32 at 10, 8 and
// 7: rain on 4096^2 96, 110 and 127 us, a 24-member ensemble step 299, 247 and
// 253 us.
template <typename T>
struct PostBlocks;
template <>
struct PostBlocks<double> {
  static constexpr int v = 6, batch = 5;
};
template <>
struct PostBlocks<float> {
  static constexpr int v = 10, batch = 8;
};
// rows per block of the staged wet-dry/dt pass (its shared-memory tile),
// and output rows per group of its copies (each group on its own mbarrier)
template <typename T>
constexpr int kStageBand = sizeof(T) == 8 ? 4 : 8;
template <typename T>
constexpr int kStageGroupRows = 2;

struct StepArgs {
  DevClock* clk;
  void* h[2];
  void* qx[2];
  void* qy[2];
  void* z;             // FP64 form: DEM; FP32 form: offsets from the tile bases
  const double* zbase; // FP32 form: FP64 base level per 32x32 tile
  int ntc;             // tiles per row
  void* n2;
  void* maxh;
  const int32_t* zone;
  const void* rates;
  int rows, cols;
  int rb, flux_blocks, flux_variant;
  double dx, hextra;
  int nsrc;
  const int32_t* src_cells;
  const double* hyg_t;
  const void* hyg_v;
  const int32_t *bc_cells, *bc_types, *bc_start, *bc_nrows;
  const void *bc_v1, *bc_v2;
  float* arrival;
  float arrival_depth;
  // tile flags of the flux kernel ([2][tiles] by buffer + [tiles] pinned),
  // forcing by tile; skip_dry: dry tiles are skipped
  uint8_t* tflag;
  uint32_t ntiles;
  TileForcing tf;
  int open_boundaries;
  bool skip_dry;
  const int32_t* maxh_neg;  // device flag: a max depth that was uploaded is negative or NaN
};

// One time step (flux/update, forcing, post kernel).  ev: optional 4
// events around the two launches.
template <typename T>
int launch_step(const StepArgs& a, cudaStream_t s, cudaEvent_t* ev);
// Blocks of the post kernel (4 warps each) for `tiles` flux tiles, `per` a warp.
inline uint32_t post_blocks(uint32_t tiles, uint32_t per) { return (tiles + 4 * per - 1) / (4 * per); }
// Tiles per warp of a post launch over n domains (tiles(m) of each): the
// fewest with which all blocks are resident, `per_sm` on an SM.  A member's last
// block is rarely full, so the blocks' sum decides, not the tiles' total: a few
// blocks above the places took a second round (48 members of 256^2 to 1024^2,
// FP64, 8-row tiles: 1272 -> 1169 us a step; no change where they fit).  Up to
// twice the even share: with nearly as many members as places, or more, a
// second round of short blocks costs less than a large member in a few blocks
// (760 members of 16x18 and one of 1024^2, FP64: 454 us a step, 5537 with one
// block for each; 1200 in FP32 632 and 4493).
template <typename F>
uint32_t post_tiles_per_warp(size_t n, uint32_t per_sm, F tiles) {
  const uint64_t places = 148 * per_sm;
  uint64_t all = 0;
  for (size_t m = 0; m < n; m++) all += tiles(m);
  const uint32_t share = (uint32_t)std::max<uint64_t>((all + 4 * places - 1) / (4 * places), 1);
  for (uint32_t per = share; per <= 2 * share; per++) {
    uint64_t blocks = 0;
    for (size_t m = 0; m < n; m++) blocks += post_blocks(tiles(m), per);
    if (blocks <= places) return per;
  }
  return share;
}
// CFL dt of the current state into the slot the next step reads.
template <typename T>
int launch_initial_dt(const StepArgs& a, cudaStream_t s);
template <typename T>
void flux_occupancy(int variant, int* per_sm);

// A batch of member domains advanced together (one step of each member per
// batched step).  Device pointers.
struct BatchArgs {
  const void* mem;  // MemberDev<T>[nm] in device memory
  int nm;
  const int32_t* tile_member;  // member of every flux tile
  const int32_t* wet_member;   // member of every wet-dry block
  BatchCtl* ctl;
  uint32_t ntiles, nwet_blocks;
  int flux_blocks, flux_variant;
  const int32_t* post_member;  // member of every post kernel block
  uint32_t npost_blocks;
  TileForcing tf;
};
// The members' clocks of the first batched step of an advance.
template <typename T>
int launch_batch_clock(const BatchArgs& a, cudaStream_t s);
template <typename T>
int launch_batch_step(const BatchArgs& a, cudaStream_t s);
// Single-launch mode: nsteps batched steps in one launch of k_batch_steps
// (the control block's ticket and status and the progress counters must be
// zero); grid: the blocks resident at once (batch_steps_grid).  Register
// budget: variant 0 or (any other) 1 of FluxBudget.
template <typename T>
int launch_batch_steps(const BatchArgs& a, MemberProgress* prog, int nsteps, int grid, cudaStream_t s);
template <typename T>
int batch_steps_grid(int variant);
template <typename T>
void batch_flux_occupancy(int variant, int* per_sm);

// Kernel attributes (shared-memory sizes) on the current device; call before
// the first launch on a device.
template <typename T>
int prepare_kernels();

extern template int prepare_kernels<double>();
extern template int prepare_kernels<float>();
extern template int launch_step<double>(const StepArgs&, cudaStream_t, cudaEvent_t*);
extern template int launch_step<float>(const StepArgs&, cudaStream_t, cudaEvent_t*);
extern template int launch_initial_dt<double>(const StepArgs&, cudaStream_t);
extern template int launch_initial_dt<float>(const StepArgs&, cudaStream_t);
extern template void flux_occupancy<double>(int, int*);
extern template void flux_occupancy<float>(int, int*);
extern template int launch_batch_clock<double>(const BatchArgs&, cudaStream_t);
extern template int launch_batch_clock<float>(const BatchArgs&, cudaStream_t);
extern template int launch_batch_step<double>(const BatchArgs&, cudaStream_t);
extern template int launch_batch_step<float>(const BatchArgs&, cudaStream_t);
extern template int launch_batch_steps<double>(const BatchArgs&, MemberProgress*, int, int, cudaStream_t);
extern template int launch_batch_steps<float>(const BatchArgs&, MemberProgress*, int, int, cudaStream_t);
extern template int batch_steps_grid<double>(int);
extern template int batch_steps_grid<float>(int);
extern template void batch_flux_occupancy<double>(int, int*);
extern template void batch_flux_occupancy<float>(int, int*);

}  // namespace tri
