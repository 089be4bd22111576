// step_tiles.cuh -- block roles and the launch of the one-kernel time step
// (kernels_f64.cu, kernels_mixed.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device.h"

namespace hb {
namespace {

constexpr int kStepBlock = 128;

// Blocks of a step kernel's grid, in order: `links` blocks of iolet links, `io`
// blocks of boundary records with such links (from record io_first), `gzs` blocks of GZS wall links, then `wall`
// blocks of boundary records without iolet links spread evenly among `bulk` blocks
// of `tiles` tiles of sites each.
struct StepTiles {
  int links, io, gzs, wall, bulk, tiles, io_first;
  uint32_t wall_share;  // of the last two kinds, 32-bit fraction rounded up
  int blocks() const { return links + io + gzs + wall + bulk; }
  // The wall blocks before block b of the last two kinds.
  __device__ __forceinline__ int walls_before(int b) const { return bulk > 0 ? (int)__umulhi((unsigned)b, wall_share) : b; }
};

// `resident`: blocks that fit an SM.  A bulk block walks up to kStepTiles tiles,
// which hides the chain from a tile's run ids to its offsets to its distributions
// and the turnover of blocks, as long as the grid keeps kStepWaves times the blocks
// that run at once (fewer leave SMs idle at the end).  One tile against four: 4M-site
// pipe FP64 234 -> 214 us a step, FP32 130 -> 122, FP16 98 -> 86; eight are slower
// again (FP64 220), and a 497k-site lattice wants two or three (36.2 -> 34.3 us; four
// 35.6).
constexpr int kStepTiles = 4, kStepWaves = 2, kStepSMs = 148;

inline StepTiles step_tiles(const StepArgs& a, int which, int resident) {
  StepTiles t{};
  auto blocks = [](int64_t n, int64_t per) { return (int)((n + per - 1) / per); };
  t.io_first = a.gen.G_noiolet;
  if (which & kLaunchIoletRecords) {
    t.links = blocks(a.iol_n, kStepBlock);
    t.io = blocks(a.gen.G - t.io_first, kStepBlock);
  }
  if (which & kLaunchWallRecords) {
    t.gzs = blocks(a.gzs_n, kStepBlock);
    t.wall = blocks(t.io_first, kStepBlock);
  }
  t.tiles = 1;
  if (which & kLaunchBulk) {
    const int n = blocks(a.n, kStepBlock);
    t.tiles = std::max(1, std::min(kStepTiles, n / (kStepSMs * resident * kStepWaves)));
    t.bulk = blocks(n, t.tiles);
  }
  if (t.bulk > 0) t.wall_share = (uint32_t)((((uint64_t)t.wall << 32) + (uint64_t)(t.wall + t.bulk) - 1) / (uint64_t)(t.wall + t.bulk));
  return t;
}

// The boundary on its own: iolet links, GZS wall links, then every record (as `io`).
inline StepTiles boundary_tiles(const StepArgs& a) {
  StepTiles t{};
  auto blocks = [](int64_t n) { return (int)((n + kStepBlock - 1) / kStepBlock); };
  t.links = blocks(a.iol_n);
  t.gzs = blocks(a.gzs_n);
  t.io = blocks(a.gen.G);
  return t;
}

// Wait for the step that wrote this step's input, then let the next step's blocks
// be launched as this one's blocks leave (a no-op in a plain launch).  Only
// constant tables may be read before it.
__device__ __forceinline__ void wait_previous_step() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch allowing the grid to start while its predecessor in the stream drains
// (the kernel itself waits, wait_previous_step).
template <class F, class... A>
void launch_dependent(F* kernel, int grid, cudaStream_t st, const A&... args) {
  if (grid <= 0) return;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kStepBlock);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace
}  // namespace hb
