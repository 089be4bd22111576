// step_tiles.cuh -- block roles and the launch of the one-kernel time step
// (kernels_f64.cu, kernels_mixed.cu).
#pragma once

#include <cuda_runtime.h>

#include "device.h"

namespace hb {
namespace {

constexpr int kStepBlock = 128;

// Blocks of a step kernel's grid, in order: `io` blocks of boundary records with
// iolet links (from record io_first), `gzs` blocks of GZS wall links, then `wall`
// blocks of boundary records without iolet links spread among `bulk` blocks of
// sites: one wall block every `period` blocks.
struct StepTiles {
  int io, gzs, wall, bulk, period, io_first;
  int blocks() const { return io + gzs + wall + bulk; }
};

// `sites` storage sites per bulk block.
inline StepTiles step_tiles(const StepArgs& a, int which, int sites = kStepBlock) {
  StepTiles t{};
  auto blocks = [](int64_t n, int per) { return (int)((n + per - 1) / per); };
  t.io_first = a.gen.G_noiolet;
  if (which & kLaunchIoletRecords) t.io = blocks(a.gen.G - t.io_first, kStepBlock);
  if (which & kLaunchWallRecords) {
    t.gzs = blocks(a.gzs_n, kStepBlock);
    t.wall = blocks(t.io_first, kStepBlock);
  }
  if (which & kLaunchBulk) t.bulk = blocks(a.n, sites);
  t.period = t.wall > 0 ? (t.wall + t.bulk) / t.wall : 1;
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
