// setup_pool.h -- short-lived device memory: of the set-up passes (geometry
// decode, storage layout) and of the transfers that reorder a field or convert
// distributions.  Stream-ordered allocations from a memory pool of the library's
// own, one per device, outside hb_device_bytes.  Freeing returns the memory to the
// pool instead of unmapping it, which made a case's set-up take from 0.3 to 1 s by
// the frees alone; the pool keeps up to kSetupPoolKeep bytes between set-ups (what
// a lattice of about eight million sites needs) and gives the rest back at the next
// synchronisation.  A transfer's scratch (kScratch) goes back at once as far as it
// made the pool hold more than kScratchKeep: unmapping 100 MB takes 0.8 ms, a fifth
// of its transfer, 600 MB 3.8 ms.  Allocations of one set-up or transfer come from a
// SetupPool object, returned on every path.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/hemeb200.h"
#include "hb_common.h"

namespace hb {

constexpr uint64_t kSetupPoolKeep = (uint64_t)4 << 30;
constexpr uint64_t kScratchKeep = (uint64_t)128 << 20;
enum PoolUse { kSetup, kScratch };

// The library's pool on `device` (created on first use; `fresh` makes a new one,
// for a device whose context was replaced since).
cudaMemPool_t setup_pool(int device, bool fresh = false);

class SetupPool {
 public:
  SetupPool(int device, cudaStream_t stream, PoolUse use = kSetup)
      : device_(device), pool_(setup_pool(device)), stream_(stream), keep_(use == kScratch ? std::max(held(), kScratchKeep) : 0) {}
  SetupPool(const SetupPool&) = delete;
  SetupPool& operator=(const SetupPool&) = delete;
  ~SetupPool() {
    for (void* p : ptrs_) cudaFreeAsync(p, stream_);
    if (keep_ && held() > keep_) {
      cudaStreamSynchronize(stream_);  // freed memory can be unmapped once its stream is through
      cudaMemPoolTrimTo(pool_, keep_);
    }
  }
  template <class T>
  T* get(size_t count) {
    void* p = nullptr;
    const size_t bytes = (count ? count : 1) * sizeof(T);
    cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, pool_, stream_);
    if (e != cudaSuccess && e != cudaErrorMemoryAllocation && ptrs_.empty()) {
      cudaGetLastError();
      pool_ = setup_pool(device_, true);
      e = cudaMallocFromPoolAsync(&p, bytes, pool_, stream_);
    }
    if (e != cudaSuccess)
      throw Error{e == cudaErrorMemoryAllocation ? HB_ERR_OOM : HB_ERR_CUDA,
                  std::string("short-lived device memory: ") + cudaGetErrorString(e)};
    ptrs_.push_back(p);
    return static_cast<T*>(p);
  }

 private:
  // Bytes the pool holds, given out or not.
  uint64_t held() const {
    uint64_t v = 0;
    if (cudaMemPoolGetAttribute(pool_, cudaMemPoolAttrReservedMemCurrent, &v) == cudaSuccess) return v;
    cudaGetLastError();
    return 0;
  }
  int device_;
  cudaMemPool_t pool_;
  cudaStream_t stream_;
  uint64_t keep_;  // 0: everything
  std::vector<void*> ptrs_;
};

}  // namespace hb
