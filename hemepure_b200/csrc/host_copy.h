// host_copy.h -- copies between device memory and the caller's pageable arrays
// through pinned pieces.
//
// A pageable cudaMemcpy runs on one host thread inside the driver, which also
// takes the page faults of a freshly allocated destination.  Here several
// threads each own a pinned piece: one piece crosses to the host while the
// others are copied to or from the caller's array, so the faults and the copies
// run in parallel with the transfer.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <initializer_list>

namespace hb {

class HostCopy {
 public:
  HostCopy();
  HostCopy(const HostCopy&) = delete;
  HostCopy& operator=(const HostCopy&) = delete;
  ~HostCopy();
  // `dst` <- `src` on `stream`.  A download is done when its call returns; after an
  // upload the caller waits for the stream before `src` changes, as it does for the
  // kernel that reads `dst` (a wait here as well: 6 us of the 130 that set 13k sites).
  void to_host(void* dst, const void* src, size_t bytes, int device, cudaStream_t stream) { run(dst, const_cast<void*>(src), bytes, true, device, stream); }
  void to_device(void* dst, const void* src, size_t bytes, int device, cudaStream_t stream) { run(const_cast<void*>(src), dst, bytes, false, device, stream); }

  // Fields of `width` values a site, [width][stride] in storage order on the device, to
  // `out` as [n][width] in reference order (`order`: storage index to reference index;
  // `order_dev` the same on the device, or null: it is then uploaded once for them all).
  // A kernel reorders them, so that the host only receives them (density, velocity and
  // stress of 4M sites: 170 ms with the reordering on the host, 12 ms so); with no device
  // memory left for the reordered copy the host reorders it.  Fields without `out` are
  // passed over.
  struct Field {
    const double* field;
    int width;
    double* out;
  };
  void fields_to_reference(std::initializer_list<Field> fields, int64_t stride, const int* order, const int* order_dev, int n,
                           int device, cudaStream_t stream);

 private:
  // Pinned pieces are the process's, not the object's: pinning takes 1 ms (5 ms as a
  // fresh allocation), which a handle that is opened, stepped and read once would pay
  // each time (first pass of a new 257k-site handle, 25 steps and its fields, 9.5 -> 4.4
  // ms).  A transfer borrows a set of kThreads pieces; further transfers beside kSets of
  // them are pageable.  A set that the cores have just read is slow to write again
  // (a 4.6 MB field 0.50 ms with one set, 0.45, 0.38, 0.33 with two to four in turn), so
  // every kTurns transfers one more joins, up to kSets; all but one are given back with
  // the last object.
  static constexpr int kThreads = 8, kSets = 4, kTurns = 8;
  static constexpr size_t kPiece = (size_t)512 << 10;
  // Up to these sizes one pageable copy: a download gains by its destination's page
  // faults taken in parallel, an upload only by the second copy.
  static constexpr size_t kDirectDown = (size_t)4 << 20, kDirectUp = (size_t)64 << 20;
  void run(void* host, void* dev, size_t bytes, bool down, int device, cudaStream_t stream);
  class Sets;
  struct Borrowed;
};

}  // namespace hb
