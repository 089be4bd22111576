// host_copy.cpp -- see host_copy.h.
#include "host_copy.h"

#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/hemeb200.h"
#include "device.h"
#include "hb_common.h"
#include "setup_pool.h"

namespace hb {

namespace {

// The device of a transfer, current in the calling thread while it runs: its kernel
// and events need it, and a thread that only reads fields may have another.
class OnDevice {
 public:
  explicit OnDevice(int device) {
    if (cudaGetDevice(&before_) != cudaSuccess) before_ = device;
    if (before_ != device) cudaSetDevice(device);
    changed_ = before_ != device;
  }
  OnDevice(const OnDevice&) = delete;
  OnDevice& operator=(const OnDevice&) = delete;
  ~OnDevice() {
    if (changed_) cudaSetDevice(before_);
  }

 private:
  int before_ = 0;
  bool changed_ = false;
};

}  // namespace

// The process's sets of pinned pieces.  The memory is the library's own, registered
// with CUDA: should the device's context have been replaced since, it is still there
// and is registered again.
class HostCopy::Sets {
 public:
  static Sets& get() {
    static Sets* s = new Sets;  // handles may be destroyed after the statics are
    return *s;
  }
  // A set for one transfer; null without memory to pin, or with kSets lent already.
  // The sets take turns, another one joining after every kTurns transfers: the device
  // writes faster into memory that no core has read of late.
  unsigned char* take() {
    unsigned char* p = nullptr;
    {
      std::lock_guard<std::mutex> lock(mu_);
      const bool grow = free_.empty() || made_ < 1 + taken_ / kTurns;
      taken_ = std::min(taken_ + 1, kSets * kTurns);
      if (grow && made_ < kSets) {
        made_++;
      } else if (!free_.empty()) {
        p = free_.front();
        free_.erase(free_.begin());
      } else {
        return nullptr;
      }
    }
    if (!p) p = map();
    if (p && !pinned(p) && cudaHostRegister(p, kBytes, cudaHostRegisterPortable) != cudaSuccess) {
      cudaGetLastError();
      munmap(p, kBytes);
      p = nullptr;
    }
    if (!p) {
      std::lock_guard<std::mutex> lock(mu_);
      made_--;
      taken_ = 0;
      if (!free_.empty()) {
        p = free_.front();
        free_.erase(free_.begin());
      }
    }
    return p;
  }
  void give(unsigned char* p) {
    std::lock_guard<std::mutex> lock(mu_);
    free_.push_back(p);
  }
  void enter() {
    std::lock_guard<std::mutex> lock(mu_);
    users_++;
  }
  void leave() {
    std::lock_guard<std::mutex> lock(mu_);
    if (--users_ > 0) return;
    taken_ = 0;
    for (; free_.size() > 1; free_.pop_back(), made_--) {
      if (cudaHostUnregister(free_.back()) != cudaSuccess) cudaGetLastError();
      munmap(free_.back(), kBytes);
    }
  }

 private:
  Sets() { free_.reserve(kSets); }  // give() runs on every path out of a transfer
  static constexpr size_t kHugePage = (size_t)2 << 20, kBytes = kThreads * kPiece;
  // Two huge pages to pin instead of a thousand, and none shared with a child process:
  // CUDA would go on copying from and to a page that the next write leaves to the child.
  static unsigned char* map() {
    void* m = mmap(nullptr, kBytes + kHugePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == MAP_FAILED) return nullptr;
    unsigned char* lo = static_cast<unsigned char*>(m);
    const size_t head = (kHugePage - (uintptr_t)lo % kHugePage) % kHugePage, tail = kHugePage - head;
    if (head) munmap(lo, head);
    if (tail) munmap(lo + head + kBytes, tail);
    madvise(lo + head, kBytes, MADV_HUGEPAGE);
    madvise(lo + head, kBytes, MADV_DONTFORK);
    return lo + head;
  }
  static bool pinned(const void* p) {
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, p) == cudaSuccess) return attr.type == cudaMemoryTypeHost;
    cudaGetLastError();
    return false;
  }
  std::mutex mu_;
  std::vector<unsigned char*> free_;
  int made_ = 0, users_ = 0, taken_ = 0;
};

// A set and the events of one transfer.
struct HostCopy::Borrowed {
  unsigned char* set = nullptr;
  cudaEvent_t done[kThreads] = {};
  bool take() {
    set = Sets::get().take();
    if (!set) return false;
    for (cudaEvent_t& e : done)
      if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        e = nullptr;
        return false;
      }
    return true;
  }
  ~Borrowed() {
    for (cudaEvent_t e : done)
      if (e) cudaEventDestroy(e);
    if (set) Sets::get().give(set);
  }
};

HostCopy::HostCopy() { Sets::get().enter(); }
HostCopy::~HostCopy() { Sets::get().leave(); }

void HostCopy::run(void* host, void* dev, size_t bytes, bool down, int device, cudaStream_t stream) {
  auto check = [](cudaError_t e) {
    if (e != cudaSuccess) throw Error{HB_ERR_CUDA, std::string("host copy: ") + cudaGetErrorString(e)};
  };
  if (bytes == 0) return;
  const OnDevice on(device);
  bool pieces = bytes > (down ? kDirectDown : kDirectUp);
  if (pieces) {
    // Memory that CUDA knows (the caller pinned or allocated it through CUDA) needs no
    // pieces, and device memory must meet the copy's own check, not the host's memcpy.
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) cudaGetLastError();
    else if (attr.type != cudaMemoryTypeUnregistered) pieces = false;
  }
  // Without pinned memory or events to spare the copy still runs, as a pageable one.
  Borrowed b;
  pieces = pieces && b.take();
  if (!pieces) {
    check(cudaMemcpyAsync(down ? host : dev, down ? dev : host, bytes, down ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice,
                          stream));
    if (down) check(cudaStreamSynchronize(stream));
    return;
  }
  const size_t count = (bytes + kPiece - 1) / kPiece;
  const int threads = (int)std::min<size_t>(kThreads, count);
  cudaError_t err[kThreads];
  auto work = [&](int k) {
    unsigned char* piece = b.set + (size_t)k * kPiece;
    cudaError_t e = cudaSetDevice(device);
    for (size_t p = k; p < count && e == cudaSuccess; p += threads) {
      unsigned char* h = static_cast<unsigned char*>(host) + p * kPiece;
      unsigned char* d = static_cast<unsigned char*>(dev) + p * kPiece;
      const size_t len = std::min(kPiece, bytes - p * kPiece);
      if (down) {
        e = cudaMemcpyAsync(piece, d, len, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaEventRecord(b.done[k], stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(b.done[k]);
        if (e == cudaSuccess) std::memcpy(h, piece, len);
      } else {
        std::memcpy(piece, h, len);
        e = cudaMemcpyAsync(d, piece, len, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaEventRecord(b.done[k], stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(b.done[k]);
      }
    }
    err[k] = e;
  };
  std::vector<std::thread> pool;
  int started = 1;
  try {
    for (; started < threads; started++) pool.emplace_back(work, started);
  } catch (...) {
    // no more threads to be had: the pieces of the missing ones follow below
  }
  work(0);
  for (auto& t : pool) t.join();
  for (int k = started; k < threads; k++) work(k);
  for (int k = 0; k < threads; k++)
    if (err[k] != cudaSuccess) {
      cudaStreamSynchronize(stream);  // no copy may still use the pieces
      check(err[k]);
    }
}

void HostCopy::fields_to_reference(std::initializer_list<Field> fields, int64_t stride, const int* order,
                                   const int* order_dev, int n, int device, cudaStream_t stream) {
  auto check = [](cudaError_t e) {
    if (e != cudaSuccess) throw Error{HB_ERR_CUDA, std::string("field download: ") + cudaGetErrorString(e)};
  };
  int width = 0;
  for (const Field& f : fields)
    if (f.out) width = std::max(width, f.width);
  if (width == 0 || n <= 0) return;
  const OnDevice on(device);
  SetupPool tmp(device, stream, kScratch);
  double* rows = nullptr;
  try {
    rows = tmp.get<double>((size_t)n * width);
    if (!order_dev) {
      int* o = tmp.get<int>((size_t)n);
      check(cudaMemcpyAsync(o, order, (size_t)n * sizeof(int), cudaMemcpyHostToDevice, stream));
      order_dev = o;
    }
  } catch (const Error& e) {
    if (e.code != HB_ERR_OOM) throw;
    cudaGetLastError();
    rows = nullptr;
  }
  std::vector<double> v(rows ? 0 : (size_t)n);
  for (const Field& f : fields) {
    if (!f.out) continue;
    if (rows) {
      launch_to_reference(f.field, stride, f.width, order_dev, n, rows, stream);
      check(cudaGetLastError());
      to_host(f.out, rows, (size_t)n * f.width * sizeof(double), device, stream);
      continue;
    }
    for (int c = 0; c < f.width; c++) {
      to_host(v.data(), f.field + (size_t)c * stride, v.size() * sizeof(double), device, stream);
      for (int s = 0; s < n; s++) f.out[(size_t)order[s] * f.width + c] = v[s];
    }
  }
}

}  // namespace hb
