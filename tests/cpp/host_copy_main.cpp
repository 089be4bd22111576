// Drives host_copy.cpp on the CPU: the CUDA runtime calls it makes are implemented
// here on host memory, with the rules that matter to it (a stream, an event and a
// kernel launch belong to a device; which device is current is a thread's own).
// Usage: host_copy_main SCENARIO; exits 0 when the scenario's checks hold.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <mutex>
#include <sstream>
#include <string>
#include <thread>
#include <vector>

#include "../../include/hemeb200.h"
#include "../../hemepure_b200/csrc/device.h"
#include "../../hemepure_b200/csrc/host_copy.h"
#include "../../hemepure_b200/csrc/setup_pool.h"

namespace {

struct FakeStream { int device; };
struct FakeEvent { int device; };
thread_local int current = 0;
thread_local cudaError_t last = cudaSuccess;
std::mutex mu;
std::map<void*, size_t> pool_blocks;
bool pool_empty = false;              // no device memory to be had
size_t pool_used = 0, pool_held = 0;  // bytes given out, and kept by the pool with those
void* own_memory = nullptr;  // a caller's buffer that CUDA knows, of this type
cudaMemoryType own_type = cudaMemoryTypeUnregistered;
std::atomic<int> copies{0};     // cudaMemcpyAsync calls
std::atomic<int> waits{0};      // cudaStreamSynchronize calls
std::map<const void*, size_t> pinned;
int pins = 0;                   // allocations and registrations of pinned memory
bool pinning_fails = false;
int events_until_failure = -1;  // calls that still succeed before one fails; -1: none fails

cudaError_t note(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
FakeStream* of(cudaStream_t s) { return reinterpret_cast<FakeStream*>(s); }
FakeEvent* of(cudaEvent_t e) { return reinterpret_cast<FakeEvent*>(e); }

void require(bool ok, const char* what) {
  if (ok) return;
  std::fprintf(stderr, "failed: %s\n", what);
  std::exit(1);
}

}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "simulated error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof(*a));
  std::lock_guard<std::mutex> lock(mu);
  a->type = p == own_memory ? own_type : pinned.count(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  copies++;
  if (own_type == cudaMemoryTypeDevice && own_memory && own_memory == (kind == cudaMemcpyDeviceToHost ? d : s))
    return note(cudaErrorInvalidValue);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { waits++; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (events_until_failure >= 0 && events_until_failure-- == 0) return note(cudaErrorMemoryAllocation);
  *e = reinterpret_cast<cudaEvent_t>(new FakeEvent{current});
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete of(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return note(e && of(e)->device == of(s)->device ? cudaSuccess : cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return note(e ? cudaSuccess : cudaErrorInvalidResourceHandle); }
cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
  std::lock_guard<std::mutex> lock(mu);
  if (pinning_fails) return note(cudaErrorMemoryAllocation);
  pins++;
  return note(pinned.emplace(p, n).second ? cudaSuccess : cudaErrorHostMemoryAlreadyRegistered);
}
cudaError_t cudaHostUnregister(void* p) {
  std::lock_guard<std::mutex> lock(mu);
  return note(pinned.erase(p) ? cudaSuccess : cudaErrorHostMemoryNotRegistered);
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::malloc(n);
  return cudaHostRegister(*p, n, 0);
}
cudaError_t cudaFreeHost(void* p) {
  cudaHostUnregister(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  if (pool_empty) return note(cudaErrorMemoryAllocation);
  *p = std::malloc(n);
  std::lock_guard<std::mutex> lock(mu);
  pool_blocks[*p] = n;
  pool_used += n;
  pool_held = std::max(pool_held, pool_used);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  std::lock_guard<std::mutex> lock(mu);
  pool_used -= pool_blocks[p];
  pool_blocks.erase(p);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) {
  std::lock_guard<std::mutex> lock(mu);
  *static_cast<uint64_t*>(v) = pool_held;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t keep) {
  std::lock_guard<std::mutex> lock(mu);
  pool_held = std::max(pool_used, std::min(pool_held, keep));
  return cudaSuccess;
}
}

namespace hb {
cudaMemPool_t setup_pool(int, bool) { return nullptr; }
// The kernel's work, refused where a launch would be: a stream of a device that is not current.
void launch_to_reference(const double* src, int64_t stride, int width, const int* st2ref, int n, double* out, void* stream) {
  if (static_cast<FakeStream*>(stream)->device != current) {
    last = cudaErrorInvalidResourceHandle;
    return;
  }
  for (int s = 0; s < n; s++)
    for (int j = 0; j < width; j++) out[(int64_t)st2ref[s] * width + j] = src[(int64_t)j * stride + s];
}
}  // namespace hb

namespace {

// A field of `n` sites, `width` values each, in storage order, and its reference order.
struct Field {
  int n, width;
  std::vector<double> storage, expect, out;
  std::vector<int> order;
  Field(int n_, int width_) : n(n_), width(width_), storage((size_t)n * width), expect(storage.size()), out(storage.size()), order(n) {
    for (int s = 0; s < n; s++) order[s] = (int)(((int64_t)s * 7919 + 13) % n);  // 7919 is prime: a permutation of n that it does not divide
    for (int j = 0; j < width; j++)
      for (int s = 0; s < n; s++) {
        storage[(size_t)j * n + s] = 10.0 * s + j;
        expect[(size_t)order[s] * width + j] = 10.0 * s + j;
      }
  }
  void fetch(hb::HostCopy& c, int device, FakeStream& st) {
    std::fill(out.begin(), out.end(), -1.0);
    c.fields_to_reference({{storage.data(), width, out.data()}}, n, order.data(), order.data(), n, device, reinterpret_cast<cudaStream_t>(&st));
  }
};

// A thread whose current device is 0 reads the fields of a handle on device 1.
void other_device() {
  for (int n : {1000, 400001}) {
    hb::HostCopy copy;
    FakeStream st{1};
    Field f(n, 3);
    current = 0;
    f.fetch(copy, 1, st);
    require(f.out == f.expect, "field of another device");
    require(current == 0, "the caller's device is left as it was");
    std::vector<double> up(f.n * 24), back(up.size());
    for (size_t k = 0; k < up.size(); k++) up[k] = (double)k;
    copy.to_device(back.data(), up.data(), up.size() * sizeof(double), 1, reinterpret_cast<cudaStream_t>(&st));
    require(up == back, "upload to another device");
    require(current == 0, "the caller's device is left as it was by an upload");
  }
}

// An event that cannot be made costs speed at most, then and later.
void event_failure() {
  for (int good : {0, 3, 7}) {
    hb::HostCopy copy;
    FakeStream st{0};
    Field f(400001, 3);
    events_until_failure = good;
    for (int pass = 0; pass < 3; pass++) {
      f.fetch(copy, 0, st);
      require(f.out == f.expect, "field after a failed event");
    }
    events_until_failure = -1;
  }
}

// A caller's pinned or managed array takes one copy of its own, and device memory
// given for an array is refused by that copy instead of being written by the host.
void own_buffers() {
  const size_t n = (size_t)12 << 20;
  std::vector<double> a(n), b(n);
  for (size_t k = 0; k < n; k++) a[k] = (double)k;
  FakeStream st{0};
  auto stream = reinterpret_cast<cudaStream_t>(&st);
  for (cudaMemoryType type : {cudaMemoryTypeHost, cudaMemoryTypeManaged, cudaMemoryTypeDevice}) {
    for (bool down : {true, false}) {
      hb::HostCopy copy;
      std::fill(b.begin(), b.end(), -1.0);
      own_type = type;
      own_memory = down ? b.data() : a.data();
      copies = 0;
      int code = 0;
      try {
        if (down) copy.to_host(b.data(), a.data(), n * sizeof(double), 0, stream);
        else copy.to_device(b.data(), a.data(), n * sizeof(double), 0, stream);
      } catch (const hb::Error& e) {
        code = e.code;
      }
      own_memory = nullptr;
      require(copies == 1, "one copy");
      if (type == cudaMemoryTypeDevice) require(code == HB_ERR_CUDA && b[0] == -1.0 && b[n - 1] == -1.0, "device memory is refused");
      else require(code == 0 && a == b, "copied");
    }
  }
}

// Handles one after the other pin once; handles side by side pin a bounded number of
// times and give all but one back; and a field arrives whatever becomes of the pinning.
void shared_pieces() {
  FakeStream st{0};
  Field f(400001, 3);
  for (int handle = 0; handle < 4; handle++) {
    hb::HostCopy copy;
    for (int pass = 0; pass < 2; pass++) {
      f.fetch(copy, 0, st);
      require(f.out == f.expect, "field of one of several handles");
    }
  }
  require(pins == 1 && pinned.size() == 1, "handles one after the other pin once");
  for (int round = 0; round < 3; round++) {
    std::vector<std::thread> threads;
    std::atomic<int> right{0};
    for (int k = 0; k < 8; k++)
      threads.emplace_back([&] {
        hb::HostCopy copy;
        FakeStream own{0};
        Field g(300007, 3);
        for (int pass = 0; pass < 3; pass++) {
          g.fetch(copy, 0, own);
          right += g.out == g.expect;
        }
      });
    for (auto& t : threads) t.join();
    require(right == 24, "fields of handles read side by side");
    require(pinned.size() == 1, "pieces beyond one set are given back");
  }
  pinned.clear();  // the context was replaced
  {
    hb::HostCopy copy;
    f.fetch(copy, 0, st);
    require(f.out == f.expect && pinned.size() == 1, "pieces are pinned again");
    pinned.clear();
    pinning_fails = true;
    for (int pass = 0; pass < 2; pass++) {
      f.fetch(copy, 0, st);
      require(f.out == f.expect, "field without pinned memory");
    }
    pinning_fails = false;
    f.fetch(copy, 0, st);
    require(f.out == f.expect && pinned.size() == 1, "pinned once it can be");
  }
}

// A transfer's device scratch goes back to what the pool held before it, or to the
// share it may keep.
void scratch_given_back() {
  FakeStream st{0};
  auto stream = reinterpret_cast<cudaStream_t>(&st);
  const size_t mb = (size_t)1 << 20;
  for (size_t before : {(size_t)0, 64 * mb, 1024 * mb}) {
    pool_held = before;
    for (size_t bytes : {mb, 100 * mb, 700 * mb, 3000 * mb}) {
      hb::SetupPool p(0, stream, hb::kScratch);
      p.get<unsigned char>(bytes);
    }
    require(pool_held <= std::max<size_t>(before, hb::kScratchKeep), "scratch is given back");
    require(pool_held >= before, "what a set-up left in the pool stays");
  }
  pool_held = 0;
  Field f((int)(hb::kScratchKeep / 24) + 1001, 3);
  hb::HostCopy copy;
  f.fetch(copy, 0, st);
  require(f.out == f.expect && pool_held <= hb::kScratchKeep, "a field's scratch is given back");
  pool_held = 0;
  { hb::SetupPool p(0, stream); p.get<unsigned char>(700 * mb); }
  require(pool_held == 700 * mb, "a set-up's memory is kept for the next");
}

// Several fields of one member: their order crosses to the device once.
void one_order() {
  FakeStream st{0};
  const int n = 10007;
  Field a(n, 1), b(n, 3), c(n, 1);
  hb::HostCopy copy;
  copies = 0;
  copy.fields_to_reference({{a.storage.data(), 1, a.out.data()}, {b.storage.data(), 3, b.out.data()}, {c.storage.data(), 1, nullptr}}, n,
                           a.order.data(), nullptr, n, 0, reinterpret_cast<cudaStream_t>(&st));
  require(a.out == a.expect && b.out == b.expect, "fields by an uploaded order");
  require(copies == 3, "one upload of the order and a download of each field asked for");
}

// A small upload is followed by its caller's kernel and wait: it does not wait itself.
// A download is done when its call returns.
void small_copies() {
  FakeStream st{0};
  auto stream = reinterpret_cast<cudaStream_t>(&st);
  std::vector<double> a(1000, 1.5), b(1000);
  hb::HostCopy copy;
  copy.to_device(b.data(), a.data(), a.size() * sizeof(double), 0, stream);
  require(a == b && waits == 0, "a small upload does not wait");
  copy.to_host(b.data(), a.data(), a.size() * sizeof(double), 0, stream);
  require(waits == 1, "a small download waits once");
}

// Without device memory for the reordered copy the host reorders the fields, to the
// same values; sizes on both sides of a piece and of the set of pieces.
void no_device_memory() {
  FakeStream st{0};
  for (int n : {1, 65535, 65536, 65537, 600011}) {
    hb::HostCopy copy;
    Field a(n, 3), b(n, 1);
    for (bool empty : {false, true}) {
      pool_empty = empty;
      std::fill(a.out.begin(), a.out.end(), -1.0);
      std::fill(b.out.begin(), b.out.end(), -1.0);
      copy.fields_to_reference({{a.storage.data(), 3, a.out.data()}, {b.storage.data(), 1, b.out.data()}}, n, a.order.data(), nullptr, n, 0,
                               reinterpret_cast<cudaStream_t>(&st));
      require(a.out == a.expect && b.out == b.expect, empty ? "fields reordered on the host" : "fields reordered on the device");
    }
    pool_empty = false;
  }
}

// Whether the mapping that holds `p` is left out of a child process ("dc" of smaps).
bool left_out_of_children(const void* p) {
  std::ifstream in("/proc/self/smaps");
  std::string line;
  bool here = false;
  while (std::getline(in, line)) {
    unsigned long lo, hi;
    if (std::sscanf(line.c_str(), "%lx-%lx ", &lo, &hi) == 2) here = lo <= (unsigned long)p && (unsigned long)p < hi;
    if (here && line.rfind("VmFlags:", 0) == 0) return line.find(" dc") != std::string::npos;
  }
  return false;
}

// A child process shares no piece with its parent: a piece written after a fork would
// otherwise move to another page than the one CUDA copies from.
void fork_safe() {
  FakeStream st{0};
  Field f(400001, 3);
  hb::HostCopy copy;
  f.fetch(copy, 0, st);
  require(f.out == f.expect && pinned.size() == 1, "a field in pieces");
  const unsigned char* p = static_cast<const unsigned char*>(pinned.begin()->first);
  require(left_out_of_children(p) && left_out_of_children(p + pinned.begin()->second - 1), "pieces are left out of child processes");
}

// A handle that goes on reading has its transfers take turns on a bounded number of
// sets, whether or not one could not be pinned, and leaves one.
void sets_in_turn() {
  FakeStream st{0};
  Field f(200003, 3);
  for (bool fails : {false, true}) {
    hb::HostCopy copy;
    size_t most = 0;
    for (int pass = 0; pass < 60; pass++) {
      pinning_fails = fails && pass > 12;
      copies = 0;
      f.fetch(copy, 0, st);
      require(f.out == f.expect && copies > 1, "a field in pieces by sets in turn");
      require(pinned.size() >= most, "no set is given up under way");
      most = pinned.size();
    }
    require(most == (fails ? 2 : 4), "sets in turn");
  }
  pinning_fails = false;
  require(pinned.size() == 1, "one set is kept");
}

}  // namespace

int main(int argc, char** argv) {
  const std::string s = argc > 1 ? argv[1] : "";
  try {
    if (s == "other_device") other_device();
    else if (s == "event_failure") event_failure();
    else if (s == "own_buffers") own_buffers();
    else if (s == "shared_pieces") shared_pieces();
    else if (s == "scratch_given_back") scratch_given_back();
    else if (s == "one_order") one_order();
    else if (s == "small_copies") small_copies();
    else if (s == "no_device_memory") no_device_memory();
    else if (s == "fork_safe") fork_safe();
    else if (s == "sets_in_turn") sets_in_turn();
    else return 2;
  } catch (const hb::Error& e) {
    std::fprintf(stderr, "error %d: %s\n", e.code, e.msg.c_str());
    return 1;
  }
  return 0;
}
