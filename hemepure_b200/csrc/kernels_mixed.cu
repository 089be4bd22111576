// kernels_mixed.cu -- collide-and-stream with shifted low-precision storage.
//
// Storage holds g_i = f_i - w_i rho0 (rho0 = 1), the deviation from the rest
// equilibrium, in FP32 or FP16 (scaled); the collision runs in FP32 on g, so
// rounding falls only on the deviation.  In shifted variables (w_i = w_inv(i)):
//   rho = 1 + sum g,  m = sum c g,
//   geq_i = w_i (drho - 3/2 |m|^2/rho + 9/2 (c_i.m)^2/rho + 3 c_i.m),
//   g*_i = g_i + omega (g_i - geq_i)             (LBGK; TRT and LES likewise),
// and every streaming rule of the FP64 kernels (bounce-back, BFL, Nash, Ladd,
// GZS) carries over unchanged because its coefficients sum to one over pairs of
// equal weight.  FP64 stays where the reference's conservation or stability
// needs it: iolet density targets (given in FP64, subtracted from rho0 in FP64),
// the Windkessel flow sums and ODE (kernels_f64.cu), the macroscopic outputs.
#include "mixed_site.cuh"

namespace hb {
namespace {

// 64 registers.  4M-site pipe, LBGK and BFL, FP32: five blocks 143.5 us a step, six
// 128.3, seven 122.7, eight 120.7; FP16: six 91, eight 85.4, ten 102.  Measured on that
// form only: bounce-back with LBGK or TRT fits, BFL spills 24 to 32 bytes, GZS 44 to 60
// and the LES forms 56 to 92.
constexpr int kMixedBlocksPerSM = 8;

// One steady-state time step in one launch (k_step of kernels_f64.cu): boundary
// records with iolet links, GZS wall links, then the other boundary records
// spread among the plain bulk sites.  Three kernels on three streams before:
// 197k-site pipe FP32 16.0 -> 10.6 us a step, 187k-site GZS bifurcation 88 -> 23,
// 1.1M-site LES stenosis 50.7 -> 48.7, 4M-site pipe FP16 92.3 -> 85.1; FP32 stays at
// 120.0.  The bulk path waits for memory (four fifths of its stalls) rather than
// issuing: two sites a thread with packed FP32 instructions halve the arithmetic but
// take 102 registers (FP32 127, FP16 93 us), and the bulk sites in a kernel of their
// own at 40 registers beside the boundary records measure 121 and 90.
template <class S, int K, int WALL>
__global__ void __launch_bounds__(kStepBlock, kMixedBlocksPerSM) k_step_m(const StepArgs a, const MixArgs m, const StepTiles t) {
  int b = blockIdx.x;
  if (b < t.links) {
    iolet_link_m<S, K, WALL, true, true>(a, m, b * kStepBlock + threadIdx.x);
    return;
  }
  b -= t.links;
  if (b < t.io) {
    const int g = t.io_first + b * kStepBlock + threadIdx.x;
    general_site_m<S, K, WALL, true, false, true, true>(a, m, g, g < a.gen.G);
    return;
  }
  b -= t.io;
  if (WALL == kGZS) {
    if (b < t.gzs) {
      gzs_link_m<S, K, true, true>(a, m, b * kStepBlock + threadIdx.x);
      return;
    }
    b -= t.gzs;
  }
  const int w = t.walls_before(b);
  if (t.walls_before(b + 1) > w) {
    const int g = w * kStepBlock + threadIdx.x;
    general_site_m<S, K, WALL, true, false, false, true>(a, m, g, g < t.io_first);
    return;
  }
  int s = (b - w) * t.tiles * kStepBlock + threadIdx.x;
  const bool po = a.run_po != nullptr;
  const int* rows = po ? a.run_po : a.run_off;
  int r = s < a.n ? __ldg(a.meta + s) : -1;
  int row[20];
  if (r >= 0) load_row(rows, r, row);
  wait_previous_step();
#pragma unroll 1
  for (int j = 0; j < t.tiles; j++) {
    const int s_next = s + kStepBlock;
    const int r_next = j + 1 < t.tiles && s_next < a.n ? __ldg(a.meta + s_next) : -1;
    if (r >= 0) {
      float g[Q];
      if (po) gather_row<S, true>(a, m, s, row, g);
      else gather_row<S, false>(a, m, s, row, g);
      bulk_collide_m<S, K, false>(a, m, s, g);
    }
    s = s_next;
    r = r_next;
    if (r >= 0) load_row(rows, r, row);
  }
}

// The other forms of the step, the first step of a state (GATHER false) and the
// output steps: the plain bulk sites and the boundary side by side (kernels_f64.cu).
// Output step of one call, FP32: 257k sites 54 -> 39 us, 2M 133 -> 117; FP16: 54 ->
// 40 and 127 -> 104.
template <class S, int K, bool GATHER, bool MACRO>
__global__ void __launch_bounds__(256) k_bulk_m(const StepArgs a, const MixArgs m) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  const int r = __ldg(a.meta + s);
  if (r < 0) return;
  bulk_site_m<S, K, GATHER, MACRO>(a, m, s, r);
}

template <class S, int K, int WALL, bool GATHER, bool MACRO>
__global__ void __launch_bounds__(kStepBlock) k_boundary_m(const StepArgs a, const MixArgs m, const StepTiles t) {
  int b = blockIdx.x;
  if (b < t.links) {
    iolet_link_m<S, K, WALL, GATHER>(a, m, b * kStepBlock + threadIdx.x);
    return;
  }
  b -= t.links;
  if (WALL == kGZS) {
    if (b < t.gzs) {
      gzs_link_m<S, K, GATHER>(a, m, b * kStepBlock + threadIdx.x);
      return;
    }
    b -= t.gzs;
  }
  const int g = b * kStepBlock + threadIdx.x;
  if (g < a.gen.G) general_site_m<S, K, WALL, GATHER, MACRO>(a, m, g);
}

template <class S, int WALL, bool GATHER>
__global__ void __launch_bounds__(256) k_to_aos_m(const StepArgs a, const MixArgs m, const int* st2ref, double* aos) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n) return;
  float g[Q];
  gather_any_m<S, WALL, GATHER>(a, m, s, g);
  const int64_t base = (int64_t)st2ref[s] * Q;
#pragma unroll
  for (int i = 0; i < Q; i++) aos[base + i] = weight(i) + (double)(g[i] * (1.0f / Store<S>::kScale));
}

template <class S>
__global__ void k_from_aos_m(const double* aos, const int* st2ref, int n, int64_t np, void* out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (int64_t)n * Q) return;
  const int s = (int)(k / Q), i = (int)(k % Q);
  Store<S>::st(static_cast<S*>(out) + (int64_t)i * np + s,
               (float)(aos[(int64_t)st2ref[s] * Q + i] - weight(i)) * Store<S>::kScale);
}

// The shifted forms' BFL coefficient c in place of the cut distance q of every link, rows
// of `n` records `pitch` apart, from
// (f*_d + (2q-1) f*_i) / (2q) = f*_d + c (f*_i - f*_d), c = 1 - 1/(2q), for q >= 1/2 and
// 2q f*_d + (1-2q) f_d = f*_d + |c| (f_d - f*_d), c = -(1-2q), otherwise.  On the device:
// the divisions of a 257k-site lattice take 0.4 ms of the 2 ms that admit it on the host.
__global__ void __launch_bounds__(256) k_bfl_coefficients(float* q, int64_t pitch, int n) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  float& v = q[blockIdx.y * pitch + g];
  const double d = 2.0 * (double)v;
  v = (float)(v < 0.5f ? -__dsub_rn(1.0, d) : __dsub_rn(1.0, __ddiv_rn(1.0, d)));
}

// GZS walls run with LBGK and TRT only (validate_case).
constexpr bool has_gzs(int k) { return k == kLBGK || k == kTRT; }

template <class S, int K, int WALL, bool GATHER, bool MACRO>
void launch_parts(const StepArgs& a, const MixArgs& m, int which, cudaStream_t st) {
  if ((which & kLaunchBulk) && a.n > 0) k_bulk_m<S, K, GATHER, MACRO><<<(a.n + 255) / 256, 256, 0, st>>>(a, m);
  if (!(which & kLaunchBoundary)) return;
  const StepTiles t = boundary_tiles(a);
  if (t.blocks() > 0) k_boundary_m<S, K, WALL, GATHER, MACRO><<<t.blocks(), kStepBlock, 0, st>>>(a, m, t);
}

template <class S, int K, int WALL>
void launch_m2(const StepArgs& a, const MixArgs& m, bool gather, bool macro, int which, cudaStream_t st) {
  if (gather && !macro) {
    const StepTiles t = step_tiles(a, which, kMixedBlocksPerSM);
    launch_dependent(k_step_m<S, K, WALL>, t.blocks(), st, a, m, t);
  } else if (gather) {
    launch_parts<S, K, WALL, true, true>(a, m, which, st);
  } else {
    // Without a gather bounce-back and BFL walls have no rule to apply.
    constexpr int W = WALL == kBFL ? kSBB : WALL;
    if (macro) launch_parts<S, K, W, false, true>(a, m, which, st);
    else launch_parts<S, K, W, false, false>(a, m, which, st);
  }
}

template <class S, int K>
void launch_m1(const StepArgs& a, const MixArgs& m, int wall, bool gather, bool macro, int which, cudaStream_t st) {
  if (wall == kSBB) launch_m2<S, K, kSBB>(a, m, gather, macro, which, st);
  else if (wall == kBFL) launch_m2<S, K, kBFL>(a, m, gather, macro, which, st);
  else if constexpr (has_gzs(K)) launch_m2<S, K, kGZS>(a, m, gather, macro, which, st);
}

template <class S>
void launch_m0(const StepArgs& a, const MixArgs& m, int kernel, int wall, bool gather, bool macro, int which, cudaStream_t st) {
  if (kernel == kLBGK) launch_m1<S, kLBGK>(a, m, wall, gather, macro, which, st);
  else if (kernel == kTRT) launch_m1<S, kTRT>(a, m, wall, gather, macro, which, st);
  else launch_m1<S, kLES>(a, m, wall, gather, macro, which, st);
}

template <class S, int WALL>
void launch_to_aos2(const StepArgs& a, const MixArgs& m, bool gather, const int* st2ref, double* aos, cudaStream_t st) {
  if (gather) k_to_aos_m<S, WALL, true><<<(a.n + 255) / 256, 256, 0, st>>>(a, m, st2ref, aos);
  else k_to_aos_m<S, WALL, false><<<(a.n + 255) / 256, 256, 0, st>>>(a, m, st2ref, aos);
}

template <class S>
void launch_to_aos1(const StepArgs& a, const MixArgs& m, int wall, bool gather, const int* st2ref, double* aos, cudaStream_t st) {
  if (wall == kBFL) launch_to_aos2<S, kBFL>(a, m, gather, st2ref, aos, st);
  else if (wall == kGZS) launch_to_aos2<S, kGZS>(a, m, gather, st2ref, aos, st);
  else launch_to_aos2<S, kSBB>(a, m, gather, st2ref, aos, st);
}

}  // namespace

void launch_step_mixed(const StepArgs& a, int precision, const void* fin, void* fout, const float* gin, float* gout,
                       int kernel, int wall, bool gather, bool macro, int which, void* stream) {
  const MixArgs m{fin, fout, gin, gout};
  cudaStream_t st = (cudaStream_t)stream;
  if (precision == HB_STORE_FP16) launch_m0<__half>(a, m, kernel, wall, gather, macro, which, st);
  else launch_m0<float>(a, m, kernel, wall, gather, macro, which, st);
}

void launch_to_aos_mixed(const StepArgs& a, int precision, const void* fin, const float* gin, int wall, bool gather,
                         const int* st2ref, double* aos, void* stream) {
  const MixArgs m{fin, nullptr, gin, nullptr};
  if (a.n <= 0) return;
  cudaStream_t st = (cudaStream_t)stream;
  if (precision == HB_STORE_FP16) launch_to_aos1<__half>(a, m, wall, gather, st2ref, aos, st);
  else launch_to_aos1<float>(a, m, wall, gather, st2ref, aos, st);
}

void launch_bfl_coefficients(float* q, int64_t pitch, int n, void* stream) {
  if (n > 0) k_bfl_coefficients<<<dim3((unsigned)((n + 255) / 256), 18), 256, 0, (cudaStream_t)stream>>>(q, pitch, n);
}

void launch_from_aos_mixed(const double* aos, const int* st2ref, int n, int64_t np, int precision, void* out, void* stream) {
  const int64_t tot = (int64_t)n * Q;
  if (tot <= 0) return;
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned blocks = (unsigned)((tot + 255) / 256);
  if (precision == HB_STORE_FP16) k_from_aos_m<__half><<<blocks, 256, 0, st>>>(aos, st2ref, n, np, out);
  else k_from_aos_m<float><<<blocks, 256, 0, st>>>(aos, st2ref, n, np, out);
}

}  // namespace hb
