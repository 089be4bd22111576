// mixed_site.cuh -- per-site routines of the shifted low-precision forms
// (g = f - w rho0 stored in FP32 or scaled FP16, FP32 collision), shared by the
// single-lattice kernels (kernels_mixed.cu) and the batched kernels
// (kernels_batch.cu).  See kernels_mixed.cu for the formulation.
//
// Every routine works on the stored scale, G = kScale * g (kScale = 1 for FP32,
// kHalfScale for FP16, a power of two, so scaling is exact): a value is converted
// but never rescaled on its way in or out.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "../../include/hemeb200.h"
#include "device.h"
#include "hb_common.h"
#include "step_tiles.cuh"

namespace hb {
namespace {

template <class S>
struct Store;

// Plain loads, not the non-coherent path: a step kernel may be launched while the
// one that wrote its input drains (step_tiles.cuh).
template <>
struct Store<float> {
  static constexpr float kScale = 1.0f;
  static __device__ __forceinline__ float ld(const float* p) { return *p; }
  static __device__ __forceinline__ void st(float* p, float v) { *p = v; }
};

template <>
struct Store<__half> {
  static constexpr float kScale = kHalfScale;
  static __device__ __forceinline__ float ld(const __half* p) { return __half2float(*p); }
  static __device__ __forceinline__ void st(__half* p, float v) { *p = __float2half_rn(v); }
};

__host__ __device__ __forceinline__ constexpr float wf(int i) { return (float)weight(i); }

// Every operation of the collision is rounded as written here, so a site has the
// same bits whichever kernel steps it.
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// Density deviation and momentum.  Opposite directions (i, i + 1) enter by their
// sum and difference.  D - D is 0 for finite values and NaN otherwise: a
// non-finite value makes every momentum component NaN.
struct Moments {
  float D, mx, my, mz;
  __device__ __forceinline__ explicit Moments(const float* g) {
    float p[9], m[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
      p[k] = vadd(g[2 * k + 1], g[2 * k + 2]);
      m[k] = vsub(g[2 * k + 1], g[2 * k + 2]);
    }
    D = vadd(g[0], vadd(vadd(vadd(p[0], p[1]), p[2]),
                        vadd(vadd(vadd(p[3], p[4]), vadd(p[5], p[6])), vadd(p[7], p[8]))));
    const float nf = vsub(D, D);
    mx = vadd(vadd(m[0], nf), vadd(vadd(m[3], m[4]), vadd(m[5], m[6])));
    my = vadd(vadd(m[1], nf), vadd(vsub(m[3], m[4]), vadd(m[7], m[8])));
    mz = vadd(vadd(m[2], nf), vadd(vsub(m[5], m[6]), vsub(m[7], m[8])));
  }
  __device__ __forceinline__ Moments(float d, float x, float y, float z) : D(d), mx(x), my(y), mz(z) {}
};

// Shifted equilibrium on the scale `scale`:
//   w_i (D - 3/2 |M|^2 / (scale + D) + 9/2 (c_i.M)^2 / (scale + D) + 3 c_i.M),
// with m = 3 M.  The weights enter as they are: the rounded 1/18 and 1/36 add up
// to a momentum scale of 1 + 7.5e-9, a rounded 3 w of 1/6 to 1 + 3.0e-8, an error
// that would grow with every step.
struct Geq {
  float mx, my, mz, t1, nh;  // 3 M; D - 3/2 |M|^2 / (scale + D); 1/2 / (scale + D)
  __device__ __forceinline__ Geq(const Moments& m, float scale) {
    mx = vmul(3.0f, m.mx);
    my = vmul(3.0f, m.my);
    mz = vmul(3.0f, m.mz);
    nh = vmul(0.5f, __frcp_rn(vadd(scale, m.D)));
    const float mm = vfma(m.mz, mz, vfma(m.my, my, vmul(m.mx, mx)));
    t1 = vfma(-mm, nh, m.D);
  }
  // 3 c_i.M of the odd direction i.
  __device__ __forceinline__ float mde(int i) const {
    switch (i) {
      case 1: return mx;
      case 3: return my;
      case 5: return mz;
      case 7: return vadd(mx, my);
      case 9: return vsub(mx, my);
      case 11: return vadd(mx, mz);
      case 13: return vsub(mx, mz);
      case 15: return vadd(my, mz);
      default: return vsub(my, mz);
    }
  }
  // The odd direction i and its opposite i + 1, which share the even part.
  __device__ __forceinline__ void pair(int i, float& a, float& b) const {
    const float w = i < 7 ? wf(1) : wf(7);
    const float e = mde(i);
    const float even = vfma(vmul(vmul(w, nh), e), e, vmul(w, t1));
    a = vfma(w, e, even);
    b = vfma(-w, e, even);
  }
  // Any direction but the rest one.
  __device__ __forceinline__ float operator()(int i) const {
    float a, b;
    pair(i - 1 + (i & 1), a, b);
    return (i & 1) ? a : b;
  }
};

// What the rounded weights 1/3, 1/18 and 1/36 add up to beyond 1 (2^-26).
constexpr float kWeightExcess = (float)((double)wf(0) + 6.0 * (double)wf(1) + 12.0 * (double)wf(7) - 1.0);

// G - geq(G).  The rest direction makes the equilibria add up to the density: the
// excess of the weights is taken off it after the difference, where it is not lost
// to rounding.  Left in, it adds 1.5e-8 of the density deviation every step, the
// largest error of long FP32 runs (velocity of a 64k-site pipe after 600 steps,
// against FP64: 3.6e-6 with it, 7e-7 without; one multiply-add a site).
__device__ __forceinline__ void non_equilibrium(const Geq& geq, const float* g, float* neq) {
  neq[0] = vfma(kWeightExcess, geq.t1, vfma(-wf(0), geq.t1, g[0]));
#pragma unroll
  for (int i = 1; i < Q; i += 2) {
    float a, b;
    geq.pair(i, a, b);
    neq[i] = vsub(g[i], a);
    neq[i + 1] = vsub(g[i + 1], b);
  }
}

// Post-collision values: G + om neq, or TRT with the rates of the even and odd parts.
__device__ __forceinline__ void relax(const float* g, const float* neq, bool trt, float om, float omm, float* out) {
  out[0] = vfma(om, neq[0], g[0]);
  if (trt) {
    const float hp = vmul(0.5f, om), hm = vmul(0.5f, omm), hn = vmul(-0.5f, omm);
#pragma unroll
    for (int i = 1; i < Q; i += 2) {
      const float s = vadd(neq[i], neq[i + 1]), d = vsub(neq[i], neq[i + 1]);
      out[i] = vfma(hm, d, vfma(hp, s, g[i]));
      out[i + 1] = vfma(hn, d, vfma(hp, s, g[i + 1]));
    }
  } else {
#pragma unroll
    for (int i = 1; i < Q; i++) out[i] = vfma(om, neq[i], g[i]);
  }
}

// Some f <= 0 (or NaN): the smallest value of each weight against -w, with D for
// the NaN that a minimum drops.
__device__ __forceinline__ bool unstable(const float* g, float D, float scale) {
  float a = fminf(fminf(g[1], g[2]), g[3]), d = fminf(fminf(g[7], g[8]), g[9]);
  a = fminf(fminf(a, g[4]), fminf(g[5], g[6]));
  d = fminf(fminf(d, g[10]), g[11]);
  d = fminf(fminf(d, g[12]), g[13]);
  d = fminf(fminf(d, g[14]), g[15]);
  d = fminf(fminf(d, g[16]), fminf(g[17], g[18]));
  return !(g[0] > -wf(0) * scale) || !(a > -wf(1) * scale) || !(d > -wf(7) * scale) || D != D;
}

// Relaxation time of the LES kernel from the squared non-equilibrium flux.
__device__ __forceinline__ float les_tau_of(const StepArgs& a, float q12sq, float vt) {
  const float tau0 = (float)a.tau;
  const float q12 = sqrtf(q12sq);
  const float ks = (float)(18.0 * 1.4142135623730950488016887242097 * 0.01);
  const float tau_les = 0.5f * (tau0 + sqrtf(tau0 * tau0 + ks * q12));
  if (a.t <= a.lifetime / 2) return (vt == tau0) ? tau_les : vt;
  if (a.t < a.lifetime) return (tau_les - vt) * 2.0f / (float)a.lifetime * (float)a.t + (2.0f * vt - tau_les);
  return tau_les;
}

// Sum of v[l] c_p c_r: the fluxes of opposite directions enter by their sum.
__device__ __forceinline__ void fluxes(const float* v, float& xx, float& xy, float& xz, float& yy, float& yz, float& zz) {
  float s[9];
#pragma unroll
  for (int k = 0; k < 9; k++) s[k] = vadd(v[2 * k + 1], v[2 * k + 2]);
  const float a = vadd(s[3], s[4]), b = vadd(s[5], s[6]), c = vadd(s[7], s[8]);
  xx = vadd(s[0], vadd(a, b));
  yy = vadd(s[1], vadd(a, c));
  zz = vadd(s[2], vadd(b, c));
  xy = vsub(s[3], s[4]);
  xz = vsub(s[5], s[6]);
  yz = vsub(s[7], s[8]);
}

__device__ __forceinline__ float flux_norm_sq(const float* neq) {
  float xx, xy, xz, yy, yz, zz;
  fluxes(neq, xx, xy, xz, yy, yz, zz);
  const float off = vfma(yz, yz, vfma(xz, xz, vmul(xy, xy)));
  return vfma(2.0f, off, vfma(zz, zz, vfma(yy, yy, vmul(xx, xx))));
}

// The site's relaxation time and rate for kernel K (LES: from its non-equilibrium part).
template <class S, int K>
__device__ __forceinline__ void site_rate(const StepArgs& a, const float* neq, int s, float& tau, float& om) {
  om = (float)a.omega;
  tau = (float)a.tau;
  if (K == kLES) {
    tau = les_tau_of(a, flux_norm_sq(neq) * (1.0f / (Store<S>::kScale * Store<S>::kScale)), (float)__ldg(a.vtau + s));
    om = -1.0f / tau;
  }
}

// Momentum flux tensor of an output step (unscaled), -(tau - 1/2) sum (gp - g) c c.
template <class S>
__device__ __forceinline__ void flux_tensor(float tau, const float* gp, const float* g, float pi[6]) {
  float df[Q];
#pragma unroll
  for (int l = 0; l < Q; l++) df[l] = gp[l] - g[l];
  fluxes(df, pi[0], pi[1], pi[2], pi[3], pi[4], pi[5]);
#pragma unroll
  for (int k = 0; k < 6; k++) pi[k] = pi[k] * (1.0f / Store<S>::kScale) * -(tau - 0.5f);
}

__device__ __forceinline__ double wss_mag_f(const float pi[6], const float nor[3]) {
  const float sx = pi[0] * nor[0] + pi[1] * nor[1] + pi[2] * nor[2];
  const float sy = pi[1] * nor[0] + pi[3] * nor[1] + pi[4] * nor[2];
  const float sz = pi[2] * nor[0] + pi[4] * nor[1] + pi[5] * nor[2];
  const float sq = sx * sx + sy * sy + sz * sz, ns = sx * nor[0] + sy * nor[1] + sz * nor[2];
  return (double)sqrtf(fmaxf(sq - ns * ns, 0.0f));
}

// The tensor as the stress caches read it (FP64, like store_pi), then tau.
__device__ __forceinline__ void store_pi_f(const StepArgs& a, int s, float tau, const float pi[6]) {
  double* o = a.pi + s;
#pragma unroll
  for (int k = 0; k < 6; k++) o[k * a.np] = (double)pi[k];
  o[6 * a.np] = (double)tau;
}

__device__ __forceinline__ bool parabolic_f(const IoletDev& I, const double x[3], uint64_t t, float v[3]) {
  const double dx = x[0] - I.pos[0], dy = x[1] - I.pos[1], dz = x[2] - I.pos[2];
  const double z = dx * I.nrm[0] + dy * I.nrm[1] + dz * I.nrm[2];
  const double rsq = (dx * dx + dy * dy + dz * dz) - z * z;
  const double r2a2 = rsq / (I.radius * I.radius);
  double mx = I.max_speed;
  if (t < I.warmup) mx *= (double)t / (double)I.warmup;
  const double s = mx * (1. - r2a2);
  v[0] = (float)(I.nrm[0] * s);
  v[1] = (float)(I.nrm[1] * s);
  v[2] = (float)(I.nrm[2] * s);
  return !(r2a2 > 1.0);
}

// The velocity of a velocity iolet's link d of general site gi (parabolic, file
// velocity or Womersley; half-way point or neighbour as for the FP64 kernels),
// evaluated in FP64 and narrowed.
__device__ __forceinline__ bool link_velocity_f(const StepArgs& a, const IoletDev& I, int io, int gi, int d, bool half,
                                                const double pos[3], float v[3]) {
  if (I.kind == kWomersley) {
    const double* A = a.wom_amp + ((int64_t)__ldg(a.gen.wom + gi) * 18 + (d - 1)) * 4 + (half ? 0 : 2);
    const double speed = __ldg(A) * a.dens_row[kRowA + io] - __ldg(A + 1) * a.dens_row[kRowB + io];
    v[0] = (float)(I.nrm[0] * -speed);
    v[1] = (float)(I.nrm[1] * -speed);
    v[2] = (float)(I.nrm[2] * -speed);
    return true;
  }
  const double h = half ? 0.5 : 1.0;
  const double x[3] = {pos[0] + h * cx(d), pos[1] + h * cy(d), pos[2] + h * cz(d)};
  if (I.kind == kParabolic) return parabolic_f(I, x, (uint64_t)(unsigned int)a.t, v);
  const double dx = x[0] - I.pos[0], dy = x[1] - I.pos[1], dz = x[2] - I.pos[2];
  const double z = dx * I.nrm[0] + dy * I.nrm[1] + dz * I.nrm[2];
  const double r2a2 = ((dx * dx + dy * dy + dz * dz) - z * z) / (I.radius * I.radius);
  const double s = a.dens_row[kRowA + io] * (1. - r2a2);
  v[0] = (float)(I.nrm[0] * s);
  v[1] = (float)(I.nrm[1] * s);
  v[2] = (float)(I.nrm[2] * s);
  return !(r2a2 > 1.0);
}

// One 20-entry row of the run table (run offsets or plane offsets).
__device__ __forceinline__ void load_row(const int* table, int r, int* row) {
  const int4* o4 = reinterpret_cast<const int4*>(table) + 5 * (int64_t)r;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const int4 v = __ldg(o4 + k);
    row[4 * k] = v.x;
    row[4 * k + 1] = v.y;
    row[4 * k + 2] = v.z;
    row[4 * k + 3] = v.w;
  }
}

// Arguments of the shifted kernels: StepArgs for the shared tables, plus typed
// storage pointers (fin/fout/gin/gout of StepArgs are unused here).  Ghost values
// are FP32 and unscaled; StepArgs' cut distances hold the BFL coefficient (below)
// except for GZS walls.
struct MixArgs {
  const void* fin;
  void* fout;
  const float* gin;
  float* gout;
};

// Gather of a plain bulk site from its run row: plane offsets i * np + run_off[i]
// (PO: one address add per load) or run offsets.
template <class S, bool PO>
__device__ __forceinline__ void gather_row(const StepArgs& a, const MixArgs& m, int s, const int* row, float* g) {
  const S* p = static_cast<const S*>(m.fin) + s;
  g[0] = Store<S>::ld(p);
#pragma unroll
  for (int i = 1; i < Q; i++) {
    if (!PO) p += a.np;
    g[i] = Store<S>::ld(p + row[i]);
  }
}

// Link masks and run of a site: a general record's own, none for a plain bulk site.
struct LinksM {
  uint32_t wall, iolet;
  int run, g;
};

__device__ __forceinline__ void load_sources_m(const StepArgs& a, const LinksM& l, int s, int* src) {
  if (l.run >= 0) {
    int off[20];
    load_row(a.run_off, l.run, off);
#pragma unroll
    for (int i = 1; i < Q; i++) src[i - 1] = s + off[i];
  } else {
#pragma unroll
    for (int i = 1; i < Q; i++) src[i - 1] = __ldg(a.gen.src + (int64_t)(i - 1) * a.gen.G + l.g);
  }
}

// Every slot's first value is one load (predicated between the ghost buffer and
// the distributions, with no branch on the link masks): the ghost of an iolet
// link, g*_d of the own site for a wall link, g*_i of the source site otherwise
// (s + run offset for a record that follows its run, else its pull table).  The
// BFL correction of wall links follows as a predicated step: both of its rules
// (gather_links, f64_site.cuh) are g*_d + |c| (X - g*_d) with the coefficient c of
// k_bfl_coefficients laid out once per link, so the kernels divide by nothing here.
template <class S, bool IO = true>
__device__ __forceinline__ void gather_links_m(const StepArgs& a, const MixArgs& m, const LinksM& l, int s, const int* src,
                                               bool bfl, float* g) {
  const GeneralDev& G = a.gen;
  const uint32_t wm = l.wall, im = IO ? l.iolet : 0u;
  const S* fin = static_cast<const S*>(m.fin);
  g[0] = Store<S>::ld(fin + s);
#pragma unroll
  for (int i = 1; i < Q; i++) {
    const int d = inv(i);
    const bool bw = (wm >> (d - 1)) & 1u, bi = (im >> (d - 1)) & 1u;
    const int64_t k = bw ? (int64_t)d * a.np + s : (int64_t)i * a.np + src[i - 1];
    float v;
    if (bi) v = m.gin[(int64_t)(d - 1) * G.G + l.g] * Store<S>::kScale;
    else v = Store<S>::ld(fin + k);
    g[i] = v;
  }
  if (bfl && wm) {
    float cv[18], fo[18];
#pragma unroll
    for (int i = 1; i < Q; i++) {
      const int d = inv(i);
      const bool corr = ((wm >> (d - 1)) & 1u) && !((wm >> (i - 1)) & 1u);
      cv[i - 1] = corr ? __ldg(G.q + (int64_t)(d - 1) * G.G + l.g) : 0.0f;
      fo[i - 1] = corr ? Store<S>::ld(fin + (int64_t)i * a.np + s) : 0.0f;
    }
    // Slot d of a corrected link is a plain gather (no wall behind the site): the
    // pre-correction values below are final ones.
#pragma unroll
    for (int i = 1; i < Q; i++) {
      const int d = inv(i);
      const float c = cv[i - 1];
      const float x = c > 0.0f ? fo[i - 1] : g[d];
      if (c != 0.0f) g[i] = vfma(fabsf(c), vsub(x, g[i]), g[i]);
    }
  }
}

template <class S, int WALL, bool GATHER>
__device__ __forceinline__ void gather_any_m(const StepArgs& a, const MixArgs& m, int s, float* g) {
  if (!GATHER) {
    const S* p = static_cast<const S*>(m.fin) + s;
#pragma unroll
    for (int i = 0; i < Q; i++) g[i] = Store<S>::ld(p + (int64_t)i * a.np);
    return;
  }
  const int r = __ldg(a.meta + s);
  LinksM l{0u, 0u, r, 0};
  if (r < 0) {
    l.g = -r - 1;
    l.wall = __ldg(a.gen.wall + l.g);
    l.iolet = __ldg(a.gen.iolet + l.g);
    l.run = __ldg(a.gen.run + l.g);
  }
  int src[18];
  load_sources_m(a, l, s, src);
  gather_links_m<S>(a, m, l, s, src, WALL == kBFL, g);
}

// Macroscopic outputs of a site from its moments (and, at a wall site, its stress).
template <class S>
__device__ __forceinline__ void store_macro(const StepArgs& a, int s, const Moments& mo, float tau, const float* gp,
                                            const float* g, bool wall, const float nor[3]) {
  const float r = Store<S>::kScale + mo.D;
  a.rho[s] = (double)(1.0f + mo.D * (1.0f / Store<S>::kScale));
  a.u[s] = (double)(mo.mx / r);
  a.u[a.np + s] = (double)(mo.my / r);
  a.u[2 * a.np + s] = (double)(mo.mz / r);
  if (!wall && !a.pi) {
    a.wss[s] = kNoValue;
    return;
  }
  float pi[6];
  flux_tensor<S>(tau, gp, g, pi);
  a.wss[s] = wall ? wss_mag_f(pi, nor) : kNoValue;
  if (a.pi) store_pi_f(a, s, tau, pi);
}

// One plain bulk site s from its gathered values.
template <class S, int K, bool MACRO>
__device__ __forceinline__ void bulk_collide_m(const StepArgs& a, const MixArgs& m, int s, const float* g) {
  float neq[Q], gp[Q];
  const Moments mo(g);
  if (unstable(g, mo.D, Store<S>::kScale)) atomicOr(a.status, kStatusUnstable);
  non_equilibrium(Geq(mo, Store<S>::kScale), g, neq);
  float tau, om;
  site_rate<S, K>(a, neq, s, tau, om);
  relax(g, neq, K == kTRT, om, (float)a.omega_minus, gp);
  S* o = static_cast<S*>(m.fout) + s;
#pragma unroll
  for (int i = 0; i < Q; i++) {
    Store<S>::st(o, gp[i]);
    o += a.np;
  }
  if (MACRO) {
    const float nor[3] = {0.0f, 0.0f, 0.0f};
    store_macro<S>(a, s, mo, tau, gp, g, false, nor);
  }
}

// One plain bulk site s (the output steps and the first step of a state).
template <class S, int K, bool GATHER, bool MACRO>
__device__ __forceinline__ void bulk_site_m(const StepArgs& a, const MixArgs& m, int s, int r) {
  float g[Q];
  if (GATHER) {
    int off[20];
    load_row(a.run_off, r, off);
    gather_row<S, false>(a, m, s, off, g);
  } else {
    const S* p = static_cast<const S*>(m.fin) + s;
#pragma unroll
    for (int i = 0; i < Q; i++) g[i] = Store<S>::ld(p + (int64_t)i * a.np);
  }
  bulk_collide_m<S, K, MACRO>(a, m, s, g);
}

// One general site gi (`live` false: no record; the thread only waits for the
// previous step).  The ghost values of its iolet links come from iolet_link_m, and
// a GZS wall link's virtual-node value from gzs_link_m, so that link's slot is not
// stored here.
template <class S, int K, int WALL, bool GATHER, bool MACRO, bool IO = true, bool PDL = false>
__device__ __forceinline__ void general_site_m(const StepArgs& a, const MixArgs& m, int gi, bool live = true) {
  const GeneralDev& G = a.gen;
  constexpr float kScale = Store<S>::kScale;
  LinksM l{0u, 0u, 0, gi};
  int s = 0;
  uint32_t keep = ~0u;
  float g[Q];
  if (live) {
    s = __ldg(G.site + gi);
    l.wall = __ldg(G.wall + gi);
    if (IO) l.iolet = __ldg(G.iolet + gi);
    if (WALL == kGZS) keep = ~__ldg(G.gzs + gi);
  }
  if (GATHER) {
    int src[18];
    if (live) {
      l.run = __ldg(G.run + gi);
      load_sources_m(a, l, s, src);
    }
    if (PDL) wait_previous_step();
    if (!live) return;
    gather_links_m<S, IO>(a, m, l, s, src, WALL == kBFL, g);
  } else {
    const S* p = static_cast<const S*>(m.fin) + s;
#pragma unroll
    for (int i = 0; i < Q; i++) g[i] = Store<S>::ld(p + (int64_t)i * a.np);
  }
  const Moments mo(g);
  if (unstable(g, mo.D, kScale)) atomicOr(a.status, kStatusUnstable);
  float neq[Q], gp[Q];
  non_equilibrium(Geq(mo, kScale), g, neq);
  float tau, om;
  site_rate<S, K>(a, neq, s, tau, om);
  relax(g, neq, K == kTRT, om, (float)a.omega_minus, gp);
  S* o = static_cast<S*>(m.fout) + s;
  Store<S>::st(o, gp[0]);
#pragma unroll
  for (int i = 1; i < Q; i++)
    if (WALL != kGZS || ((keep >> (i - 1)) & 1u)) Store<S>::st(o + (int64_t)i * a.np, gp[i]);
  if (IO && l.iolet) {
    const int cpl = __ldg(G.cpl + gi);
    if (cpl >= 0) {
      const IoletDev& I = a.iolets[__ldg(G.io + gi)];
      const float r = kScale + mo.D;
      const float ux = mo.mx / r, uy = mo.my / r, uz = mo.mz / r;
      a.cpl_buf[cpl] = (double)ux * (-I.nrm[0]) + (double)uy * (-I.nrm[1]) + (double)uz * (-I.nrm[2]);
    }
  }
  if (MACRO) {
    const float nor[3] = {__ldg(G.nrm + gi), __ldg(G.nrm + G.G + gi), __ldg(G.nrm + 2 * G.G + gi)};
    store_macro<S>(a, s, mo, tau, gp, g, l.wall != 0u, nor);
  }
}

// A link's direction is known at run time only: opposite directions by pairs, as
// in f64_site.cuh.
__constant__ float kVelocityF[9][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0}, {1, -1, 0}, {1, 0, 1}, {1, 0, -1}, {0, 1, 1}, {0, 1, -1}};

struct PairF {
  float o, e;  // of the odd and of the even direction
};

__device__ __forceinline__ PairF pick_pair_m(const float* v, int p) {
  PairF x{v[1], v[2]};
#pragma unroll
  for (int k = 1; k < 9; k++) {
    x.o = k == p ? v[2 * k + 1] : x.o;
    x.e = k == p ? v[2 * k + 2] : x.e;
  }
  return x;
}

__device__ __forceinline__ float pair_weight_m(int p) { return p < 3 ? wf(1) : wf(7); }

// Equilibria of the pair (Geq::pair).
__device__ __forceinline__ PairF geq_pair(const Geq& c, int p) {
  const float w = pair_weight_m(p);
  const float e = vfma(kVelocityF[p][0], c.mx, vfma(kVelocityF[p][1], c.my, vmul(kVelocityF[p][2], c.mz)));
  const float even = vfma(vmul(vmul(w, c.nh), e), e, vmul(w, c.t1));
  return PairF{vfma(w, e, even), vfma(-w, e, even)};
}

// The virtual-node value of entry k of the GZS link list, one thread per link
// (gzs_link_f64 in FP32 on the stored scale).
template <class S, int K, bool GATHER, bool PDL = false>
__device__ __forceinline__ void gzs_link_m(const StepArgs& a, const MixArgs& m, int k) {
  const GeneralDev& G = a.gen;
  constexpr float kScale = Store<S>::kScale;
  const bool live = k < a.gzs_n;
  int gi = 0, d = 1, s = 0, i = 0, nb = 0;
  uint32_t im = 0;
  float q = 1.0f;
  bool extrapolate = false;
  if (live) {
    gi = __ldg(a.gzs_rec + k);
    d = __ldg(a.gzs_dir + k);
    i = (d & 1) ? d + 1 : d - 1;
    s = __ldg(G.site + gi);
    im = __ldg(G.iolet + gi);
    const int run = __ldg(G.run + gi);
    q = __ldg(G.q + (int64_t)(d - 1) * G.G + gi);
    extrapolate = q < 0.75f && !((im >> (i - 1)) & 1u);
    nb = s;
    if (extrapolate) nb = run >= 0 ? s + __ldg(a.run_off + 20 * run + d) : __ldg(G.src + (int64_t)(d - 1) * G.G + gi);
  }
  if (PDL) wait_previous_step();
  if (!live) return;
  float g[Q], gn[Q];
  gather_any_m<S, kGZS, GATHER>(a, m, s, g);
  gather_any_m<S, kGZS, GATHER>(a, m, nb, gn);
  const Moments mo(g);
  const Geq geq(mo, kScale);
  const float rho = kScale + mo.D;
  const int p = (d - 1) >> 1;
  const bool odd = d & 1;  // link d is the pair's odd direction
  PairF n = pick_pair_m(g, p);
  {
    const PairF eq = geq_pair(geq, p);
    n.o -= eq.o;
    n.e -= eq.e;
  }
  const float fac = 1.0f - 1.0f / q;
  float mw0 = mo.mx * fac, mw1 = mo.my * fac, mw2 = mo.mz * fac;
  if (extrapolate) {
    const Moments mn(gn);
    const float k2 = (1.0f - q) * rho * (q - 1.0f) / (q + 1.0f) / (kScale + mn.D);
    mw0 = q * mw0 + k2 * mn.mx;
    mw1 = q * mw1 + k2 * mn.my;
    mw2 = q * mw2 + k2 * mn.mz;
    const PairF x = pick_pair_m(gn, p), eq = geq_pair(Geq(mn, kScale), p);
    n.o = q * n.o + (1.0f - q) * (x.o - eq.o);
    n.e = q * n.e + (1.0f - q) * (x.e - eq.e);
  } else if (q < 0.75f) {  // behind the site: a velocity iolet
    const int io = __ldg(G.io + gi);
    const double p3[3] = {(double)__ldg(G.xyz + gi), (double)__ldg(G.xyz + G.G + gi), (double)__ldg(G.xyz + 2 * G.G + gi)};
    float nv[3];
    if (!link_velocity_f(a, a.iolets[io], io, gi, i, false, p3, nv)) {
      atomicOr(a.status, kStatusIoletRadius);
      nv[0] = nv[1] = nv[2] = 0.0f;
    }
    const float k2 = (1.0f - q) * rho * (q - 1.0f) / (q + 1.0f);
    mw0 = q * mw0 + k2 * nv[0];
    mw1 = q * mw1 + k2 * nv[1];
    mw2 = q * mw2 + k2 * nv[2];
  }
  const PairF eqw = geq_pair(Geq(Moments(mo.D, mw0, mw1, mw2), kScale), p);
  const float fi = odd ? n.e : n.o, gw_i = (odd ? eqw.e : eqw.o) + fi;
  float v;
  if (K == kTRT) {
    const float sym = 0.5f * (float)a.omega * (n.o + n.e), asym = 0.5f * (float)a.omega_minus * (n.o - n.e);
    v = odd ? gw_i + sym - asym : gw_i + sym + asym;
  } else {
    v = gw_i + fi * (float)a.omega;
  }
  Store<S>::st(static_cast<S*>(m.fout) + (int64_t)d * a.np + s, v);
}

// The ghost value of entry k of the iolet link list, one thread per link
// (iolet_link_f64 in FP32; the imposed velocity and density in FP64).
template <class S, int K, int WALL, bool GATHER, bool PDL = false>
__device__ __forceinline__ void iolet_link_m(const StepArgs& a, const MixArgs& m, int k) {
  const GeneralDev& G = a.gen;
  constexpr float kScale = Store<S>::kScale;
  const bool live = k < a.iol_n;
  const int gi = live ? __ldg(a.iol_rec + k) : 0, d = live ? __ldg(a.iol_dir + k) : 1;
  LinksM l{0u, 0u, 0, gi};
  int s = 0, src[18];
  if (live) {
    s = __ldg(G.site + gi);
    l.wall = __ldg(G.wall + gi);
    l.iolet = __ldg(G.iolet + gi);
    l.run = __ldg(G.run + gi);
    if (GATHER) load_sources_m(a, l, s, src);
  }
  if (PDL) wait_previous_step();
  if (!live) return;
  float g[Q];
  if (GATHER) gather_links_m<S>(a, m, l, s, src, WALL == kBFL, g);
  else {
    const S* p = static_cast<const S*>(m.fin) + s;
#pragma unroll
    for (int i = 0; i < Q; i++) g[i] = Store<S>::ld(p + (int64_t)i * a.np);
  }
  const Moments mo(g);
  const int io = __ldg(G.io + gi), p = (d - 1) >> 1;
  const bool odd = d & 1;
  const IoletDev& I = a.iolets[io];
  float v;
  if (is_velocity_iolet(I.kind)) {
    float neq[Q], tau, om, w[3];
    non_equilibrium(Geq(mo, kScale), g, neq);
    site_rate<S, K>(a, neq, s, tau, om);
    const PairF x = pick_pair_m(g, p), n = pick_pair_m(neq, p);
    float post = odd ? x.o : x.e;
    if (K == kTRT) {
      post = vfma(0.5f * om, vadd(n.o, n.e), post);
      post = vfma((odd ? 0.5f : -0.5f) * (float)a.omega_minus, vsub(n.o, n.e), post);
    } else {
      post = vfma(om, odd ? n.o : n.e, post);
    }
    const double pos[3] = {(double)__ldg(G.xyz + gi), (double)__ldg(G.xyz + G.G + gi), (double)__ldg(G.xyz + 2 * G.G + gi)};
    if (!link_velocity_f(a, I, io, gi, d, true, pos, w)) {
      atomicOr(a.status, kStatusIoletRadius);
      w[0] = w[1] = w[2] = 0.0f;
    }
    const float rho = 1.0f + mo.D * (1.0f / kScale);
    const float wc = w[0] * kVelocityF[p][0] + w[1] * kVelocityF[p][1] + w[2] * kVelocityF[p][2];
    const float corr = 2.0f * pair_weight_m(p) * rho * (odd ? wc : -wc) * 3.0f;
    v = post * (1.0f / kScale) - corr;
  } else {
    const float r = kScale + mo.D;
    const float ux = mo.mx / r, uy = mo.my / r, uz = mo.mz / r;
    const double rb = a.dens_row[io];
    const float drb = (float)(rb - 1.0);
    const float rbf = (float)rb;
    const float nx = (float)I.nrm_f[0], ny = (float)I.nrm_f[1], nz = (float)I.nrm_f[2];
    const float comp = ux * nx + uy * ny + uz * nz;
    const PairF eq = geq_pair(Geq(Moments(drb, nx * comp * rbf, ny * comp * rbf, nz * comp * rbf), 1.0f), p);
    v = odd ? eq.e : eq.o;  // the direction opposite to the link
  }
  m.gout[(int64_t)(d - 1) * G.G + gi] = v;
}

}  // namespace
}  // namespace hb
