// f64_site.cuh -- per-site device routines of the FP64 collide-and-stream step
// (kernels_f64.cu).  Every translation unit that includes it is compiled with
// -fmad=false: each product and sum is rounded separately, in the association
// order of the reference's SSE3 build.
#pragma once

#include <cuda_runtime.h>

#include "device.h"
#include "hb_common.h"
#include "step_tiles.cuh"

namespace hb {
namespace {

// ---------------------------------------------------------------------------
// Lattice maths in the reference's SSE3 order (src/lb/lattices/Lattice.h:51-110, 374-448).
// ---------------------------------------------------------------------------

// The reference multiplies every component by every f; the products with a zero
// component add +-0 and are left out here (a third of a site's FP64 operations:
// they cannot be folded by the compiler, as 0 * inf is NaN).  rho - rho is 0 for
// finite distributions and NaN otherwise, which keeps a non-finite value's effect
// on all three components.  A sum begun at -0.0 takes its first term unchanged.
// (Step time: 4M-site pipe 218.0 -> 214.2 us, 497k-site LES stenosis 44.0 -> 41.8 us.)
__device__ __forceinline__ void moments(const double* f, double& rho, double& mx, double& my, double& mz) {
  double dl = f[0], dh = f[18];
  double xl = -0.0, xh = cx(18) ? (double)cx(18) * f[18] : -0.0;
  double yl = -0.0, yh = cy(18) ? (double)cy(18) * f[18] : -0.0;
  double zl = -0.0, zh = cz(18) ? (double)cz(18) * f[18] : -0.0;
#pragma unroll
  for (int d = 0; d < 18; d += 2) {
    if (d) dl = dl + f[d];
    dh = dh + f[d + 1];
    if (cx(d)) xl = xl + (double)cx(d) * f[d];
    if (cx(d + 1)) xh = xh + (double)cx(d + 1) * f[d + 1];
    if (cy(d)) yl = yl + (double)cy(d) * f[d];
    if (cy(d + 1)) yh = yh + (double)cy(d + 1) * f[d + 1];
    if (cz(d)) zl = zl + (double)cz(d) * f[d];
    if (cz(d + 1)) zh = zh + (double)cz(d + 1) * f[d + 1];
  }
  rho = dl + dh;
  const double nf = rho - rho;
  mx = (xl + xh) + nf;
  my = (yl + yh) + nf;
  mz = (zl + zh) + nf;
}

struct FeqConst {
  double rho, mx, my, mz, t1, nh;
  __device__ __forceinline__ FeqConst(double r, double x, double y, double z) : rho(r), mx(x), my(y), mz(z) {
    const double th = (3. / 2.) * (mx * mx + my * my + mz * mz);
    const double d1 = 1. / rho;
    nh = (9. / 2.) * d1;
    t1 = rho - th * d1;
  }
  __device__ __forceinline__ double mde(int i) const {
    double e = -0.0;
    if (cx(i)) e = e + (double)cx(i) * mx;
    if (cy(i)) e = e + (double)cy(i) * my;
    if (cz(i)) e = e + (double)cz(i) * mz;
    return e;
  }
  __device__ __forceinline__ double operator()(int i) const {
    if (i == 0) return weight(0) * t1;
    const double e = mde(i);
    return weight(i) * ((t1 + nh * (e * e)) + 3. * e);
  }
  // f[i] - feq(i) for every direction; the opposite of an odd i is i + 1, whose
  // momentum component is -e exactly, so the two share the even part.
  __device__ __forceinline__ void neq(const double* f, double* fneq) const {
    fneq[0] = f[0] - (*this)(0);
#pragma unroll
    for (int i = 1; i < Q; i += 2) {
      const double e = mde(i), even = t1 + nh * (e * e), odd = 3. * e;
      fneq[i] = f[i] - weight(i) * (even + odd);
      fneq[i + 1] = f[i + 1] - weight(i + 1) * (even - odd);
    }
  }
};

// Sum over l of v[l] c_p c_r in index order (a momentum flux component).
__device__ __forceinline__ double flux(const double* v, int p, int r) {
  double acc = -0.0;
#pragma unroll
  for (int l = 0; l < Q; l++)
    if (cc(p, l) * cc(r, l)) acc += (double)(cc(p, l) * cc(r, l)) * v[l];
  return acc;
}

// Relaxation time of the LES kernel (LBGKLESSpongeLayer::CalculateTau and
// compute_tau_smagorinsky, src/lb/kernels/LBGKLESSpongeLayer.h:122-182).
__device__ __forceinline__ double les_tau(const StepArgs& a, const double* fneq, double vt) {
  const double tau0 = a.tau;
  double q12 = 0.0;
#pragma unroll
  for (int p = 0; p < 3; p++)
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const double qij = flux(fneq, p < r ? p : r, p < r ? r : p);
      q12 += qij * qij;
    }
  q12 = sqrt(q12);
  constexpr double kSmag = 18.0 * 1.4142135623730950488016887242097 * 1.0 * 0.1 * 0.1;
  const double tau_les = 1. / 2. * (tau0 + sqrt((tau0 * 1.0 * 1.0) * (tau0 * 1.0 * 1.0) + kSmag * q12) / (1.0 * 1.0));
  if (a.t <= a.lifetime / 2) return (vt == tau0) ? tau_les : vt;
  if (a.t < a.lifetime) return (tau_les - vt) * 2.0 / (double)a.lifetime * (double)a.t + (2.0 * vt - tau_les);
  return tau_les;
}

// Relaxation time of the LBGK and TRT sponge-layer kernels (CalculateTau,
// src/lb/kernels/LBGKSpongeLayer.h:124-140, TRTSpongeLayer.h:157-172): the site's
// sponge time for the first half of the lifetime, then a linear return to tau0.
__device__ __forceinline__ double sponge_tau(const StepArgs& a, double vt) {
  const double tau0 = a.tau;
  if (a.t <= a.lifetime / 2) return vt;
  if (a.t < a.lifetime) return (tau0 - vt) * 2.0 / (double)a.lifetime * (double)a.t + (2.0 * vt - tau0);
  return tau0;
}

// Post-collision value of direction i for kernel K (LBGK.h:64-72, TRT.h:80-109,
// and the sponge-layer kernels).  `omega_site` is the site's -1/tau for LBGK,
// LES and LBGKSL, and its antisymmetric rate for TRTSL, whose symmetric rate stays
// the global omega (TRTSpongeLayer.h:86-115).
template <int K>
__device__ __forceinline__ double collide_one(const StepArgs& a, const double* f, const double* fneq, double omega_site, int i) {
  if (K == kTRT || K == kTRTSL) {
    const double omm = K == kTRT ? a.omega_minus : omega_site;
    if (i == 0) return f[0] + (0.5 * a.omega * (fneq[0] + fneq[0])) - (0.5 * omm * (fneq[0] - fneq[0]));
    const int j = inv(i);
    const int lo = i < j ? i : j, hi = i < j ? j : i;
    const double sym = 0.5 * a.omega * (fneq[lo] + fneq[hi]);
    const double asym = 0.5 * omm * (fneq[lo] - fneq[hi]);
    return i == lo ? (f[i] + sym + asym) : (f[i] + sym - asym);
  }
  return f[i] + fneq[i] * omega_site;
}

// The site's relaxation time and the rate collide_one takes for kernel K.
template <int K>
__device__ __forceinline__ void site_rates(const StepArgs& a, const double* fneq, int s, double& tau, double& om) {
  tau = a.tau;
  om = a.omega;
  if (K == kLES) {
    tau = les_tau(a, fneq, __ldg(a.vtau + s));
    om = -1.0 / tau;
  } else if (K == kLBGKSL) {
    tau = sponge_tau(a, __ldg(a.vtau + s));
    om = -1.0 / tau;
  } else if (K == kTRTSL) {
    tau = sponge_tau(a, __ldg(a.vtau + s));
    const double tau_minus = 0.5 + a.lambda / (tau - 0.5);
    om = -1.0 / tau_minus;
  }
}

// Wall-shear-stress magnitude (Lattice::CalculateWallShearStressMagnitude,
// CalculatePiTensor; src/lb/lattices/Lattice.h:1122-1156, 1353-1383).
__device__ __forceinline__ double wss_mag(double tau, const double* fpost, const double* f, const double nor[3]) {
  double pi[3][3], df[Q];
#pragma unroll
  for (int l = 0; l < Q; l++) df[l] = fpost[l] - f[l];
#pragma unroll
  for (int p = 0; p < 3; p++)
#pragma unroll
    for (int r = 0; r <= p; r++) pi[p][r] = flux(df, p, r) * -(tau - 0.5);
  pi[0][1] = pi[1][0];
  pi[0][2] = pi[2][0];
  pi[1][2] = pi[2][1];
  double sv[3] = {0.0, 0.0, 0.0}, sq = 0.0, ns = 0.0;
#pragma unroll
  for (int p = 0; p < 3; p++) {
#pragma unroll
    for (int r = 0; r < 3; r++) sv[p] += pi[p][r] * nor[r];
    sq += sv[p] * sv[p];
    ns += sv[p] * nor[p];
  }
  return sqrt(sq - ns * ns);
}

// Non-equilibrium momentum flux tensor of an output step, stored for the stress
// caches: the lower triangle in CalculatePiTensor's order and rounding
// (src/lb/lattices/Lattice.h:1353-1383) as xx, xy, xz, yy, yz, zz, then tau.
__device__ __forceinline__ void store_pi(const StepArgs& a, int s, double tau, const double* fpost, const double* f) {
  double pi[3][3], df[Q];
#pragma unroll
  for (int l = 0; l < Q; l++) df[l] = fpost[l] - f[l];
#pragma unroll
  for (int p = 0; p < 3; p++)
#pragma unroll
    for (int r = 0; r <= p; r++) pi[p][r] = flux(df, p, r) * -(tau - 0.5);
  double* o = a.pi + s;
  o[0] = pi[0][0];
  o[a.np] = pi[1][0];
  o[2 * a.np] = pi[2][0];
  o[3 * a.np] = pi[1][1];
  o[4 * a.np] = pi[2][1];
  o[5 * a.np] = pi[2][2];
  o[6 * a.np] = tau;
}

// InOutLetParabolicVelocity::GetVelocity (src/lb/iolets/InOutLetParabolicVelocity.cc:30-58).
__device__ __forceinline__ bool parabolic(const IoletDev& I, const double x[3], uint64_t t, double v[3]) {
  const double dx = x[0] - I.pos[0], dy = x[1] - I.pos[1], dz = x[2] - I.pos[2];
  const double z = dx * I.nrm[0] + dy * I.nrm[1] + dz * I.nrm[2];
  const double rsq = (dx * dx + dy * dy + dz * dz) - z * z;
  const double r2a2 = rsq / (I.radius * I.radius);
  double mx = I.max_speed;
  if (t < I.warmup) mx *= (double)t / (double)I.warmup;
  const double s = mx * (1. - r2a2);
  v[0] = I.nrm[0] * s;
  v[1] = I.nrm[1] * s;
  v[2] = I.nrm[2] * s;
  return !(r2a2 > 1.0);
}

// InOutLetVelocity::GetVelocity of a velocity iolet for link d of general site g:
// at the Ladd half-way point pos + c_d / 2 (half) or at the neighbour pos + c_d
// (the GZS extrapolation).  Parabolic: the profile above.  File velocity
// (src/lb/iolets/InOutLetFileVelocity.cc:104-128): the same profile with the
// step's peak speed from the iolet row.  Womersley
// (src/lb/iolets/InOutLetWomersleyVelocity.cc:25-41): Re(A exp(i omega t)) along
// -normal, A from the link table and exp(i omega t) from the iolet row, the
// product's real part rounded as the host's complex multiply rounds it.
// Returns false for a point outside a parabolic profile's radius.
__device__ __forceinline__ bool link_velocity(const StepArgs& a, const IoletDev& I, int io, int g, int d, bool half,
                                              const double pos[3], double v[3]) {
  if (I.kind == kWomersley) {
    const double* A = a.wom_amp + ((int64_t)__ldg(a.gen.wom + g) * 18 + (d - 1)) * 4 + (half ? 0 : 2);
    const double re = __ldg(A), im = __ldg(A + 1);
    const double speed = re * a.dens_row[kRowA + io] - im * a.dens_row[kRowB + io];
    v[0] = I.nrm[0] * -speed;
    v[1] = I.nrm[1] * -speed;
    v[2] = I.nrm[2] * -speed;
    return true;
  }
  double x[3] = {pos[0], pos[1], pos[2]};
  if (half) {
    x[0] += 0.5 * cx(d);
    x[1] += 0.5 * cy(d);
    x[2] += 0.5 * cz(d);
  } else {
    x[0] += cx(d);
    x[1] += cy(d);
    x[2] += cz(d);
  }
  if (I.kind == kParabolic) return parabolic(I, x, (uint64_t)(unsigned int)a.t, v);
  const double dx = x[0] - I.pos[0], dy = x[1] - I.pos[1], dz = x[2] - I.pos[2];
  const double z = dx * I.nrm[0] + dy * I.nrm[1] + dz * I.nrm[2];
  const double rsq = (dx * dx + dy * dy + dz * dz) - z * z;
  const double r2a2 = rsq / (I.radius * I.radius);
  const double s = a.dens_row[kRowA + io] * (1. - r2a2);
  v[0] = I.nrm[0] * s;
  v[1] = I.nrm[1] * s;
  v[2] = I.nrm[2] * s;
  return !(r2a2 > 1.0);
}

// Distributions and ghosts are read with plain loads: the step kernel is launched
// while the one that wrote them may still be running and waits for it inside
// (griddepcontrol), which orders plain loads but not the non-coherent ones.
__device__ __forceinline__ double ld(const double* p) { return *p; }

__device__ __forceinline__ void load_run_offsets(const StepArgs& a, int r, int* off) {
  const int4* o4 = reinterpret_cast<const int4*>(a.run_off) + 5 * r;
#pragma unroll
  for (int k = 0; k < 5; k++) {
    const int4 v = __ldg(o4 + k);
    off[4 * k] = v.x;
    off[4 * k + 1] = v.y;
    off[4 * k + 2] = v.z;
    off[4 * k + 3] = v.w;
  }
}

// Link masks and run of a site: a general record's own, none for a plain bulk site.
struct Links {
  uint32_t wall, iolet;
  int run, g;
};

// The source of every slot i of site s before any boundary rule: s + run_off[run][i]
// for a site whose bulk slots follow its run (L1-resident offsets), else the
// record's pull table entry (which holds the record's own site for a slot that a
// boundary rule fills).
__device__ __forceinline__ void load_sources(const StepArgs& a, const Links& l, int s, int* src) {
  if (l.run >= 0) {
    int off[20];
    load_run_offsets(a, l.run, off);
#pragma unroll
    for (int i = 1; i < Q; i++) src[i - 1] = s + off[i];
  } else {
#pragma unroll
    for (int i = 1; i < Q; i++) src[i - 1] = __ldg(a.gen.src + (int64_t)(i - 1) * a.gen.G + l.g);
  }
}

// Every slot's first value is one load whose address needs no branch: the
// ghost of an iolet link, f*_d of the own site for a wall link, f*_i of the
// source site otherwise.  All eighteen loads are issued together, and a warp
// issues them once whatever its sites' link masks; the BFL correction of wall
// links follows as a predicated step.  (4M-site pipe, boundary kernel alone:
// branching per link 0.0599 ms, pull table for every record 0.0554 ms, run
// offsets where they apply 0.0541 ms.)
template <int WALL, bool IO = true>
__device__ __forceinline__ void gather_links(const StepArgs& a, const Links& l, int s, const int* src, double* f) {
  const GeneralDev& G = a.gen;
  const uint32_t wm = l.wall, im = IO ? l.iolet : 0u;
  const int g = l.g;
  f[0] = ld(a.fin + s);
#pragma unroll
  for (int i = 1; i < Q; i++) {
    const int d = inv(i);
    const bool bw = (wm >> (d - 1)) & 1u, bi = (im >> (d - 1)) & 1u;
    const double* p = bi ? a.gin + (int64_t)(d - 1) * G.G + g
                         : a.fin + (bw ? (int64_t)d * a.np + s : (int64_t)i * a.np + src[i - 1]);
    f[i] = ld(p);
  }
  if (WALL == kBFL && wm) {
    // BFL on wall link d with no wall behind (slot i = inv(d)): q >= 1/2 takes
    // (f*_d + (2q-1) f*_i) / (2q); q < 1/2 keeps f*_d and takes the post-step
    // 2q f*_d + (1-2q) f[d] (slot d is never corrected itself, as link i has no
    // wall).  Every cut distance and own-site value is loaded before any
    // arithmetic, so they share one round trip with the gather (4M-site pipe,
    // boundary kernel alone 0.0545 -> 0.0429 ms together with 128 registers).
    float qv[18];
    double fo[18];
#pragma unroll
    for (int i = 1; i < Q; i++) {
      const int d = inv(i);
      const bool corr = ((wm >> (d - 1)) & 1u) && !((wm >> (i - 1)) & 1u);
      qv[i - 1] = corr ? __ldg(G.q + (int64_t)(d - 1) * G.G + g) : 1.0f;
      fo[i - 1] = corr ? ld(a.fin + (int64_t)i * a.np + s) : 0.0;
    }
#pragma unroll
    for (int i = 1; i < Q; i++) {
      const int d = inv(i);
      const bool corr = ((wm >> (d - 1)) & 1u) && !((wm >> (i - 1)) & 1u);
      if (corr) {
        const double q = (double)qv[i - 1];
        if (!(q < 0.5)) f[i] = (f[i] + (2.0 * q - 1) * fo[i - 1]) / (2.0 * q);
        else f[i] = 2.0 * q * f[i] + (1.0 - 2.0 * q) * f[d];
      }
    }
  }
}

// Pre-collision f of any site (GZS neighbours, materialisation).
template <int WALL, bool GATHER>
__device__ __forceinline__ void gather_any(const StepArgs& a, int s, double* f) {
  if (!GATHER) {
#pragma unroll
    for (int i = 0; i < Q; i++) f[i] = ld(a.fin + (int64_t)i * a.np + s);
    return;
  }
  const int r = __ldg(a.meta + s);
  Links l{0u, 0u, r, 0};
  if (r < 0) {
    l.g = -r - 1;
    l.wall = __ldg(a.gen.wall + l.g);
    l.iolet = __ldg(a.gen.iolet + l.g);
    l.run = __ldg(a.gen.run + l.g);
  }
  int src[18];
  load_sources(a, l, s, src);
  gather_links<WALL>(a, l, s, src, f);
}

__device__ __forceinline__ void flag_unstable(const StepArgs& a, const double* f) {
  bool bad = false;
#pragma unroll
  for (int i = 0; i < Q; i++) bad |= !(f[i] > 0.0);
  if (bad) atomicOr(a.status, kStatusUnstable);
}

// ---------------------------------------------------------------------------
// Per-site steps
// ---------------------------------------------------------------------------

// One plain bulk site s whose run's offsets are `off` (GATHER).
template <int K, bool GATHER, bool MACRO>
__device__ __forceinline__ void bulk_site_f64(const StepArgs& a, int s, const int* off) {
  double f[Q];
  f[0] = ld(a.fin + s);
#pragma unroll
  for (int i = 1; i < Q; i++) f[i] = ld(a.fin + (int64_t)i * a.np + (GATHER ? s + off[i] : s));
  flag_unstable(a, f);
  double rho, mx, my, mz;
  moments(f, rho, mx, my, mz);
  const FeqConst feq(rho, mx, my, mz);
  double fneq[Q];
  feq.neq(f, fneq);
  double om, tau;
  site_rates<K>(a, fneq, s, tau, om);
#pragma unroll
  for (int i = 0; i < Q; i++) a.fout[(int64_t)i * a.np + s] = collide_one<K>(a, f, fneq, om, i);
  if (MACRO) {
    a.rho[s] = rho;
    a.u[s] = mx / rho;
    a.u[a.np + s] = my / rho;
    a.u[2 * a.np + s] = mz / rho;
    a.wss[s] = kNoValue;
    if (a.pi) {
      double fp[Q];
#pragma unroll
      for (int i = 0; i < Q; i++) fp[i] = collide_one<K>(a, f, fneq, om, i);
      store_pi(a, s, tau, fp, f);
    }
  }
}

// One general (boundary or irregular) site record g; `live` false: no record (the
// thread only waits for the previous step).  The ghost values of its iolet links
// come from iolet_link_f64, and a GZS wall link's virtual-node value from
// gzs_link_f64, so that link's slot is not stored here.
template <int K, int WALL, bool GATHER, bool MACRO, bool IO = true, bool PDL = false>
__device__ __forceinline__ void general_site_f64(const StepArgs& a, int g, bool live = true) {
  const GeneralDev& G = a.gen;
  Links l{0u, 0u, 0, g};
  int s = 0;
  uint32_t keep = ~0u;
  double f[Q];
  if (GATHER) {
    int src[18];
    if (live) {
      s = __ldg(G.site + g);
      l.wall = __ldg(G.wall + g);
      if (IO) l.iolet = __ldg(G.iolet + g);
      l.run = __ldg(G.run + g);
      load_sources(a, l, s, src);
      if (WALL == kGZS) keep = ~__ldg(G.gzs + g);
    }
    if (PDL) wait_previous_step();
    if (!live) return;
    gather_links<WALL, IO>(a, l, s, src, f);
  } else {
    s = __ldg(G.site + g);
    l.wall = __ldg(G.wall + g);
    if (IO) l.iolet = __ldg(G.iolet + g);
    if (WALL == kGZS) keep = ~__ldg(G.gzs + g);
#pragma unroll
    for (int i = 0; i < Q; i++) f[i] = ld(a.fin + (int64_t)i * a.np + s);
  }
  const uint32_t wm = l.wall, im = l.iolet;
  flag_unstable(a, f);
  double rho, mx, my, mz;
  moments(f, rho, mx, my, mz);
  const double ux = mx / rho, uy = my / rho, uz = mz / rho;
  const FeqConst feq(rho, mx, my, mz);
  double fneq[Q];
  feq.neq(f, fneq);
  double om, tau;
  site_rates<K>(a, fneq, s, tau, om);
  double fp[Q];
#pragma unroll
  for (int i = 0; i < Q; i++) fp[i] = collide_one<K>(a, f, fneq, om, i);
  a.fout[s] = fp[0];
#pragma unroll
  for (int i = 1; i < Q; i++)
    if (WALL != kGZS || ((keep >> (i - 1)) & 1u)) a.fout[(int64_t)i * a.np + s] = fp[i];

  const int cpl = im ? __ldg(G.cpl + g) : -1;
  if (cpl >= 0) {
    const IoletDev& I = a.iolets[__ldg(G.io + g)];
    a.cpl_buf[cpl] = ux * (-I.nrm[0]) + uy * (-I.nrm[1]) + uz * (-I.nrm[2]);
  }
  if (MACRO) {
    a.rho[s] = rho;
    a.u[s] = ux;
    a.u[a.np + s] = uy;
    a.u[2 * a.np + s] = uz;
    if (wm) {
      const double nor[3] = {(double)__ldg(G.nrm + g), (double)__ldg(G.nrm + G.G + g), (double)__ldg(G.nrm + 2 * G.G + g)};
      a.wss[s] = wss_mag(tau, fp, f, nor);
    } else {
      a.wss[s] = kNoValue;
    }
    if (a.pi) store_pi(a, s, tau, fp, f);
  }
}

// A link's direction is known at run time only.  Directions 2p + 1 (odd) and 2p + 2
// (even) are opposite, so nine pairs are told apart instead of eighteen
// directions, and the velocities come from a constant table: selecting each
// direction and converting compared components took half of a GZS link's
// instructions (594k-site bifurcation, TRT: step 95.2 -> 84.3 us, FP32 of
// 187k sites 24.5 -> 19.1).
__constant__ double kVelocity[9][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0}, {1, -1, 0}, {1, 0, 1}, {1, 0, -1}, {0, 1, 1}, {0, 1, -1}};

struct Pair {
  double o, e;  // of the odd and of the even direction
};

__device__ __forceinline__ Pair pick_pair(const double* v, int p) {
  Pair x{v[1], v[2]};
#pragma unroll
  for (int k = 1; k < 9; k++) {
    x.o = k == p ? v[2 * k + 1] : x.o;
    x.e = k == p ? v[2 * k + 2] : x.e;
  }
  return x;
}

__device__ __forceinline__ double pair_weight(int p) { return p < 3 ? weight(1) : weight(7); }

// Equilibria of the pair (FeqConst::neq).
__device__ __forceinline__ Pair feq_pair(const FeqConst& c, int p) {
  const double e = kVelocity[p][0] * c.mx + kVelocity[p][1] * c.my + kVelocity[p][2] * c.mz;
  const double even = c.t1 + c.nh * (e * e), odd = 3. * e, w = pair_weight(p);
  return Pair{w * (even + odd), w * (even - odd)};
}

// The virtual-node value of entry k of the GZS link list (wall link d of general
// record g; GuoZhengShiDelegate::StreamLink, src/lb/streamers/GuoZhengShiDelegate.h:127-293),
// stored in f*_d of the record's site.  One thread per link: the site and the
// neighbour its virtual node extrapolates from are gathered together, where a
// thread per record walked its links one after the other, each with a gather of its
// own inlined: 18 gathers of code, most of its time waiting for instructions
// (594k-site bifurcation, TRT: step 215 -> 105 us).  Walking a record's links
// in a rolled loop that gathers the site once is slower (96 -> 135 us: too few
// threads for so long a chain), and so are a record's links side by side in a warp
// (101 us).
template <int K, bool GATHER, bool PDL = false>
__device__ __forceinline__ void gzs_link_f64(const StepArgs& a, int k) {
  const GeneralDev& G = a.gen;
  const bool live = k < a.gzs_n;
  const int g = live ? __ldg(a.gzs_rec + k) : 0, d = live ? __ldg(a.gzs_dir + k) : 1;
  int s = 0, run = 0, i = 0, nb = 0;
  uint32_t wm = 0, im = 0;
  double q = 1.0;
  bool extrapolate = false;
  if (live) {
    i = (d & 1) ? d + 1 : d - 1;
    s = __ldg(G.site + g);
    wm = __ldg(G.wall + g);
    im = __ldg(G.iolet + g);
    run = __ldg(G.run + g);
    q = (double)__ldg(G.q + (int64_t)(d - 1) * G.G + g);
    extrapolate = q < 0.75 && !((im >> (i - 1)) & 1u);
    nb = s;
    if (extrapolate) nb = run >= 0 ? s + __ldg(a.run_off + 20 * run + d) : __ldg(G.src + (int64_t)(d - 1) * G.G + g);
  }
  if (PDL) wait_previous_step();
  if (!live) return;
  double f[Q], fn[Q];
  gather_any<kGZS, GATHER>(a, s, f);
  gather_any<kGZS, GATHER>(a, nb, fn);
  double rho, mx, my, mz;
  moments(f, rho, mx, my, mz);
  const FeqConst feq(rho, mx, my, mz);
  const int p = (d - 1) >> 1;
  const bool odd = d & 1;  // link d is the pair's odd direction
  Pair n = pick_pair(f, p);
  {
    const Pair eq = feq_pair(feq, p);
    n.o -= eq.o;
    n.e -= eq.e;
  }
  const double fac = 1. - 1. / q;
  double mw0 = mx * fac, mw1 = my * fac, mw2 = mz * fac;
  if (extrapolate) {
    double rn, mnx, mny, mnz;
    moments(fn, rn, mnx, mny, mnz);
    const double vn0 = mnx / rn, vn1 = mny / rn, vn2 = mnz / rn;
    mw0 = q * mw0 + (1. - q) * rho * (vn0 * (q - 1) / (q + 1));
    mw1 = q * mw1 + (1. - q) * rho * (vn1 * (q - 1) / (q + 1));
    mw2 = q * mw2 + (1. - q) * rho * (vn2 * (q - 1) / (q + 1));
    const Pair x = pick_pair(fn, p), eq = feq_pair(FeqConst(rn, mnx, mny, mnz), p);
    n.o = q * n.o + (1. - q) * (x.o - eq.o);
    n.e = q * n.e + (1. - q) * (x.e - eq.e);
  } else if (q < 0.75) {  // behind the site: a velocity iolet
    const int io = __ldg(G.io + g);
    const double p3[3] = {(double)__ldg(G.xyz + g), (double)__ldg(G.xyz + G.G + g), (double)__ldg(G.xyz + 2 * G.G + g)};
    double nv[3];
    if (!link_velocity(a, a.iolets[io], io, g, i, false, p3, nv)) {
      atomicOr(a.status, kStatusIoletRadius);
      nv[0] = nv[1] = nv[2] = 0.0;
    }
    mw0 = q * mw0 + (1. - q) * rho * (nv[0] * (q - 1) / (q + 1));
    mw1 = q * mw1 + (1. - q) * rho * (nv[1] * (q - 1) / (q + 1));
    mw2 = q * mw2 + (1. - q) * rho * (nv[2] * (q - 1) / (q + 1));
  }
  const Pair eqw = feq_pair(FeqConst(rho, mw0, mw1, mw2), p);
  const double fnw_i = odd ? n.e : n.o, fw_i = (odd ? eqw.e : eqw.o) + fnw_i;
  double v;
  if (K == kTRT) {
    const double sym = 0.5 * a.omega * (n.o + n.e);
    const double asym = 0.5 * a.omega_minus * (n.o - n.e);
    v = odd ? (fw_i + sym - asym) : (fw_i + sym + asym);
  } else {
    v = fw_i + fnw_i * a.omega;
  }
  a.fout[(int64_t)d * a.np + s] = v;
}

// Post-collision value of direction d, known at run time only (collide_one).
template <int K>
__device__ __forceinline__ double collide_at(const StepArgs& a, const double* f, const double* fneq, double omega_site, int d) {
  const int p = (d - 1) >> 1;
  const bool odd = d & 1;
  const Pair x = pick_pair(f, p), n = pick_pair(fneq, p);
  if (K == kTRT || K == kTRTSL) {
    const double omm = K == kTRT ? a.omega_minus : omega_site;
    const double sym = 0.5 * a.omega * (n.o + n.e);
    const double asym = 0.5 * omm * (n.o - n.e);
    return odd ? (x.o + sym + asym) : (x.e + sym - asym);
  }
  return odd ? x.o + n.o * omega_site : x.e + n.e * omega_site;
}

// The ghost value of entry k of the iolet link list: link d of general record g.
// One thread per link: with a thread per record, the few blocks of iolet records
// evaluated up to eighteen links' profiles and divisions one after the other and
// set the time of a small lattice's step (13k-site pipe 7.7 -> 5.5 us, 63k-site pipe
// with a velocity inlet 13.4 -> 8.4, 197k-site pipe FP32 10.6 -> 7.4).
template <int K, int WALL, bool GATHER, bool PDL = false>
__device__ __forceinline__ void iolet_link_f64(const StepArgs& a, int k) {
  const GeneralDev& G = a.gen;
  const bool live = k < a.iol_n;
  const int g = live ? __ldg(a.iol_rec + k) : 0, d = live ? __ldg(a.iol_dir + k) : 1;
  Links l{0u, 0u, 0, g};
  int s = 0, src[18];
  if (live) {
    s = __ldg(G.site + g);
    l.wall = __ldg(G.wall + g);
    l.iolet = __ldg(G.iolet + g);
    l.run = __ldg(G.run + g);
    if (GATHER) load_sources(a, l, s, src);
  }
  if (PDL) wait_previous_step();
  if (!live) return;
  double f[Q];
  if (GATHER) gather_links<WALL>(a, l, s, src, f);
  else {
#pragma unroll
    for (int i = 0; i < Q; i++) f[i] = ld(a.fin + (int64_t)i * a.np + s);
  }
  const int io = __ldg(G.io + g);
  const IoletDev& I = a.iolets[io];
  double rho, mx, my, mz;
  moments(f, rho, mx, my, mz);
  double v;
  if (is_velocity_iolet(I.kind)) {
    // LaddIoletDelegate::StreamLink (src/lb/streamers/LaddIoletDelegate.h:37-86).
    double fneq[Q], om, tau, w[3];
    FeqConst(rho, mx, my, mz).neq(f, fneq);
    site_rates<K>(a, fneq, s, tau, om);
    const double pos[3] = {(double)__ldg(G.xyz + g), (double)__ldg(G.xyz + G.G + g), (double)__ldg(G.xyz + 2 * G.G + g)};
    if (!link_velocity(a, I, io, g, d, true, pos, w)) {
      atomicOr(a.status, kStatusIoletRadius);
      w[0] = w[1] = w[2] = 0.0;
    }
    w[0] *= rho;
    w[1] *= rho;
    w[2] *= rho;
    const int p = (d - 1) >> 1;
    const double sign = (d & 1) ? 1.0 : -1.0;
    const double wc = w[0] * (sign * kVelocity[p][0]) + w[1] * (sign * kVelocity[p][1]) + w[2] * (sign * kVelocity[p][2]);
    v = collide_at<K>(a, f, fneq, om, d) - 2. * pair_weight(p) * wc / kCs2;
  } else {
    // NashZerothOrderPressureDelegate::StreamLink (src/lb/streamers/NashZerothOrderPressureDelegate.h:36-76).
    const double rb = a.dens_row[io];
    const double nx = I.nrm_f[0], ny = I.nrm_f[1], nz = I.nrm_f[2];
    const double comp = (mx / rho) * nx + (my / rho) * ny + (mz / rho) * nz;
    const Pair eq = feq_pair(FeqConst(rb, nx * comp * rb, ny * comp * rb, nz * comp * rb), (d - 1) >> 1);
    v = (d & 1) ? eq.e : eq.o;  // the direction opposite to the link
  }
  a.gout[(int64_t)(d - 1) * G.G + g] = v;
}

}  // namespace
}  // namespace hb
