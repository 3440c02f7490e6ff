// ref_stepper.cu - the reference's src/physics Kerr API batched on the GPU.
//
//   k_kerr_potentials  <- physics::kerrPotentials       (src/physics/kerr.cpp:69-97)
//   k_kerr_step_mino   <- physics::kerrStepMino         (src/physics/kerr.cpp:99-134)
//   k_kerr_trace_rays  <- physics::KerrRaytracer::trace (src/physics/raytracer.h:324-378)
//
// First-order Mino-time form with sign flips, CGS units, the reference's
// expression order; compiled with -fmad=false so every FP64 operation rounds
// once as on the CPU. What differs from the host is sin^2 and cos^2, by an ulp
// or two: the potentials take them from CUDA's sincos, the steps and the trace's
// sign test from sin2_cos2 below. One thread per state; inputs and outputs are
// structure-of-arrays.
#include <cuda_runtime.h>

#include "ieee_fp64.cuh"
#include "launch.h"

namespace {

constexpr double kC = 2.99792458e10;
constexpr double kC2 = kC * kC;
constexpr double kG = 6.67430e-8;
constexpr double kPI = 3.141592653589793;

struct Pot {
  double rPot, dRdr, thetaPot, dThetadtheta;
};
struct St {
  double r, theta, phi, t, signR, signTheta;
};
struct Cs {
  double e, lz, q;
};
struct Dv {
  double dr, dtheta, dphi, dt;
};

__device__ __forceinline__ double mx(double a, double b) { return (a < b) ? b : a; }

__device__ __forceinline__ Pot potentials(double r, double theta, double mass, double a, const Cs &c) {
  const double mGeom = kG * mass / kC2;
  const double rr = r * r;
  const double aa = a * a;
  double sinTheta, cosTheta;
  sincos(theta, &sinTheta, &cosTheta);
  const double sin2 = mx(sinTheta * sinTheta, 1e-12);
  const double cos2 = cosTheta * cosTheta;
  const double delta = rr - (2.0 * mGeom * r) + aa;
  const double aFactor = ((rr + aa) * c.e) - (a * c.lz);
  const double lzMinusAe = c.lz - (a * c.e);
  Pot p;
  p.rPot = (aFactor * aFactor) - (delta * (c.q + (lzMinusAe * lzMinusAe)));
  const double dAdR = 2.0 * r * c.e;
  const double dDeltaDr = (2.0 * r) - (2.0 * mGeom);
  p.dRdr = (2.0 * aFactor * dAdR) - (dDeltaDr * (c.q + (lzMinusAe * lzMinusAe)));
  p.thetaPot = c.q + (aa * c.e * c.e * cos2) - (c.lz * c.lz / sin2);
  p.dThetadtheta = -(2.0 * aa * c.e * c.e * cosTheta * sinTheta) + (2.0 * c.lz * c.lz * cosTheta / (sin2 * sinTheta));
  return p;
}

// sin^2 and cos^2 of |x| < 2^10. The angle less the nearest multiple of pi / 2,
// which is taken in two parts, as r + rl; Taylor's series on |r| <= pi / 4 to
// r^17 and r^16, summed in pairs (G. Estrin's scheme). Sine and cosine were within
// 0.83 ulp each at 2e7 arguments; tests/test_gpu_ray_angles.py has the step's. CUDA's
// sincos has a branch for large arguments: four calls a step keep its stages in
// blocks of their own, and the polar motion is the step's longest chain.
__device__ __forceinline__ void sin2_cos2(double x, double &s2, double &c2) {
  const double t = fma(x, 0x1.45f306dc9c883p-1, 0x1.8p52);  // 2 / pi
  const bool odd = __double2loint(t) & 1;
  const double k = t - 0x1.8p52;
  constexpr double hi = 0x1.921fb54442d18p0, lo = 0x1.1a62633145c07p-54;  // pi / 2
  const double r1 = fma(-k, hi, x), r = fma(-k, lo, r1), rl = fma(-k, lo, r1 - r);
  const double z = r * r, z2 = z * z, z4 = z2 * z2;
  const double S = fma(fma(fma(1 / 355687428096000.0, z, -1 / 1307674368000.0), z2,
                           fma(1 / 6227020800.0, z, -1 / 39916800.0)),
                       z4, fma(fma(1 / 362880.0, z, -1 / 5040.0), z2, fma(1 / 120.0, z, -1 / 6.0)));
  const double C = fma(fma(1 / 20922789888000.0, z2, fma(-1 / 87178291200.0, z, 1 / 479001600.0)), z4,
                       fma(fma(-1 / 3628800.0, z, 1 / 40320.0), z2, fma(-1 / 720.0, z, 1 / 24.0)));
  const double w = fma(-0.5, z, 1.0), e = fma(-0.5, z, 1.0 - w);
  const double s = r + fma(r * z, S, rl * w), c = w + fma(z2, C, fma(-r, rl, e));
  const double ss = s * s, cc = c * c;
  s2 = odd ? cc : ss;
  c2 = odd ? ss : cc;
}

// What a step's derivatives and the trace's sign test need of a state.
struct Stage {
  double rr, sin2, delta, aFactor, rPot, thetaPot;
};
__device__ __forceinline__ Stage stage_at(const St &s, double mass, double a, const Cs &c) {
  const double mGeom = kG * mass / kC2;
  const double r = s.r;
  const double rr = r * r;
  const double aa = a * a;
  double sin2, cos2;
  if (fabs(s.theta) < 1024.0) {
    sin2_cos2(s.theta, sin2, cos2);
  } else {
    double sinTheta, cosTheta;
    sincos(s.theta, &sinTheta, &cosTheta);
    sin2 = sinTheta * sinTheta;
    cos2 = cosTheta * cosTheta;
  }
  sin2 = mx(sin2, 1e-12);
  const double delta = rr - (2.0 * mGeom * r) + aa;
  const double aFactor = ((rr + aa) * c.e) - (a * c.lz);
  const double lzMinusAe = c.lz - (a * c.e);
  const double rPotRaw = (aFactor * aFactor) - (delta * (c.q + (lzMinusAe * lzMinusAe)));
  const double thetaPotRaw = c.q + (aa * c.e * c.e * cos2) - (c.lz * c.lz / sin2);
  return Stage{rr, sin2, delta, aFactor, rPotRaw, thetaPotRaw};
}

// kerrMinoDerivatives (kerr.cpp:40-66). The reference recomputes the full
// potentials (including the unused derivatives) and sin(theta) twice; the
// values that feed the result are identical here.
__device__ __forceinline__ Dv mino_derivs(const St &s, double mass, double a, const Cs &c) {
  const Stage w = stage_at(s, mass, a, c);
  const double aa = a * a;
  const double rPot = mx(w.rPot, 0.0);
  const double thetaPot = mx(w.thetaPot, 0.0);
  const double deltaSafe = mx(w.delta, 1e-12);
  Dv d;
  d.dr = s.signR * sqrt(rPot);
  d.dtheta = s.signTheta * sqrt(thetaPot);
  d.dphi = (c.lz / w.sin2) - (a * c.e) + (a * w.aFactor / deltaSafe);
  d.dt = (((w.rr + aa) * w.aFactor) / deltaSafe) + (a * (c.lz - (a * c.e * w.sin2)));
  return d;
}

// kerrStepMino with CUDA's operators: every input.
__device__ __noinline__ St step_mino_any(const St &state, double mass, double a, const Cs &c, double dlam) {
  St next = state;
  const Dv k1 = mino_derivs(state, mass, a, c);
  St s2 = state;
  s2.r += 0.5 * dlam * k1.dr;
  s2.theta += 0.5 * dlam * k1.dtheta;
  s2.phi += 0.5 * dlam * k1.dphi;
  s2.t += 0.5 * dlam * k1.dt;
  const Dv k2 = mino_derivs(s2, mass, a, c);
  St s3 = state;
  s3.r += 0.5 * dlam * k2.dr;
  s3.theta += 0.5 * dlam * k2.dtheta;
  s3.phi += 0.5 * dlam * k2.dphi;
  s3.t += 0.5 * dlam * k2.dt;
  const Dv k3 = mino_derivs(s3, mass, a, c);
  St s4 = state;
  s4.r += dlam * k3.dr;
  s4.theta += dlam * k3.dtheta;
  s4.phi += dlam * k3.dphi;
  s4.t += dlam * k3.dt;
  const Dv k4 = mino_derivs(s4, mass, a, c);
  next.r += dlam * (k1.dr + (2.0 * k2.dr) + (2.0 * k3.dr) + k4.dr) / 6.0;
  next.theta += dlam * (k1.dtheta + (2.0 * k2.dtheta) + (2.0 * k3.dtheta) + k4.dtheta) / 6.0;
  next.phi += dlam * (k1.dphi + (2.0 * k2.dphi) + (2.0 * k3.dphi) + k4.dphi) / 6.0;
  next.t += dlam * (k1.dt + (2.0 * k2.dt) + (2.0 * k3.dt) + k4.dt) / 6.0;
  const double lo = 1e-6, hi = kPI - 1e-6;
  next.theta = (next.theta < lo) ? lo : ((hi < next.theta) ? hi : next.theta);
  return next;
}

// ---- the same step with the branch-free quotients and roots (ieee_fp64.cuh) -------
//
// The same operations on the same values in the same order, so the same bits
// (both take sin^2 and cos^2 from sin2_cos2, for the sign test too):
//   * the quotients by sin^2 share one reciprocal, those by Delta another;
//   * products with 2 are exact, so fma(2, x, y) rounds as y + 2 x;
//   * the first stage's potentials are those the trace loop tests for sign
//     flips (kerr.cpp evaluates them twice).
// It is bound by one ray's chain of FP64 operations: 4096 rays of up to 1500
// steps take 4.53 ms with the operators, 1.56 ms without their branches and
// 1.45 ms with sin2_cos2 in place of sincos as well (one B200; 300,000 rays of
// 1000 steps: 14.3, 8.7 and 8.4 ms).
// Operands must stay far from the ends of the exponent range: consts_ok() once
// per ray, r and the stages' potentials per step; a step that fails is redone
// by step_mino_any.

__device__ __forceinline__ bool magnitude_in(double x, int lo, int hi) {  // 2^lo <= |x| < 2^hi
  const unsigned e = (unsigned)(__double2hiint(x) & 0x7fffffff) >> 20;
  return e - (unsigned)(1023 + lo) < (unsigned)(hi - lo);
}
__device__ __forceinline__ bool zero_or_in(double x, int lo, int hi) { return x == 0.0 || magnitude_in(x, lo, hi); }

struct Geo {
  double twoM, a, aa, e, lz, q, ae, kTh, lzae2, lz2, alz;  // per ray
};

__device__ __forceinline__ Geo geo_of(double mass, double a, const Cs &c) {
  Geo g;
  const double mGeom = kG * mass / kC2;
  g.twoM = 2.0 * mGeom;
  g.a = a;
  g.aa = a * a;
  g.e = c.e;
  g.lz = c.lz;
  g.q = c.q;
  g.ae = a * c.e;
  g.kTh = g.aa * c.e * c.e;
  const double d = c.lz - g.ae;
  g.lzae2 = c.q + (d * d);
  g.lz2 = c.lz * c.lz;
  g.alz = a * c.lz;
  return g;
}

__device__ __forceinline__ bool consts_ok(const Geo &g, double dlam) {
  return zero_or_in(g.twoM, -200, 200) && zero_or_in(g.a, -200, 200) && zero_or_in(g.e, -50, 50) &&
         zero_or_in(g.lz, -200, 200) && zero_or_in(g.q, -400, 400) && zero_or_in(dlam, -200, 66);
}

// max(x, 1e-12), by the bits.
__device__ __forceinline__ double at_least_tiny(double x) {
  return __double_as_longlong(x) < __double_as_longlong(1e-12) ? 1e-12 : x;
}

// What a stage needs at (r, theta), before the signs.
struct Raw {
  double R, Th, y2, yd, A, rr, sin2, delta, theta;
};

__device__ __forceinline__ Raw raw_at(double r, double theta, const Geo &g) {
  Raw w;
  double sin2, cos2;
  sin2_cos2(theta, sin2, cos2);
  w.theta = theta;
  w.rr = r * r;
  w.sin2 = at_least_tiny(sin2);
  const double delta = w.rr - (g.twoM * r) + g.aa;
  w.A = ((w.rr + g.aa) * g.e) - g.alz;
  w.R = (w.A * w.A) - (delta * g.lzae2);
  w.y2 = bhk::rcp_near(w.sin2);
  w.Th = g.q + (g.kTh * cos2) - bhk::div_by(g.lz2, w.sin2, w.y2);
  w.delta = at_least_tiny(delta);
  w.yd = bhk::rcp_near(w.delta);
  return w;
}

// |R| and |Theta| finite and below 2^860: no product of the stage overflowed.
// The angle within sin2_cos2's range.
__device__ __forceinline__ bool raw_ok(const Raw &w) {
  return (__double2hiint(w.R) & 0x7fffffff) < ((1023 + 860) << 20) &&
         (__double2hiint(w.Th) & 0x7fffffff) < ((1023 + 860) << 20) &&
         (__double2hiint(w.theta) & 0x7fffffff) < ((1023 + 10) << 20);
}

// sqrt(max(x, 0)).
__device__ __forceinline__ double root_of_positive(double x) {
  const double s = bhk::sqrt_rn(x);
  return __double2hiint(x) < 0 ? 0.0 : s;
}

template <bool TIME>
__device__ __forceinline__ Dv rates(const Raw &w, double signR, double signTheta, const Geo &g) {
  Dv d;
  d.dr = signR * root_of_positive(w.R);
  d.dtheta = signTheta * root_of_positive(w.Th);
  d.dphi = bhk::div_by(g.lz, w.sin2, w.y2) - g.ae + bhk::div_by(g.a * w.A, w.delta, w.yd);
  d.dt = TIME ? bhk::div_by((w.rr + g.aa) * w.A, w.delta, w.yd) + (g.a * (g.lz - (g.ae * w.sin2))) : 0.0;
  return d;
}

// One step from s (signs already flipped) whose potentials are w1; ok = false
// where the result is not to be used. TIME: the coordinate time as well.
template <bool TIME>
__device__ __forceinline__ St step_mino_fast(const St &s, const Raw &w1, const Geo &g, double dlam, bool &ok) {
  const double hh = 0.5 * dlam;
  const Dv k1 = rates<TIME>(w1, s.signR, s.signTheta, g);
  const Raw w2 = raw_at(s.r + hh * k1.dr, s.theta + hh * k1.dtheta, g);
  const Dv k2 = rates<TIME>(w2, s.signR, s.signTheta, g);
  const Raw w3 = raw_at(s.r + hh * k2.dr, s.theta + hh * k2.dtheta, g);
  const Dv k3 = rates<TIME>(w3, s.signR, s.signTheta, g);
  const Raw w4 = raw_at(s.r + dlam * k3.dr, s.theta + dlam * k3.dtheta, g);
  const Dv k4 = rates<TIME>(w4, s.signR, s.signTheta, g);
  ok = raw_ok(w1) && raw_ok(w2) && raw_ok(w3) && raw_ok(w4);
  St n = s;
#define BHK_SUM(f) bhk::div_6(dlam * (fma(2.0, k3.f, fma(2.0, k2.f, k1.f)) + k4.f))
  n.r += BHK_SUM(dr);
  n.theta += BHK_SUM(dtheta);
  n.phi += BHK_SUM(dphi);
  if (TIME) n.t += BHK_SUM(dt);
#undef BHK_SUM
  const double lo = 1e-6, hi = kPI - 1e-6;
  n.theta = (n.theta < lo) ? lo : ((hi < n.theta) ? hi : n.theta);
  return n;
}

__global__ void k_kerr_potentials(int64_t n, const double *__restrict__ r, const double *__restrict__ th,
                                  double mass, double a, BhkConstsSoA c, double *rp, double *drp, double *tp,
                                  double *dtp) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const Cs cs{c.e[i], c.lz[i], c.q[i]};
    const Pot p = potentials(r[i], th[i], mass, a, cs);
    if (rp) rp[i] = p.rPot;
    if (drp) drp[i] = p.dRdr;
    if (tp) tp[i] = p.thetaPot;
    if (dtp) dtp[i] = p.dThetadtheta;
  }
}

__global__ void k_kerr_step_mino(int64_t n, BhkStateSoA s, double mass, double a, BhkConstsSoA c,
                                 const double *__restrict__ dlam, double dlam_scalar) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const St st{s.r[i], s.theta[i], s.phi[i], s.t[i], s.sr[i], s.sth[i]};
    const Cs cs{c.e[i], c.lz[i], c.q[i]};
    const double h = dlam ? dlam[i] : dlam_scalar;
    const Geo g = geo_of(mass, a, cs);
    bool ok = consts_ok(g, h) && magnitude_in(st.r, -200, 200);
    St nx = st;
    if (ok) nx = step_mino_fast<true>(st, raw_at(st.r, st.theta, g), g, h, ok);
    if (!ok) nx = step_mino_any(st, mass, a, cs, h);
    s.r[i] = nx.r;
    s.theta[i] = nx.theta;
    s.phi[i] = nx.phi;
    s.t[i] = nx.t;
    s.sr[i] = nx.signR;
    s.sth[i] = nx.signTheta;
  }
}

// kerrRedshift (src/physics/kerr.h:361-378) for geometric mass m.
__device__ __forceinline__ double redshift_z(double r, double theta, double m, double a) {
  const double rS = 2.0 * m;
  const double cosTheta = cos(theta);
  const double sigma = (r * r) + (a * a * cosTheta * cosTheta);
  const double factor = 1.0 - ((rS * r) / sigma);
  if (factor <= 0.0) return __longlong_as_double(0x7ff0000000000000LL);
  return (1.0 / sqrt(factor)) - 1.0;
}

__global__ void k_kerr_trace_rays(int64_t n, BhkStateSoA init, BhkConstsSoA c, double mass, double a,
                                  double rH, double rEsc, double step, int32_t maxSteps, int32_t *status,
                                  int32_t *steps, double *dist, double *rf, double *thf, double *phf,
                                  double *red) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    St state{init.r[i], init.theta[i], init.phi[i], init.t[i], init.sr[i], init.sth[i]};
    const Cs cs{c.e[i], c.lz[i], c.q[i]};
    int32_t st = 0, taken = 0;
    double total = 0.0;
    const Geo g = geo_of(mass, a, cs);
    const bool fine = consts_ok(g, step);
    const double rStop = rH * 1.001;
    for (int32_t k = 0; k < maxSteps; ++k) {
      if (state.r <= rStop) { st = 2; break; }
      if (state.r >= rEsc) { st = 1; break; }
      bool ok = fine && magnitude_in(state.r, -200, 200);
      St next = state;
      if (ok) {
        const Raw w = raw_at(state.r, state.theta, g);
        if (w.R < 0.0) next.signR = -next.signR;
        if (w.Th < 0.0) next.signTheta = -next.signTheta;
        next = step_mino_fast<false>(next, w, g, step, ok);
      }
      if (!ok) {
        const Stage w = stage_at(state, mass, a, cs);
        next = state;
        if (w.rPot < 0.0) next.signR = -next.signR;
        if (w.thetaPot < 0.0) next.signTheta = -next.signTheta;
        next = step_mino_any(next, mass, a, cs, step);
      }
      state = next;
      total += step;
      ++taken;
    }
    if (st == 0) st = (taken >= maxSteps) ? 4 : 1;
    double rs = 1.0;
    if (state.r > (rH * 1.001)) rs = 1.0 + redshift_z(state.r, state.theta, kG * mass / kC2, a);
    if (status) status[i] = st;
    if (steps) steps[i] = taken;
    if (dist) dist[i] = total;
    if (rf) rf[i] = state.r;
    if (thf) thf[i] = state.theta;
    if (phf) phf[i] = state.phi;
    if (red) red[i] = rs;
  }
}

int grid_for(int64_t n, int block) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t want = (n + block - 1) / block;
  const int64_t cap = (int64_t)sms * 16;
  return (int)((want < cap) ? (want > 0 ? want : 1) : cap);
}

}  // namespace

extern "C" int bhk_kerr_potentials(int64_t n, const double *r, const double *theta, double mass, double a,
                                   BhkConstsSoA c, double *rp, double *drp, double *tp, double *dtp,
                                   void *stream) {
  if (n <= 0) return 0;
  k_kerr_potentials<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(n, r, theta, mass, a, c, rp, drp, tp, dtp);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int bhk_kerr_step_mino(int64_t n, BhkStateSoA s, double mass, double a, BhkConstsSoA c,
                                  const double *dlam, double dlam_scalar, void *stream) {
  if (n <= 0) return 0;
  k_kerr_step_mino<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(n, s, mass, a, c, dlam, dlam_scalar);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int bhk_kerr_trace_rays(int64_t n, BhkStateSoA init, BhkConstsSoA c, double mass, double a,
                                   double r_horizon, double r_escape, double step, int32_t max_steps,
                                   int32_t *status, int32_t *steps, double *dist, double *rf, double *thf,
                                   double *phf, double *redshift, void *stream) {
  if (n <= 0) return 0;
  k_kerr_trace_rays<<<grid_for(n, 128), 128, 0, (cudaStream_t)stream>>>(
      n, init, c, mass, a, r_horizon, r_escape, step, max_steps, status, steps, dist, rf, thf, phf, redshift);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
