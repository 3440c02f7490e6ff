// trace_image_fp64.cu - FP64 image-plane Kerr tracer (sm_100a).
//
// One ray per lane in a persistent grid: each warp keeps 32 rays in
// registers; lanes whose rays cross the equator or terminate (horizon, disk,
// escape, step budget) are held until the warp serves them together
// (frame_source.cuh), and take new rays from a global work counter with one
// warp-aggregated atomicAdd (ballot + popc). The integration
// follows the reference trace loop order (src/physics/raytracer.h:338-365): step budget, horizon test, escape
// test, step; then the equatorial-crossing test, located inside the step by
// Hermite interpolation (hermite.cuh) on the bracket of the
// src/physics/event_detection.h:127-180 pattern.
//
// Built with -fmad=false: bit-identical to the FP64 CPU oracle.
#include <cuda_runtime.h>

#include <cstdio>

#include "frame_source.cuh"
#include "rt.cuh"
#include "sky.cuh"
#include "hermite.cuh"
#include "image_fp64.cuh"
#include "launch.h"

namespace bhk {

constexpr unsigned kFull = 0xffffffffu;

struct RayFp64 {
  RayC c;
  Yd y;
  Yd k1;        // rhs(y); DP45: its FSAL stage
  double h;     // next step; DP45: next trial step
  double inten;
  long long pix;
  int f;  // frame of the current ray (batch launches)
  int steps;
  int attempts;
  int ncross;
  double drift;  // largest Carter-constant residual the projection removed
};

// RK4's step at y, DP45's first trial step.
__device__ __forceinline__ double mino_step(const BhkImageParams &p, const Yd &y) {
  const double hh = p.step_coeff * dmin_(y.r, p.step_rcap);
  const double sigma = (y.r * y.r) + ((p.a2 * y.u) * y.u);
  return div_rn(hh, sigma);
}

__device__ __forceinline__ void init_ray(const BhkImageParams &p, long long pix, RayFp64 &R) {
  const long long i = pix % p.width, j = pix / p.width;
  const double alpha = p.alpha_min + ((double)i + 0.5) * p.dalpha;
  const double beta = p.beta_min + ((double)j + 0.5) * p.dbeta;
  R.c.a = p.a;
  R.c.a2 = p.a2;
  R.c.lam = -alpha * p.sin_o;
  const double eta = (beta * beta) + (((alpha * alpha) - (p.a * p.a)) * p.cos_o) * p.cos_o;
  R.c.qTh = eta + (R.c.lam * R.c.lam);
  const double qR = (p.form == 1) ? eta : R.c.qTh;
  R.c.K = qR + ((R.c.lam - R.c.a) * (R.c.lam - R.c.a));
  R.y.r = p.r_obs;
  R.y.u = p.cos_o;
  R.y.phi = 0.0;
  const double Rv = pot_R(R.y.r, R.c);
  R.y.pr = 0.0 - sqrt((Rv < 0.0) ? 0.0 : Rv);  // no -0, which is_neg takes for negative
  R.y.pu = beta * p.sin_o + 0.0;
  R.steps = 0;
  R.attempts = 0;
  R.ncross = 0;
  R.inten = 0.0;
  R.pix = pix;
  project(R.y, R.c);  // idempotent from here on (see iterate)
  R.drift = 0.0;
  R.h = mino_step(p, R.y);
  R.k1 = rhs(R.y, R.c);
}

// The step in which a lane's ray crosses u = 0, y0 -> y1 (y1 before the
// projection) with k0 = rhs(y0), k1 = rhs(y1), kept in shared memory until
// the warp locates its held lanes' crossings together (trace_loop).
struct HeldSteps {
  double v[17][128];
};

__device__ __forceinline__ void hold_step(HeldSteps &hs, const Yd &y0, const Yd &k0, const Yd &y1, const Yd &k1,
                                          double h) {
  const int t = threadIdx.x;
  hs.v[0][t] = y0.r, hs.v[1][t] = y0.u, hs.v[2][t] = y0.phi, hs.v[3][t] = y0.pr, hs.v[4][t] = y0.pu;
  hs.v[5][t] = k0.pr, hs.v[6][t] = k0.pu, hs.v[7][t] = k0.phi;
  hs.v[8][t] = y1.r, hs.v[9][t] = y1.u, hs.v[10][t] = y1.phi, hs.v[11][t] = y1.pr, hs.v[12][t] = y1.pu;
  hs.v[13][t] = k1.pr, hs.v[14][t] = k1.pu, hs.v[15][t] = k1.phi;
  hs.v[16][t] = h;
}

__device__ __forceinline__ void held_crossing(const HeldSteps &hs, double &r_c, double &phi_c) {
  const int t = threadIdx.x;
  const bhh_dev::Ends e{hs.v[0][t], hs.v[1][t], hs.v[2][t],  hs.v[3][t],  hs.v[4][t],  hs.v[5][t],
                        hs.v[6][t], hs.v[7][t], hs.v[8][t],  hs.v[9][t],  hs.v[10][t], hs.v[11][t],
                        hs.v[12][t], hs.v[13][t], hs.v[14][t], hs.v[15][t]};
  bhh_dev::hermite_crossing(e, hs.v[16][t], r_c, phi_c);
}

// Records a crossing at (r_c, phi_c) when it lies on the disk; returns true
// when the ray stops there (last allowed crossing).
__device__ __forceinline__ bool on_crossing(const BhkImageParams &p, const BhkImageOut &o, RayFp64 &R,
                                            double r_c, double phi_c) {
  if (!(r_c >= p.r_in && r_c <= p.r_out)) return false;
  const int k = R.ncross;
  const long long off = (long long)k * p.n_pix + R.pix;
  const double g = disk_g(r_c, p.a, R.c.lam);
  if (o.r_hit) o.r_hit[off] = r_c;
  if (o.phi_hit) o.phi_hit[off] = phi_of_psi(phi_c, r_c, p);
  if (o.g) o.g[off] = g;
  const double q = p.r_in / r_c;
  const double g2 = g * g;
  R.inten = R.inten + ((((g2 * g2) * q) * q) * q);
  if (k == 0 && o.flux) o.flux[R.pix] = nt_flux(r_c, p.nt_isco, p.nt_flux_peak);
  R.ncross = k + 1;
  return R.ncross >= p.max_cross;
}

__device__ __forceinline__ void finish(const BhkImageParams &p, const BhkImageOut &o, const RayFp64 &R,
                                       int cls) {
  const long long pix = R.pix;
  if (o.cls) o.cls[pix] = cls;
  if (o.steps) o.steps[pix] = R.steps;
  if (o.n_cross) o.n_cross[pix] = R.ncross;
  if (R.ncross == 0 && o.flux) o.flux[pix] = 0.0;
  for (int k = R.ncross; k < p.max_cross; ++k) {
    const long long off = (long long)k * p.n_pix + pix;
    if (o.r_hit) o.r_hit[off] = 0.0;
    if (o.phi_hit) o.phi_hit[off] = 0.0;
    if (o.g) o.g[off] = 0.0;
  }
  double th = 0.0, ph = 0.0, inten = R.inten;
  if (cls == 2) {
    const double u = R.y.u;
    th = acos((u < -1.0) ? -1.0 : ((1.0 < u) ? 1.0 : u));
    ph = phi_of_psi(R.y.phi, R.y.r, p);
    if (p.sky) {  // dphi/dtau = dpsi/dtau + a p_r / Delta  (phi = psi + a G(r), G' = 1 / Delta)
      const Yd k = rhs(R.y, R.c);
      const double delta = ((R.y.r * R.y.r) - (2.0 * R.y.r)) + p.a2;
      const double dphi = k.phi + (p.a * R.y.pr) / delta;
      inten = inten + bhsky::radiance(p.sky, p.sky_size, R.y.r, u, ph, R.y.pr, R.y.pu, dphi);
    }
  }
  if (o.intensity) o.intensity[pix] = inten;
  if (o.theta_inf) o.theta_inf[pix] = th;
  if (o.phi_inf) o.phi_inf[pix] = ph;
  if (o.carter_drift) o.carter_drift[pix] = R.drift;
}

// One iteration of the trace loop for an active ray; returns the class when
// the ray terminates, kCross when the step crosses the equator (the step is
// held in hs), kRun otherwise.
// DRIFT: keep the largest Carter-constant residual the projection removes (a
// separate instantiation, so the plain kernels carry none of it).
template <int INTEG, bool DRIFT = false>
__device__ __forceinline__ int iterate(const BhkImageParams &p, HeldSteps &hs, RayFp64 &R) {
  if (INTEG == 0) {
    if (R.steps >= p.max_steps) return 3;
    if (R.y.r <= p.r_hor) return 0;
    if (R.y.r >= p.r_esc) return 2;
    Yd yn = rk4(R.y, R.h, R.c, R.k1);
    ++R.steps;
    const bool cross = (R.y.u * yn.u) < 0.0;
    if (cross) hold_step(hs, R.y, R.k1, yn, rhs(yn, R.c), R.h);
    if (DRIFT)
      R.drift = dmax_(R.drift, project(yn, R.c, true));
    else
      project(yn, R.c);
    R.y = yn;
    R.h = mino_step(p, yn);  // beside the projection's roots, which the step and the accelerations do not need
    R.k1 = rhs(yn, R.c);
    return cross ? bhsrc::kCross : bhsrc::kRun;
  } else {
    const long long max_attempts = 4LL * p.max_steps + 64;
    if (R.steps >= p.max_steps || R.attempts >= max_attempts) return 3;
    if (R.y.r <= p.r_hor) return 0;
    if (R.y.r >= p.r_esc) return 2;
    ++R.attempts;
    const DPRes d = dp45(R.y, R.h, R.c, R.k1, p.rtol, p.atol, true);
    // Accepted and rejected lanes run the same instructions: a rejected lane
    // keeps its state and re-projects it, which is exact no-op because every
    // state is already on its first integrals (projected at set-up).
    const bool acc = d.err <= 1.0;
    const bool cross = acc && (R.y.u * d.y5.u) < 0.0;
    if (acc) ++R.steps;
    if (cross) hold_step(hs, R.y, R.k1, d.y5, d.k7, R.h);
    R.y = acc ? d.y5 : R.y;
    R.k1 = acc ? d.k7 : R.k1;
    const double drift = project(R.y, R.c, DRIFT);
    if (DRIFT && acc) R.drift = dmax_(R.drift, drift);
    R.k1.r = R.y.pr;  // projection moves only the momenta
    R.k1.u = R.y.pu;
    R.h = R.h * step_factor(d.err, acc);
    return cross ? bhsrc::kCross : bhsrc::kRun;
  }
}

// The persistent loop shared by the single-frame and batch kernels. A lane
// whose ray crosses the equator or ends is held (see kHold) until the warp
// serves its held lanes together: crossings are located, outputs of ended
// rays written, and new work items taken with one warp-aggregated atomicAdd
// on the counter (ballot + popc).
template <int INTEG, bool DRIFT = false, class Src>
__device__ __forceinline__ void trace_loop(const Src &src, unsigned long long *__restrict__ counter, int refill) {
  __shared__ HeldSteps hs;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lanemask_lt = (1u << lane) - 1u;
  const unsigned long long total = (unsigned long long)src.total();
  RayFp64 R;
  int st = bhsrc::kEmpty;
  bool exhausted = false;
  int waited = bhsrc::kHold;  // the first pass fills every lane
  const int turns = refill * (INTEG == 0 ? bhsrc::kTurnsRk4 : bhsrc::kTurnsDp45);
  for (;;) {
    const unsigned running = __ballot_sync(kFull, st == bhsrc::kRun);
    const unsigned held = __ballot_sync(kFull, st != bhsrc::kRun && !(st == bhsrc::kEmpty && exhausted));
    if (held) {
      waited += __popc(held) * turns;
      if (waited >= bhsrc::kHold || !running) {
        waited = 0;
        if (st == bhsrc::kCross) {
          double r_c, phi_c;
          held_crossing(hs, r_c, phi_c);
          st = on_crossing(src.params(R.f), src.out(R.f), R, r_c, phi_c) ? 1 : bhsrc::kRun;
        }
        if (st >= 0) {
          finish(src.params(R.f), src.out(R.f), R, st);
          src.pixel_done(R.f);
          st = bhsrc::kEmpty;
        }
        const unsigned need = __ballot_sync(kFull, st == bhsrc::kEmpty && !exhausted);
        if (need) {
          const int leader = __ffs(need) - 1;
          unsigned long long base = 0;
          if ((int)lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(need));
          base = __shfl_sync(kFull, base, leader);
          if (st == bhsrc::kEmpty && !exhausted) {
            const unsigned long long mine = base + (unsigned long long)__popc(need & lanemask_lt);
            if (mine < total) {
              long long pix;
              const int f = src.frame_of((long long)mine, pix);
              init_ray(src.params(f), pix, R);
              R.f = f;
              st = bhsrc::kRun;
            } else {
              exhausted = true;
            }
          }
        }
      }
    } else if (!running) {
      break;
    }
    for (int k = 0; k < turns; ++k)
      if (st == bhsrc::kRun) st = iterate<INTEG, DRIFT>(src.params(R.f), hs, R);
  }
}

template <int INTEG, bool DRIFT>
__global__ void __launch_bounds__(128, 4) k_trace_image_fp64(const __grid_constant__ BhkImageParams p,
                                                          const __grid_constant__ BhkImageOut o,
                                                          unsigned long long *__restrict__ counter, int refill) {
  trace_loop<INTEG, DRIFT>(bhsrc::SingleSrc<INTEG == 0>{p, o}, counter, refill);
}

template <int INTEG, bool DRIFT>
__global__ void __launch_bounds__(128, 4) k_trace_list_fp64(const __grid_constant__ BhkImageParams p,
                                                         const __grid_constant__ BhkImageOut o,
                                                         const int *__restrict__ list,
                                                         const unsigned int *__restrict__ count,
                                                         unsigned long long *__restrict__ counter, int refill) {
  trace_loop<INTEG, DRIFT>(bhsrc::ListSrc{p, o, list, count}, counter, refill);
}

template <int INTEG, bool DRIFT>
__global__ void __launch_bounds__(128, 4) k_trace_batch_fp64(const __grid_constant__ BhkBatchDev b,
                                                          unsigned long long *__restrict__ counter, int refill) {
  if (threadIdx.x == 0) atomicMin(b.start_ns, bhsrc::globaltimer_ns());
  trace_loop<INTEG, DRIFT>(bhsrc::BatchSrc{b}, counter, refill);
}

// ---- along-ray radiative transfer -------------------------------------------

// The samples of one accepted step y0 -> y1 (derivatives k0, k1 at its ends,
// length h in Mino time): at most ds_max apart in affine length. 0 where the
// step stays beyond r_max: on t in [0, 1] the cubic Hermite r(t) >= min(r0,
// r1) - (4/27) |h| (|r0'| + |r1'|).
__device__ __forceinline__ int rt_count(const BhkImageParams &p, const BhkRtParams &q, const Yd &y0, const Yd &k0,
                                        const Yd &y1, const Yd &k1, double h) {
  const double rm = 0.5 * (y0.r + y1.r) + 0.125 * h * (k0.r - k1.r);
  const double um = 0.5 * (y0.u + y1.u) + 0.125 * h * (k0.u - k1.u);
  const double sig_m = rm * rm + p.a2 * um * um;
  const double rlow = (y0.r < y1.r ? y0.r : y1.r) - (4.0 / 27.0) * fabs(h) * (fabs(k0.r) + fabs(k1.r));
  if (rlow > q.r_max) return 0;
  double ns = ceil(div_rn(sig_m * h, q.ds_max));
  ns = ns < 1.0 ? 1.0 : (ns > 64.0 ? 64.0 : ns);
  return ns > 0.0 ? (int)ns : 0;  // no number: none, as an integer it would be INT_MIN in the warp's sum
}

using RtWarp = bhrt::WarpSamples<double>;

// Leaves a step for the warp's samples.
__device__ __forceinline__ void rt_hold(RtWarp &w, const Yd &y0, const Yd &k0, const Yd &y1, const Yd &k1, double h,
                                        int nsub, double lam) {
  const int l = threadIdx.x & 31;
  w.step[0][l] = y0.r, w.step[1][l] = k0.r, w.step[2][l] = y1.r, w.step[3][l] = k1.r;
  w.step[4][l] = y0.u, w.step[5][l] = k0.u, w.step[6][l] = y1.u, w.step[7][l] = k1.u;
  w.step[8][l] = y0.phi, w.step[9][l] = k0.phi, w.step[10][l] = y1.phi, w.step[11][l] = k1.phi;
  w.step[12][l] = h, w.step[13][l] = (double)nsub, w.step[14][l] = lam;
}

// Sample m of lane l's step, its position by cubic Hermite interpolation in
// Mino time: the source term over the segment, the fraction absorbed and the
// optical depth (all zero outside the medium).
__device__ __forceinline__ void rt_sample(const BhkImageParams &p, const BhkRtParams &q, RtWarp &w, int l, int m,
                                          int slot) {
  const double h = w.step[12][l], ns = w.step[13][l];
  const double dt = div_rn(h, ns);
  const double t = div_rn((double)m + 0.5, ns);
  const double t2 = t * t, t3 = t2 * t;
  const double h00 = 2.0 * t3 - 3.0 * t2 + 1.0, h10 = t3 - 2.0 * t2 + t;
  const double h01 = -2.0 * t3 + 3.0 * t2, h11 = t3 - t2;
  const double r = h00 * w.step[0][l] + h10 * h * w.step[1][l] + h01 * w.step[2][l] + h11 * h * w.step[3][l];
  const double u = h00 * w.step[4][l] + h10 * h * w.step[5][l] + h01 * w.step[6][l] + h11 * h * w.step[7][l];
  const double psi = h00 * w.step[8][l] + h10 * h * w.step[9][l] + h01 * w.step[10][l] + h11 * h * w.step[11][l];
  const double dl = (r * r + p.a2 * u * u) * dt;  // affine length of the sample, M
  double src = 0.0, om = 0.0, ts = 0.0, n, th, b;
  if (bhrt::sample(q, r, u, psi, p, n, th, b)) {
    const double g = bhrt::redshift(p.a, r, u, w.step[14][l]);
    if (g > 0.0) {
      double j, al;
      bhrt::synchrotron(q, n, th, b, div_rn(q.nu, g), j, al);
      const double jo = g * g * j, ao = al < INFINITY ? div_rn(al, g) : al;  // div_rn wants finite operands
      const double ds = dl * q.length_cm;
      ts = ao * ds;
      om = (ts < 1.0e-4) ? ts * (1.0 - 0.5 * ts) : -expm1(-ts);
      src = (ao > 0.0) ? (jo / ao) * om : jo * ds;
    }
  }
  w.res[0][slot] = src;
  w.res[1][slot] = om;
  w.res[2][slot] = ts;
}

// A warp traces up to `slots` rays at a time and samples the medium for all
// of them together (bhrt::warp_samples). With fewer rays than the resident
// lanes, slots < 32 spreads them over more warps: the steps cost the same per
// warp, and a warp's samples fill its lanes either way.
__global__ void __launch_bounds__(128, 3) k_trace_rt_fp64(const __grid_constant__ BhkImageParams p,
                                                          const __grid_constant__ BhkRtParams q,
                                                          double *__restrict__ i_nu, double *__restrict__ tau_out,
                                                          int *__restrict__ cls_out, int *__restrict__ steps_out,
                                                          unsigned long long *__restrict__ counter, int slots) {
  __shared__ RtWarp warps[4];
  RtWarp &w = warps[threadIdx.x >> 5];
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lanemask_lt = (1u << lane) - 1u;
  const long long max_attempts = 4LL * p.max_steps + 64;
  RayFp64 R;
  double I = 0.0, T = 1.0, tau = 0.0;
  int st = bhsrc::kEmpty;
  bool exhausted = (int)lane >= slots;
  int waited = bhsrc::kHold;
  for (;;) {
    const unsigned running = __ballot_sync(kFull, st == bhsrc::kRun);
    const unsigned held = __ballot_sync(kFull, st != bhsrc::kRun && !(st == bhsrc::kEmpty && exhausted));
    if (held) {
      waited += __popc(held);
      if (waited >= bhsrc::kHold || !running) {
        waited = 0;
        if (st >= 0) {
          if (i_nu) i_nu[R.pix] = I;
          if (tau_out) tau_out[R.pix] = tau;
          if (cls_out) cls_out[R.pix] = st;
          if (steps_out) steps_out[R.pix] = R.steps;
          st = bhsrc::kEmpty;
        }
        const unsigned need = __ballot_sync(kFull, st == bhsrc::kEmpty && !exhausted);
        if (need) {
          const int leader = __ffs(need) - 1;
          unsigned long long base = 0;
          if ((int)lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(need));
          base = __shfl_sync(kFull, base, leader);
          if (st == bhsrc::kEmpty && !exhausted) {
            const long long mine = (long long)(base + (unsigned long long)__popc(need & lanemask_lt));
            if (mine < p.n_pix) {
              init_ray(p, bhsrc::tile_pixel(mine, p.width, p.n_pix), R);
              I = 0.0, T = 1.0, tau = 0.0;
              st = bhsrc::kRun;
            } else {
              exhausted = true;
            }
          }
        }
      }
    } else if (!running) {
      break;
    }
    int nsub = 0;
    bool acc = false;
    if (st == bhsrc::kRun) {
      if (R.steps >= p.max_steps || R.attempts >= max_attempts) {
        st = 3;
      } else if (R.y.r <= p.r_hor) {
        st = 0;
      } else if (R.y.r >= p.r_esc) {
        st = 2;
      } else {
        ++R.attempts;
        const DPRes d = dp45(R.y, R.h, R.c, R.k1, p.rtol, p.atol, true);
        acc = d.err <= 1.0;
        if (acc) {
          ++R.steps;
          nsub = rt_count(p, q, R.y, R.k1, d.y5, d.k7, R.h);
          if (nsub) rt_hold(w, R.y, R.k1, d.y5, d.k7, R.h, nsub, R.c.lam);
          R.y = d.y5;
          R.k1 = d.k7;
          project(R.y, R.c);
          R.k1.r = R.y.pr;
          R.k1.u = R.y.pu;
        }
        R.h = R.h * step_factor(d.err, acc);
      }
    }
    bhrt::warp_samples(
        w, nsub, [&](int l, int m, int slot) { rt_sample(p, q, w, l, m, slot); },
        [&](int slot) {
          I = I + T * w.res[0][slot];
          T = T * (1.0 - w.res[1][slot]);
          tau = tau + w.res[2][slot];
        });
    if (acc && T < q.min_transmit) st = 4;
  }
}

}  // namespace bhk

namespace {
thread_local char g_err[256] = {0};
int set_err(cudaError_t e, const char *what) {
  snprintf(g_err, sizeof(g_err), "%s: %s", what, cudaGetErrorString(e));
  return -1;
}
}  // namespace

extern "C" const char *bhk_last_error(void) { return g_err; }

extern "C" int bhk_trace_image_fp64(const BhkImageParams *p, const BhkImageOut *o, unsigned long long *counter,
                                    BhkLaunch launch, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return set_err(e, "work-counter reset");
  const bool drift = o->carter_drift != nullptr;
  auto k = p->integrator == 0 ? (drift ? bhk::k_trace_image_fp64<0, true> : bhk::k_trace_image_fp64<0, false>)
                              : (drift ? bhk::k_trace_image_fp64<1, true> : bhk::k_trace_image_fp64<1, false>);
  k<<<launch.grid, launch.block, 0, s>>>(*p, *o, counter, launch.refill);
  e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(e, "k_trace_image_fp64 launch");
  return 0;
}

extern "C" int bhk_trace_list_fp64(const BhkImageParams *p, const BhkImageOut *o, const int *list,
                                   const unsigned int *count, unsigned long long *counter, BhkLaunch L,
                                   void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return set_err(e, "work-counter reset");
  const bool drift = o->carter_drift != nullptr;
  auto k = p->integrator == 0 ? (drift ? bhk::k_trace_list_fp64<0, true> : bhk::k_trace_list_fp64<0, false>)
                              : (drift ? bhk::k_trace_list_fp64<1, true> : bhk::k_trace_list_fp64<1, false>);
  k<<<L.grid, L.block, 0, s>>>(*p, *o, list, count, counter, L.refill);
  e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(e, "k_trace_list_fp64 launch");
  return 0;
}

extern "C" int bhk_trace_image_fp64_occupancy(int integrator, int block, int *blocks_per_sm) {
  cudaError_t e = (integrator == 0)
                      ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, bhk::k_trace_image_fp64<0, false>,
                                                                      block, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, bhk::k_trace_image_fp64<1, false>,
                                                                      block, 0);
  if (e != cudaSuccess) return set_err(e, "occupancy query");
  return 0;
}

extern "C" int bhk_trace_batch_fp64(const BhkBatchDev *b, int integrator, unsigned long long *counter, BhkLaunch L,
                                    void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return set_err(e, "work-counter reset");
  auto k = integrator == 0 ? (b->drift ? bhk::k_trace_batch_fp64<0, true> : bhk::k_trace_batch_fp64<0, false>)
                           : (b->drift ? bhk::k_trace_batch_fp64<1, true> : bhk::k_trace_batch_fp64<1, false>);
  k<<<L.grid, L.block, 0, s>>>(*b, counter, L.refill);
  e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(e, "k_trace_batch_fp64 launch");
  return 0;
}

extern "C" int bhk_trace_batch_fp64_occupancy(int integrator, int block, int *blocks_per_sm) {
  cudaError_t e = (integrator == 0)
                      ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, bhk::k_trace_batch_fp64<0, false>,
                                                                      block, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, bhk::k_trace_batch_fp64<1, false>,
                                                                      block, 0);
  if (e != cudaSuccess) return set_err(e, "occupancy query");
  return 0;
}

extern "C" int bhk_trace_rt_fp64(const BhkImageParams *p, const BhkRtParams *q, double *i_nu, double *tau,
                                 int32_t *cls, int32_t *steps, unsigned long long *counter, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return set_err(e, "work-counter reset");
  int dev = 0, sms = 0, per_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bhk::k_trace_rt_fp64, 128, 0)) != cudaSuccess)
    return set_err(e, "k_trace_rt_fp64 occupancy");
  const bhrt::Slots L = bhrt::slots_for(p->n_pix, (long long)sms * per_sm);
  bhk::k_trace_rt_fp64<<<L.grid, 128, 0, s>>>(*p, *q, i_nu, tau, cls, steps, counter, L.slots);
  e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(e, "k_trace_rt_fp64 launch");
  return 0;
}

namespace bhk {

// Paths of image-plane rays (the Blender bridge's geodesic export): one
// thread per ray, classical RK4 with the image tracer's affine step rule,
// the position written before the first step and after every step until the
// ray reaches the horizon or escape radius or max_points are written.
__global__ void __launch_bounds__(128) k_trace_paths_fp64(const __grid_constant__ BhkImageParams p,
                                                          float *__restrict__ xyz, int32_t *__restrict__ counts,
                                                          int max_points) {
  const long long pix = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (pix >= p.n_pix) return;
  RayFp64 R;
  init_ray(p, pix, R);
  float *out = xyz + pix * (long long)max_points * 3;
  int n = 0;
  for (;;) {
    const double s = sqrt(dmax_(0.0, (1.0 - R.y.u) * (1.0 + R.y.u)));
    const double ph = phi_of_psi(R.y.phi, R.y.r, p);
    out[3 * n + 0] = (float)(R.y.r * s * cos(ph));
    out[3 * n + 1] = (float)(R.y.r * s * sin(ph));
    out[3 * n + 2] = (float)(R.y.r * R.y.u);
    ++n;
    if (n >= max_points || R.y.r <= p.r_hor || R.y.r >= p.r_esc) break;
    const double hh = p.step_coeff * dmin_(R.y.r, p.step_rcap);
    const double h = div_rn(hh, (R.y.r * R.y.r) + ((p.a2 * R.y.u) * R.y.u));
    R.y = rk4(R.y, h, R.c, rhs(R.y, R.c));
    project(R.y, R.c);
  }
  counts[pix] = n;
}

}  // namespace bhk

extern "C" int bhk_trace_paths_fp64(const BhkImageParams *p, float *xyz, int32_t *counts, int max_points,
                                    void *stream) {
  if (p->n_pix <= 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long blocks = (p->n_pix + 127) / 128;
  bhk::k_trace_paths_fp64<<<(unsigned)blocks, 128, 0, s>>>(*p, xyz, counts, max_points);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_err(e, "k_trace_paths_fp64 launch");
  return 0;
}
