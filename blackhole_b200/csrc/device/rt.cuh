// rt.cuh - the medium and the emission of the along-ray radiative transfer
// (FP64, device): grid sampling, the emitter's redshift, thermal synchrotron
// emission and absorption, and one front-to-back segment of the formal
// solution.
//
// Physics restated from the reference: synchrotronThermalEmissivity /
// synchrotronThermalAbsorption (src/physics/rte_integrator.h:291-356:
// Mahadevan 1996 with K_2(1/Theta) ~ 2 Theta^2, the branch the reference
// builds without Boost), planckFunction (:221-230), grTransformEmission /
// Absorption (:480-512: j g^2, alpha / g), rteStep (:138-187: exact for
// constant coefficients, (1 - e^-tau) ~ tau (1 - tau/2) below tau = 1e-4),
// here in front-to-back form (I += T S (1 - e^-tau), T *= e^-tau), the
// reference GPU kernel's order (src/cuda/device_physics.cuh:1988-2173).
#pragma once

#include "azimuth_cell.h"
#include "ieee_fp64.cuh"
#include "launch.h"

namespace bhrt {

// ---- one warp's samples of the medium --------------------------------------------
//
// An accepted step has 0 to 64 samples, few steps have many, and a sample costs
// more than the step. Looped over by the step's own lane they ran at 19 of 32
// lanes (FP64, 160^2 rays) while the warp waited for the lane with the most.
// Here the warp takes the samples of all its lanes' steps together, 32 at a
// time, whichever lanes they belong to: the owner leaves its step in shared
// memory, any lane evaluates the sample, and the owner adds up its own results
// in their order along the ray (the sums round as before). With the cheaper
// sample (divisions by constants as products, no 64-bit remainder) the FP64
// transfer of 160^2 rays went from 8.2 to 2.5 ms, of 32^2 rays from 5.8 to 1.1.
template <class T>
struct WarpSamples {
  T step[15][32];  // the owners' steps
  T res[3][32];    // results of the 32 samples in hand
  int incl[32];    // inclusive sum of the lanes' sample counts
};

// Calls eval(owner lane, m, slot) for every sample of the warp and add(slot) on
// the owner, in order, for each of its nsub samples. Whole warps only.
template <class W, class Eval, class Add>
__device__ __forceinline__ void warp_samples(W &w, int nsub, Eval eval, Add add) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int incl = nsub;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(kAll, incl, o);
    if (lane >= o) incl += up;
  }
  const int total = __shfl_sync(kAll, incl, 31);
  if (total == 0) return;
  w.incl[lane] = incl;
  __syncwarp();
  for (int base = 0; base < total; base += 32) {
    const int s = base + lane;
    if (s < total) {
      int lo = 0;  // the first lane whose inclusive sum exceeds s
#pragma unroll
      for (int half = 16; half; half >>= 1)
        if (w.incl[lo + half - 1] <= s) lo += half;
      eval(lo, s - (lo ? w.incl[lo - 1] : 0), lane);
    }
    __syncwarp();
    for (int i = max(incl - nsub, base); i < min(incl, base + 32); ++i) add(i - base);
    __syncwarp();
  }
}

// Rays a warp traces at a time and CTAs of 4 warps of a transfer of n rays:
// all resident warps get rays, each as few as that leaves, but not under
// kMinSlots (16^2 rays, mixed: 0.39 ms at 4, 0.45 ms at 8; from 64^2 on equal).
constexpr int kMinSlots = 4;
struct Slots {
  int slots, grid;
};
inline Slots slots_for(long long n, long long resident_ctas) {
  const long long warps = 4 * (resident_ctas > 0 ? resident_ctas : 1);
  long long s = (n + warps - 1) / warps;
  s = s < kMinSlots ? kMinSlots : (s > 32 ? 32 : s);
  const long long need = (n + 4 * s - 1) / (4 * s);
  const long long grid = need < resident_ctas ? need : resident_ctas;
  return Slots{(int)s, (int)(grid > 0 ? grid : 1)};
}

constexpr double kE = 4.80320425e-10;     // esu
constexpr double kMe = 9.1093837015e-28;  // g
constexpr double kC = 2.99792458e10;      // cm / s
constexpr double kKb = 1.380649e-16;      // erg / K
constexpr double kH = 6.62607015e-27;     // erg s (2 pi hbar)
constexpr double kTwoPi = 6.283185307179586;

// Trilinear (n_e, Theta_e, |B|) at (r, theta, phi), phi = psi + a (G(r) - G(r_obs))
// (image_fp64.cuh); false outside [r_min, r_max].
__device__ __forceinline__ bool sample(const BhkRtParams &q, double r, double u, double psi, const BhkImageParams &p,
                                       double &n, double &th, double &b) {
  if (!(r >= q.r_min && r <= q.r_max)) return false;
  double phi = psi;
  if (p.a != 0.0) {
    const double c = bhk::div_rn((r - p.r_plus) * (p.r_obs - p.r_minus), (r - p.r_minus) * (p.r_obs - p.r_plus));
    phi = psi + bhk::div_rn(p.a * log(c), p.r_plus - p.r_minus);
  }
  const double fr = log(bhk::div_rn(r, q.r_min)) * q.fr_scale;
  int i0 = (int)floor(fr);
  i0 = i0 < 0 ? 0 : (i0 > q.n_r - 2 ? q.n_r - 2 : i0);
  double tr = fr - (double)i0;
  tr = tr < 0.0 ? 0.0 : (tr > 1.0 ? 1.0 : tr);
  const double theta = acos(u < -1.0 ? -1.0 : (u > 1.0 ? 1.0 : u));
  const double ft = (theta * (1.0 / 3.141592653589793)) * (double)q.n_th - 0.5;
  int j0 = (int)floor(ft);
  j0 = j0 < 0 ? 0 : (j0 > q.n_th - 2 ? q.n_th - 2 : j0);
  double tt = ft - (double)j0;
  tt = tt < 0.0 ? 0.0 : (tt > 1.0 ? 1.0 : tt);
  const double fp = (phi * (1.0 / kTwoPi)) * (double)q.n_ph;
  const double fl = floor(fp);
  const double tp = fp - fl;
  const int k0 = azimuth_cell(fl, q.n_ph, q.inv_n_ph);
  const int k1 = k0 + 1 == q.n_ph ? 0 : k0 + 1;
  const float4 *c = reinterpret_cast<const float4 *>(q.cells);
  double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int di = 0; di < 2; ++di)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj)
#pragma unroll
      for (int dk = 0; dk < 2; ++dk) {
        const double w = (di ? tr : 1.0 - tr) * (dj ? tt : 1.0 - tt) * (dk ? tp : 1.0 - tp);
        const long long idx = ((long long)(i0 + di) * q.n_th + (j0 + dj)) * q.n_ph + (dk ? k1 : k0);
        const float4 v = __ldg(c + idx);
        acc[0] = acc[0] + w * (double)v.x;
        acc[1] = acc[1] + w * (double)v.y;
        acc[2] = acc[2] + w * (double)v.z;
      }
  n = acc[0];
  th = acc[1];
  b = acc[2];
  return true;
}

// Redshift nu_obs / nu_emit of an emitter on a circular orbit of angular
// velocity Omega = 1 / (r^(3/2) + a) at (r, theta) for a photon of lambda;
// 0 where that orbit is not timelike.
__device__ __forceinline__ double redshift(double a, double r, double u, double lam) {
  const double u2 = u * u;
  const double s2 = (1.0 - u) * (1.0 + u);
  const double sig = r * r + a * a * u2;
  const double delta = r * r - 2.0 * r + a * a;
  const double A = (r * r + a * a) * (r * r + a * a) - a * a * delta * s2;
  const double om = bhk::div_rn(1.0, r * bhk::sqrt_rn(r) + a);
  const double inv_sig = bhk::div_rn(1.0, sig);
  const double gtt = -(1.0 - 2.0 * r * inv_sig);
  const double gtp = -2.0 * a * r * s2 * inv_sig;
  const double gpp = A * s2 * inv_sig;
  const double norm = -(gtt + 2.0 * gtp * om + gpp * om * om);
  if (!(norm > 0.0)) return 0.0;
  const double den = 1.0 - om * lam;  // over sqrt(norm)
  return den > 0.0 ? bhk::div_rn(bhk::sqrt_rn(norm), den) : 0.0;
}

// Planck B_nu(T) (reference planckFunction).
__device__ __forceinline__ double planck(double nu, double temp) {
  const double x = bhk::div_rn(kH * nu, kKb * temp);
  const double den = (x > 500.0) ? exp(x) : expm1(x);
  if (!(den > 0.0)) return 0.0;
  return ((2.0 * kH / (kC * kC)) * nu * nu * nu) / den;
}

// Emission and absorption in the emitter's frame at frequency nu_e (the
// table holds ln(j / (n_e nu_B)), interpolated bilinearly).
__device__ __forceinline__ void synchrotron(const BhkRtParams &q, double n, double theta_e, double b, double nu_e,
                                            double &j, double &alpha) {
  j = 0.0;
  alpha = 0.0;
  if (!(n > 0.0 && theta_e > 0.0 && b > 0.0 && nu_e > 0.0)) return;
  const double nu_b = (kE / (kTwoPi * kMe * kC)) * b;
  const double nu_s = 1.5 * nu_b * theta_e * theta_e;
  // an infinite Theta_e or |B| (div_rn wants finite operands) is the table's lower end, as x = 0 is
  const double lx = nu_s < INFINITY ? log(bhk::div_rn(nu_e, nu_s)) : -INFINITY;
  // beyond the table: exp(-1.89 x^(1/3)) below any use; a quotient past the range is no number
  if (!(lx <= q.lx1)) return;
  const double lt = log(theta_e);
  double ft = (lt - q.lt0) * q.lt_scale;
  double fx = (lx - q.lx0) * q.lx_scale;
  // a coordinate that is no number takes node 0 too: as an integer it would be INT_MIN
  ft = ft > 0.0 ? (ft > (double)(q.n_lt - 1) ? (double)(q.n_lt - 1) : ft) : 0.0;
  fx = fx > 0.0 ? (fx > (double)(q.n_lx - 1) ? (double)(q.n_lx - 1) : fx) : 0.0;
  int i0 = (int)floor(ft), k0 = (int)floor(fx);
  i0 = i0 > q.n_lt - 2 ? q.n_lt - 2 : i0;
  k0 = k0 > q.n_lx - 2 ? q.n_lx - 2 : k0;
  const double ti = ft - (double)i0, tk = fx - (double)k0;
  const float *L = q.lut;
  const double v00 = (double)__ldg(L + i0 * q.n_lx + k0), v01 = (double)__ldg(L + i0 * q.n_lx + k0 + 1);
  const double v10 = (double)__ldg(L + (i0 + 1) * q.n_lx + k0), v11 = (double)__ldg(L + (i0 + 1) * q.n_lx + k0 + 1);
  const double J = ((1.0 - ti) * ((1.0 - tk) * v00 + tk * v01)) + (ti * ((1.0 - tk) * v10 + tk * v11));
  j = n * nu_b * exp(J);
  const double bnu = planck(nu_e, theta_e * (kMe * kC * kC / kKb));
  alpha = bnu > 0.0 ? j / bnu : 0.0;
}

}  // namespace bhrt

// ---- FP32 variants (the mixed-precision transfer) ------------------------------
//
// The same physics in FP32 with the emission and the source function carried
// as logarithms: ln j = ln n_e + ln nu_B + J (J the table value), Kirchhoff
// alpha = j / B_nu, so the observed source function g^3 B_nu and the
// observed opacity alpha / g never leave the FP32 exponent range (j itself
// reaches 1e-40 and below, under FP32's normal range).

namespace bhrt {

struct MediumF {
  const float4 *cells;
  const float *lut;
  int n_r, n_th, n_ph, n_lt, n_lx;
  float r_min, r_max, fr_scale;  // (n_r - 1) / log(r_max / r_min)
  float lt0, lt_scale, lx0, lx1, lx_scale;
  float ln_nu, ln_len, ds_max, min_transmit;
  float inv_n_ph;
  float x_coef;        // h nu / (m_e c^2): x = x_coef / (g Theta_e)
  float ln_nub_gauss;  // ln(e / (2 pi m_e c)): ln nu_B per ln gauss
  float ln_2h_c2;      // ln(2 h / c^2)
};

__host__ __device__ inline MediumF medium_f(const BhkRtParams &q) {
  MediumF m;
  m.cells = reinterpret_cast<const float4 *>(q.cells);
  m.lut = q.lut;
  m.n_r = q.n_r;
  m.n_th = q.n_th;
  m.n_ph = q.n_ph;
  m.n_lt = q.n_lt;
  m.n_lx = q.n_lx;
  m.r_min = (float)q.r_min;
  m.r_max = (float)q.r_max;
  m.fr_scale = (float)(q.inv_log_range * (double)(q.n_r - 1));
  m.lt0 = (float)q.lt0;
  m.lt_scale = (float)((double)(q.n_lt - 1) / (q.lt1 - q.lt0));
  m.lx0 = (float)q.lx0;
  m.lx1 = (float)q.lx1;
  m.lx_scale = (float)((double)(q.n_lx - 1) / (q.lx1 - q.lx0));
  m.ln_nu = (float)log(q.nu);
  m.ln_len = (float)log(q.length_cm);
  m.ds_max = (float)q.ds_max;
  m.min_transmit = (float)q.min_transmit;
  m.inv_n_ph = 1.0f / (float)q.n_ph;
  m.x_coef = (float)(kH * q.nu / (kMe * kC * kC));
  m.ln_nub_gauss = (float)log(kE / (kTwoPi * kMe * kC));
  m.ln_2h_c2 = (float)log(2.0 * kH / (kC * kC));
  return m;
}

#ifdef __CUDACC__
// Issue slots bound a transfer, most of them its samples': fmodf and eight
// 64-bit indices here took 5 % of the 512^2 frame (2.84 -> 2.70 ms), and eight
// 64-bit addresses again (2.58 -> 2.45). Off, the type of a byte offset into
// the cells, is 32 bits up to 2^28 cells.
template <class Off>
__device__ __forceinline__ bool sample_f(const MediumF &q, float r, float u, float phi, float &n, float &th,
                                         float &b) {
  if (!(r >= q.r_min && r <= q.r_max)) return false;
  const float fr = __logf(r / q.r_min) * q.fr_scale;
  const int i0 = min(max((int)floorf(fr), 0), q.n_r - 2);
  const float tr = fminf(fmaxf(fr - (float)i0, 0.0f), 1.0f);
  const float theta = acosf(fminf(fmaxf(u, -1.0f), 1.0f));
  const float ft = theta * (0.31830988618f * (float)q.n_th) - 0.5f;
  const int j0 = min(max((int)floorf(ft), 0), q.n_th - 2);
  const float tt = fminf(fmaxf(ft - (float)j0, 0.0f), 1.0f);
  const float fp = phi * (0.15915494309f * (float)q.n_ph);
  const float fl = floorf(fp);
  const float tp = fp - fl;
  const int k0 = azimuth_cell(fl, q.n_ph, q.inv_n_ph);
  const int k1 = (k0 + 1 == q.n_ph) ? 0 : k0 + 1;
  const char *cells = reinterpret_cast<const char *>(q.cells);
  const Off c00 = ((Off)i0 * (Off)q.n_th + (Off)j0) * (Off)q.n_ph * 16u, row = (Off)q.n_th * (Off)q.n_ph * 16u,
            col = (Off)q.n_ph * 16u, o0 = c00 + (Off)k0 * 16u, o1 = c00 + (Off)k1 * 16u;
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
#pragma unroll
  for (int di = 0; di < 2; ++di)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj)
#pragma unroll
      for (int dk = 0; dk < 2; ++dk) {
        const float w = (di ? tr : 1.0f - tr) * (dj ? tt : 1.0f - tt) * (dk ? tp : 1.0f - tp);
        const float4 v =
            __ldg(reinterpret_cast<const float4 *>(cells + ((dk ? o1 : o0) + (di ? row : 0u) + (dj ? col : 0u))));
        a0 = fmaf(w, v.x, a0);
        a1 = fmaf(w, v.y, a1);
        a2 = fmaf(w, v.z, a2);
      }
  n = a0;
  th = a1;
  b = a2;
  return true;
}

// FP32 redshift of the circular-orbit emitter (see redshift above).
__device__ __forceinline__ float redshift_f(float a, float r, float u, float lam) {
  const float u2 = u * u;
  const float s2 = (1.0f - u) * (1.0f + u);
  const float sig = fmaf(r, r, a * a * u2);
  const float delta = fmaf(r, r - 2.0f, a * a);
  const float rr = fmaf(r, r, a * a);
  const float A = fmaf(rr, rr, -a * a * delta * s2);
  const float om = 1.0f / fmaf(r, sqrtf(r), a);
  const float inv_sig = 1.0f / sig;
  const float gtt = -(1.0f - 2.0f * r * inv_sig);
  const float gtp = -2.0f * a * r * s2 * inv_sig;
  const float gpp = A * s2 * inv_sig;
  const float norm = -(gtt + om * fmaf(gpp, om, 2.0f * gtp));
  if (!(norm > 0.0f)) return 0.0f;
  const float den = (1.0f - om * lam) * rsqrtf(norm);
  return den > 0.0f ? 1.0f / den : 0.0f;
}

// ln(j_obs) - ln(S_obs) and ln(S_obs) of one sample: S_obs = g^3 B_nu(nu/g),
// alpha_obs = (j / B_nu) / g. Returns false where there is no emission.
__device__ __forceinline__ bool ln_emission_f(const MediumF &q, float n, float theta_e, float b, float g,
                                              float &ln_alpha_obs, float &ln_s_obs) {
  if (!(n > 0.0f && theta_e > 0.0f && b > 0.0f && g > 0.0f)) return false;
  const float ln_g = __logf(g);
  const float ln_nu_e = q.ln_nu - ln_g;
  const float ln_nub = __logf(b) + q.ln_nub_gauss;
  const float lt = __logf(theta_e);
  const float lx = ln_nu_e - 0.40546511f - ln_nub - 2.0f * lt;  // ln(nu_e / nu_s), nu_s = 3/2 nu_B Theta^2
  if (lx > q.lx1) return false;
  const float ft = fminf(fmaxf((lt - q.lt0) * q.lt_scale, 0.0f), (float)(q.n_lt - 1));
  const float fx = fminf(fmaxf((lx - q.lx0) * q.lx_scale, 0.0f), (float)(q.n_lx - 1));
  const int i0 = min((int)ft, q.n_lt - 2), k0 = min((int)fx, q.n_lx - 2);
  const float ti = ft - (float)i0, tk = fx - (float)k0;
  const float *L = q.lut + i0 * q.n_lx + k0;
  const float J = (1.0f - ti) * fmaf(tk, __ldg(L + 1) - __ldg(L), __ldg(L)) +
                  ti * fmaf(tk, __ldg(L + q.n_lx + 1) - __ldg(L + q.n_lx), __ldg(L + q.n_lx));
  const float ln_j = __logf(n) + ln_nub + J;
  // ln B_nu(nu_e, T) = ln(2 h / c^2) + 3 ln nu_e - ln(e^x - 1), x = h nu_e / (k T) = x_coef / (g Theta_e)
  const float x = __fdividef(q.x_coef, g * theta_e);
  const float ln_em1 = x > 20.0f ? x : __logf(expm1f(x));
  const float ln_bnu = q.ln_2h_c2 + 3.0f * ln_nu_e - ln_em1;
  ln_alpha_obs = ln_j - ln_bnu - ln_g;
  ln_s_obs = 3.0f * ln_g + ln_bnu;
  return true;
}
#endif

}  // namespace bhrt
