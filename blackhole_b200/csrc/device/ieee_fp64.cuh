// ieee_fp64.cuh - FP64 quotients and square roots without branches.
//
// The FP64 tracers round every operation as the CPU oracle does, so their
// quotients and roots are the IEEE ones. CUDA's operators expand to a
// sequence with a slow-path branch each; with some twenty of them in one
// step, the branches cut the step into basic blocks, and the independent
// divisions of its stages run one after another. Here a quotient is
//   y = 1/b from the hardware's approximation (2^-20) and one third-order
//       Newton step, y (1 + e + e^2) with e = 1 - b y,
//   q = a y,  q + (a - b q) y
// with the remainder exact in one FMA: the correction step of P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34 (1990) 111-119, likewise the root g + (x - g^2) / (2 g).
// Before the last rounding the value is within 2^-51 ulp of the exact one, so
// the result is the correctly rounded one unless the exact value lies that
// close to the midpoint of two doubles. They serve operands whose quotient
// and remainder stay in the normal range (|a|, |b| in 1e-290 .. 1e300, or a
// = 0). Beyond it a quotient may be NaN or 0 where the operator's is not: a / b
// with an infinite a or b, or a zero or subnormal b, is NaN, and the root of
// infinity is NaN. The step controller rejects that like the overflow it stands
// for; elsewhere the callers keep such operands out.
//
// What it bought (one B200, outputs bit for bit the same): the FP64 pipe was
// 57 % busy in a DP45 frame, "wait" (fixed latency) the first stall. 640 x 360
// DP45, three crossings: 4.36 ms with CUDA's operators, 3.21 ms here; 64 x 48
// DP45: 0.97 and 0.61 ms; 256^2 RK4: 8.45 and 6.72 ms; the FP64 transfer of
// 160^2 rays: 9.4 and 8.2 ms.
#pragma once

namespace bhk {

// The sign bit: x < 0 for every x but -0 (and NaN), on the integer pipe.
__device__ __forceinline__ bool is_neg(double x) { return __double2hiint(x) < 0; }

// 1 / b to 0.51 ulp, and a / b from it.
__device__ __forceinline__ double rcp_near(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  double e = fma(-b, y, 1.0);
  e = fma(e, e, e);
  return fma(y, e, y);
}
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}

// a / b.
__device__ __forceinline__ double div_rn(double a, double b) { return div_by(a, b, rcp_near(b)); }

// a / 5 and a / 6, the reciprocal in two parts: a quotient by 5 or 3 lies a
// tenth of an ulp or more from any midpoint of two doubles (a multiple of the
// half ulp that is not 5 or 3 times a midpoint is one half ulp off at least),
// and the sum before its one rounding is within 2^-50 ulp of it.
__device__ __forceinline__ double div_5(double a) { return fma(a, 1.0 / 5.0, a * -0x1.999999999999ap-57); }
__device__ __forceinline__ double div_6(double a) { return fma(a, 1.0 / 6.0, a * 0x1.5555555555555p-57); }

// sqrt(x) for x > 1e-290; a smaller x (0 among them) is returned as it is: the
// callers compare the root with bounds that all such values, and their roots,
// lie on the same side of. The compare is of the high words. Root and half
// reciprocal are refined side by side (R. E. Goldschmidt's scheme), a chain of
// seven dependent operations.
__device__ __forceinline__ double sqrt_rn(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double g0 = x * y, h0 = 0.5 * y;
  const double e = fma(-g0, y, 1.0);
  const double t = fma(0.375, e, 0.5) * e;
  const double g = fma(g0, t, g0);
  const double s = fma(fma(-g, g, x), fma(h0, t, h0), g);
  return __double2hiint(x) > 0x03cfffff ? s : x;
}

// The FP32 root, the same way; 0 is its own root, arguments below 1e-30 are
// scaled by an even power of two. tests/test_gpu_exact_ops.py: equal to sqrtf at all
// 2^31 floats.
__device__ __forceinline__ float sqrt_rn_f(float x) {
  const bool tiny = x < 1e-30f;
  const float v = tiny ? x * 0x1p100f : x;
  float y;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(v));
  const float g = v * y;
  float s = fmaf(fmaf(-g, g, v), 0.5f * y, g);
  s = tiny ? s * 0x1p-50f : s;
  return x == 0.0f || x == INFINITY ? x : s;
}

}  // namespace bhk
