// azimuth_cell.h - the azimuthal cell of a medium. Plain arithmetic for the
// device and for the host test.
#pragma once

#include <algorithm>
#include <cmath>

#ifdef __CUDACC__
#define BHRT_HD __host__ __device__ __forceinline__
#define BHRT_CLAMP(k, top) min(max(k, 0), top)
#else
#define BHRT_HD inline
#define BHRT_CLAMP(k, top) std::clamp(k, 0, top)
#endif

namespace bhrt {

// Cell fl (a whole number; negative and past the last one after turns) of n < 2^22
// around the axis, inv_n = 1 / n: fl modulo n. Whole turns by the rounded quotient are
// taken off in one exact rounding, which leaves 2^-22 (FP32) or 2^-51 (FP64) of fl or
// half a turn, whichever is more: twice, exact for |fl| < 2^44 and 2^102 (beyond, and for
// what is no number, some cell). A step over the pole, accepted at a wide tolerance,
// turns 10^12 radians. Without branches, n and inv_n where they lie in the launch's
// constants: the 512^2 mixed image 2.30 ms, as with one quotient that held up to 2^23;
// with them by value 2.35, with fmodf behind a test 2.34 to 2.47 where that was placed.
template <class T>
BHRT_HD int azimuth_cell(T fl, const int &n, const T &inv_n) {
  using std::fma, std::rint;
  const T turn = (T)n, rest = fma(-turn, rint(fl * inv_n), fl);
  int k = (int)fma(-turn, rint(rest * inv_n), rest);
  k += k < 0 ? n : (k >= n ? -n : 0);
  return BHRT_CLAMP(k, n - 1);
}

}  // namespace bhrt
