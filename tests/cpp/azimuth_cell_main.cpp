// Checks bhrt::azimuth_cell on the host against the exact remainder: 1 to 2^24
// azimuths, whole numbers of every magnitude that it serves and of either sign, and
// beside multiples of the number of azimuths.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "azimuth_cell.h"

namespace {

uint64_t state = 0x243F6A8885A308D3ull;
uint64_t next() {
  state ^= state << 13, state ^= state >> 7, state ^= state << 17;
  return state;
}

template <class T>
bool wrong(T v, int n) {
  long long want = (long long)std::fmod((double)v, (double)n);  // exact
  if (want < 0) want += n;
  return bhrt::azimuth_cell(v, n, T(1) / (T)n) != want;
}

template <class T>
long long check(int top) {
  long long bad = 0;
  for (int n : {1, 2, 3, 5, 7, 10, 63, 64, 100, 4096, 65535, 65537, 1000003, 1 << 22, 1 << 24})
    for (int e = 0; e <= top; ++e)
      for (int k = 0; k < 2000; ++k) {
        const T v = std::floor(std::ldexp((T)(next() >> 11) * (T)0x1p-53, e));
        const T m = std::floor(v / (T)n) * (T)n;  // at a whole turn or, rounded, near one
        for (T w : {v, m, m - 1, m + 1}) bad += wrong<T>(w, n) + wrong<T>(-w, n);
      }
  return bad;
}

}  // namespace

int main() {
  const long long f = check<float>(44), d = check<double>(102);
  if (f || d) std::printf("wrong cells: %lld in FP32, %lld in FP64\n", f, d);
  return f || d ? 1 : 0;
}
