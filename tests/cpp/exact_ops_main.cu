// Counts arguments at which the branch-free operations of ieee_fp64.cuh differ from
// CUDA's IEEE ones. Prints five counts: sqrt_rn_f over every float >= 0 and NaN;
// div_rn, sqrt_rn, div_5 and div_6 over pseudo-random operands of their range.
#include <cmath>
#include <cstdio>

#include "ieee_fp64.cuh"

__device__ unsigned long long mix(unsigned long long x) {  // splitmix64
  unsigned long long z = x + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// 53 random bits, sign, and an exponent in [lo, hi)
__device__ double operand(unsigned long long k, int lo, int hi) {
  const unsigned long long a = mix(2 * k), b = mix(2 * k + 1);
  const long long e = 1023 + lo + (long long)(b % (unsigned)(hi - lo));
  return __longlong_as_double((long long)((a & 0x800fffffffffffffull) | (unsigned long long)e << 52));
}

__global__ void floats(unsigned long long* bad) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 31);
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const float x = __uint_as_float((unsigned)i), a = bhk::sqrt_rn_f(x), b = sqrtf(x);
    if (__float_as_uint(a) != __float_as_uint(b) && !(isnan(a) && isnan(b))) atomicAdd(bad, 1ull);
  }
}

__global__ void doubles(unsigned long long n, unsigned long long* bad) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    // the quotient and its remainder stay normal: exponents within 2^+-450
    const double a = operand(3 * i, -450, 450), b = operand(3 * i + 1, -450, 450), x = fabs(operand(3 * i + 2, -960, 960));
    if (bhk::div_rn(a, b) != a / b) atomicAdd(bad, 1ull);
    if (bhk::sqrt_rn(x) != sqrt(x)) atomicAdd(bad + 1, 1ull);
    if (bhk::div_5(a) != a / 5.0) atomicAdd(bad + 2, 1ull);
    if (bhk::div_6(a) != a / 6.0) atomicAdd(bad + 3, 1ull);
  }
}

int main() {
  unsigned long long* bad = nullptr;
  if (cudaMalloc(&bad, 5 * sizeof(*bad)) != cudaSuccess || cudaMemset(bad, 0, 5 * sizeof(*bad)) != cudaSuccess) return 2;
  floats<<<1184, 256>>>(bad);
  doubles<<<1184, 256>>>(1ull << 28, bad + 1);
  unsigned long long h[5];
  if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("%llu %llu %llu %llu %llu\n", h[0], h[1], h[2], h[3], h[4]);
  return 0;
}
