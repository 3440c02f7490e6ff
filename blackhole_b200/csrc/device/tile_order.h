// tile_order.h - the order in which the tracers take a frame's pixels. Plain
// integer code for the device and for the host test.
#pragma once

#ifdef __CUDACC__
#define BHSRC_HD __host__ __device__ __forceinline__
#else
#define BHSRC_HD inline
#endif

namespace bhsrc {

// Pixel w of a frame in the order the tracers take them: bands of 4 rows, in
// a band 8 x 4 tiles, so that a warp's 32 rays are neighbours in both
// directions and reach the disk, the hole or the sky at about the same step.
// Row order where a band of 4 rows, or the frame, is beyond 32 bits.
BHSRC_HD long long tile_pixel(long long w, int width, long long n_pix) {
  if (n_pix > 0x7fffffffLL || width > 0x3fffffff) return w;
  const unsigned W = (unsigned)width, n = (unsigned)n_pix, q = (unsigned)w;
  const unsigned band = q / (4u * W), r0 = 4u * band;
  const unsigned left = n / W - r0, rows = left < 4u ? left : 4u;
  const unsigned in = q - r0 * W;
  const unsigned tiled = (W & ~7u) * rows;
  unsigned x, y;
  if (in < tiled) {
    const unsigned t = in / (8u * rows), i = in - t * 8u * rows;
    x = 8u * t + (i & 7u);
    y = i >> 3;
  } else {
    const unsigned rest = W & 7u, i = in - tiled;
    y = i / rest;
    x = (W & ~7u) + i - y * rest;
  }
  return (long long)(r0 + y) * width + x;
}

}  // namespace bhsrc
