// frame_source.cuh - where a persistent tracer's work items come from.
//
// The tracing loop hands out global work indices w = 0, 1, ... from one
// counter. SingleSrc maps them to the pixels of one frame whose parameters
// live in kernel parameter space; BatchSrc maps them through a device frame
// table (prefix sums of the frames' pixel counts) so that one launch traces
// frames of uneven size, spin, inclination and observer radius back to back,
// and records when each frame's last pixel finished.
#pragma once

#include "launch.h"
#include "tile_order.h"

namespace bhsrc {

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The persistent tracers hold a lane whose ray needs rare work -- a crossing
// to locate, outputs to write, a new ray to set up -- until the warp's held
// lanes have waited kHold lane-iterations in all, then do that work for all
// of them at once: it takes a warp about half an iteration, however many of
// its lanes take part. Served as it came up, one or two lanes at a time, it
// kept 22 to 25 of 32 lanes busy. One B200, kHold = 1 / 16 / 64 / 128 / 512:
// 48 uneven frames, mixed DP45 (4.2 M rays): 23.9 / 16.3 / 15.3 / 15.2 / 14.8
// ms; 1920 x 1080 camera frame: 3.84 / 2.11 / 1.86 / 1.83 / 1.81 ms; 640 x 360
// FP64 DP45: 3.02 / 3.03 / 2.91 / 2.91 / 2.99 ms; 64 x 48 FP64 DP45, where a
// held ray is a late one: 0.66 / 0.62 / 0.62 / 0.65 / 0.79 ms. Served at once
// and in row order (before): 21.6, 3.27, 3.21 and 0.61 ms.
constexpr int kHold = 64;

// Steps between two looks at the warp's held lanes (times the launch's refill
// interval). The votes cost a warp its lanes' reconvergence and some thirty
// cycles of the step's latency each time: every step / every 8 or 32, one B200,
// 64 x 48 RK4: mixed 2.07 / 1.31 ms, FP64 3.39 / 2.63; 64 x 48 DP45: mixed 0.24 /
// 0.20, FP64 0.62 / 0.57; 48 uneven mixed frames 13.95 / 13.28.
constexpr int kTurnsRk4 = 32, kTurnsDp45 = 8;

// Lane states of the persistent tracers.
enum : int { kEmpty = -1, kRun = -2, kCross = -3, kCrossStop = -4 };  // >= 0: ended with that class

// tile_pixel for a frame of one wave (every ray has a lane from the start), with
// its tiles shuffled (a bijection of [0, 2^k) by two xor shifts and a product
// with an odd number, repeated until it falls below the number of tiles): rays
// that run long -- past the hole and out again, twice the others' RK4 steps --
// are neighbours, and in order one SM got six such warps while most had none
// (256^2 RK4: FP64 6.1 ms, shuffled 5.4; mixed 3.0 and 2.65).
// Frames of several waves keep their order: there a warp takes new rays from
// two tiles at a time, and neighbours stay together.
__device__ __forceinline__ long long wave_pixel(long long w, const BhkImageParams &p) {
  if (p.n_pix <= (long long)gridDim.x * blockDim.x) {
    const unsigned T = (unsigned)(p.n_pix >> 5);
    unsigned t = (unsigned)(w >> 5);
    if (t < T && T > 1) {
      const int k = 32 - __clz((int)(T - 1)), half = (k + 1) / 2;
      const unsigned mask = (1u << k) - 1u;
      do {
        t ^= t >> half;
        t = (t * 0x9E3779B1u) & mask;
        t ^= t >> half;
      } while (t >= T);
      w = (long long)(t << 5 | (unsigned)(w & 31));
    }
  }
  return tile_pixel(w, p.width, p.n_pix);
}

// WAVE: the order of wave_pixel (RK4, whose steps depend on where a ray ends).
template <bool WAVE>
struct SingleSrc {
  const BhkImageParams &p;
  const BhkImageOut &o;
  __device__ __forceinline__ long long total() const { return p.n_pix; }
  __device__ __forceinline__ int frame_of(long long w, long long &pix) const {
    pix = WAVE ? wave_pixel(w, p) : tile_pixel(w, p.width, p.n_pix);
    return 0;
  }
  __device__ __forceinline__ const BhkImageParams &params(int) const { return p; }
  __device__ __forceinline__ const BhkImageOut &out(int) const { return o; }
  __device__ __forceinline__ void pixel_done(int) const {}
};

// The pixels of one frame named by a device list whose length a previous
// kernel wrote (the surrogate renderer's integrator fallback).
struct ListSrc {
  const BhkImageParams &p;
  const BhkImageOut &o;
  const int *list;
  const unsigned int *count;
  __device__ __forceinline__ long long total() const { return (long long)*count; }
  __device__ __forceinline__ int frame_of(long long w, long long &pix) const {
    pix = list[w];
    return 0;
  }
  __device__ __forceinline__ const BhkImageParams &params(int) const { return p; }
  __device__ __forceinline__ const BhkImageOut &out(int) const { return o; }
  __device__ __forceinline__ void pixel_done(int) const {}
};

struct BatchSrc {
  const BhkBatchDev &b;
  __device__ __forceinline__ long long total() const { return b.n_total; }
  // Largest f with prefix[f] <= w (binary search; prefix[0] = 0).
  __device__ __forceinline__ int frame_of(long long w, long long &pix) const {
    int lo = 0, hi = b.n_frames - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (b.prefix[mid] <= w)
        lo = mid;
      else
        hi = mid - 1;
    }
    pix = tile_pixel(w - b.prefix[lo], b.frames[lo].p.width, b.frames[lo].p.n_pix);
    return lo;
  }
  __device__ __forceinline__ const BhkImageParams &params(int f) const { return b.frames[f].p; }
  __device__ __forceinline__ const BhkImageOut &out(int f) const { return b.frames[f].o; }
  // The lane that finishes a frame's last pixel stamps the frame's end time.
  __device__ __forceinline__ void pixel_done(int f) const {
    const unsigned int n = (unsigned int)b.frames[f].p.n_pix;
    if (atomicAdd(&b.done[f], 1u) + 1u == n) b.end_ns[f] = globaltimer_ns();
  }
};

}  // namespace bhsrc
