// postprocess.cu - bloom and tone mapping of an RGBA float4 framebuffer, the
// bridge's post-processing (src/blender_bridge/cuda_postprocess.cu:237-275).
//
// The reference's pipeline, per frame:
//   bright = bright_pass(fb)            luminance excess over the threshold
//   accum  = sum over r in {4, 8, 16, 32} of V_r(H_r(bright))
//   fb    += strength * accum
//   fb     = tone(fb)                   exposure, vignette, ACES, gamma 1/2.2
// with H_r / V_r the normalized Gaussian of half-width r (sigma = r / 2),
// clamped at the image edges. Each scale blurs the bright-pass itself (the
// reference re-extracts it between scales).
//
// Here that is three launches instead of nineteen:
//   k_post_rows : bright-pass fused into the four horizontal blurs. A tile of
//                 16 rows x 64 columns (+ 32-column halos) in shared memory,
//                 two rows side by side (pitch 129 pairs: a half-warp's 8 row
//                 pairs x 2 runs fall in distinct banks); two warps a channel,
//                 a thread has 8 outputs of a row pair and stores them from
//                 its registers, a warp 128 bytes of a row. The framebuffer's
//                 own channels leave as planes too.
//   k_post_cols : the four vertical blurs of one channel, summed in the
//                 reference's order (r = 4, 8, 16, 32), added to that
//                 channel's plane; a thread has 8 rows of two neighbouring
//                 columns; the next scale's plane arrives by 16-byte cp.async
//                 meanwhile, no more rows of it than the scale reaches.
//   k_post_tone : the tone map of the three planes into the caller's
//                 framebuffer.
// Both blurs multiply and add two values per instruction (fma.rn.f32x2, each
// half rounded as the scalar one): issue slots, not the FP32 lanes, bound the
// scalar version (79 and 68 % issue at 42 and 34 % of the FMA pipe). 1920 x
// 1080, strength 0.5, per launch from a cold L2: rows 76 -> 61 us in pairs,
// -> 52 in these tiles (1.15 waves of 32 x 128 tiles, all channels in turn,
// became 2.8 waves of a third of the work); columns 101 -> 54 in pairs, -> 47
// with a channel a CTA (2 CTAs of 256 threads at 126 registers became 7 of
// 128); tone, without a 64-bit division per pixel, 30 -> 29 (three powf, 84 %
// issue). The multiplications alone fill the FP32 pipe for 24 us a blur.
// The horizontal results travel through 12 float planes (4 scales x RGB,
// structure of arrays, rows padded to 64 columns), the composite through three
// more: the tone map reads a neighbour's colour (below), which an in-place
// pass would race on. Bytes per pixel: rows 16 in + 60 out, columns 60 in +
// 12 out, tone 12 in + 16 out.
//
// The tone map's red and blue come from pixel (rx, ry) = (int(u w), int(v h))
// with u = px / w, v = py / h rounded to float (cuda_postprocess.cu:165-176,
// chromatic aberration at strength 0): for most widths a few columns take
// them from the pixel to their left (fl(fl(px / w) w) < px). That index is
// kept bit for bit; the colour read there is the composite before tone
// mapping.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "launch.h"

namespace {

// Rows of tiles in a grid's second dimension; taller images take the third.
constexpr unsigned kMaxY = 65535;

constexpr int kHalo = 32;  // the largest blur half-width
constexpr int kRun = 8;    // outputs per thread along the blur direction

// Rows pass tile: two warps (of 64 columns) a channel.
constexpr int kRowsY = 16;
constexpr int kRowsX = 64;
constexpr int kRowsW = kRowsX + 2 * kHalo;
constexpr int kRowsPitch = kRowsW + 1;          // in row pairs
constexpr int kRowPairs = kRowsY / 2;
constexpr int kRowsLanes = kRowPairs * (kRowsX / kRun);  // threads of a channel
constexpr int kRowsThreads = 3 * kRowsLanes;

// Columns pass tile.
constexpr int kColsX = 32;
constexpr int kColsY = 64;
constexpr int kColsH = kColsY + 2 * kHalo;
constexpr int kColsThreads = kColsX / 2 * (kColsY / kRun);
constexpr int kColsBuf = kColsH * kColsX;

// Floats between rows of a plane: whole tiles of 64 columns, so that every row
// starts on 256 bytes, where 15 such planes take no more than 16 floats a
// pixel; narrower images the widest padding of 32, 16, 8 or 4 floats (a 16-byte
// copy) that does, and 4 where none does (some below 42 columns). At 64 for all, a
// column of 50 million rows would take 192 GB.
constexpr int plane_pitch(int w) {
  int pad = 64;
  while (pad > 4 && 15ll * ((w + (pad - 1ll)) / pad * pad) > 16ll * w) pad /= 2;
  return (w + pad - 1) / pad * pad;
}
constexpr int kBase = 12;  // planes kBase + c: the framebuffer's channels, then the composite's

// Scale index and offset of the normalized taps (2r + 1 each) of half-width R.
__host__ __device__ constexpr int scale_of(int R) { return R == 4 ? 0 : R == 8 ? 1 : R == 16 ? 2 : 3; }
__host__ __device__ constexpr int tap_off(int R) { return R == 4 ? 0 : R == 8 ? 9 : R == 16 ? 26 : 59; }

// The taps, each twice: both halves of a packed product.
struct Taps2 {
  float2 w[124];
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

__device__ __forceinline__ float bright_scale(float4 c, float threshold) {
  const float lum = 0.2126f * c.x + 0.7152f * c.y + 0.0722f * c.z;
  const float excess = fmaxf(0.0f, lum - threshold);
  return lum > 0.001f ? excess / lum : 0.0f;
}

// acc[j] += sum_t w[t] src[(j + t) * stride], t = 0..2R in order: the blur of
// R taps either side of output j, src pointing at output 0's first tap, for
// two values at a time. The 8 values that a tap meets slide through registers.
template <int R>
__device__ __forceinline__ void blur_run(const float2 *src, int stride, const float2 *w, float2 (&acc)[kRun]) {
  float2 v[kRun];
#pragma unroll
  for (int j = 0; j < kRun; ++j) v[j] = src[j * stride];
#pragma unroll
  for (int t = 0; t <= 2 * R; ++t) {
#pragma unroll
    for (int j = 0; j < kRun; ++j) acc[j] = fma2(w[t], v[(t + j) % kRun], acc[j]);
    if (t < 2 * R) v[t % kRun] = src[(t + kRun) * stride];
  }
}

__global__ void __launch_bounds__(kRowsThreads, 5) k_post_rows(const __grid_constant__ Taps2 taps,
                                                               const float4 *__restrict__ fb, int w, int h, int pitch,
                                                               float threshold, float *__restrict__ planes) {
  __shared__ float2 sm[3 * kRowPairs * kRowsPitch];  // bright-pass
  const int x0 = blockIdx.x * kRowsX, y0 = (blockIdx.y + kMaxY * blockIdx.z) * kRowsY;
  const int64_t plane = (int64_t)h * pitch;
  constexpr int kPairs = kRowPairs * kRowsW, kInFlight = 3;  // 6 pixels a thread
#pragma unroll 1
  for (int k0 = 0; k0 < kPairs; k0 += kInFlight * kRowsThreads) {
    float4 v[kInFlight][2];
#pragma unroll
    for (int k = 0; k < kInFlight; ++k) {
      const int e = k0 + k * kRowsThreads + threadIdx.x, rp = e / kRowsW, col = e - rp * kRowsW;
      const int x = min(max(x0 - kHalo + col, 0), w - 1);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int y = y0 + 2 * rp + i;
        v[k][i] = e < kPairs && y < h ? fb[(int64_t)y * w + x] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
#pragma unroll
    for (int k = 0; k < kInFlight; ++k) {
      const int e = k0 + k * kRowsThreads + threadIdx.x, rp = e / kRowsW, col = e - rp * kRowsW;
      if (e >= kPairs) continue;
      const float s0 = bright_scale(v[k][0], threshold), s1 = bright_scale(v[k][1], threshold);
      sm[(0 * kRowPairs + rp) * kRowsPitch + col] = make_float2(v[k][0].x * s0, v[k][1].x * s1);
      sm[(1 * kRowPairs + rp) * kRowsPitch + col] = make_float2(v[k][0].y * s0, v[k][1].y * s1);
      sm[(2 * kRowPairs + rp) * kRowsPitch + col] = make_float2(v[k][0].z * s0, v[k][1].z * s1);
      const int x = x0 - kHalo + col;
      if (col >= kHalo && col < kHalo + kRowsX && x < w) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int y = y0 + 2 * rp + i;
          float *base = planes + kBase * plane + (int64_t)y * pitch + x;
          if (y < h) base[0] = v[k][i].x, base[plane] = v[k][i].y, base[2 * plane] = v[k][i].z;
        }
      }
    }
  }
  const int c = threadIdx.x / kRowsLanes, lane = threadIdx.x % kRowsLanes;
  const int rp = lane % kRowPairs, run = lane / kRowPairs;
  __syncthreads();
  // A warp has 8 row pairs x 4 neighbouring runs: its stores fill whole 32-byte
  // sectors, 128 bytes of a row at a time.
  const int y = y0 + 2 * rp, x = x0 + run * kRun;
  const float2 *src = sm + (c * kRowPairs + rp) * kRowsPitch + kHalo + run * kRun;
  float *dst = planes + c * plane + (int64_t)y * pitch + x;
  const bool left = x < pitch, right = x + 4 < pitch, top = y < h, low = y + 1 < h;
  auto scale = [&](auto rtag) {
    constexpr int R = decltype(rtag)::value, si = scale_of(R);
    float2 acc[kRun] = {};
    asm volatile("" ::: "memory");  // one scale's window at a time in registers
    blur_run<R>(src - R, 1, taps.w + tap_off(R), acc);
    float4 *out = reinterpret_cast<float4 *>(dst + 3 * si * plane);
    if (left && top) out[0] = make_float4(acc[0].x, acc[1].x, acc[2].x, acc[3].x);
    if (right && top) out[1] = make_float4(acc[4].x, acc[5].x, acc[6].x, acc[7].x);
    if (left && low) out[pitch / 4] = make_float4(acc[0].y, acc[1].y, acc[2].y, acc[3].y);
    if (right && low) out[pitch / 4 + 1] = make_float4(acc[4].y, acc[5].y, acc[6].y, acc[7].y);
  };
  scale(std::integral_constant<int, 4>{});
  scale(std::integral_constant<int, 8>{});
  scale(std::integral_constant<int, 16>{});
  scale(std::integral_constant<int, 32>{});
}

// Rows y0 - R .. y0 + kColsY - 1 + R (clamped) of one channel's plane of scale
// si, kColsX columns from x0 (those inside the plane), into a shared buffer, by
// cp.async.
__device__ __forceinline__ void cols_fetch(float *buf, const float *__restrict__ planes, int c, int si, int x0,
                                           int y0, int pitch, int h) {
  const int R = 4 << si;
  constexpr int kVecs = kColsX / 4;
  const float *src = planes + (int64_t)(si * 3 + c) * h * pitch + x0 + 4 * (threadIdx.x % kVecs);
  float *dst = buf + 4 * (threadIdx.x % kVecs);
  if (x0 + 4 * (int)(threadIdx.x % kVecs) >= pitch) return;
  for (int row = threadIdx.x / kVecs; row < kColsY + 2 * R; row += kColsThreads / kVecs) {
    const int y = min(max(y0 - R + row, 0), h - 1);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst + row * kColsX)),
                 "l"(src + (int64_t)y * pitch)
                 : "memory");
  }
}

__global__ void __launch_bounds__(kColsThreads, 7) k_post_cols(const __grid_constant__ Taps2 taps,
                                                               float *__restrict__ planes, int h, int pitch,
                                                               float strength) {
  extern __shared__ float cols_sm[];  // two buffers of [kColsH][kColsX]: scale si in buffer si % 2
  const int x0 = blockIdx.x * kColsX, y0 = (blockIdx.y + kMaxY * (blockIdx.z / 3)) * kColsY, c = blockIdx.z % 3;
  const int lane = threadIdx.x % (kColsX / 2), grp = threadIdx.x / (kColsX / 2);
  auto fetch = [&](int si) {
    if (si < 4) cols_fetch(cols_sm + (si % 2) * kColsBuf, planes, c, si, x0, y0, pitch, h);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  fetch(0);
  fetch(1);
  float2 tot[kRun] = {};
  auto scale = [&](auto rtag) {
    constexpr int R = decltype(rtag)::value, si = scale_of(R);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this scale landed, the next may be in flight
    __syncthreads();
    const float2 *buf = reinterpret_cast<const float2 *>(cols_sm + (si % 2) * kColsBuf);
    float2 acc[kRun] = {};
    blur_run<R>(buf + grp * kRun * (kColsX / 2) + lane, kColsX / 2, taps.w + tap_off(R), acc);
#pragma unroll
    for (int j = 0; j < kRun; ++j) tot[j].x += acc[j].x, tot[j].y += acc[j].y;
    if (si < 2) __syncthreads();  // every warp is done with the buffer
    fetch(si + 2);
  };
  scale(std::integral_constant<int, 4>{});
  scale(std::integral_constant<int, 8>{});
  scale(std::integral_constant<int, 16>{});
  scale(std::integral_constant<int, 32>{});
  if (x0 + 2 * lane >= pitch) return;
  float *base = planes + (int64_t)(kBase + c) * h * pitch + x0 + 2 * lane;
#pragma unroll
  for (int j = 0; j < kRun; ++j) {
    const int y = y0 + grp * kRun + j;
    if (y >= h) break;
    float2 *p = reinterpret_cast<float2 *>(base + (int64_t)y * pitch);
    const float2 b = *p;
    *p = make_float2(b.x + tot[j].x * strength, b.y + tot[j].y * strength);
  }
}

// ACES filmic curve, the fit of K. Narkowicz (2015), clamped to [0, 1].
__device__ __forceinline__ float aces(float x) {
  const float y = (x * (2.51f * x + 0.03f)) / (x * (2.43f * x + 0.59f) + 0.14f);
  return fminf(fmaxf(y, 0.0f), 1.0f);
}

// Exposure, vignette, ACES, gamma 1/2.2, in the reference's order.
__device__ __forceinline__ float tone_channel(float x, float exposure, float vignette) {
  return powf(fmaxf(aces((x * exposure) * vignette), 0.0f), 1.0f / 2.2f);
}

// A thread has one column of ROWS rows, so that u and the column index are
// worked out once: 4 (1920 x 1080: 30 -> 28 us), but 1 where one wave of threads
// holds the image and a thread's own chain of powf is the time (100 x 60 with
// bloom: 44 and 41 us a call).
// PLANAR: the composite is in three planes, otherwise a copy of the framebuffer.
template <bool PLANAR, int ROWS>
__global__ void __launch_bounds__(256) k_post_tone(const float *__restrict__ src, int w, int h, int pitch, float exposure,
                                                   float4 *__restrict__ fb) {
  const int64_t plane = (int64_t)h * pitch;
  // red and blue of one pixel
  auto red_blue = [&](int64_t i) {
    if (PLANAR) return make_float2(src[i], src[2 * plane + i]);
    const float4 v = reinterpret_cast<const float4 *>(src)[i];
    return make_float2(v.x, v.z);
  };
  const int px = blockIdx.x * 64 + (threadIdx.x & 63);
  const unsigned y0 = ((blockIdx.y + kMaxY * blockIdx.z) * 4 + (threadIdx.x >> 6)) * ROWS;  // passes 2^31 by a slice
  if (px >= w) return;
  const float u = __fdiv_rn((float)px, (float)w);
  const int rx = min(max((int)__fmul_rn(u, (float)w), 0), w - 1);
  const float du = u - 0.5f;
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    if (y0 + k >= (unsigned)h) break;
    const int py = (int)(y0 + k);
    const int64_t i = (int64_t)py * w + px;
    const float v = __fdiv_rn((float)py, (float)h);
    const int ry = min(max((int)__fmul_rn(v, (float)h), 0), h - 1);
    const float2 rb = red_blue((int64_t)ry * pitch + rx);
    const int64_t g = (int64_t)py * pitch + px;
    const float gch = PLANAR ? src[plane + g] : src[4 * g + 1];
    const float dv = v - 0.5f;
    // fused as written, for the same values at every ROWS
    const float dist = sqrtf(__fmaf_rn(du, du, __fmul_rn(dv, dv)));
    const float vig = sqrtf(fmaxf(1.0f - dist * dist * 0.5f, 0.0f));
    fb[i] = make_float4(tone_channel(rb.x, exposure, vig), tone_channel(gch, exposure, vig),
                        tone_channel(rb.y, exposure, vig), 1.0f);
  }
}

}  // namespace

// 15 padded planes, or a copy of the framebuffer where the bloom is off; -1: the
// image is too wide for the blurs' 32-bit columns.
extern "C" int64_t bhk_post_scratch_floats(int w, int h, float strength) {
  if (strength == 0.0f) return (int64_t)4 * w * h;
  if (w > INT32_MAX - 2 * kRowsX) return -1;
  return (int64_t)(kBase + 3) * plane_pitch(w) * h;
}

extern "C" int bhk_post_process(float *fb, int w, int h, const BhkPostTaps *taps, float threshold, float strength,
                                float exposure, float *scratch, void *stream) {
  if (w <= 0 || h <= 0) return 0;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  float4 *f4 = reinterpret_cast<float4 *>(fb);
  auto tiles = [&](unsigned tx, unsigned ty, unsigned channels) {
    const unsigned rows = ((unsigned)h + ty - 1) / ty;
    return dim3(((unsigned)w + tx - 1) / tx, std::min(rows, kMaxY), (rows + kMaxY - 1) / kMaxY * channels);
  };
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev) != cudaSuccess)
    return -1;
  const int64_t wave = (int64_t)sms * per_sm;
  const int pitch = strength != 0.0f ? plane_pitch(w) : 0;
  auto tone = [&](auto planar, const float *src) {
    constexpr bool kPlanar = decltype(planar)::value;
    const int row = kPlanar ? pitch : w;
    if ((int64_t)w * h <= wave)
      k_post_tone<kPlanar, 1><<<tiles(64, 4, 1), 256, 0, st>>>(src, w, h, row, exposure, f4);
    else
      k_post_tone<kPlanar, 4><<<tiles(64, 16, 1), 256, 0, st>>>(src, w, h, row, exposure, f4);
  };
  if (strength != 0.0f) {
    constexpr int smem = sizeof(float) * 2 * kColsBuf;
    if (cudaFuncSetAttribute(k_post_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return -1;
    Taps2 t2;
    for (int i = 0; i < 124; ++i) t2.w[i] = make_float2(taps->w[i], taps->w[i]);
    k_post_rows<<<tiles(kRowsX, kRowsY, 1), kRowsThreads, 0, st>>>(t2, f4, w, h, pitch, threshold, scratch);
    k_post_cols<<<tiles(kColsX, kColsY, 3), kColsThreads, smem, st>>>(t2, scratch, h, pitch, strength);
    tone(std::true_type{}, scratch + (int64_t)kBase * pitch * h);
  } else {
    if (cudaMemcpyAsync(scratch, fb, sizeof(float4) * w * h, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return -1;
    tone(std::false_type{}, scratch);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
