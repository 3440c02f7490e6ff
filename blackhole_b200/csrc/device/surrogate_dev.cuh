// surrogate_dev.cuh - device pieces shared by the network's inference kernel
// (surrogate.cu) and its training kernels (surrogate_train.cu): activations,
// input features, the swizzled shared-memory store, tensor maps.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <mutex>

#include "surrogate_net.h"
#include "umma.cuh"

namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;
// Waits on other warps' progress run out after the caller's limit (default
// 2 s; bh_surrogate_set_wait_limit) and record an error code. Work this
// thread itself started (TMA loads, MMAs) is then drained with a fixed limit
// before TMEM is freed and the CTA exits: it completes on its own.
constexpr uint64_t kDrainNs = 1000000000ull;

enum : int { kErrProducer = 11, kErrMma = 12, kErrDone = 13 };

__device__ __forceinline__ float tanh_approx(float x) {
  float r;
  asm("tanh.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// SiLU(y) = y sigmoid(y) with sigmoid(y) = (1 + tanh(y/2)) / 2: one MUFU
// operation per element (training and inference use the same form).
__device__ __forceinline__ float silu(float y) {
  const float h = 0.5f * y;
  return fmaf(h, tanh_approx(h), h);
}

__device__ __forceinline__ float silu_grad(float y) {
  const float s = fmaf(0.5f, tanh_approx(0.5f * y), 0.5f);
  return s * (1.0f + y * (1.0f - s));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// SiLU of two pre-activations given as halves hy = y / 2 (FP32), returned as
// packed FP16: hy (1 + tanh hy) = y sigmoid(y), with one tanh.approx.f16x2
// (one MUFU operation for both) and one f16x2 FMA. The activation is the next
// layer's FP16 operand, so nothing is unpacked; FP16 keeps 11 significant
// bits, as many as the MUFU tanh delivers.
__device__ __forceinline__ uint32_t silu_f16x2(float hy_lo, float hy_hi) {
  const uint32_t h = pack_f16(hy_lo, hy_hi);
  uint32_t t, r;
  asm("tanh.approx.f16x2 %0, %1;" : "=r"(t) : "r"(h));
  asm("fma.rn.f16x2 %0, %1, %2, %2;" : "=r"(r) : "r"(t), "r"(h));
  return r;
}

// 2^(k/3), k = 0..15: Fourier frequencies in units of pi.
__constant__ float c_freq[BHS_FOURIER] = {1.0f,
                     1.2599210498948732f,
                     1.5874010519681994f,
                     2.0f,
                     2.5198420997897464f,
                     3.1748021039363987f,
                     4.0f,
                     5.0396841995794928f,
                     6.3496042078727974f,
                     8.0f,
                     10.079368399158986f,
                     12.699208415745595f,
                     16.0f,
                     20.158736798317971f,
                     25.398416831491190f,
                     32.0f};

// Fourier features of one input x: (sin, cos)(pi 2^(k/3) x), k = 0..15,
// interleaved. Frequencies k = 0, 1, 2 come from sincospif; every further
// one doubles the angle of the one three below (sin 2t = 2 s c,
// cos 2t = (c - s)(c + s)), which keeps the absolute error near 1e-6.
__device__ __forceinline__ void fourier_pairs(float x, float (&v)[2 * BHS_FOURIER]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) sincospif(c_freq[k] * x, &v[2 * k], &v[2 * k + 1]);
#pragma unroll
  for (int k = 3; k < BHS_FOURIER; ++k) {
    const float sn = v[2 * (k - 3)], cs = v[2 * (k - 3) + 1];
    v[2 * k] = 2.0f * sn * cs;
    v[2 * k + 1] = (cs - sn) * (cs + sn);
  }
}

// The network's scaled inputs: x = (alpha/15, beta/15, 2a - 1, 2 cos theta - 1)
// and the constants of motion lambda/15, eta/225.
__device__ __forceinline__ void scaled_inputs(float4 q, float (&x)[4], float& lam, float& eta) {
  x[0] = q.x * (1.0f / 15.0f);
  x[1] = q.y * (1.0f / 15.0f);
  x[2] = 2.0f * q.z - 1.0f;
  x[3] = 2.0f * q.w - 1.0f;
  const float st = sqrtf(fmaxf(0.0f, 1.0f - q.w * q.w));
  lam = -q.x * st * (1.0f / 15.0f);
  eta = (q.y * q.y + (q.x * q.x - q.z * q.z) * q.w * q.w) * (1.0f / 225.0f);
}

// Regression output j (head column 3 + j, target column 2 + j) counts when:
// j = 0..2, 6: a first disk hit; j = 3..5: a second hit; j = 7..9: escaped.
__device__ __forceinline__ bool reg_mask(int j, int cls, int nc) {
  if (j <= 2 || j == 6) return nc >= 1;
  if (j <= 5) return nc >= 2;
  return cls == 2;
}

// K steps (16 columns each) of layer 0's last 64-column chunk that can hold a
// nonzero term: features 128..133 lie in the first.
constexpr int kFeatTailSteps = (BHS_FEATURES_USED - 128 + 15) / 16;
static_assert(BHS_FEATURES_USED > 128 && BHS_FEATURES_USED <= 144, "feature tail within one K step");

__device__ __forceinline__ int layer_k(int l) { return l == 0 ? BHS_FEATURES : BHS_HIDDEN; }
__device__ __forceinline__ int layer_chunks(int l) { return layer_k(l) / kBK; }

// One 16-byte unit (8 BF16, unit j of 8 in a 64-column chunk) of row r of a
// K-major 128-byte-swizzled tile chunk at shared address cb.
__device__ __forceinline__ void st_unit(uint32_t cb, int r, int j, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  const uint32_t addr = cb + (uint32_t)r * 128u + ((uint32_t)(j ^ (r & 7)) << 4);
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// ---- tensor maps -------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
        cudaSuccess &&
      q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// K-major 16-bit matrix [rows][ld] (K valid columns), box {64, box_rows}, 128-byte swizzle.
bool make_map(CUtensorMap* m, const void* base, int64_t rows, int K, int ld, int box_rows,
              CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0 || (ld * 2) % 16 != 0) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t es[2] = {1, 1};
  return fn(m, type, 2, const_cast<void*>(base), dims, strides, box, es,
       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace
