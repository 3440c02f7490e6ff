// One training batch of the learned transfer function in three launches:
//
//   k_train_pass    every 128-row tile through the whole network and back:
//                   features, four hidden layers, head, loss, and the loss
//                   gradient of every pre-activation, BF16 operands and FP32
//                   accumulation. One CTA per tile; the tile's activations (A
//                   operand of the next product) stay in shared memory, its
//                   accumulators in tensor memory.
//   k_train_dw      dW_l = dY_l^T X_l for all layers at once, split over the
//                   batch: both operands straight from the row-major arrays as
//                   MN-major tiles, so nothing is transposed anywhere.
//   k_train_collect the partial sums into the gradient vector.
//
// What bounds it (batch 16384, one B200): 23 GFLOP, 14 us of tensor time at
// the measured rate. One GEMM launch per product (twenty launches, a tile's
// loads, MMAs and its row-by-row epilogue one after another, every activation
// and gradient also written transposed) took 300 us; this takes 84: 45 in the
// pass, 22 in the weight gradients, 8 in the collection, the rest between
// them. The pass is bound by the tile's chain of nine products and epilogues
// and, inside the epilogues, by the L2: its 128 tiles move in step, and write
// and read back 100 MB of FP32 pre-activations and stream 115 MB of weights (a
// layer whose pre-activations stay in tensor memory takes 3.9 K cycles, the
// others 7). With 8 epilogue warps and an mbarrier arrival per thread the
// pass took 60.
#include <algorithm>
#include <cstdio>
#include <cstring>

#include "surrogate_dev.cuh"

namespace {

constexpr int kTile = 128;
constexpr int kChunk = kTile * kBK * 2;         // 16 KB: 64 columns of a tile, 128-byte swizzle
constexpr int kWStage = BHS_HIDDEN * kBK * 2;   // 32 KB: 64 columns of a weight matrix
constexpr int kWRing = 4;
constexpr int kBiases = 4 * BHS_HIDDEN + BHS_HEAD;
constexpr int kEpiWarps = 16;                   // per TMEM lane quarter four, 16 columns of each chunk
constexpr int kPassThreads = 32 * (kEpiWarps + 3);  // + producer, MMA issuer, store warp
constexpr int kPassSmem = 4 * kChunk + kWRing * kWStage + kBiases * 4 + 64 + 1024 + 256;

// Tensor maps of a plan, all {64, rows} boxes with the 128-byte swizzle.
enum : int { kMapW = 0, kMapWT = 5, kMapF = 9, kMapH = 10, kMapDY = 14, kMapDout = 18, kMaps = 19 };
struct TrainMaps {
  CUtensorMap m[kMaps];
};
static_assert(sizeof(CUtensorMap) == 128 && kMaps <= 24, "BhsTrainPlan::maps");

struct PassArgs {
  const float* in;
  const float* targets;
  int targets16;  // targets start on 16 bytes
  const float* params;
  __nv_bfloat16* dout;
  float* y[3];
  float* bias_part;
  float* loss;
  int64_t B;
  int* err;
  uint64_t wait_ns;
  int64_t bias_off[BHS_LAYERS];
};

__device__ __forceinline__ void tma_store_2d(const void* tmap, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(src),
               "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Loss of one row and its gradient d with respect to the 16 head outputs o:
// cross entropy of the class and the squared error of the masked targets.
__device__ __forceinline__ void row_loss(const float (&o)[BHS_HEAD], const float (&t)[BHS_TARGETS], float invB,
                                         float (&d)[BHS_HEAD], float (&acc)[4]) {
  const int cls = (int)t[0], nc = (int)t[1];
#pragma unroll
  for (int i = 0; i < BHS_HEAD; ++i) d[i] = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = 0.0f;
  if (cls >= 0) {
    const float m = fmaxf(o[0], fmaxf(o[1], o[2]));
    const float e0 = expf(o[0] - m), e1 = expf(o[1] - m), e2 = expf(o[2] - m);
    const float Z = e0 + e1 + e2;
    const float oc = cls == 0 ? o[0] : (cls == 1 ? o[1] : o[2]);
    acc[0] = -(oc - m - logf(Z));
    d[0] = (e0 / Z - (cls == 0 ? 1.f : 0.f)) * invB;
    d[1] = (e1 / Z - (cls == 1 ? 1.f : 0.f)) * invB;
    d[2] = (e2 / Z - (cls == 2 ? 1.f : 0.f)) * invB;
    const int am = (o[1] > o[0] && o[1] >= o[2]) ? 1 : ((o[2] > o[0] && o[2] > o[1]) ? 2 : 0);
    acc[2] = am == cls ? 1.f : 0.f;
    acc[3] = 1.f;
  }
#pragma unroll
  for (int j = 0; j < 10; ++j) {
    if (reg_mask(j, cls, nc)) {
      const float e = o[3 + j] - t[2 + j];
      acc[1] += e * e;
      d[3 + j] = 2.0f * e * invB;
    }
  }
}

// The tile's stages: products s = 0..3 the hidden layers, 4 the head, 5 the
// gradient of layer 3's activations, 6..8 of layers 2..0's. Operand set s
// (features, H_0..H_3, dout, dY_3..dY_1) feeds product s; set 9 (dY_0) only
// leaves. Accumulators alternate between two halves of tensor memory, so the
// product after an epilogue starts on the 64-column chunks that are done.
// Product 5 goes beside layer 3's pre-activations, which its epilogue still
// needs: product 6 alone waits for all of that epilogue.
//
// An operand set is read by a product and copied to HBM, both of which see
// its chunks' `ready` phases; the epilogue completes a chunk's next phase only
// after both have passed the last one (acc_full and `stored` follow it). Set 5
// has no copy and set 9 no product, so they have barriers of their own
// (dout_ready, out_ready): on the shared ones a reader that does not wait for
// them could fall two phases behind, which looks like none.
__device__ __forceinline__ int set_chunks(int s) { return s == 0 ? 3 : (s == 5 ? 1 : 4); }
__device__ __forceinline__ uint32_t acc_col(int s) { return (0x14Au >> s) & 1u ? 256u : 0u; }  // s = 1, 3, 6, 8

__global__ void __launch_bounds__(kPassThreads, 1)
    k_train_pass(const __grid_constant__ TrainMaps M, const __grid_constant__ PassArgs A) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = umma::smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
  const uint32_t act = raw + pad;
  const uint32_t ring = act + 4u * kChunk;
  float* sb = reinterpret_cast<float*>(smem_raw + pad + 4 * kChunk + kWRing * kWStage);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + pad + 4 * kChunk + kWRing * kWStage + kBiases * 4 + 64);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kWRing + 12);
  const uint32_t b0 = umma::smem_u32(bars);
  auto full = [&](int i) { return b0 + 8u * i; };
  auto empty = [&](int i) { return b0 + 8u * (kWRing + i); };
  auto ready = [&](int c) { return b0 + 8u * (2 * kWRing + c); };  // chunk c of operand sets 0..4, 6..8 is written
  const uint32_t acc_full = b0 + 8u * (2 * kWRing + 4);
  const uint32_t stored = b0 + 8u * (2 * kWRing + 5);  // the operand set has been read by its copy to HBM
  const uint32_t drained = b0 + 8u * (2 * kWRing + 6);
  const uint32_t dout_ready = b0 + 8u * (2 * kWRing + 7);               // set 5 (one chunk) is written
  auto out_ready = [&](int c) { return b0 + 8u * (2 * kWRing + 8 + c); };  // chunk c of set 9 is written
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t tiles = A.B / kTile;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kWRing; ++i) {
      umma::mbar_init(full(i), 1);
      umma::mbar_init(empty(i), 1);
    }
    for (int c = 0; c < 4; ++c) {
      umma::mbar_init(ready(c), kEpiWarps);
      umma::mbar_init(out_ready(c), kEpiWarps);
    }
    umma::mbar_init(dout_ready, kEpiWarps);
    umma::mbar_init(acc_full, 1);
    umma::mbar_init(stored, 1);
    umma::mbar_init(drained, 1);
    umma::fence_mbar_init();
    for (int i = 0; i < kMaps; ++i) umma::tma_prefetch_desc(&M.m[i]);
  }
  for (int i = threadIdx.x; i < kBiases; i += kPassThreads)
    sb[i] = A.params[A.bias_off[i / BHS_HIDDEN] + i % BHS_HIDDEN];
  if (warp == 0) {
    umma::tmem_alloc(umma::smem_u32(tmem_slot), 512);
    umma::tmem_relinquish();
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {  // weight producer
      uint32_t it = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x)
        for (int s = 0; ok && s < 9; ++s) {
          const CUtensorMap* map = s < 5 ? &M.m[kMapW + s] : &M.m[kMapWT + (8 - s)];  // WT: layers 1..4 at 0..3
          const uint32_t bytes = s == 4 ? BHS_HEAD * kBK * 2 : kWStage;
          for (int c = 0; c < set_chunks(s); ++c, ++it) {
            const int st = (int)(it % kWRing);
            if (it >= (uint32_t)kWRing && !umma::mbar_wait(empty(st), ((it / kWRing) - 1) & 1, A.wait_ns)) {
              atomicExch(A.err, kErrProducer);
              ok = false;
              break;
            }
            umma::mbar_arrive_expect_tx(full(st), bytes);
            umma::tma_load_2d(ring + (uint32_t)st * kWStage, map, full(st), c * kBK, 0);
          }
        }
      for (uint32_t i = it > (uint32_t)kWRing ? it - kWRing : 0u; i < it; ++i)
        umma::mbar_wait(full((int)(i % kWRing)), (i / kWRing) & 1, kDrainNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      uint32_t it = 0, seen[4] = {0u, 0u, 0u, 0u}, tiles_seen = 0;
      bool ok = true;
      auto wait_on = [&](uint32_t bar, uint32_t phases) {
        if (ok && !umma::mbar_wait(bar, phases & 1u, A.wait_ns)) {
          atomicExch(A.err, kErrMma);
          ok = false;
        }
      };
      auto wait_ready = [&](int c) { wait_on(ready(c), seen[c]++); };
      for (int64_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x, ++tiles_seen) {
        for (int s = 0; ok && s < 9; ++s) {
          const uint32_t idesc = umma::idesc_bf16_f32(kTile, s == 4 ? BHS_HEAD : BHS_HIDDEN);
          const uint32_t d = tmem + acc_col(s);
          if (s == 6)
            for (int c = 0; c < 4; ++c) wait_ready(c);
          for (int c = 0; ok && c < set_chunks(s); ++c, ++it) {
            if (s == 5)
              wait_on(dout_ready, tiles_seen);
            else if (s != 6)
              wait_ready(c);
            const int st = (int)(it % kWRing);
            if (ok && !umma::mbar_wait(full(st), (it / kWRing) & 1, A.wait_ns)) {
              atomicExch(A.err, kErrMma);
              ok = false;
            }
            if (!ok) break;
            umma::tc_fence_after();
            const uint64_t ad = umma::sw128_desc(act + (uint32_t)c * kChunk);
            const uint64_t bd = umma::sw128_desc(ring + (uint32_t)st * kWStage);
            // columns past the last feature, and past the 16 head outputs, are zero
            const int ksteps = s == 0 && c == 2 ? kFeatTailSteps : (s == 5 ? 1 : kBK / 16);
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              if (k < ksteps) umma::mma_bf16(d, ad + 2u * k, bd + 2u * k, idesc, (c > 0 || k > 0) ? 1u : 0u);
            umma::mma_commit(empty(st));
          }
          if (ok) umma::mma_commit(acc_full);
        }
      }
      umma::mma_commit(drained);
      umma::mbar_wait(drained, 0, kDrainNs);
    }
  } else if (warp == 2) {
    if (lane == 0) {  // copies each operand set to HBM as its chunks are written
      uint32_t seen[4] = {0u, 0u, 0u, 0u}, tiles_seen = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x, ++tiles_seen)
        for (int s = 0; ok && s < 10; ++s) {
          if (s == 5) continue;  // dout is written to HBM by the epilogue itself
          const CUtensorMap* map = s == 0 ? &M.m[kMapF] : (s < 5 ? &M.m[kMapH + s - 1] : &M.m[kMapDY + 9 - s]);
          for (int c = 0; c < set_chunks(s); ++c) {
            if (!umma::mbar_wait(s == 9 ? out_ready(c) : ready(c), (s == 9 ? tiles_seen : seen[c]++) & 1u,
                                 A.wait_ns)) {
              atomicExch(A.err, kErrDone);
              ok = false;
              break;
            }
            for (int half = 0; half < 2; ++half)
              tma_store_2d(map, act + (uint32_t)c * kChunk + (uint32_t)half * (kChunk / 2), c * kBK,
                           (int)(tile * kTile) + 64 * half);
          }
          if (!ok) continue;
          bulk_commit();
          bulk_wait_read();
          umma::mbar_arrive(stored);
        }
      bulk_wait();
    }
  } else {  // epilogue: TMEM lane quarter q (warp % 4); columns 16 hf .. 16 hf + 15 of every chunk
    const int hf = (warp - 3) >> 2;
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t tacc = tmem + ((uint32_t)(q * 32) << 16);
    uint32_t acc_seen = 0, stores = 0, stores_seen = 0;
    bool ok = true;
    auto arrive_on = [&](uint32_t bar) {  // one arrival a warp: an arrival is an atomic on one word
      umma::fence_async_smem();
      umma::tc_fence_before();
      __syncwarp();
      if (lane == 0) umma::mbar_arrive(bar);
    };
    auto chunk_done = [&](int c) { arrive_on(ready(c)); };
    // the copy of the last set has read the tile's buffer
    auto wait_stored = [&]() {
      if (stores == stores_seen) return;
      ok = __all_sync(0xffffffffu, umma::mbar_wait(stored, stores_seen & 1u, A.wait_ns));
      ++stores_seen;
    };
    auto wait_acc = [&]() {
      ok = __all_sync(0xffffffffu, umma::mbar_wait(acc_full, acc_seen & 1u, A.wait_ns));
      ++acc_seen;
      umma::tc_fence_after();
    };
    // 16 values of this row into chunk c, as BF16
    auto put16 = [&](int c, const float (&v)[16]) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
        st_unit(act + (uint32_t)c * kChunk, r, 2 * hf + u, pack_bf16(v[8 * u], v[8 * u + 1]),
                pack_bf16(v[8 * u + 2], v[8 * u + 3]), pack_bf16(v[8 * u + 4], v[8 * u + 5]),
                pack_bf16(v[8 * u + 6], v[8 * u + 7]));
    };
    // sums over the warp's 32 rows of 16 BF16 columns from unit u0 of chunk c: lanes l and l + 16 get column l
    auto column_sum = [&](int c, int u0) {
      float s = 0.0f;
      const int col = lane & 15;
      const uint32_t base = act + (uint32_t)c * kChunk + 2u * (uint32_t)(col & 7);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int row = q * 32 + (lane & 16) + i;
        const uint32_t a = base + (uint32_t)row * 128u + ((uint32_t)((u0 + (col >> 3)) ^ (row & 7)) << 4);
        uint16_t h;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(a) : "memory");
        s += __uint_as_float((uint32_t)h << 16);
      }
      return s + __shfl_xor_sync(0xffffffffu, s, 16);
    };
    for (int64_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
      const int64_t row = tile * kTile + r;
      float* bias_out = A.bias_part + (tile * 4 + q) * kBiases;
      {  // features: warp group hf the pairs of input hf (32 columns), group 3 the rest (chunk 2) as well
        wait_stored();
        if (!ok) break;
        float x[4], lam, eta, v[2 * BHS_FOURIER];
        scaled_inputs(reinterpret_cast<const float4*>(A.in)[row], x, lam, eta);
        fourier_pairs(hf == 0 ? x[0] : (hf == 1 ? x[1] : (hf == 2 ? x[2] : x[3])), v);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          st_unit(act + (uint32_t)(hf >> 1) * kChunk, r, 4 * (hf & 1) + u, pack_bf16(v[8 * u], v[8 * u + 1]),
                  pack_bf16(v[8 * u + 2], v[8 * u + 3]), pack_bf16(v[8 * u + 4], v[8 * u + 5]),
                  pack_bf16(v[8 * u + 6], v[8 * u + 7]));
        if (hf == 3) {
          st_unit(act + 2u * kChunk, r, 0, pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(lam, eta), 0u);
          for (int u = 1; u < 8; ++u) st_unit(act + 2u * kChunk, r, u, 0u, 0u, 0u, 0u);
        }
        for (int c = 0; c < 3; ++c) chunk_done(c);
        ++stores;
      }
      for (int l = 0; l < 4; ++l) {  // hidden layers
        wait_acc();
        if (ok) wait_stored();
        if (!ok) break;
        const uint32_t acc = tacc + acc_col(l);
        const float* b = sb + l * BHS_HIDDEN;
        float4* ys = l < 3 ? reinterpret_cast<float4*>(A.y[l]) + tile * (kTile * BHS_HIDDEN / 4) : nullptr;
        float va[16], vb[16];
        tmem_ld16_nowait(acc + 16u * hf, va);
        umma::tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float(&v)[16] = (c & 1) ? vb : va;
          if (c < 3) tmem_ld16_nowait(acc + 64u * (c + 1) + 16u * hf, (c & 1) ? va : vb);
          const int col = 64 * c + 16 * hf;
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const float4 bb = reinterpret_cast<const float4*>(b + col)[g];
            v[4 * g] += bb.x, v[4 * g + 1] += bb.y, v[4 * g + 2] += bb.z, v[4 * g + 3] += bb.w;
            if (l < 3) ys[(col / 4 + g) * kTile + r] = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = silu(v[i]);
          put16(c, v);
          chunk_done(c);
          if (c < 3) umma::tmem_wait_ld();
        }
        ++stores;
      }
      if (!ok) break;
      float t[BHS_TARGETS];
      if (hf == 0) {
        if (A.targets16) {
          const float4* tp = reinterpret_cast<const float4*>(A.targets) + row * 4;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 f = tp[i];
            t[4 * i] = f.x, t[4 * i + 1] = f.y, t[4 * i + 2] = f.z, t[4 * i + 3] = f.w;
          }
        } else {
#pragma unroll
          for (int i = 0; i < BHS_TARGETS; ++i) t[i] = A.targets[row * BHS_TARGETS + i];
        }
      }
      wait_acc();
      if (ok) wait_stored();
      if (!ok) break;
      if (hf == 0) {  // head outputs, loss, dout
        float o[16], d[16], part[4];
        tmem_ld16_nowait(tacc + acc_col(4), o);
        umma::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < BHS_HEAD; ++i) o[i] += sb[4 * BHS_HIDDEN + i];
        row_loss(o, t, 1.0f / (float)A.B, d, part);
        uint32_t pk[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) pk[i] = pack_bf16(d[2 * i], d[2 * i + 1]);
        st_unit(act, r, 0, pk[0], pk[1], pk[2], pk[3]);
        st_unit(act, r, 1, pk[4], pk[5], pk[6], pk[7]);
        uint4* g = reinterpret_cast<uint4*>(A.dout + row * BHS_HEAD_PAD);
        g[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        g[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        __syncwarp();
        const float s = column_sum(0, 0);
        if (lane < 16) bias_out[4 * BHS_HIDDEN + lane] = s;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float v = part[i];
#pragma unroll
          for (int x = 16; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
          if (lane == 0 && v != 0.0f) atomicAdd(A.loss + i, v);
        }
      }
      arrive_on(dout_ready);
      for (int s = 5; s < 9; ++s) {  // dY_l = (dY_(l+1) W_(l+1)) * SiLU'(Y_l)
        const int l = 8 - s;
        const float4* ys = l < 3 ? reinterpret_cast<const float4*>(A.y[l]) + tile * (kTile * BHS_HIDDEN / 4) : nullptr;
        float4 yn[4];  // the next chunk's pre-activations, read ahead
        if (l < 3) {
#pragma unroll
          for (int g = 0; g < 4; ++g) yn[g] = ys[(4 * hf + g) * kTile + r];
        }
        wait_acc();
        if (ok) wait_stored();
        if (!ok) break;
        const uint32_t acc = tacc + acc_col(s);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          const int col = 64 * c + 16 * hf;
          float v[16], y[16];
          tmem_ld16_nowait(acc + (uint32_t)col, v);
          if (l == 3) {
            tmem_ld16_nowait(tacc + acc_col(3) + (uint32_t)col, y);
          } else {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              y[4 * g] = yn[g].x, y[4 * g + 1] = yn[g].y, y[4 * g + 2] = yn[g].z, y[4 * g + 3] = yn[g].w;
              if (c < 3) yn[g] = ys[((col + 64) / 4 + g) * kTile + r];
            }
          }
          umma::tmem_wait_ld();
          if (l == 3) {
#pragma unroll
            for (int i = 0; i < 16; ++i) y[i] += sb[3 * BHS_HIDDEN + col + i];
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] *= silu_grad(y[i]);
          put16(c, v);
          arrive_on(s == 8 ? out_ready(c) : ready(c));
          const float s1 = column_sum(c, 2 * hf);
          if (lane < 16) bias_out[l * BHS_HIDDEN + col + lane] = s1;
        }
        ++stores;
      }
    }
    if (!ok && lane == 0) atomicExch(A.err, kErrDone);
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

// ---- weight gradients ------------------------------------------------------------

constexpr int kDwRows = 512;                      // batch rows per split (layer 4: twice as many)
constexpr int kDwRing = 3;
constexpr int kDwBox = 64 * 128;                  // 8 KB: 64 rows x 64 columns
constexpr int kDwStage = 8 * kDwBox;              // A: 256 columns, B: up to 256
constexpr int kDwThreads = 192;
constexpr int kDwSmem = kDwRing * kDwStage + 1024 + 256;

struct DwArgs {
  float* part[BHS_LAYERS];
  int64_t B;
  int splits;  // of layers 0..3
  int* err;
  uint64_t wait_ns;
};

// Shared-memory descriptor of an MN-major operand in {64 columns, 64 rows}
// boxes with the 128-byte swizzle: 64 consecutive M (or N) values per 128-byte
// row, one row per K; the next 64 M values a box (8 KB) on (leading byte
// offset), the next 8 K values 1024 bytes on (stride byte offset). 16 values
// of K further is 2048 bytes.
__device__ __forceinline__ uint64_t mn_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(kDwBox >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

// One CTA: 256 x N products of up to 512 rows, M = 256 as two accumulators.
// Blocks [0, 4 splits) are layers 0..3 (dY_l^T X_l, N = the layer's input
// width), the rest layer 4, as its transpose H_3^T dout so that M is 256 there
// too (N = 64 columns of dout, 16 of them used).
__global__ void __launch_bounds__(kDwThreads, 1)
    k_train_dw(const __grid_constant__ TrainMaps M, const __grid_constant__ DwArgs A) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = umma::smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
  const uint32_t base = raw + pad;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + pad + kDwRing * kDwStage);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kDwRing + 1);
  const uint32_t b0 = umma::smem_u32(bars);
  auto full = [&](int i) { return b0 + 8u * i; };
  auto empty = [&](int i) { return b0 + 8u * (kDwRing + i); };
  const uint32_t done = b0 + 8u * (2 * kDwRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int l = min((int)blockIdx.x / A.splits, 4);
  const int sp = (int)blockIdx.x - l * A.splits;
  const int rows = l == 4 ? 2 * kDwRows : kDwRows;
  const int r0 = sp * rows;
  const int nch = (int)(min((int64_t)rows, A.B - r0) / 64);
  const int N = l == 4 ? 64 : layer_k(l);
  const int nbox = N / 64;
  const CUtensorMap* ma = l == 4 ? &M.m[kMapH + 3] : &M.m[kMapDY + l];
  const CUtensorMap* mb = l == 4 ? &M.m[kMapDout] : (l == 0 ? &M.m[kMapF] : &M.m[kMapH + l - 1]);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kDwRing; ++i) {
      umma::mbar_init(full(i), 1);
      umma::mbar_init(empty(i), 1);
    }
    umma::mbar_init(done, 1);
    umma::fence_mbar_init();
    umma::tma_prefetch_desc(ma);
    umma::tma_prefetch_desc(mb);
  }
  if (warp == 0) {
    umma::tmem_alloc(umma::smem_u32(tmem_slot), 512);
    umma::tmem_relinquish();
  }
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    int issued = 0;
    for (int i = 0; i < nch; ++i) {
      const int st = i % kDwRing;
      if (i >= kDwRing && !umma::mbar_wait(empty(st), ((i / kDwRing) - 1) & 1, A.wait_ns)) {
        atomicExch(A.err, kErrProducer);
        break;
      }
      const uint32_t sa = base + (uint32_t)(st * kDwStage);
      umma::mbar_arrive_expect_tx(full(st), (uint32_t)((4 + nbox) * kDwBox));
      for (int x = 0; x < 4; ++x) umma::tma_load_2d(sa + (uint32_t)(x * kDwBox), ma, full(st), 64 * x, r0 + 64 * i);
      for (int x = 0; x < nbox; ++x)
        umma::tma_load_2d(sa + (uint32_t)((4 + x) * kDwBox), mb, full(st), 64 * x, r0 + 64 * i);
      issued = i + 1;
    }
    for (int i = max(0, issued - kDwRing); i < issued; ++i) umma::mbar_wait(full(i % kDwRing), (i / kDwRing) & 1, kDrainNs);
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = umma::idesc_bf16_f32(128, N) | (1u << 15) | (1u << 16);  // A and B MN-major
    for (int i = 0; i < nch; ++i) {
      const int st = i % kDwRing;
      if (!umma::mbar_wait(full(st), (i / kDwRing) & 1, A.wait_ns)) {
        atomicExch(A.err, kErrMma);
        break;
      }
      umma::tc_fence_after();
      const uint32_t sa = base + (uint32_t)(st * kDwStage), sbb = sa + 4u * kDwBox;
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          umma::mma_bf16(tmem + 256u * h, mn_desc(sa + (uint32_t)(2 * h * kDwBox + 2048 * k)),
                         mn_desc(sbb + (uint32_t)(2048 * k)), idesc, (i > 0 || k > 0) ? 1u : 0u);
      umma::mma_commit(empty(st));
    }
    umma::mma_commit(done);
  }
  __syncwarp();
  const bool ok = umma::mbar_wait(done, 0, A.wait_ns);
  if (!ok) {
    atomicExch(A.err, kErrDone);
    umma::mbar_wait(done, 0, kDrainNs);
  }
  umma::tc_fence_after();
  if (warp >= 2) {
    // partials as [half][columns / 4][128 rows][4]: a warp stores 32 consecutive float4
    const int q = warp & 3;
    const int cols = l == 4 ? BHS_HEAD : N;
    float4* out = reinterpret_cast<float4*>(A.part[l]) + (int64_t)sp * (BHS_HIDDEN * cols / 4);
    for (int h = 0; h < 2; ++h) {
      const uint32_t t = tmem + 256u * h + ((uint32_t)(q * 32) << 16);
      for (int c = 0; c < cols; c += 16) {
        float v[16];
        tmem_ld16_nowait(t + (uint32_t)c, v);
        umma::tmem_wait_ld();
#pragma unroll
        for (int g = 0; g < 4; ++g)
          out[(int64_t)(h * (cols / 4) + c / 4 + g) * 128 + q * 32 + lane] =
              ok ? make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

// ---- gradient vector ---------------------------------------------------------------

struct CollectArgs {
  const float* part[BHS_LAYERS];
  const float* bias_part;
  float* grad;
  int splits, splits4;
  int bias_rows;  // B / 32
  int64_t w_off[BHS_LAYERS], b_off[BHS_LAYERS];
  int blocks[BHS_LAYERS + 1];  // first block of each layer, then of the biases
};

__global__ void __launch_bounds__(256) k_train_collect(const __grid_constant__ CollectArgs A) {
  __shared__ float red[8][33];
  if ((int)blockIdx.x >= A.blocks[BHS_LAYERS]) {  // biases: 32 columns, 8 groups of partial rows
    const int col = ((int)blockIdx.x - A.blocks[BHS_LAYERS]) * 32 + (threadIdx.x & 31), grp = threadIdx.x >> 5;
    float s = 0.0f;
    if (col < kBiases) {
#pragma unroll 8
      for (int i = grp; i < A.bias_rows; i += 8) s += A.bias_part[(int64_t)i * kBiases + col];
    }
    red[grp][threadIdx.x & 31] = s;
    __syncthreads();
    if (grp == 0 && col < kBiases) {
      for (int i = 1; i < 8; ++i) s += red[i][threadIdx.x];
      A.grad[A.b_off[col / BHS_HIDDEN] + col % BHS_HIDDEN] = s;
    }
    return;
  }
  int l = 0;
  while (l < BHS_LAYERS - 1 && (int)blockIdx.x >= A.blocks[l + 1]) ++l;
  const int cols = l == 4 ? BHS_HEAD : layer_k(l);
  const int n4 = BHS_HIDDEN * cols / 4;
  const int i = ((int)blockIdx.x - A.blocks[l]) * 256 + threadIdx.x;  // [half][cg][row]
  if (i >= n4) return;
  const float4* P = reinterpret_cast<const float4*>(A.part[l]) + i;
  const int splits = l == 4 ? A.splits4 : A.splits;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int sp = 0; sp < splits; ++sp) {
    const float4 v = P[(int64_t)sp * n4];
    s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
  }
  const int row = i & 127, hc = i >> 7, half = hc / (cols / 4), c4 = 4 * (hc - half * (cols / 4));
  const int m = half * 128 + row;
  float* g = A.grad + A.w_off[l];
  if (l == 4) {  // stored transposed
    g[(c4 + 0) * BHS_HIDDEN + m] = s.x;
    g[(c4 + 1) * BHS_HIDDEN + m] = s.y;
    g[(c4 + 2) * BHS_HIDDEN + m] = s.z;
    g[(c4 + 3) * BHS_HIDDEN + m] = s.w;
  } else {
    float* p = g + m * cols + c4;
    p[0] = s.x, p[1] = s.y, p[2] = s.z, p[3] = s.w;
  }
}

}  // namespace

extern "C" int bhs_train_splits(int layer, int64_t batch) {
  const int rows = layer == BHS_LAYERS - 1 ? 2 * kDwRows : kDwRows;
  return (int)((batch + rows - 1) / rows);
}

extern "C" int bhs_train_plan(const BhsTrainBuffers* b, int64_t batch, BhsTrainPlan* plan) {
  TrainMaps m;
  bool ok = true;
  for (int l = 0; l < BHS_LAYERS; ++l)
    ok = ok && make_map(&m.m[kMapW + l], b->wb[l], bhs_layer_n(l), bhs_layer_k(l), bhs_layer_k(l), bhs_layer_n(l));
  for (int l = 1; l < BHS_LAYERS; ++l) {
    const int n = l == BHS_LAYERS - 1 ? BHS_HEAD_PAD : BHS_HIDDEN;
    ok = ok && make_map(&m.m[kMapWT + l - 1], b->wt[l], BHS_HIDDEN, n, n, BHS_HIDDEN);
  }
  ok = ok && make_map(&m.m[kMapF], b->F, batch, BHS_FEATURES, BHS_FEATURES, 64);
  ok = ok && make_map(&m.m[kMapDout], b->dout, batch, BHS_HEAD_PAD, BHS_HEAD_PAD, 64);
  for (int l = 0; l < 4; ++l) {
    ok = ok && make_map(&m.m[kMapH + l], b->h[l], batch, BHS_HIDDEN, BHS_HIDDEN, 64);
    ok = ok && make_map(&m.m[kMapDY + l], b->dy[l], batch, BHS_HIDDEN, BHS_HIDDEN, 64);
  }
  if (!ok) {
    std::fprintf(stderr, "blackhole_b200: tensor map encoding failed\n");
    return -1;
  }
  std::memcpy(plan->maps, &m, sizeof(m));
  plan->batch = batch;
  return 0;
}

extern "C" int bhs_launch_train(const BhsTrainBuffers* b, const BhsTrainPlan* plan, const float* inputs,
                                const float* targets, float* grad, float* loss, int* d_err, uint64_t wait_ns,
                                cudaStream_t stream) {
  const int64_t B = plan->batch;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaFuncSetAttribute(k_train_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, kPassSmem) != cudaSuccess ||
      cudaFuncSetAttribute(k_train_dw, cudaFuncAttributeMaxDynamicSharedMemorySize, kDwSmem) != cudaSuccess)
    return -1;
  TrainMaps m;
  std::memcpy(&m, plan->maps, sizeof(m));
  PassArgs p{};
  p.in = inputs;
  p.targets = targets;
  p.targets16 = (reinterpret_cast<uintptr_t>(targets) & 15u) == 0 ? 1 : 0;
  p.params = b->params;
  p.dout = b->dout;
  for (int i = 0; i < 3; ++i) p.y[i] = b->y[i];
  p.bias_part = b->bias_part;
  p.loss = loss;
  p.B = B;
  p.err = d_err;
  p.wait_ns = wait_ns;
  for (int l = 0; l < BHS_LAYERS; ++l) p.bias_off[l] = bhs_bias_offset(l);
  k_train_pass<<<(unsigned)std::min<int64_t>(sms, B / kTile), kPassThreads, kPassSmem, stream>>>(m, p);
  if (cudaGetLastError() != cudaSuccess) return -1;

  DwArgs w{};
  CollectArgs c{};
  for (int l = 0; l < BHS_LAYERS; ++l) {
    w.part[l] = b->part[l];
    c.part[l] = b->part[l];
    c.w_off[l] = bhs_weight_offset(l);
    c.b_off[l] = bhs_bias_offset(l);
  }
  w.B = B;
  w.splits = bhs_train_splits(0, B);
  w.err = d_err;
  w.wait_ns = wait_ns;
  const int splits4 = bhs_train_splits(BHS_LAYERS - 1, B);
  k_train_dw<<<(unsigned)(4 * w.splits + splits4), kDwThreads, kDwSmem, stream>>>(m, w);
  if (cudaGetLastError() != cudaSuccess) return -1;

  c.bias_part = b->bias_part;
  c.grad = grad;
  c.splits = w.splits;
  c.splits4 = splits4;
  c.bias_rows = (int)(B / 32);
  int blocks = 0;
  for (int l = 0; l < BHS_LAYERS; ++l) {
    c.blocks[l] = blocks;
    const int cols = l == BHS_LAYERS - 1 ? BHS_HEAD : bhs_layer_k(l);
    blocks += (BHS_HIDDEN * cols / 4 + 255) / 256;
  }
  c.blocks[BHS_LAYERS] = blocks;
  blocks += (kBiases + 31) / 32;
  k_train_collect<<<(unsigned)blocks, 256, 0, stream>>>(c);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
