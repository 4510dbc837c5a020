// mlp.cuh -- what the warm-start network's kernels share: its parameter layout, GELU, and
// the tcgen05 building blocks (descriptors, MMA issue, commit and bounded wait, TMEM loads).
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

#include "tcphase.h"

namespace delta {

namespace {

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __halves2bfloat162(__float2bfloat16(lo), __float2bfloat16(hi));
  return *reinterpret_cast<const uint32_t *>(&v);
}

// GELU, tanh form (Hendrycks & Gimpel 2016), with the hardware tanh (tanh.approx.f32,
// relative error about 2^-11, below the BF16 rounding that follows).
__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kGeluK = 0.7978845608028654f;  // sqrt(2/pi)
constexpr float kGeluC = 0.044715f;
__device__ __forceinline__ float gelu(float x) {
  const float u = x * fmaf(kGeluC * kGeluK, x * x, kGeluK);
  const float h = 0.5f * x;
  return fmaf(h, tanh_hw(u), h);
}
__device__ __forceinline__ float gelu_grad(float x) {
  const float x2 = x * x;
  const float th = tanh_hw(x * fmaf(kGeluC * kGeluK, x2, kGeluK));
  const float sech2 = fmaf(-th, th, 1.f);
  const float q = 0.5f * x * sech2 * kGeluK * fmaf(3.f * kGeluC, x2, 1.f);
  return fmaf(0.5f, 1.f + th, q);
}

// gelu and gelu_grad of two values with the packed FP32 operations of sm_100 (one issue slot
// for both), the same operations in the same order: every multiply-add is written out in both
// forms, so each lane rounds as the scalar form does.  The tcgen05 kernels' epilogues are
// bound by issue slots and the tanh unit.
__device__ __forceinline__ float2 splat2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 gelu2(float2 x) {
  const float2 u = __fmul2_rn(x, __ffma2_rn(splat2(kGeluC * kGeluK), __fmul2_rn(x, x), splat2(kGeluK)));
  const float2 h = __fmul2_rn(splat2(0.5f), x);
  return __ffma2_rn(h, make_float2(tanh_hw(u.x), tanh_hw(u.y)), h);
}
__device__ __forceinline__ float2 gelu_grad2(float2 x) {
  const float2 x2 = __fmul2_rn(x, x);
  const float2 u = __fmul2_rn(x, __ffma2_rn(splat2(kGeluC * kGeluK), x2, splat2(kGeluK)));
  const float2 th = make_float2(tanh_hw(u.x), tanh_hw(u.y));
  const float2 sech2 = __ffma2_rn(make_float2(-th.x, -th.y), th, splat2(1.f));
  const float2 p = __fmul2_rn(__fmul2_rn(__fmul2_rn(splat2(0.5f), x), sech2), splat2(kGeluK));
  const float2 q = __fmul2_rn(p, __ffma2_rn(splat2(3.f * kGeluC), x2, splat2(1.f)));
  return __ffma2_rn(splat2(0.5f), __fadd2_rn(splat2(1.f), th), q);
}
__device__ __forceinline__ uint32_t pack_bf16(float2 v) { return pack_bf16(v.x, v.y); }

// Adam (Kingma & Ba 2015) on FP32 master weight i with gradient gi; refreshes the BF16 copy.
__device__ __forceinline__ void adam_update(int64_t i, float gi, float *w, float *m, float *v, float lr, float b1,
                                            float b2, float eps, float c1, float c2, __nv_bfloat16 *wb) {
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] = wi;
  if (wb) wb[i] = __float2bfloat16(wi);
}

// parameter layout: 32 (18 used) -> 128 -> 128 -> 128 -> 4
constexpr int kIn = 32, kHid = 128, kOut = 4;
constexpr int64_t kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
                  kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kHid, kOffW4 = kOffB3 + kHid,
                  kOffB4 = kOffW4 + kOut * kHid, kNumParams = (kOffB4 + kOut + 7) / 8 * 8;
constexpr int kTcRows = 128;          // pairs per tile = MMA M
constexpr uint32_t kTmemCols = 128;   // FP32 accumulator columns (N of the hidden layers)
constexpr int kTcW4Rows = 16;         // W4 padded to N = 16
constexpr uint32_t kTcSpin = 1u << 22;  // mbarrier polls before giving up

// byte offset of the 16-byte chunk (row r, k-chunk kc) in a canonical K-major tile
__device__ __forceinline__ uint32_t tc_chunk(int r, int kc, int K) {
  return (uint32_t)((r >> 3) * (16 * K) + kc * 128 + (r & 7) * 16);
}

__device__ __forceinline__ uint64_t tc_desc(uint32_t smem_addr, uint32_t sbo) {
  // start address >> 4 [0,14), LBO >> 4 [16,30) = 128 B, SBO >> 4 [32,46), version 1 at
  // bit 46, base offset 0, no swizzle
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: F32 accumulator, BF16 A and B, both K-major, M x N
__host__ __device__ constexpr uint32_t tc_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void tc_commit(uint64_t *mbar) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(mbar);
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(a) : "memory");
}

// bounded wait for the mbarrier phase with parity `phase`; false on time-out
__device__ __forceinline__ bool tc_wait(uint64_t *mbar, uint32_t phase, uint32_t spin) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(mbar);
  for (uint32_t it = 0; it < spin; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// 32 consecutive FP32 accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float v[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// copy a row-major [rows][K] BF16 matrix (global, 16-byte aligned rows) into the canonical
// layout; rows at or beyond `valid_rows` are zero
__device__ __forceinline__ void tc_stage(__nv_bfloat16 *dst, const __nv_bfloat16 *src, int rows, int valid_rows,
                                         int K) {
  const int chunks = K / 8;
  for (int e = threadIdx.x; e < rows * chunks; e += blockDim.x) {
    const int r = e / chunks, kc = e % chunks;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (r < valid_rows) v = __ldg(reinterpret_cast<const uint4 *>(src + (size_t)r * K + kc * 8));
    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(dst) + tc_chunk(r, kc, K)) = v;
  }
}

}  // namespace

}  // namespace delta
