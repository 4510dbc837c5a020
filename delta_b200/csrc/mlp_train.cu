// mlp_train.cu -- one training step of the warm-start network in two kernels: forward,
// loss and gradients of a batch on the tensor cores (tcgen05), then the sum of the CTAs'
// gradients with Adam.
//
// The step's least traffic is its rows (81 bytes each); layer by layer it moved the
// activations, pre-activations and their gradients through memory (about 7 KB a row, 27
// launches).  Here a tile of 128 rows stays on its SM from the features to the weight
// gradients:
//
// - shared memory holds the weights, the tile's features, the three hidden activations
//   (BF16), the gradient of one pre-activation (BF16) and of the output (BF16).  One copy
//   of each serves every product: the canonical layout without swizzle (8 x 8 core matrices)
//   is K-major along the columns and MN-major along the rows, so dW = dZ^T H and dH = dZ W
//   read the forward tiles with the transpose bits of the instruction descriptor;
// - TMEM (512 columns, FP32) holds dW3 and dW2 over all of the CTA's tiles (128 columns
//   each), one layer's pre-activation and one layer's dH.  Pre-activations are not kept:
//   the backward pass runs Z2 = H1 W2^T and Z1 = X W1^T again (the same MMAs, the same bits);
// - dW1 (32 columns) and dW4 (16) are formed per tile and added up in registers, and the
//   bias gradients are column sums of the BF16 tiles, taken while the MMAs run.
//
// Rounding: activations and their gradients are BF16 where the layer-by-layer path rounds
// them, everything else FP32.  The partial gradients of the CTAs are added in a fixed order.
// Bound by the chain of a tile (seven MMA groups, each followed by its epilogue: 768 GELU
// and GELU' a row).  Batch 65,536: 442 us a step layer by layer, 72 us now.
#include <cuda_bf16.h>

#include <algorithm>

#include "internal.h"
#include "mlp.cuh"

namespace delta {

namespace {

constexpr int kTrThreads = 512;  // warp w: TMEM lanes (rows) 32 (w % 4).., columns 32 (w / 4)..
constexpr int64_t kPartStride = kNumParams + 8;  // a CTA's gradients, then its loss

struct TrainSmem {
  __nv_bfloat16 w1[kHid * kIn];        // [out][in] tiles, as k_mlp_infer_tc's
  __nv_bfloat16 w2[kHid * kHid];
  __nv_bfloat16 w3[kHid * kHid];
  __nv_bfloat16 w4[kTcW4Rows * kHid];  // rows 4..15 zero
  __nv_bfloat16 x[2][kTcRows * kIn];   // [row][feature]; the tile at work and the next one
  __nv_bfloat16 h[3][kTcRows * kHid];  // [row][unit]
  __nv_bfloat16 dz[kTcRows * kHid];    // [row][unit]
  __nv_bfloat16 dy[kTcRows * kTcW4Rows];  // [row][output]; columns 4..15 zero
  float bias[3 * kHid + 8];
  uint64_t mbar;
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(TrainSmem) <= 227 * 1024, "one CTA per SM");

// TMEM columns
constexpr uint32_t kColDW3 = 0, kColDW2 = 128, kColZ = 256, kColD = 384;
constexpr uint32_t kColDW1 = kColD, kColDW4 = kColD + 32, kColY = kColD + 64;

// Operand descriptors.  K-major: 8-row groups `16 K` bytes apart, 8-column groups 128 bytes
// apart.  MN-major (the same tile read along its rows): the leading offset is between 8-row
// groups (K), the stride between 8-column groups (M or N).
__device__ __forceinline__ uint64_t tc_desc_mn(uint32_t smem_addr, uint32_t lbo) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
}
constexpr uint32_t kTransA = 1u << 15, kTransB = 1u << 16;

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// D[128 rows][N] (+)= A[128][K] B[N][K]^T, both K-major tiles
__device__ __forceinline__ void mma_kk(uint32_t d, const void *A, const void *B, int K, int N) {
  const uint32_t a0 = saddr(A), b0 = saddr(B);
  for (int s = 0; s < K / 16; ++s)
    tc_mma(d, tc_desc(a0 + 256u * s, 16u * K), tc_desc(b0 + 256u * s, 16u * K), tc_idesc(kTcRows, N), s > 0);
}
// D[128 rows][N] = A[128][K] W[K][N]: A a K-major tile, W a tile of K rows and N columns
__device__ __forceinline__ void mma_kn(uint32_t d, const void *A, const void *W, int K, int N) {
  const uint32_t a0 = saddr(A), b0 = saddr(W);
  for (int s = 0; s < K / 16; ++s)
    tc_mma(d, tc_desc(a0 + 256u * s, 16u * K), tc_desc_mn(b0 + 2u * 16u * N * s, 16u * N),
           tc_idesc(kTcRows, N) | kTransB, s > 0);
}
// D[128][N] (+)= A^T B over the tile's 128 rows: A a tile of 128 columns, B one of N columns
__device__ __forceinline__ void mma_tn(uint32_t d, const void *A, const void *B, int N, bool accumulate) {
  const uint32_t a0 = saddr(A), b0 = saddr(B);
  for (int s = 0; s < kTcRows / 16; ++s)
    tc_mma(d, tc_desc_mn(a0 + 2u * 16u * kHid * s, 16u * kHid), tc_desc_mn(b0 + 2u * 16u * N * s, 16u * N),
           tc_idesc(kHid, N) | kTransA | kTransB, accumulate || s > 0);
}

__device__ __forceinline__ void tc_ld8(uint32_t taddr, float v[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = __uint_as_float(r[k]);
}

// Makes the CTA's shared-memory stores and TMEM reads visible to the MMAs that follow.
__device__ __forceinline__ void tr_publish() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Waits (bounded) for everything thread 0 has issued and committed; false on time-out.
// (`phase` is thread 0's.)
__device__ __forceinline__ bool tr_wait(TrainSmem &sm, TcPhase &phase) {
  if (threadIdx.x == 0 && !phase.wait([&](uint32_t parity) { return tc_wait(&sm.mbar, parity, kTcSpin); })) sm.abort = 1;
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return sm.abort == 0;
}

// H = bf16(gelu(Z + b)) of this thread's 32 columns of its row
__device__ __forceinline__ void epilogue_forward(uint32_t tz, const float *bias, int r, int c0, __nv_bfloat16 *h) {
  float v[32];
  tc_ld32(tz + (uint32_t)c0, v);
  char *dst = reinterpret_cast<char *>(h);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      w[k] = pack_bf16(gelu2(__fadd2_rn(make_float2(v[8 * q + 2 * k], v[8 * q + 2 * k + 1]),
                                        *reinterpret_cast<const float2 *>(bias + c0 + 8 * q + 2 * k))));
    *reinterpret_cast<uint4 *>(dst + tc_chunk(r, c0 / 8 + q, kHid)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// dZ = bf16(dH gelu'(Z + b)) of this thread's 32 columns of its row
__device__ __forceinline__ void epilogue_backward(uint32_t td, uint32_t tz, const float *bias, int r, int c0,
                                                  __nv_bfloat16 *dz) {
  char *dst = reinterpret_cast<char *>(dz);
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float d[16], z[16];
    const int c = c0 + 16 * p;
    tc_ld16(td + (uint32_t)c, d);
    tc_ld16(tz + (uint32_t)c, z);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int j = 8 * q + 2 * k;
        w[k] = pack_bf16(__fmul2_rn(make_float2(d[j], d[j + 1]),
                                    gelu_grad2(__fadd2_rn(make_float2(z[j], z[j + 1]),
                                                          *reinterpret_cast<const float2 *>(bias + c + j)))));
      }
      *reinterpret_cast<uint4 *>(dst + tc_chunk(r, c / 8 + q, kHid)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// Adds the columns of the dZ tile: this thread 8 columns (chunk (tid / 8) % 16) of the rows
// = tid (mod 8) of 4 of the 16 row groups; 8 threads read 128 contiguous bytes.
__device__ __forceinline__ void column_sums(const __nv_bfloat16 *dz, float s[8]) {
  const int r8 = threadIdx.x & 7, kc = (threadIdx.x >> 3) & 15, grp = threadIdx.x >> 7;
  const char *src = reinterpret_cast<const char *>(dz);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint4 v = *reinterpret_cast<const uint4 *>(src + tc_chunk(8 * (grp + 4 * g) + r8, kc, kHid));
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s[2 * k] += __uint_as_float(w[k] << 16);
      s[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
    }
  }
}

__global__ void __launch_bounds__(kTrThreads, 1)
    k_train_grad(int64_t M, const __nv_bfloat16 *__restrict__ X, const float *__restrict__ T,
                 const uint8_t *__restrict__ valid, float inv_n, const float *__restrict__ params,
                 const __nv_bfloat16 *__restrict__ wb, float *__restrict__ part, int *__restrict__ err) {
  extern __shared__ __align__(128) unsigned char tr_smem_raw[];
  TrainSmem &sm = *reinterpret_cast<TrainSmem *>(tr_smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t tiles = (M + kTcRows - 1) / kTcRows;
  // a feature chunk (16 of a row's 64 bytes) per thread; zero past the last row
  auto feature_chunk = [&](int64_t tile) {
    const int64_t row = tile * kTcRows + (tid >> 2);
    return tile < tiles && row < M ? __ldg(reinterpret_cast<const uint4 *>(X + kIn * row) + (tid & 3))
                                   : make_uint4(0u, 0u, 0u, 0u);
  };
  auto store_chunk = [&](__nv_bfloat16 *x, uint4 v) {
    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(x) + tc_chunk(tid >> 2, tid & 3, kIn)) = v;
  };
  const uint4 first = feature_chunk(blockIdx.x);
  tc_stage(sm.w1, wb + kOffW1, kHid, kHid, kIn);
  tc_stage(sm.w2, wb + kOffW2, kHid, kHid, kHid);
  tc_stage(sm.w3, wb + kOffW3, kHid, kHid, kHid);
  tc_stage(sm.w4, wb + kOffW4, kTcW4Rows, kOut, kHid);
  for (int e = tid; e < kHid; e += kTrThreads) {
    sm.bias[e] = params[kOffB1 + e];
    sm.bias[kHid + e] = params[kOffB2 + e];
    sm.bias[2 * kHid + e] = params[kOffB3 + e];
  }
  if (tid < kOut) sm.bias[3 * kHid + tid] = params[kOffB4 + tid];
  store_chunk(sm.x[0], first);
  if (tid < kTcRows * kTcW4Rows / 8)
    *reinterpret_cast<uint4 *>(reinterpret_cast<char *>(sm.dy) + 16 * tid) = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    sm.abort = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&sm.mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&sm.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tr_publish();
  const uint32_t tmem = sm.tmem_base;
  const int r = (warp & 3) * 32 + lane, part_c = warp >> 2, c0 = 32 * part_c;
  const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  TcPhase phase;
  float db[3][8] = {}, dw1[8] = {}, dw4[4] = {}, db4[4] = {}, loss = 0.f;
  // the last tile's dW1 (8 columns a thread) and dW4 (threads of the first 4 warps)
  auto add_small = [&]() {
    float v[8];
    tc_ld8(tlane + kColDW1 + 8u * part_c, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) dw1[k] += v[k];
    if (part_c == 0) {
      tc_ld8(tlane + kColDW4, v);
#pragma unroll
      for (int k = 0; k < kOut; ++k) dw4[k] += v[k];
    }
  };
  bool ok = true;
  int it = 0;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
    const __nv_bfloat16 *x = sm.x[it & 1];
    const uint4 next = feature_chunk(tile + gridDim.x);
    const int64_t row = tile * kTcRows + r;
    const bool live = part_c == 0 && row < M && valid[row] != 0;
    const float4 t4 = live ? __ldg(reinterpret_cast<const float4 *>(T) + row) : make_float4(0.f, 0.f, 0.f, 0.f);
    // forward
    tr_publish();
    if (tid == 0) {
      mma_kk(tmem + kColZ, x, sm.w1, kIn, kHid);
      tc_commit(&sm.mbar);
    }
    if (!(ok = tr_wait(sm, phase))) break;
    if (it > 0) add_small();
    epilogue_forward(tlane + kColZ, sm.bias, r, c0, sm.h[0]);
    tr_publish();
    if (tid == 0) {
      mma_kk(tmem + kColZ, sm.h[0], sm.w2, kHid, kHid);
      tc_commit(&sm.mbar);
    }
    if (!(ok = tr_wait(sm, phase))) break;
    epilogue_forward(tlane + kColZ, sm.bias + kHid, r, c0, sm.h[1]);
    tr_publish();
    if (tid == 0) {
      mma_kk(tmem + kColZ, sm.h[1], sm.w3, kHid, kHid);
      tc_commit(&sm.mbar);
    }
    if (!(ok = tr_wait(sm, phase))) break;
    epilogue_forward(tlane + kColZ, sm.bias + 2 * kHid, r, c0, sm.h[2]);
    tr_publish();
    if (tid == 0) {
      mma_kk(tmem + kColY, sm.h[2], sm.w4, kHid, kTcW4Rows);
      tc_commit(&sm.mbar);
    }
    if (!(ok = tr_wait(sm, phase))) break;
    // dY = bf16(2 (Y - T) / n) and the loss, one row per thread of the first 4 warps
    if (part_c == 0) {
      float y[8];
      tc_ld8(tlane + kColY, y);
      const float t[4] = {t4.x, t4.y, t4.z, t4.w};
      float g[4];
#pragma unroll
      for (int k = 0; k < kOut; ++k) {
        const float d = live ? (y[k] + sm.bias[3 * kHid + k]) - t[k] : 0.f;
        const __nv_bfloat16 b = __float2bfloat16(2.f * d * inv_n);
        g[k] = __bfloat162float(b);
        db4[k] += g[k];
        loss += d * d * inv_n;
      }
      *reinterpret_cast<uint2 *>(reinterpret_cast<char *>(sm.dy) + tc_chunk(r, 0, kTcW4Rows)) =
          make_uint2(pack_bf16(g[0], g[1]), pack_bf16(g[2], g[3]));
    }
    // backward: layer 4, 3, 2, 1
    tr_publish();
    if (tid == 0) {
      mma_kn(tmem + kColD, sm.dy, sm.w4, kTcW4Rows, kHid);
      tc_commit(&sm.mbar);
    }
    if (!(ok = tr_wait(sm, phase))) break;
    epilogue_backward(tlane + kColD, tlane + kColZ, sm.bias + 2 * kHid, r, c0, sm.dz);
    tr_publish();
    if (tid == 0) {
      mma_kn(tmem + kColD, sm.dz, sm.w3, kHid, kHid);
      mma_kk(tmem + kColZ, sm.h[0], sm.w2, kHid, kHid);
      mma_tn(tmem + kColDW3, sm.dz, sm.h[1], kHid, it > 0);
      tc_commit(&sm.mbar);
    }
    column_sums(sm.dz, db[2]);
    if (!(ok = tr_wait(sm, phase))) break;
    epilogue_backward(tlane + kColD, tlane + kColZ, sm.bias + kHid, r, c0, sm.dz);
    tr_publish();
    if (tid == 0) {
      mma_kn(tmem + kColD, sm.dz, sm.w2, kHid, kHid);
      mma_kk(tmem + kColZ, x, sm.w1, kIn, kHid);
      mma_tn(tmem + kColDW2, sm.dz, sm.h[0], kHid, it > 0);
      tc_commit(&sm.mbar);
    }
    column_sums(sm.dz, db[1]);
    if (!(ok = tr_wait(sm, phase))) break;
    epilogue_backward(tlane + kColD, tlane + kColZ, sm.bias, r, c0, sm.dz);
    store_chunk(sm.x[(it + 1) & 1], next);
    tr_publish();
    // (waited for with the next tile's first layer, or below)
    if (tid == 0) {
      mma_tn(tmem + kColDW1, sm.dz, x, kIn, false);
      mma_tn(tmem + kColDW4, sm.h[2], sm.dy, kTcW4Rows, false);
    }
    column_sums(sm.dz, db[0]);
  }
  // the last tile's products
  if (ok) {
    __syncthreads();
    if (tid == 0) tc_commit(&sm.mbar);
    ok = tr_wait(sm, phase);
  }
  // after a time-out thread 0 waits once more, bounded, for the commit that was late (it
  // tracks every MMA issued before it): nothing is in flight when the TMEM is freed, unless
  // that wait runs out too, which the flag reports
  if (!ok && tid == 0) {
    const bool drained = phase.drain([&](uint32_t parity) { return tc_wait(&sm.mbar, parity, kTcSpin); });
    atomicMax(err, drained ? kTcLate : kTcLost);
  }
  float *out = part + (int64_t)blockIdx.x * kPartStride;
  if (ok) {
    add_small();
    float v[32];
    float4 *o3 = reinterpret_cast<float4 *>(out + kOffW3 + kHid * r + c0);
    tc_ld32(tlane + kColDW3 + (uint32_t)c0, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) o3[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    float4 *o2 = reinterpret_cast<float4 *>(out + kOffW2 + kHid * r + c0);
    tc_ld32(tlane + kColDW2 + (uint32_t)c0, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) o2[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    float4 *o1 = reinterpret_cast<float4 *>(out + kOffW1 + kIn * r + 8 * part_c);
    o1[0] = make_float4(dw1[0], dw1[1], dw1[2], dw1[3]);
    o1[1] = make_float4(dw1[4], dw1[5], dw1[6], dw1[7]);
    if (part_c == 0)
      for (int k = 0; k < kOut; ++k) out[kOffW4 + kHid * k + r] = dw4[k];
    // bias gradients and the loss: sums over the threads of a column, through the (now idle)
    // activation tiles
    float *red = reinterpret_cast<float *>(sm.h[0]);
#pragma unroll
    for (int l = 0; l < 3; ++l)
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float s = db[l][k];
        for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((tid & 7) == 0) red[((tid >> 7) * 3 + l) * kHid + 8 * ((tid >> 3) & 15) + k] = s;
      }
    float *red4 = red + 12 * kHid;
    if (part_c == 0) {
      float s[5] = {db4[0], db4[1], db4[2], db4[3], loss};
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        if (lane == 0) red4[5 * warp + k] = s[k];
      }
    }
    __syncthreads();
    const int64_t off[3] = {kOffB1, kOffB2, kOffB3};
    if (tid < 3 * kHid) {
      const int l = tid / kHid, c = tid % kHid;
      float s = 0.f;
      for (int g = 0; g < 4; ++g) s += red[(g * 3 + l) * kHid + c];
      out[off[l] + c] = s;
    } else if (tid < 3 * kHid + 5) {
      const int k = tid - 3 * kHid;
      float s = 0.f;
      for (int w = 0; w < 4; ++w) s += red4[5 * w + k];
      out[k < kOut ? kOffB4 + k : kNumParams] = s;
    }
  } else {
    for (int64_t e = tid; e < kPartStride; e += kTrThreads) out[e] = __int_as_float(0x7fc00000);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// grads = the CTAs' partial gradients added in order (a block of 8 warps takes 32 consecutive
// parameters, warp w adds CTAs w, w + 8, ..., warp 0 the 8 sums), the loss likewise, then
// Adam on the 32 parameters (k_adam's update).  Bound by reading the partials from L2.
__global__ void __launch_bounds__(256) k_train_update(int ctas, const float *__restrict__ part, float *w, float *g,
                                                      float *m, float *v, float lr, float b1, float b2, float eps,
                                                      float c1, float c2, __nv_bfloat16 *wb, float *loss) {
  __shared__ float ws[8][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  const bool pad = i >= kOffB4 + kOut && i < kNumParams;  // never written by a CTA
  float s = 0.f;
  if (i <= kNumParams && !pad)
    for (int j = wid; j < ctas; j += 8) s += part[j * kPartStride + i];
  ws[wid][lane] = s;
  __syncthreads();
  if (wid != 0 || i > kNumParams) return;
  float t = ws[0][lane];
#pragma unroll
  for (int k = 1; k < 8; ++k) t += ws[k][lane];
  if (i == kNumParams) {
    *loss = t;
    return;
  }
  g[i] = t;
  adam_update(i, t, w, m, v, lr, b1, b2, eps, c1, c2, wb);
}

}  // namespace

}  // namespace delta

using namespace delta;

extern "C" delta_status delta_mlp_train_step(delta_ctx *ctx, int64_t M, const void *X_bf16, const float *T,
                                             const uint8_t *valid, float inv_n, float *w, void *w_bf16, float *g,
                                             float *m, float *v, float lr, float b1, float b2, float eps,
                                             int64_t step, float *loss) {
  if (!ctx || M <= 0 || !X_bf16 || !T || !valid || !w || !w_bf16 || !g || !m || !v || !loss || step < 1)
    return set_error(DELTA_ERR_INVALID, "delta_mlp_train_step: bad argument");
  if (((reinterpret_cast<uintptr_t>(X_bf16) | reinterpret_cast<uintptr_t>(T) | reinterpret_cast<uintptr_t>(w_bf16)) & 15))
    return set_error(DELTA_ERR_INVALID, "delta_mlp_train_step: X, T and w_bf16 must be 16-byte aligned");
  if (ctx->mlp_engine != DELTA_MLP_TCGEN05)
    return set_error(DELTA_ERR_UNSUPPORTED, "delta_mlp_train_step: built for the tcgen05 engine");
  cudaError_t e;
  if (!ctx->gemm_err) {
    if ((e = cudaMalloc(&ctx->gemm_err, sizeof(int))) != cudaSuccess) return cuda_error(e, "train flag");
    if ((e = cudaMemsetAsync(ctx->gemm_err, 0, sizeof(int), ctx->stream)) != cudaSuccess)
      return cuda_error(e, "train flag");
  }
  const int ctas = (int)std::min<int64_t>((M + kTcRows - 1) / kTcRows, kNumSMs);
  void *buf;
  delta_status st = ctx_scratch(ctx, 28, sizeof(float) * (size_t)ctas * kPartStride, &buf);
  if (st != DELTA_OK) return st;
  static thread_local int configured_device = -1;
  if (configured_device != ctx->device) {
    e = cudaFuncSetAttribute(k_train_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem));
    if (e != cudaSuccess) return cuda_error(e, "train shared memory");
    configured_device = ctx->device;
  }
  float *part = static_cast<float *>(buf);
  k_train_grad<<<ctas, kTrThreads, sizeof(TrainSmem), ctx->stream>>>(
      M, (const __nv_bfloat16 *)X_bf16, T, valid, inv_n, w, (const __nv_bfloat16 *)w_bf16, part, ctx->gemm_err);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_error(e, "train gradients");
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_train_update<<<(unsigned)((kNumParams + 1 + 31) / 32), 256, 0, ctx->stream>>>(
      ctas, part, w, g, m, v, lr, b1, b2, eps, c1, c2, (__nv_bfloat16 *)w_bf16, loss);
  ctx->launches += 2;
  return cuda_error(cudaGetLastError(), "train update");
}
