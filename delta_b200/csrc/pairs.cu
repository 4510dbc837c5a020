// pairs.cu -- pair-list narrowphase kernels (one thread per triangle pair).
//
// Input planes a[9*ld], b[9*ld] (plane 3*vertex+coord), outputs p[3*ld], q[3*ld],
// dist[n], flags[n].  Every warp reads 18 consecutive 256-byte segments, one per plane,
// and writes 7 more, so the loads and stores are fully coalesced.  Replaces the
// per-pair loops of bf()/penalty() (bf.cpp:95-118, penalty.cpp:187-210) and the SIMD
// pair-list kernels ispc_bf / ispc_pen (bf.ispc:3, penalty.ispc:154).
#include <type_traits>

#include "internal.h"
#include "tri_bf64.cuh"
#include "tri_cert.cuh"
#include "tri_gjk.cuh"
#include "tri_ref.cuh"

namespace delta {

enum { M_BF = 0, M_PENALTY = 1, M_PENALTY_ITER = 2, M_GJK = 3, M_HYBRID_PAIR = 4, M_BF_CERT = 5 };

// Launch bounds of the pair kernel: FP64 GJK is held to 128 registers (2^22 pairs: 1.29 ms
// unbounded, 1.02 at 3 blocks, 1.00 at 4, 1.11 at 5).  The FP64 penalty kernels are bound by the FP64 pipe (44 divisions a pair) once enough warps are
// resident: unbounded (144-176 registers) one block of 256 fitted an SM.  2^22 pairs,
// before / 2 / 3 / 4 / 5 blocks of 128 per SM: penalty 549 / 412 / 412 / 381 / 415 us,
// adaptive penalty 693 / 520 / 520 / 493 / 513, hybrid 551 / 529 / 416 / 433 / 559.  The
// FP32 kernels keep their registers.
template <class R, int M>
struct PairBounds {
  static constexpr int kThreads = 256, kMinBlocks = 1;
};
template <>
struct PairBounds<xf64, M_PENALTY> {
  static constexpr int kThreads = 128, kMinBlocks = 4;
};
template <>
struct PairBounds<xf64, M_PENALTY_ITER> {
  static constexpr int kThreads = 128, kMinBlocks = 4;
};
template <>
struct PairBounds<xf64, M_HYBRID_PAIR> {
  static constexpr int kThreads = 128, kMinBlocks = 3;
};
template <>
struct PairBounds<xf64, M_GJK> {
  static constexpr int kThreads = 128, kMinBlocks = 4;
};

// A warp walks the list 32 pairs at a time and meets at __syncwarp after each group: the
// lanes of a divergent solver would otherwise drift apart over the iterations of a
// grid-stride loop and run as several partial warps (measured: 4x slower when each
// thread takes ~50 pairs).
template <class R, int M>
__global__ void __launch_bounds__(PairBounds<R, M>::kThreads, PairBounds<R, M>::kMinBlocks)
    k_pairs(int64_t n, const double *__restrict__ a, const double *__restrict__ b, int64_t ld, double max_error,
            double *__restrict__ p, double *__restrict__ q, double *__restrict__ dist, uint8_t *__restrict__ flags) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
    const int64_t i = base + lane;
    if (i >= n) {
      __syncwarp();
      continue;
    }
    R A[3][3], B[3][3];
#pragma unroll
    for (int v = 0; v < 3; ++v)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        A[v][k] = from_f64<R>(__ldg(a + (3 * v + k) * ld + i));
        B[v][k] = from_f64<R>(__ldg(b + (3 * v + k) * ld + i));
      }
    R pq[6];
    int flag = 0;
    const R me = from_f64<R>(max_error);
    if constexpr (M == M_BF) {
      bf_solve_lean(A, B, pq);
    } else if constexpr (M == M_PENALTY) {
      penalty_ref(A, B, me, false, pq, flag);
    } else if constexpr (M == M_PENALTY_ITER) {
      penalty_ref(A, B, me, true, pq, flag);
    } else if constexpr (M == M_GJK) {
      gjk_ref(A, B, pq);
    } else {  // per-pair hybrid: penalty, bf when the pair reports failure
      penalty_ref(A, B, me, false, pq, flag);
      if (flag) bf_solve_lean(A, B, pq);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      p[k * ld + i] = to_f64(pq[k]);
      q[k * ld + i] = to_f64(pq[3 + k]);
    }
    dist[i] = to_f64(pq_distance(pq));
    if (flags) flags[i] = (uint8_t)flag;
    __syncwarp();
  }
}

// The points pq and distance of FP64 bf's pair i, to the pair list's outputs.
__device__ __forceinline__ void bf64_write(const xf64 pq[6], int64_t i, int64_t ld, double *p, double *q, double *dist,
                                           uint8_t *flags) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    p[k * ld + i] = pq[k].v;
    q[k * ld + i] = pq[3 + k].v;
  }
  dist[i] = pq_distance(pq).v;
  if (flags) flags[i] = 0;
}

// A thread per pair, 8 blocks of 128 per SM (64 registers).  Bound by the FP64 pipe and the
// lanes' divergence: 2^22 pairs 1083 us before, 744 now (762 when 92 registers took 808 and
// 48 took 859).
constexpr int kBfThreads = 128;
__global__ void __launch_bounds__(kBfThreads, 8)
    k_pairs_bf64(int64_t n, const double *__restrict__ a, const double *__restrict__ b, int64_t ld,
                 double *__restrict__ p, double *__restrict__ q, double *__restrict__ dist,
                 uint8_t *__restrict__ flags) {
  __shared__ BfTile<kBfThreads> tile;
  const int col = threadIdx.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = base + col;
    if (i < n) {
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        tile.v[k][col] = __ldg(a + k * ld + i);
        tile.v[9 + k][col] = __ldg(b + k * ld + i);
      }
      xf64 pq[6];
      tile.solve(col, pq);
      bf64_write(pq, i, ld, p, q, dist, flags);
    }
    __syncwarp();
  }
}

// Short lists: five warps to 32 pairs (a lane per pair), warps 0..2 one edge of A each,
// warps 3..4 one face each; then the first warp takes the minima in the same order.  A
// pair's chain of 15 dependent evaluations shrinks to 3.
constexpr int kBfSplitWarps = 5;
__global__ void __launch_bounds__(32 * kBfSplitWarps, 6)
    k_pairs_bf64_split(int64_t n, const double *__restrict__ a, const double *__restrict__ b, int64_t ld,
                       double *__restrict__ p, double *__restrict__ q, double *__restrict__ dist,
                       uint8_t *__restrict__ flags) {
  __shared__ BfTile<32> tile;
  __shared__ double s_d[kBfSplitWarps][32], s_p0[kBfSplitWarps][32], s_p1[kBfSplitWarps][32];
  __shared__ uint8_t s_id[kBfSplitWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t base = (int64_t)blockIdx.x * 32; base < n; base += (int64_t)gridDim.x * 32) {
    const int64_t i = base + lane, ii = i < n ? i : n - 1;
    for (int k = w; k < 18; k += kBfSplitWarps)
      tile.v[k][lane] = k < 9 ? __ldg(a + k * ld + ii) : __ldg(b + (k - 9) * ld + ii);
    __syncthreads();
    BfBest best;
    best.start();
    if (w < 3) tile.edges(w, lane, best);
    else tile.faces(w - 3, lane, best);
    s_d[w][lane] = best.d.v;
    s_p0[w][lane] = best.p0.v;
    s_p1[w][lane] = best.p1.v;
    s_id[w][lane] = (uint8_t)best.id;
    __syncthreads();
    if (w == 0 && i < n) {
      BfBest e, f;
      e.start();
      f.start();
#pragma unroll
      for (int g = 0; g < 3; ++g) e.take(xf64(s_d[g][lane]), xf64(s_p0[g][lane]), xf64(s_p1[g][lane]), s_id[g][lane]);
#pragma unroll
      for (int g = 3; g < 5; ++g) f.take(xf64(s_d[g][lane]), xf64(s_p0[g][lane]), xf64(s_p1[g][lane]), s_id[g][lane]);
      xf64 pq[6];
      tile.points(lane, e, f, pq);
      bf64_write(pq, i, ld, p, q, dist, flags);
    }
    __syncthreads();
  }
}

// FP32 GJK.  The iteration counts are heavy-tailed there (mean about 6; 7% of the
// microbenchmark's pairs take more than 10, up to 36), so with one pair per lane a warp ran
// for its slowest pair.  Here a warp owns `per_warp` consecutive pairs, and lanes that are
// done wait only until kGjkRefill of them are; these write their results and take the
// warp's next pairs.  2^22 pairs: 18.4 ms with the simplex indexed in local memory and
// always 36 iterations, 1.91 ms with registers and repeated states left out, 1.01 ms here.
// (In FP64 the counts are even, 3 to 7, and the plain loop is faster: 1.00 against 1.53 ms.)
constexpr int kGjkRefill = 12;
constexpr int kGjkThreads = 128;
__global__ void __launch_bounds__(kGjkThreads)
    k_pairs_gjk32(int64_t n, int64_t per_warp, const double *__restrict__ a, const double *__restrict__ b, int64_t ld,
                  double *__restrict__ p, double *__restrict__ q, double *__restrict__ dist,
                  uint8_t *__restrict__ flags) {
  const int lane = threadIdx.x & 31;
  int64_t next = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per_warp;
  const int64_t end = next + per_warp < n ? next + per_warp : n;
  if (next >= end) return;
  float A[3][3], B[3][3];
  Gjk<float> g;
  int64_t i = -1;  // this lane's pair
  bool more = false;
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, !more);
    if (__popc(idle) >= kGjkRefill || next >= end) {
      if (!more) {
        if (i >= 0) {
          float pq[6];
          g.points(A, B, pq);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            p[k * ld + i] = to_f64(pq[k]);
            q[k * ld + i] = to_f64(pq[3 + k]);
          }
          dist[i] = to_f64(pq_distance(pq));
          if (flags) flags[i] = 0;
        }
        i = next + __popc(idle & ((1u << lane) - 1u));
        if (i < end) {
#pragma unroll
          for (int v = 0; v < 3; ++v)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              A[v][k] = from_f64<float>(__ldg(a + (3 * v + k) * ld + i));
              B[v][k] = from_f64<float>(__ldg(b + (3 * v + k) * ld + i));
            }
          more = g.start(A, B);
        } else {
          i = -1;
        }
      }
      __syncwarp();
      next += __popc(idle);
      if (__all_sync(0xffffffffu, i < 0)) return;
    }
    if (more) more = g.step(A, B);
    __syncwarp();
  }
}

// bf_cert: warps walk the pair list 32 pairs at a time (the certificate's candidate queue
// is shared by the warp).
template <int W>
__global__ void __launch_bounds__(32 * W) k_pairs_cert(int64_t n, const double *__restrict__ a,
                                                       const double *__restrict__ b, int64_t ld,
                                                       double *__restrict__ p, double *__restrict__ q,
                                                       double *__restrict__ dist, uint8_t *__restrict__ flags) {
  __shared__ CertWarpSmem sm[W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + warp) * 32; base < n; base += nwarps * 32) {
    const int64_t i = base + lane;
    const bool valid = i < n;
    const int64_t ii = valid ? i : n - 1;
    double A[3][3], B[3][3];
#pragma unroll
    for (int v = 0; v < 3; ++v)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        A[v][k] = __ldg(a + (3 * v + k) * ld + ii);
        B[v][k] = __ldg(b + (3 * v + k) * ld + ii);
      }
    double out[6];
    const int evals = bf_cert_warp(A, B, valid, out, sm[warp]);
    if (valid) {
      xf64 pq[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) pq[k] = xf64(out[k]);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p[k * ld + i] = out[k];
        q[k * ld + i] = out[3 + k];
      }
      dist[i] = pq_distance(pq).v;
      if (flags) flags[i] = (uint8_t)evals;
    }
  }
}

// The certified kernel over an index list: pairs idx[0 .. *count) of the pair list (the
// count is read on the device, so the list can be built by an earlier kernel on the
// stream without a host round trip).  With `stage`, entry j's coordinates are read from
// stage[stage_at(j, c)] (a's 9, then b's; one contiguous tile per warp) instead of being
// gathered from a and b; results go to pair idx[j] of p, q, dist.
template <int W>
__global__ void __launch_bounds__(32 * W) k_pairs_cert_indexed(const uint32_t *__restrict__ count,
                                                               const uint32_t *__restrict__ idx,
                                                               const double *__restrict__ a,
                                                               const double *__restrict__ b, int64_t ld,
                                                               const double *__restrict__ stage,
                                                               double *__restrict__ p, double *__restrict__ q,
                                                               double *__restrict__ dist) {
  __shared__ CertWarpSmem sm[W];
  const int64_t n = *count;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t base = ((int64_t)blockIdx.x * (blockDim.x >> 5) + warp) * 32; base < n; base += nwarps * 32) {
    const bool valid = base + lane < n;
    const int64_t j = valid ? base + lane : n - 1;
    const int64_t i = idx[j];
    double A[3][3], B[3][3];
#pragma unroll
    for (int v = 0; v < 3; ++v)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        A[v][k] = stage ? __ldg(stage + stage_at(j, 3 * v + k)) : __ldg(a + (3 * v + k) * ld + i);
        B[v][k] = stage ? __ldg(stage + stage_at(j, 9 + 3 * v + k)) : __ldg(b + (3 * v + k) * ld + i);
      }
    double out[6];
    bf_cert_warp(A, B, valid, out, sm[warp]);
    if (valid) {
      xf64 pq[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) pq[k] = xf64(out[k]);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p[k * ld + i] = out[k];
        q[k * ld + i] = out[3 + k];
      }
      dist[i] = pq_distance(pq).v;
    }
  }
}

// cfg.blocks_per_sm > 0 caps the grid at that many blocks per SM (a grid-stride loop);
// 0 launches one thread per pair
template <class R, int M>
static cudaError_t launch_one(cudaStream_t s, int64_t n, const double *a, const double *b, int64_t ld, double me,
                              double *p, double *q, double *dist, uint8_t *flags, PairLaunch cfg) {
  int threads = cfg.threads == 64 || cfg.threads == 128 ? cfg.threads : 256;
  if (threads > PairBounds<R, M>::kThreads) threads = PairBounds<R, M>::kThreads;
  int64_t blocks = (n + threads - 1) / threads;
  if (cfg.blocks_per_sm > 0 && blocks > (int64_t)kNumSMs * cfg.blocks_per_sm) blocks = (int64_t)kNumSMs * cfg.blocks_per_sm;
  if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
  if (blocks < 1) blocks = 1;
  k_pairs<R, M><<<(unsigned)blocks, threads, 0, s>>>(n, a, b, ld, me, p, q, dist, flags);
  return cudaGetLastError();
}

// Pairs of a warp of k_pairs_gjk32: enough warps for one wave of 16 per SM, in whole
// groups of 32; at most 512 (262,143 pairs: 117 us with 96 a warp, 148 with 64, 144 with
// 256; 2^22: 1.01 ms with 512, 1.28 with 128, 1.07 with 1024).
static cudaError_t launch_gjk32(cudaStream_t s, int64_t n, const double *a, const double *b, int64_t ld, double *p,
                                double *q, double *dist, uint8_t *flags, PairLaunch cfg) {
  const int threads = cfg.threads == 64 ? 64 : kGjkThreads, warps = threads / 32;
  int64_t per = n / (16 * kNumSMs);
  if (per > 512) per = 512;
  if (cfg.blocks_per_sm > 0) {
    const int64_t least = n / ((int64_t)kNumSMs * cfg.blocks_per_sm * warps);
    if (per < least) per = least;
  }
  per = (per / 32 > 0 ? per / 32 : 1) * 32;
  int64_t blocks = (n + warps * per - 1) / (warps * per);
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  k_pairs_gjk32<<<(unsigned)(blocks > 0 ? blocks : 1), threads, 0, s>>>(n, per, a, b, ld, p, q, dist, flags);
  return cudaGetLastError();
}

// Below this the split kernel is the faster one (us, whole / split): 4,097 pairs 16.9 / 8.8,
// 20,000 17.0 / 11.7, 65,537 23.1 / 20.3, 98,000 29.3 / 27.2, 131,000 33.4 / 33.4, 196,000
// 46.9 / 47.7, 262,143 55.9 / 62.1.
constexpr int64_t kBfSplitPairs = 1 << 17;
static cudaError_t launch_bf64(cudaStream_t s, int64_t n, const double *a, const double *b, int64_t ld, double *p,
                               double *q, double *dist, uint8_t *flags, PairLaunch cfg) {
  const bool split = n < kBfSplitPairs;
  const int threads = cfg.threads == 64 ? 64 : kBfThreads, pairs = split ? 32 : threads;
  int64_t blocks = (n + pairs - 1) / pairs;
  if (cfg.blocks_per_sm > 0 && blocks > (int64_t)kNumSMs * cfg.blocks_per_sm) blocks = (int64_t)kNumSMs * cfg.blocks_per_sm;
  if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
  if (blocks < 1) blocks = 1;
  if (split) k_pairs_bf64_split<<<(unsigned)blocks, 32 * kBfSplitWarps, 0, s>>>(n, a, b, ld, p, q, dist, flags);
  else k_pairs_bf64<<<(unsigned)blocks, threads, 0, s>>>(n, a, b, ld, p, q, dist, flags);
  return cudaGetLastError();
}

template <class R>
static cudaError_t launch_prec(int method, cudaStream_t s, int64_t n, const double *a, const double *b, int64_t ld,
                               double me, double *p, double *q, double *dist, uint8_t *flags, PairLaunch cfg) {
  switch (method) {
    case M_BF:
      if constexpr (std::is_same_v<R, float>) return launch_one<R, M_BF>(s, n, a, b, ld, me, p, q, dist, flags, cfg);
      else return launch_bf64(s, n, a, b, ld, p, q, dist, flags, cfg);
    case M_PENALTY: return launch_one<R, M_PENALTY>(s, n, a, b, ld, me, p, q, dist, flags, cfg);
    case M_PENALTY_ITER: return launch_one<R, M_PENALTY_ITER>(s, n, a, b, ld, me, p, q, dist, flags, cfg);
    case M_GJK:
      if constexpr (std::is_same_v<R, float>) return launch_gjk32(s, n, a, b, ld, p, q, dist, flags, cfg);
      else return launch_one<R, M_GJK>(s, n, a, b, ld, me, p, q, dist, flags, cfg);
    case M_HYBRID_PAIR: return launch_one<R, M_HYBRID_PAIR>(s, n, a, b, ld, me, p, q, dist, flags, cfg);
    default: return cudaErrorInvalidValue;
  }
}

template <int W>
static cudaError_t launch_cert(cudaStream_t s, int64_t n, const double *a, const double *b, int64_t ld, double *p,
                               double *q, double *dist, uint8_t *flags, PairLaunch cfg) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pairs_cert<W>, 32 * W, 0);
  if (e != cudaSuccess) return e;
  int64_t blocks = (n + 32 * W - 1) / (32 * W);
  const int64_t per = cfg.blocks_per_sm > 0 ? cfg.blocks_per_sm : 8;
  const int64_t cap = (int64_t)kNumSMs * (per_sm > 0 ? per_sm : 1) * per;
  if (blocks > cap) blocks = cap;
  k_pairs_cert<W><<<(unsigned)(blocks > 0 ? blocks : 1), 32 * W, 0, s>>>(n, a, b, ld, p, q, dist, flags);
  return cudaGetLastError();
}

int pair_max_threads(int method, int precision) {
  if (method == M_BF_CERT) return 128;
  return (method == M_BF && precision == 0) ? kBfThreads : 256;
}

int pair_kernel_threads(int method, int precision) {
  return precision == 0 || method == M_GJK || method == M_BF_CERT ? 128 : 256;
}

cudaError_t launch_pairs_cfg(int method, int precision, cudaStream_t s, int64_t n, const double *a, const double *b,
                             int64_t ld, double max_error, double *p, double *q, double *dist, uint8_t *flags,
                             PairLaunch cfg) {
  if (method == M_BF_CERT) {
    if (cfg.threads == 64) return launch_cert<2>(s, n, a, b, ld, p, q, dist, flags, cfg);
    return launch_cert<4>(s, n, a, b, ld, p, q, dist, flags, cfg);
  }
  if (precision == 0) return launch_prec<xf64>(method, s, n, a, b, ld, max_error, p, q, dist, flags, cfg);
  return launch_prec<float>(method, s, n, a, b, ld, max_error, p, q, dist, flags, cfg);
}

cudaError_t launch_cert_indexed(cudaStream_t s, const uint32_t *count, int64_t max_count, const uint32_t *idx,
                                const double *a, const double *b, int64_t ld, double *p, double *q, double *dist,
                                PairLaunch cfg, const double *stage) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pairs_cert_indexed<4>, 128, 0);
  if (e != cudaSuccess) return e;
  int64_t blocks = (max_count + 127) / 128;
  const int64_t per = cfg.blocks_per_sm > 0 ? cfg.blocks_per_sm : 8;
  const int64_t cap = (int64_t)kNumSMs * (per_sm > 0 ? per_sm : 1) * per;
  if (blocks > cap) blocks = cap;
  k_pairs_cert_indexed<4><<<(unsigned)(blocks > 0 ? blocks : 1), 128, 0, s>>>(count, idx, a, b, ld, stage, p, q, dist);
  return cudaGetLastError();
}

cudaError_t launch_pairs(int method, int precision, cudaStream_t s, int64_t n, const double *a, const double *b,
                         int64_t ld, double max_error, double *p, double *q, double *dist, uint8_t *flags) {
  return launch_pairs_cfg(method, precision, s, n, a, b, ld, max_error, p, q, dist, flags, default_pair_launch(method));
}

}  // namespace delta
