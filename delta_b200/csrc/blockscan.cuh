// blockscan.cuh -- exclusive prefix sums of the time step's short count arrays (hash-grid
// buckets, per-body slave lists, per-pair contact counts) by one CTA: one graph node
// instead of cub's two (an init and a decoupled look-back scan), each of which costs its
// launch latency in a replayed step.  Longer arrays go to cub's device-wide scan.
#pragma once
#include <cub/cub.cuh>

#include "pdl.cuh"

#include <cstdint>

namespace delta {

constexpr int kBlockScanThreads = 1024, kBlockScanItems = 8;
// Up to two tiles of 8,192 entries.  Microseconds a scan, cub's two kernels / this one (200 in
// a row in a graph): 257 entries 2.7 / 2.1, 8,192 4.1 / 2.8, 10,001 4.1 / 4.3, 16,384 4.1 / 4.8,
// 24,576 4.1 / 6.7, 32,768 4.1 / 8.6.  A replayed step, whose other kernels are dependent
// launches, loses about 1 us more with cub's: of 16,000 bodies (as many counts) it takes 28.8 /
// 28.5, of 24,000 35.8 / 37.9, of 32,000 36.0 / 40.0.  (With a run of 8 entries per thread, whose
// 64-byte strides cost the CTA's loads and stores 8 sectors a request, one full tile took 7 us
// of a hopper step.)
constexpr int64_t kBlockScanMax = 2 * (int64_t)kBlockScanThreads * kBlockScanItems;

// out[i] = in[0] + ... + in[i-1] (integer sums: exact in any order).  A warp takes 256
// consecutive entries of a tile in 8 rounds of 32, so that its loads and stores are whole
// lines; the rounds' scans run side by side, the warps' totals are scanned by the first
// warp, and the running total is carried from tile to tile.
template <class T>
__global__ void __launch_bounds__(kBlockScanThreads) k_block_exclusive_scan(const T *__restrict__ in,
                                                                            T *__restrict__ out, int64_t n) {
  dep_sync();
  __shared__ T wsum[kBlockScanThreads / 32], carry;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = T(0);
  for (int64_t base = 0; base < n; base += (int64_t)kBlockScanThreads * kBlockScanItems) {
    const int64_t i0 = base + (int64_t)w * 32 * kBlockScanItems + lane;
    T v[kBlockScanItems], own[kBlockScanItems];
#pragma unroll
    for (int j = 0; j < kBlockScanItems; ++j) v[j] = own[j] = i0 + 32 * j < n ? in[i0 + 32 * j] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int j = 0; j < kBlockScanItems; ++j) {
        const T y = __shfl_up_sync(0xffffffffu, v[j], o);
        if (lane >= o) v[j] += y;
      }
    T total = T(0);  // of the rounds before j, then of the warp
#pragma unroll
    for (int j = 0; j < kBlockScanItems; ++j) {
      const T t = __shfl_sync(0xffffffffu, v[j], 31);
      v[j] += total - own[j];
      total += t;
    }
    if (lane == 0) wsum[w] = total;
    __syncthreads();
    if (w == 0) {
      const T s = wsum[lane];
      T x = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      wsum[lane] = x - s + carry;
      __syncwarp();
      if (lane == 31) carry += x;
    }
    __syncthreads();
    const T before = wsum[w];
#pragma unroll
    for (int j = 0; j < kBlockScanItems; ++j)
      if (i0 + 32 * j < n) out[i0 + 32 * j] = v[j] + before;
    __syncthreads();  // wsum is written again by the next tile
  }
}

// Exclusive sum of n entries: one CTA for n <= kBlockScanMax, else cub's device scan with
// the given temporary storage (sized by cub for n).
template <class T>
inline cudaError_t exclusive_sum(void *temp, size_t &temp_bytes, const T *in, T *out, int64_t n, cudaStream_t s,
                                 bool dep = false) {
  if (n <= kBlockScanMax) return launch_dep(dep, k_block_exclusive_scan<T>, 1, kBlockScanThreads, 0, s, in, out, n);
  return cub::DeviceScan::ExclusiveSum(temp, temp_bytes, in, out, n, s);
}

}  // namespace delta
