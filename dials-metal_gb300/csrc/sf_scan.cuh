// Scans: a block's, and a device-wide one whose count lives on the device, so
// that a pipeline of kernels never has to read a size back to the host. Two
// launches on a fixed grid: per-block chunk sums, then each block rescans its
// chunk with its offset, which it takes from its own block scan of the chunk
// sums.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sf_launch.cuh"

namespace sf {

constexpr int kScanBlocks = 512;
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr uint32_t kScanStep = kScanThreads * kScanItems;  // values a block step
static_assert(kScanBlocks <= kScanThreads, "a chunk sum a thread in the offset scan");

// Block-wide exclusive scan of one value per thread; returns the exclusive
// prefix and writes the block total to *total (all threads see it).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *total) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o)
      incl += t;
  }
  if (lane == 31)
    s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < nwarps ? s_warp[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o)
        wi += t;
    }
    if (lane < nwarps)
      s_warp[lane] = wi - w;
    if (lane == 31)
      s_total = wi;
  }
  __syncthreads();
  const uint32_t r = s_warp[warp] + incl - v;
  *total = s_total;
  __syncthreads();
  return r;
}

// This block's share [lo, hi) of n values, in whole steps (so a share starts
// 16-byte aligned when the array does).
__device__ __forceinline__ void scan_chunk(uint32_t n, uint32_t *lo, uint32_t *hi) {
  const uint32_t per = (n + gridDim.x - 1) / gridDim.x;
  const uint32_t chunk = (per + kScanStep - 1) / kScanStep * kScanStep;
  *lo = (uint32_t)min((unsigned long long)n, (unsigned long long)blockIdx.x * chunk);
  *hi = (uint32_t)min((unsigned long long)n, (unsigned long long)*lo + chunk);
}

// An exclusive scan of pairs of counts (two 32-bit halves of a 64-bit value,
// whose sums stay below 2^32 each) by a Scan object:
//   skip()             nothing to do (an error earlier in the pipeline)
//   size()             how many items there are (on the device)
//   first(i)           item i's pair, in the first pass
//   load(i)            the same, in the second
//   sums_done()        after the first pass's items, by every thread
//   store(i, v, e)     item i's pair and the sum of those before it
//   totals(t)          the sum of all, by one thread in the second pass
// size() may not depend on what totals() or store() writes.
__device__ __forceinline__ unsigned long long block_exclusive_scan64(unsigned long long v,
                                                                     unsigned long long *total) {
  __shared__ unsigned long long s_warp[32];
  __shared__ unsigned long long s_total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  unsigned long long incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o)
      incl += t;
  }
  if (lane == 31)
    s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long w = lane < nwarps ? s_warp[lane] : 0ull;
    unsigned long long wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o)
        wi += t;
    }
    if (lane < nwarps)
      s_warp[lane] = wi - w;
    if (lane == 31)
      s_total = wi;
  }
  __syncthreads();
  const unsigned long long r = s_warp[warp] + incl - v;
  *total = s_total;
  __syncthreads();
  return r;
}

template <class Scan>
static __global__ void __launch_bounds__(kScanThreads)
scan_pair_sums(Scan scan, unsigned long long *__restrict__ block_sums) {
  previous_done();
  if (scan.skip())
    return;
  uint32_t lo, hi;
  scan_chunk(scan.size(), &lo, &hi);
  unsigned long long acc = 0;
  for (uint32_t i = lo + threadIdx.x; i < hi; i += kScanThreads)
    acc += scan.first(i);
  scan.sums_done();
  unsigned long long total;
  (void)block_exclusive_scan64(acc, &total);
  if (threadIdx.x == 0)
    block_sums[blockIdx.x] = total;
}

template <class Scan>
static __global__ void __launch_bounds__(kScanThreads)
scan_pair_apply(Scan scan, const unsigned long long *__restrict__ block_sums) {
  previous_done();
  if (scan.skip())
    return;
  // This block's offset: the chunk sums of the blocks before it.
  __shared__ unsigned long long s_carry;
  unsigned long long all;
  const unsigned long long be =
      block_exclusive_scan64(threadIdx.x < kScanBlocks ? block_sums[threadIdx.x] : 0ull, &all);
  if (threadIdx.x == blockIdx.x)
    s_carry = be;
  if (blockIdx.x == 0 && threadIdx.x == 0)
    scan.totals(all);
  __syncthreads();
  uint32_t lo, hi;
  scan_chunk(scan.size(), &lo, &hi);
  unsigned long long carry = s_carry;
  for (uint32_t base = lo; base < hi; base += kScanStep) {  // block-uniform
    // A thread's kScanItems consecutive items.
    const uint32_t i = base + threadIdx.x * kScanItems;
    unsigned long long v[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      v[k] = i + k < hi ? scan.load(i + k) : 0ull;
      sum += v[k];
    }
    unsigned long long total;
    unsigned long long e = carry + block_exclusive_scan64(sum, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      if (i + k < hi)
        scan.store(i + k, v[k], e);
      e += v[k];
    }
    carry += total;
  }
}

// block_sums holds kScanBlocks values.
template <class Scan>
cudaError_t scan_pairs(const Scan &scan, unsigned long long *block_sums, cudaStream_t stream) {
  launch_after(scan_pair_sums<Scan>, kScanBlocks, kScanThreads, 0, stream, scan, block_sums);
  launch_after(scan_pair_apply<Scan>, kScanBlocks, kScanThreads, 0, stream, scan, block_sums);
  return cudaGetLastError();
}

} // namespace sf
