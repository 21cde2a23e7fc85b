// How the kernels that order signal pixels split a frame's items (mask words,
// candidates): blocks of kScanT threads, kScanPer consecutive items a thread,
// on a (block, frame) grid.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace sf {

constexpr int kScanT = 256;                    // threads of a scan block
constexpr int kScanPer = 8;                    // consecutive items per thread
constexpr int kScanChunk = kScanT * kScanPer;  // items per block pass

// This block's share [lo, hi) of a frame's n items, in whole passes.
__device__ __forceinline__ void chunk_of(size_t n, size_t *lo, size_t *hi) {
  size_t chunk = (n + gridDim.x - 1) / gridDim.x;
  chunk = (chunk + kScanChunk - 1) / kScanChunk * kScanChunk;
  *lo = min(n, (size_t)blockIdx.x * chunk);
  *hi = min(n, *lo + chunk);
}

// Sum of the block's predecessors' counts in its frame, and the frame's
// total.
__device__ __forceinline__ uint32_t block_base(const uint32_t *__restrict__ block_sums,
                                               uint32_t *total) {
  __shared__ uint32_t s_base, s_total;
  if (threadIdx.x < 32) {
    const uint32_t *bs = block_sums + (size_t)blockIdx.y * gridDim.x;
    uint32_t b = 0, t = 0;
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += 32) {
      const uint32_t v = bs[i];
      b += i < blockIdx.x ? v : 0u;
      t += v;
    }
    for (int o = 16; o; o >>= 1) {
      b += __shfl_xor_sync(0xffffffffu, b, o);
      t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (threadIdx.x == 0) {
      s_base = b;
      s_total = t;
    }
  }
  __syncthreads();
  *total = s_total;
  return s_base;
}

} // namespace sf
