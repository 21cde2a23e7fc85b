// What the kernels that walk strips of a frame share (sf_lattice.cu,
// sf_dispersion.cu): a batch's division into each frame's own strips x runs,
// and the asynchronous copies that stage pixel rows in shared memory.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sf_stream.cuh"

namespace sf {

// Division of 32-bit numerators by a divisor fixed for a launch (tile
// counts), by one multiply-high and shifts: the round-up method of
// Granlund & Montgomery, "Division by invariant integers using
// multiplication" (PLDI 1994), with its add-and-shift step for multipliers of
// 33 bits. Exact for every numerator and divisor below 2^32.
struct FastDiv {
  uint32_t d, m, s1, s2;
};

inline FastDiv make_fastdiv(uint32_t d) {
  int l = 0;
  while ((1ull << l) < d)
    l++;
  FastDiv f;
  f.d = d;
  f.m = (uint32_t)(((((unsigned long long)1 << l) - d) << 32) / d + 1);
  f.s1 = l < 1 ? (uint32_t)l : 1u;
  f.s2 = l > 1 ? (uint32_t)(l - 1) : 0u;
  return f;
}

__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv &f) {
  const uint32_t t = __umulhi(n, f.m);
  return (t + ((n - t) >> f.s1)) >> f.s2;
}

// Where each frame's share of a launch's warps (lat_stage01: strips x runs)
// or tile groups (lat_tiles: tile rows x groups of 32 tiles) starts, and how
// many make one of its rows: every frame of a batch, mixed shapes or not,
// gets exactly its own.
struct FrameSpans {
  int start[kMaxBatch + 1];
  FastDiv by_row[kMaxBatch];
};

// The frame whose span holds item g (start[f] <= g < start[f + 1]); g below
// start[nframes].
__device__ __forceinline__ int span_frame(const FrameSpans &S, int nframes, int g) {
  int lo = 0, hi = nframes;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (S.start[mid] <= g)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
// One piece of 4 pixels: 16 bytes of a 32-bit frame, 8 of a 16-bit one.
template <typename Pix> __device__ __forceinline__ void cp_async_piece(void *dst, const void *src) {
  if (sizeof(Pix) == 4)
    cp_async16(dst, src);
  else
    cp_async8(dst, src);
}
template <typename Pix> __device__ __forceinline__ void fill_piece_masked(void *dst) {
  if (sizeof(Pix) == 4)
    *reinterpret_cast<uint4 *>(dst) = make_uint4(~0u, ~0u, ~0u, ~0u);
  else
    *reinterpret_cast<uint2 *>(dst) = make_uint2(~0u, ~0u);
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

} // namespace sf
