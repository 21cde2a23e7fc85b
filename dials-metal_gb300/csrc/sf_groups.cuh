// What the kernels that decide a mask's pixels and write them out in order
// share (sf_extended.cu, sf_dispersion.cu). A mask row is cut into runs of 4
// words (128 pixels), numbered along the rows; a block takes whole bands of 8
// rows, so that its runs, and the pixels it counts, are consecutive.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "sf_common.cuh"
#include "sf_launch.cuh"
#include "sf_scan.cuh"
#include "sf_stream.cuh"

namespace sf {

constexpr int kScanT = 256;   // threads of a block
constexpr int kRunWords = 4;  // words of a run
constexpr int kBandRows = 8;  // rows of a band

__host__ __device__ inline int runs_per_row(int width) {
  return (((width + 31) >> 5) + kRunWords - 1) / kRunWords;
}

// This block's rows [lo, hi) of a frame, whole bands.
__device__ __forceinline__ void band_share(int height, int *lo, int *hi) {
  const int bands = (height + kBandRows - 1) / kBandRows;
  const int share = (bands + (int)gridDim.x - 1) / (int)gridDim.x * kBandRows;
  *lo = min(height, (int)blockIdx.x * share);
  *hi = min(height, *lo + share);
}

// The grid: blocks a frame, and the frames. A block of 8 warps takes enough
// bands for 128 runs (four a warp's round in the last pass: blocks of one band
// left six of its warps idle) while the batch still makes kMinBlocks blocks,
// else a band; at most kCountBlocks over the batch. (16 blocks an SM: 32 frames of
// 2162 x 2068 at kernel 2 take 490 us, 513 with 1024 blocks; 16 of 3262 x 3108 at
// kernel 4 647 and 700.)
constexpr int kMinBlocks = 16 * 152;
inline dim3 band_grid(int nframes, int height, int width) {
  const int bands = (height + kBandRows - 1) / kBandRows, rpr = runs_per_row(width);
  const int per = std::max(1, std::min((128 + rpr - 1) / rpr, bands * nframes / kMinBlocks));
  return dim3((unsigned)std::min((bands + per - 1) / per, kCountBlocks / nframes),
              (unsigned)nframes);
}

// The k-th set bit (from 0) of a word that has more than k.
__device__ __forceinline__ int select_bit(uint32_t w, uint32_t k) {
  int at = 0;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const uint32_t c = __popc(w & ((1u << s) - 1u));
    if (k >= c) {
      k -= c;
      w >>= s;
      at += s;
    }
  }
  return at;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o)
      v += t;
  }
  return v;
}

// Results kept between the two kernels, the passing pixels' backgrounds and
// populations: `keep` places a run. What did not fit is summed again.
struct Kept {
  uint2 *res;
  uint32_t stride, keep;  // places a frame, and a run
};
inline Kept make_kept(const StreamBuffers &b, int h, int w) {
  return {b.res, b.res_stride,
          (uint32_t)(b.res_stride / ((size_t)h * (size_t)runs_per_row(w)))};
}

// The places of a warp's group of runs [run0, min(run0 + 32, end)) whose results are
// kept together: what lies beyond belongs to the next group. (The last group of a
// block's bands is mostly a partial one: 8 of the 72 runs of a band 1030 wide.)
__device__ __forceinline__ uint32_t group_places(const Kept &kept, uint32_t run0, uint32_t end) {
  return min(32u, end - run0) * kept.keep;
}

// The window's mean as the records hold it: float(RN_double(S / n)) is
// RN_float(S / n) for S below 2^24 (sf_common.cuh), and 16-bit frames divide in
// float. A window short of valid pixels has the mean 0 (dext.cc:204).
template <typename Pix>
__device__ __forceinline__ float window_mean(uint32_t n, unsigned long long S,
                                             uint32_t min_local) {
  if (n < min_local)
    return 0.0f;
  return sizeof(Pix) == 2 || S < (1ull << 24)
             ? __fdiv_rn(__uint2float_rn((uint32_t)S), __uint2float_rn(n))
             : __double2float_rn(__ddiv_rn(__ull2double_rn(S), (double)n));
}

// A lane's run: its row, first word and words (zeros past the row's end).
struct LaneRun {
  int y, word;
  uint32_t w[kRunWords];
};
__device__ __forceinline__ LaneRun load_run(const uint32_t *bits, uint32_t run, uint32_t end,
                                            uint32_t rpr, uint32_t wpr) {
  LaneRun r;
  const uint32_t y = run / rpr, first = (run - y * rpr) * kRunWords;
  r.y = (int)y;
  r.word = (int)first;
#pragma unroll
  for (int k = 0; k < kRunWords; k++)
    r.w[k] = run < end && first + k < wpr ? bits[(size_t)y * wpr + first + k] : 0u;
  return r;
}
__device__ __forceinline__ uint32_t run_pixels(const LaneRun &r) {
  uint32_t c = 0;
#pragma unroll
  for (int k = 0; k < kRunWords; k++)
    c += (uint32_t)__popc(r.w[k]);
  return c;
}

// The set pixels of a warp's 32 consecutive runs (a lane each; incl the
// inclusive prefix of their counts), in order, 32 / kLanes at a time with
// kLanes lanes each: visit(live, q, rank, owner, k, bit, y, x), q the pixel's
// place among them, rank its place in its run, owner the lane that holds the
// run, k its word there. The whole warp calls it.
template <int kLanes, class Visit>
__device__ __forceinline__ void visit_pixels(const LaneRun &r, uint32_t incl, int lane,
                                             Visit visit) {
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t excl = incl - run_pixels(r);
  for (uint32_t q0 = 0; q0 < total; q0 += 32 / kLanes) {  // warp-uniform
    const uint32_t q = q0 + lane / kLanes;
    const bool live = q < total;
    int owner = 0;
#pragma unroll
    for (int s = 16; s; s >>= 1)
      owner += __shfl_sync(0xffffffffu, incl, owner + s - 1) <= q ? s : 0;
    owner &= 31;
    const uint32_t rank = q - __shfl_sync(0xffffffffu, excl, owner);
    uint32_t left = rank, word = 0;
    int k = 0;
#pragma unroll
    for (int i = 0; i < kRunWords; i++) {
      const uint32_t x = __shfl_sync(0xffffffffu, r.w[i], owner), c = (uint32_t)__popc(x);
      word = k == i ? x : word;
      if (k == i && i + 1 < kRunWords && left >= c) {
        left -= c;
        k = i + 1;
      }
    }
    const int bit = live ? select_bit(word, left) : 0;
    const int y = __shfl_sync(0xffffffffu, r.y, owner);
    const int x = (__shfl_sync(0xffffffffu, r.word, owner) + k) * 32 + bit;
    visit(live, q, rank, owner, k, bit, y, x);
  }
}

// The count and sum of the clipped window around (x, y), each lane its own: valid
// pixels, and outside the mask `out` where one is given. A row's pixels are loaded
// together. (A 4362 x 4148 frame at kernel 3 whose capacity is just above its 114
// thousand records takes 107 us, by the whole warp a window after another 184.)
struct WindowSum {
  unsigned long long S;
  uint32_t n;
};
template <typename Pix>
__device__ __noinline__ WindowSum sum_window(const Pix *image, const uint32_t *out, int height,
                                             int width, int half, int y, int x) {
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5;
  const int xl = x - half;
  uint32_t inside = 0;  // bit c: column xl + c is the window's and the frame's
#pragma unroll
  for (int c = 0; c < 2 * (kMaxHalf + 2) + 1; c++)
    inside |= c <= 2 * half && xl + c >= 0 && xl + c < width ? 1u << c : 0u;
  WindowSum r = {0ull, 0u};
  for (int yy = max(0, y - half); yy <= min(height - 1, y + half); yy++) {
    uint32_t in = inside;
    if (out) {
      const uint32_t *row = out + (size_t)yy * wpr;
      const int w0 = xl >> 5;  // (-1 left of the frame)
      const uint32_t a = w0 >= 0 ? row[w0] : 0u, b = w0 + 1 < (int)wpr ? row[w0 + 1] : 0u;
      in &= ~__funnelshift_r(a, b, xl & 31);
    }
    const Pix *at = image + ((ptrdiff_t)yy * width + xl);
    uint32_t v[2 * (kMaxHalf + 2) + 1];
#pragma unroll
    for (int c = 0; c < 2 * (kMaxHalf + 2) + 1; c++)
      v[c] = in >> c & 1u ? (uint32_t)__ldg(at + c) : Traits<Pix>::kMasked;
#pragma unroll
    for (int c = 0; c < 2 * (kMaxHalf + 2) + 1; c++) {
      const bool ok = v[c] < Traits<Pix>::kMasked;
      r.n += ok ? 1u : 0u;
      r.S += ok ? v[c] : 0u;
    }
  }
  return r;
}

// The mask's pixels as records, ascending by index (src/spots/dext.cc:212-220
// emits in scan order), each at its place from the blocks' counts, and, when
// asked for, each word's place. Their results come from their run's places
// (kByRun), or from those of the warp's 32 runs together; a pixel beyond them
// has its window summed again (half its half-width, `excluded` the mask that
// its pixels are outside of, if any). With cand_sums (the blocks' counts of
// candidates) a frame of more than cand_limit of them reports an overflowing
// count; with a fault recorded (a device wait that ran out) every count says so.
template <typename Pix, bool kByRun>
__global__ void __launch_bounds__(kScanT, 6)
scatter_pixels(const __grid_constant__ FramePtrs F, const uint32_t *bits_all, size_t words,
               const uint32_t *excluded_all, int half, Kept kept, uint32_t min_local,
               const uint32_t *block_sums, const uint32_t *cand_sums, uint32_t cand_limit,
               const uint32_t *fault, sf_signal_pixel *__restrict__ out_all,
               size_t out_stride, uint32_t capacity, uint32_t *__restrict__ count_out,
               uint32_t *__restrict__ prefix_all) {
  previous_done();
  const int f = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Pix *image = reinterpret_cast<const Pix *>(F.image[f]);
  const int height = F.h[f], width = F.w[f];
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5, rpr = (uint32_t)runs_per_row(width);
  const uint32_t *bits = bits_all + (size_t)f * words;
  const uint32_t *excluded = excluded_all ? excluded_all + (size_t)f * words : nullptr;
  const uint2 *res = kept.res + (size_t)f * kept.stride;
  sf_signal_pixel *out = out_all + (size_t)f * out_stride;
  // Each warp's share of the block's runs, in order, and its pixels' first
  // place: the blocks before this one's pixels, the warps before it's. All that
  // is counted first and meets at one barrier (32 frames of 4362 x 4148: 98 us;
  // 104 with the blocks' counts added up by one warp before the runs' were).
  struct Part {
    uint32_t before, total, cand, mine;
  };
  __shared__ Part s_part[kScanT / 32];
  int row_lo, row_hi;
  band_share(height, &row_lo, &row_hi);
  const uint32_t run_lo = (uint32_t)row_lo * rpr, run_hi = (uint32_t)row_hi * rpr;
  const uint32_t share = ((run_hi - run_lo + kScanT - 1) / kScanT) * 32u;
  const uint32_t lo = min(run_hi, run_lo + (uint32_t)warp * share), end = min(run_hi, lo + share);
  Part part = {0u, 0u, 0u, 0u};
  LaneRun r = load_run(bits, lo + lane, end, rpr, wpr);
  const size_t first_block = (size_t)f * gridDim.x;
  for (uint32_t i = threadIdx.x; i < (blockIdx.x ? blockIdx.x : gridDim.x); i += kScanT) {
    const uint32_t v = block_sums[first_block + i];
    part.before += v;
    if (blockIdx.x == 0 && cand_sums)
      part.cand += cand_sums[first_block + i];
  }
  if (blockIdx.x == 0) {
    part.total = part.before;
    part.before = 0;
  }
  part.mine = run_pixels(r);
  for (uint32_t run0 = lo + 32; run0 < end; run0 += 32)
    part.mine += run_pixels(load_run(bits, run0 + lane, end, rpr, wpr));
  part.before = __reduce_add_sync(0xffffffffu, part.before);
  part.mine = __reduce_add_sync(0xffffffffu, part.mine);
  if (blockIdx.x == 0) {
    part.total = __reduce_add_sync(0xffffffffu, part.total);
    part.cand = __reduce_add_sync(0xffffffffu, part.cand);
  }
  if (lane == 0)
    s_part[warp] = part;
  __syncthreads();
  uint32_t pos = 0;
#pragma unroll
  for (int k = 0; k < kScanT / 32; k++)
    pos += s_part[k].before + (k < warp ? s_part[k].mine : 0u);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    uint32_t total = 0, cand = 0;
#pragma unroll
    for (int k = 0; k < kScanT / 32; k++) {
      total += s_part[k].total;
      cand += s_part[k].cand;
    }
    count_out[f] = fault && *fault ? kCountFault : cand > cand_limit ? 0xFFFFFFFFu : total;
  }
  if (!prefix_all && part.mine == 0)
    return;  // whole warp
  for (uint32_t run0 = lo; run0 < end; run0 += 32) {
    if (run0 != lo)
      r = load_run(bits, run0 + lane, end, rpr, wpr);
    const uint32_t incl = warp_inclusive(run_pixels(r), lane);
    if (prefix_all) {
      uint32_t at = pos + incl - run_pixels(r);
#pragma unroll
      for (int k = 0; k < kRunWords; k++) {
        if (run0 + lane < end && (uint32_t)r.word + k < wpr)
          prefix_all[(size_t)f * words + (size_t)r.y * wpr + r.word + k] = at;
        at += (uint32_t)__popc(r.w[k]);
      }
    }
    visit_pixels<1>(r, incl, lane,
                    [&](bool live, uint32_t q, uint32_t rank, int owner, int, int, int y, int x) {
                      const uint32_t index = (uint32_t)y * (uint32_t)width + (uint32_t)x;
                      const uint32_t held = kByRun ? kept.keep : group_places(kept, run0, end);
                      const uint32_t place = kByRun ? rank : q;
                      const size_t at =
                          (size_t)(run0 + (kByRun ? (uint32_t)owner : 0u)) * kept.keep + place;
                      uint2 b = make_uint2(0u, 0u);
                      uint32_t value = 0;
                      if (live) {
                        value = (uint32_t)__ldg(image + index);
                        if (place < held)
                          b = res[at];
                      }
                      if (live && place >= held) {
                        const WindowSum w = sum_window(image, excluded, height, width, half, y, x);
                        b = make_uint2(__float_as_uint(window_mean<Pix>(w.n, w.S, min_local)), w.n);
                      }
                      if (live && pos + q < capacity) {
                        sf_signal_pixel rec;
                        rec.index = index;
                        rec.value = value;
                        rec.background = __uint_as_float(b.x);
                        rec.population = (uint16_t)b.y;
                        rec.reserved = 0;
                        out[pos + q] = rec;
                      }
                    });
    pos += __shfl_sync(0xffffffffu, incl, 31);
  }
}

} // namespace sf
