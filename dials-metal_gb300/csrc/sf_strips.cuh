// What the kernels that walk strips of a frame share (sf_extended.cu,
// sf_dispersion.cu). A warp walks down a strip of 360 output columns (or 112) for
// a run of rows. Lane l owns 12 columns (4); lanes 1-30 (2-29) write, and the others
// hold the columns on either side of the strip that their windows reach into.
// Each pixel row is staged in shared memory by cp.async a row or two ahead and
// stays there until it leaves the window.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "sf_launch.cuh"
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

// Where each frame's share of a launch's warps (strips x runs) starts, and its
// strips a run: every frame of a batch, mixed shapes or not, gets exactly its
// own.
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


// Columns a lane owns (C below): wide strips, and narrow ones for launches too
// small to fill the device with wide ones.
constexpr int kWideCols = 12, kNarrowCols = 4;
// Lanes at either end that hold the columns which the others' windows, and the
// erosion of their decisions, reach into: up to 7.
template <int C> constexpr int kHalo = C == kNarrowCols ? 2 : 1;
template <int C> constexpr int kStripOut = C * (32 - 2 * kHalo<C>);  // output columns a warp
template <int C> constexpr int kStripStride = C * 32;  // pixels a staged row
constexpr int kStripWarps = 2;         // warps a block
// A sum of pixels of which m are masked: the valid ones' sum (81 x 65533 is below
// 2^24) less m << 24. masked_of is -m, the place of a window's constants before
// the end of their table; a masked pixel is negative and its square wraps to 0.
constexpr uint32_t kCountShift = 24;
constexpr uint32_t kSumMask = (1u << kCountShift) - 1u;
constexpr uint32_t kMaskedPixel = 0u - (1u << kCountShift);
__device__ __forceinline__ int masked_of(uint32_t sum) { return (int)sum >> kCountShift; }

// Windows of 2K + 1 pixels square, with E rows of decisions either side of an
// output row (0: none).
template <int K> struct StripG {
  static constexpr int W0 = 2 * K + 1;
  static constexpr int N0 = W0 * W0;
  // Rows in flight ahead of the current one, the staged rows (from the one
  // leaving the window to the last in flight) and the blocks an SM that those
  // of 32-bit frames leave room for. One row's arithmetic takes longer than a
  // load, so few rows ahead and more warps.
  static constexpr int Ahead = K == 4 ? 1 : 2;
  static constexpr int Slots = W0 + Ahead + 1;
  static constexpr int Occ = K == 2 ? 8 : K == 3 ? 7 : 6;
  // Valid 32-bit pixels saturate at Cap, or rows whose windows hold a larger one
  // are summed apart, so that a window's sum of squares stays below 2^32. Below Big
  // a window's sum S is below sqrt(N0 Big) = 2^13, and both sides of the 32-bit tests (16 n Q; S (16 S + c) + 32, c < kMaxC16)
  // below 2^31: their difference's sign bit is the decision.
  static constexpr uint32_t Cap = K == 2 ? 13107 : K == 3 ? 9362 : 7281;
  static constexpr uint32_t Big = (1u << 26) / N0;
  static_assert((unsigned long long)Cap * Cap * N0 < (1ull << 32) && Cap * Cap >= Big,
                "exact squares, and a saturated pixel makes its window big");
};
constexpr uint32_t kMaxC16 = 1u << 17;

// The sign bits of x(c) for the lane's columns c, two chains of shifts.
template <int C, class X> __device__ __forceinline__ uint32_t sign_bits(X x) {
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int c = C / 2 - 1; c >= 0; c--) {
    lo = __funnelshift_l(x(c), lo, 1);
    hi = __funnelshift_l(x(c + C / 2), hi, 1);
  }
  return hi << (C / 2) | lo;
}

// A row into and another out of a lane's column sums and sums of squares.
template <int C>
__device__ __forceinline__ void add_rows(uint32_t Vn[C], uint32_t Vq[C],
                                         const uint32_t v[C], const uint32_t o[C]) {
#pragma unroll
  for (int c = 0; c < C; c++) {
    Vn[c] += v[c] - o[c];
    const uint32_t u = o[c] * o[c] - Vq[c];  // (two multiply-adds)
    Vq[c] = v[c] * v[c] - u;
  }
}

template <int K, typename Pix, int C> constexpr size_t strip_smem() {
  return (size_t)kStripWarps * StripG<K>::Slots * kStripStride<C> * sizeof(Pix);
}

// A valid pixel's value, 32-bit ones saturated at kCap, or a masked one's.
template <typename Pix, uint32_t kCap> __device__ __forceinline__ uint32_t pack_pixel(uint32_t v) {
  if (sizeof(Pix) == 2)
    return v >= 0xFFFEu ? kMaskedPixel : v;
  return v >= 0xFFFFFFFEu ? kMaskedPixel : min(v, kCap);
}

// A lane's staged pixels, packed. 32-bit rows are packed in place when
// they arrive (kRaw reads them first), 16-bit rows whenever they are read.
template <typename Pix, int C, uint32_t kCap, bool kRaw>
__device__ __forceinline__ void read_row(Pix *slot, int lane, uint32_t v[C]) {
  if constexpr (sizeof(Pix) == 2) {
    const uint2 *src = reinterpret_cast<const uint2 *>(slot + C * lane);
#pragma unroll
    for (int i = 0; i < C / 4; i++) {
      const uint2 x = src[i];
      v[4 * i] = pack_pixel<Pix, kCap>(x.x & 0xFFFFu);
      v[4 * i + 1] = pack_pixel<Pix, kCap>(x.x >> 16);
      v[4 * i + 2] = pack_pixel<Pix, kCap>(x.y & 0xFFFFu);
      v[4 * i + 3] = pack_pixel<Pix, kCap>(x.y >> 16);
    }
  } else {
    uint4 *src = reinterpret_cast<uint4 *>(slot + C * lane);
#pragma unroll
    for (int i = 0; i < C / 4; i++) {
      uint4 x = src[i];
      if (kRaw) {
        x.x = pack_pixel<Pix, kCap>(x.x), x.y = pack_pixel<Pix, kCap>(x.y);
        x.z = pack_pixel<Pix, kCap>(x.z), x.w = pack_pixel<Pix, kCap>(x.w);
        src[i] = x;
      }
      v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
    }
  }
}

// One warp's strip and run: where it reads and writes.
struct StripRun {
  int frame, height, width, bytes_per_row;
  int X, cx;      // the strip's and this lane's first column
  int ra, rb;     // output rows
  bool writer, first_of_pair;
  int pair_byte;  // this lane's first mask byte (lane pairs share C / 4)
  uint32_t inside;  // bit c: the lane's column c lies in the frame
};

// False (for the whole warp) past the last strip.
template <int C>
__device__ __forceinline__ bool strip_run(const FramePtrs &F, int nframes, const FrameSpans &S,
                                          int run_rows, StripRun &r) {
  const int lane = threadIdx.x & 31;
  const int gw = blockIdx.x * kStripWarps + (threadIdx.x >> 5);
  if (gw >= S.start[nframes])
    return false;
  const int f = span_frame(S, nframes, gw);
  const uint32_t local = (uint32_t)(gw - S.start[f]);
  const int ry = (int)fast_div(local, S.by_row[f]);
  const int sx = (int)(local - (uint32_t)ry * S.by_row[f].d);
  r.frame = f;
  r.height = F.h[f];
  r.width = F.w[f];
  r.bytes_per_row = ((r.width + 31) >> 5) * 4;
  r.X = kStripOut<C> * sx;
  r.cx = r.X + C * (lane - kHalo<C>);
  r.ra = ry * run_rows;
  r.rb = min(r.height, r.ra + run_rows);
  r.writer = lane >= kHalo<C> && lane < 32 - kHalo<C>;
  r.first_of_pair = ((lane - kHalo<C>) & 1) == 0;
  r.pair_byte = (r.X + 2 * C * ((lane - kHalo<C>) >> 1)) >> 3;
  r.inside = (r.cx < 0 || r.cx >= r.width)
                   ? 0u
                   : (r.cx + C <= r.width ? (1u << C) - 1u : ((1u << (r.width - r.cx)) - 1u));
  return true;
}

// The strip's pixel rows [pbeg, pend), fetched in turn into slots of the ring.
// Where the frame's rows are whole aligned pieces of 4 pixels a lane copies
// pieces l, l + 32 .. (a warp's copy covers 128 pixels), else pixels a lane apart. Bit u of `inside`: its u-th piece or pixel lies in the frame;
// what lies off it is staged as masked.
template <typename Pix, int C> struct RowReader {
  const Pix *next_row;
  int next_p, pend, width, lane;
  uint32_t inside;
  bool aligned, whole;  // whole: every lane's pieces lie in the frame's columns

  __device__ __forceinline__ RowReader(const Pix *image, const StripRun &r, int pbeg, int rows)
      : next_p(pbeg), pend(min(r.height, pbeg + rows)), width(r.width),
        lane(threadIdx.x & 31), inside(0) {
    aligned = width % 4 == 0 && reinterpret_cast<uintptr_t>(image) % (4 * sizeof(Pix)) == 0;
    const int x0 = r.X - kHalo<C> * C;  // the staged row's first column
#pragma unroll
    for (int u = 0; u < C; u++) {
      const int c = aligned ? x0 + 4 * lane + 128 * u : x0 + lane + 32 * u;
      const bool in = aligned ? u < C / 4 && c >= 0 && c + 4 <= width : c >= 0 && c < width;
      inside |= in ? 1u << u : 0u;
    }
    whole = __all_sync(0xffffffffu, aligned && inside == (1u << C / 4) - 1u);
    next_row = image + (ptrdiff_t)pbeg * width + x0 + (aligned ? 4 * lane : lane);
  }
  __device__ __forceinline__ void fetch(Pix *slot) {
    const uint32_t in = next_p >= 0 && next_p < pend ? inside : 0u;
    if (whole && next_p >= 0 && next_p < pend) {
#pragma unroll
      for (int u = 0; u < C / 4; u++)
        cp_async_piece<Pix>(slot + 4 * lane + 128 * u, next_row + 128 * u);
    } else if (aligned) {
      Pix *dst = slot + 4 * lane;
#pragma unroll
      for (int u = 0; u < C / 4; u++) {
        if ((in >> u) & 1u)
          cp_async_piece<Pix>(dst + 128 * u, next_row + 128 * u);
        else
          fill_piece_masked<Pix>(dst + 128 * u);
      }
    } else {
      Pix *dst = slot + lane;
#pragma unroll
      for (int u = 0; u < C; u++) {
        if constexpr (sizeof(Pix) == 4) {
          if ((in >> u) & 1u)
            cp_async4(dst + 32 * u, next_row + 32 * u);
          else
            dst[32 * u] = (Pix)~0u;
        } else {
          dst[32 * u] = (in >> u) & 1u ? __ldg(next_row + 32 * u) : (Pix)~0u;
        }
      }
    }
    next_row += width;
    next_p++;
  }
};

// A lane's C mask bits of a row into the mask: lane pairs write three bytes, the
// first lane two and the second the third, or with C = 4 the first lane one.
// The whole warp calls it; `row` is the row's pair_byte in a mask row that has
// `left` bytes from there.
template <int C>
__device__ __forceinline__ void write_bits(const StripRun &r, uint8_t *row, int left,
                                           uint32_t bits) {
  static_assert(C == kWideCols || C == kNarrowCols, "whole bytes a lane pair");
  const uint32_t next = __shfl_down_sync(0xffffffffu, bits, 1);
  if (!r.writer)
    return;
  if (C == kNarrowCols) {
    if (r.first_of_pair && left > 0)
      row[0] = (uint8_t)(bits | next << C);
  } else if (r.first_of_pair) {
    if (left > 0)
      row[0] = (uint8_t)bits;
    if (left > 1)
      row[1] = (uint8_t)((bits >> 8) | (next & 0xFu) << 4);
  } else if (left > 2) {
    row[2] = (uint8_t)(bits >> 4);
  }
}

// The column sums V of a lane and, by shuffles, of the K columns either side
// of its own, summed over the 2K + 1 columns around each of its own.
template <int K, int C>
__device__ __forceinline__ void window_sums(const uint32_t V[C], uint32_t h[C]) {
  uint32_t e[C + 2 * K];
#pragma unroll
  for (int c = 0; c < C; c++)
    e[K + c] = V[c];
#pragma unroll
  for (int k = 0; k < K; k++) {
    e[k] = __shfl_up_sync(0xffffffffu, V[C - K + k], 1);
    e[K + C + k] = __shfl_down_sync(0xffffffffu, V[k], 1);
  }
  h[0] = 0u;
#pragma unroll
  for (int k = 0; k <= 2 * K; k++)
    h[0] += e[k];
#pragma unroll
  for (int c = 1; c < C; c++)
    h[c] = h[c - 1] + e[c + 2 * K] - e[c - 1];
}

// Host: strips of a frame w wide (whole mask rows), and the run length and
// spans of a launch. run_rows 0: runs that fill `slots` resident warps
// kStripWaves times over, so that warps of unequal cost even out (one wave
// left a third of the warps' time idle), as long as a run keeps kLongRun
// rows (each run reads some rows more than it writes); else once, down to
// runs of kMinRunRows: a launch that cannot fill the device is a warp's walk
// long. (One frame of 1065 x 1030: the strips take 21 us with 2 to 4 rows, 26
// with 8; one of 430 x 393 whose windows need 64-bit sums is 92 us in all with 2,
// 110 with 4, 145 with 8.)
constexpr int kMinRunRows = 2;
constexpr int kLongRun = 64;
constexpr int kStripWaves = 4;

template <int C> inline int strips_of(int w) {
  return ((w + 31) / 32 * 32 + kStripOut<C> - 1) / kStripOut<C>;
}

inline int strip_run_rows(int tallest, long long strips, int slots, int run_rows) {
  const long long runs = std::max(1ll, slots / std::max(1ll, strips));
  const int once = (int)((tallest + runs - 1) / runs);
  if (run_rows <= 0)
    run_rows = std::min(once, std::max(kLongRun, (once + kStripWaves - 1) / kStripWaves));
  else if (once < kShortRun)
    run_rows = std::min(run_rows, once);
  return std::max(run_rows, kMinRunRows);
}

// Whether a launch takes narrow strips: where wide ones would fill `slots` resident
// warps with runs of fewer than kNarrowRun rows, and a warp's walk sets its time.
// (Wide and narrow, kernel 4 in a captured graph: one frame of 1065 x 1030, 2 rows,
// 40 and 34 us; of 2162 x 2068, 7 rows, 45 and 44; two of those 56 and 60.)
constexpr int kNarrowRun = 8;
inline bool narrow_strips(const FramePtrs &F, int nframes, int slots) {
  long long rows = 0;
  for (int f = 0; f < nframes; f++)
    rows += (long long)strips_of<kWideCols>(F.w[f]) * F.h[f];
  return rows < (long long)kNarrowRun * slots;
}

template <int C>
inline int strip_spans(const FramePtrs &F, int nframes, int slots, int run_rows, FrameSpans *S) {
  long long strips = 0;
  int tallest = 0;
  for (int f = 0; f < nframes; f++) {
    strips += strips_of<C>(F.w[f]);
    tallest = std::max(tallest, F.h[f]);
  }
  run_rows = strip_run_rows(tallest, strips, slots, run_rows);
  S->start[0] = 0;
  for (int f = 0; f < nframes; f++) {
    S->start[f + 1] = S->start[f] + strips_of<C>(F.w[f]) * ((F.h[f] + run_rows - 1) / run_rows);
    S->by_row[f] = make_fastdiv((uint32_t)strips_of<C>(F.w[f]));
  }
  return run_rows;
}

} // namespace sf
