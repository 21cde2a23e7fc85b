// Internal interface of the streaming threshold: one frame or a batch of
// frames, of one shape or of several, of either pixel type, per launch sequence.
//
//   sf_extended.cu    dispersion_extended (the reference's algorithm); stage 0 and
//                     the erosion on strips, or (sf_lattice.cu) on a lattice
//   sf_dispersion.cu  the plain dispersion algorithm
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "sf_common.cuh"

namespace sf {

// The current device's SM count (152 until a device answers).
int device_sms();

// Frames one launch sequence takes.
constexpr int kMaxBatch = 64;

// A launch's frames and each one's shape. Every buffer is laid out for the
// largest, and each frame uses its own rows of it.
struct FramePtrs {
  const uint32_t *image[kMaxBatch];
  int h[kMaxBatch], w[kMaxBatch];
};

// Mask words of frame f (its own rows of ceil(w / 32) words).
__host__ __device__ inline size_t frame_words(const FramePtrs &F, int f) {
  return (size_t)((F.w[f] + 31) >> 5) * (size_t)F.h[f];
}

// Blocks over a batch of the kernels that count a mask's pixels (the size of
// block_sums and of cand_sums).
constexpr int kCountBlocks = 8192;

// A frame's signal count when its launch met a device fault (kCtrFault):
// no list, whatever the capacity.
constexpr uint32_t kCountFault = 0xFFFFFFFEu;

struct StreamBuffers {
  uint32_t *bits;          // final strong masks (output), frame f at bits + f * words
  size_t words;            // mask words per frame
  uint32_t *prefix;        // per-word list positions (output) or null
  uint2 *res;              // kept results, frame f at res + f * res_stride
  uint32_t res_stride;
  uint32_t *block_sums;    // per-block counts of strong pixels
  uint32_t capacity;
  sf_signal_pixel *out;    // ascending lists (output), frame f at out + f * out_stride
  size_t out_stride;
  uint32_t *count_out;     // one count per frame
  // dispersion_extended:
  uint32_t *cand;          // candidate masks, laid out as bits
  uint32_t *cand_sums;     // per-block counts of candidates
  uint32_t cand_limit;     // a frame of more candidates reports an overflowing count
  // The lattice path:
  uint32_t *tiles;         // its tile list, nframes * lattice_tiles
  uint32_t *counters;      // kCounterWords
};

// Tiles of the lattice path's exact check a frame has.
size_t lattice_tiles(int h, int w);

// Events recorded on the stream between the kernels when profiling.
struct StreamMarks {
  cudaEvent_t start, stage01, stage2, order;
};

// Whether the streaming path takes these parameters. 16-bit frames' tests are
// the reference's float sequences, whatever the parameters; 32-bit ones are
// bounded by integers first, which need a right side of at least zero and of
// a bounded size. The tile path (sf_threshold.cu) has the others.
bool streaming_path(const LaunchParams &P, int pixel_bytes);

// A launch that fills the device once with runs of fewer rows takes those whatever
// run length it is given: longer ones only leave warps without work. (One frame of
// 1065 x 1030 in a captured graph, L2 cold: 35 us so, 60 with the 64 rows that a
// tuned plan gave it.) Run lengths from here on are the tuner's to choose.
constexpr int kShortRun = 16;

// run_rows 0: the default geometry. marks may be null. h and w are the batch's
// envelope.
cudaError_t launch_extended(const FramePtrs &frames, int nframes, int h, int w, int pixel_bytes,
                            const LaunchParams &P, const StreamBuffers &b, int run_rows,
                            cudaStream_t stream, const StreamMarks *marks = nullptr);
cudaError_t launch_dispersion(const FramePtrs &frames, int nframes, int h, int w,
                              int pixel_bytes, const LaunchParams &P, const StreamBuffers &b, int run_rows,
                              cudaStream_t stream, const StreamMarks *marks = nullptr);

// The run length the default geometry picks for a batch of 32-bit frames of
// one shape under dispersion_extended (the tuner's start).
int stream_default_run_rows(const LaunchParams &P, int h, int w, int nframes);

} // namespace sf
