// Stage 0 and the erosion of the streaming threshold for the reference's own
// window (kernel 3,3: 7 x 7 stage-0 windows, erosion by 2), in two kernels:
//
//   lat_stage01  stage 0 on a lattice of every third row and every third
//                column only, and the erosion of that lattice: an upper bound
//                of the eroded mask, written as the candidate mask
//   lat_verify   the exact stage 0 and erosion on the 8 x 28 tiles that hold
//                a candidate of the bound; the candidates that fail leave the
//                mask, which is then the reference's candidate mask
//
// Why the bound holds. The erosion (src/spots/dext.cc:117-142) keeps a valid
// pixel only if every in-frame pixel of its 5 x 5 neighbourhood is signal or
// masked after stage 0. ANDing over only the lattice pixels of the
// neighbourhood can keep more pixels, never fewer. Every 5 x 5 neighbourhood
// holds 1 to 4 lattice pixels, and next to a masked band or the frame's edge
// a valid pixel still sees a 3 x 3 block of in-frame valid pixels, so a
// lattice pixel; the bound passes about 1.7 times the exact candidates, all in
// and around spots.
//
// The lattice decisions are an upper bound too: a window counts as signal
// when the lower of the two integer bounds of sf_lattice.cuh says it may be,
// and when its sums may not be exact. Valid pixels are summed saturated at
// kLatCap (2^15 - 1), so every packed sum is exact for the saturated values;
// a window whose saturated sum S is below kLatCap - 1 holds no saturated
// pixel, its sum of squares is at most S^2 < 2^30, and its decision is that
// of the reference. A window with a larger S is taken as signal, and the tile
// check decides it exactly.
//
// The tile check decides the stage-0 windows of the rows within 2 of a candidate
// (the only ones whose decision can clear one), four next to one another a lane.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include <cudaTypedefs.h>

#include "sf_common.cuh"
#include "sf_lattice.cuh"
#include "sf_strips.cuh"
#include "sf_tma.cuh"

namespace sf {
namespace {

constexpr int kLatK = 3;                    // stage-0 half-width
constexpr int kLatN0 = 49;                  // pixels of a stage-0 window
constexpr int kLatCols = 12;                // columns a lane owns
constexpr int kLatOutLanes = 30;            // lanes 1-30 write; lanes 0 and 31 are their halos
constexpr int kLatOut = kLatCols * kLatOutLanes;  // 360 output columns a warp
constexpr int kLatWarps = 4;                // warps a block
constexpr int kLatOcc = 5;                  // blocks an SM the kernel is built for
constexpr uint32_t kLatPS = 26;             // masked count above a 26-bit sum
constexpr uint32_t kLatMask = (1u << kLatPS) - 1u;
constexpr uint32_t kLatCap = 32767;         // valid pixels saturate here

static_assert(kLatOut % 24 == 0, "lane pairs write whole bytes");

static_assert(kLatN0 * kLatCap < (1u << kLatPS), "saturated sums stay below the count field");

// The 12 bound bits of a lane from the lattice bits b0-b4 at its columns
// -1, 2, 5, 8 and 11 (b0 is the lane before's column 11): column c keeps the
// lattice columns within 2 of it.
__host__ __device__ constexpr uint32_t lat_bound12(uint32_t b) {
  const uint32_t b0 = b & 1u, b1 = (b >> 1) & 1u, b2 = (b >> 2) & 1u, b3 = (b >> 3) & 1u,
                 b4 = (b >> 4) & 1u;
  const uint32_t a = b0 & b1, d = b1 & b2, e = b2 & b3, g = b3 & b4;
  return a * 0x003u | b1 << 2 | d * 0x018u | b2 << 5 | e * 0x0C0u | b3 << 8 | g * 0x600u |
         b4 << 11;
}

// One pixel row of a lane: its 12 pixels packed (masked as a lone count bit
// whose square wraps to 0, valid saturated at kLatCap), the row sums of 7
// columns at the lattice columns 2, 5, 8, 11, and the masked bits of the 12
// columns. The windows reach one column into the lane before (its column 11,
// by a shuffle) and three into the lane after (its first triple, likewise):
// lanes 0 and 31 hold the halo columns of the warp's 30 writing lanes.
// 16-bit frames (Pix = uint16_t) are summed as the reference sums them: in
// 32 bits, the sum of squares modulo 2^32 (src/spots/dext.hh:31-33); their
// pixels need no saturation (49 of them sum below 2^22).
template <typename Pix>
__device__ __forceinline__ void lat_row(const uint32_t v[kLatCols], int lane, uint32_t hn[4],
                                        uint32_t hq[4], uint32_t *m12) {
  constexpr bool k16 = sizeof(Pix) == 2;
  uint32_t ns[kLatCols], q[kLatCols];
#pragma unroll
  for (int i = 0; i < kLatCols; i++) {
    if (k16)
      ns[i] = v[i] >= 0xFFFEu ? (1u << kLatPS) : v[i];
    else
      ns[i] = v[i] >= 0xFFFFFFFEu ? (1u << kLatPS) : min(v[i], kLatCap);
    q[i] = ns[i] * ns[i];
  }
  // Triples of columns [3a, 3a + 2], then the 7-column windows.
  uint32_t gn[4], gq[4];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    gn[a] = ns[3 * a] + ns[3 * a + 1] + ns[3 * a + 2];
    gq[a] = q[3 * a] + q[3 * a + 1] + q[3 * a + 2];
  }
  const uint32_t ln = __shfl_sync(0xffffffffu, ns[kLatCols - 1], (lane + 31) & 31);
  const uint32_t lq = __shfl_sync(0xffffffffu, q[kLatCols - 1], (lane + 31) & 31);
  const uint32_t rn = __shfl_sync(0xffffffffu, gn[0], (lane + 1) & 31);
  const uint32_t rq = __shfl_sync(0xffffffffu, gq[0], (lane + 1) & 31);
  hn[0] = ln + gn[0] + gn[1];
  hq[0] = lq + gq[0] + gq[1];
  hn[1] = ns[2] + gn[1] + gn[2];
  hq[1] = q[2] + gq[1] + gq[2];
  hn[2] = ns[5] + gn[2] + gn[3];
  hq[2] = q[5] + gq[2] + gq[3];
  hn[3] = ns[8] + gn[3] + rn;
  hq[3] = q[8] + gq[3] + rq;
  // A valid packed 32-bit-frame pixel is below 2^15, so shifting it right by
  // 26 - c (c <= 11) leaves nothing: the shifted words add up to the masked
  // bits. A 16-bit pixel can reach 2^16, so its count bit is isolated first.
  uint32_t m = 0;
#pragma unroll
  for (int c = 0; c < kLatCols; c++)
    m += k16 ? (ns[c] >> kLatPS) << c : ns[c] >> (kLatPS - c);
  *m12 = m;
}

// Each warp's pixel rows are staged in shared memory by cp.async (RowReader,
// sf_strips.cuh), kRingSlots - 1 rows ahead, 12 columns a lane from column X - 12
// (X the strip's first output column).
constexpr int kRingSlots = 4;
template <typename Pix>
constexpr size_t ring_bytes() {
  return (size_t)kLatWarps * kRingSlots * kStripStride<kLatCols> * sizeof(Pix);
}

template <int kOcc, typename Pix>
__global__ void __launch_bounds__(kLatWarps * 32, kOcc)
lat_stage01(const __grid_constant__ FramePtrs F, int nframes,
            const __grid_constant__ FrameSpans S, int run_rows,
            const __grid_constant__ StreamTables T,
            const __grid_constant__ LaunchParams P, uint8_t *__restrict__ final_bytes,
            size_t mask_bytes, uint32_t *__restrict__ counters) {
  previous_done();
  if (blockIdx.x == 0 && threadIdx.x < kCounterWords)
    counters[threadIdx.x] = 0u;  // for the next two kernels
  constexpr bool k16 = sizeof(Pix) == 2;
  extern __shared__ __align__(16) unsigned char lat_ring_raw[];
  Pix *lat_ring = reinterpret_cast<Pix *>(lat_ring_raw);
  // Lower-bound constants by masked count m (window count 49 - m).
  __shared__ uint2 tab[kLatN0 + 1];
  __shared__ uint16_t lut[32];
  for (int m = threadIdx.x; m <= kLatN0; m += blockDim.x)
    tab[m] = make_uint2(T.nk[kLatN0 - m], T.clo[kLatN0 - m]);
  if (threadIdx.x < 32)
    lut[threadIdx.x] = (uint16_t)lat_bound12(threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gw = blockIdx.x * kLatWarps + warp;
  if (gw >= S.start[nframes])
    return;  // whole warp
  // This warp's frame, strip and run (each frame has its own strips x runs).
  const int f = span_frame(S, nframes, gw);
  const uint32_t local = (uint32_t)(gw - S.start[f]);
  const int ry = (int)fast_div(local, S.by_row[f]);
  const int sx = (int)(local - (uint32_t)ry * S.by_row[f].d);
  const int height = F.h[f], width = F.w[f];
  const Pix *image = reinterpret_cast<const Pix *>(F.image[f]);
  const int bytes_per_row = ((width + 31) >> 5) * 4;
  uint8_t *fin = final_bytes + (size_t)f * mask_bytes;
  // Lane l holds columns X + 12 (l - 1) .. + 11: lanes 1-30 the strip's
  // 360, lane 0 the 12 before it, lane 31 the 12 after it.
  const int cx = kLatOut * sx + kLatCols * (lane - 1);
  // This lane's first mask byte (lane pairs 1-2, 3-4, .. share three
  // bytes), and the bits of its columns inside the frame.
  const int pair_byte = (kLatOut * sx + 24 * ((lane - 1) >> 1)) >> 3;
  const bool writer = lane >= 1 && lane <= kLatOutLanes;
  const bool first_of_pair = (lane & 1) != 0;
  const uint32_t inside =
      (cx < 0 || cx >= width) ? 0u
                              : (cx + kLatCols <= width ? 0xFFFu : ((1u << (width - cx)) - 1u));
  const int ra = ry * run_rows;
  const int rb = min(height, ra + run_rows);
  const int ja = ra / 3;
  const int ntrip = (rb - ra + 2) / 3;

  // U = h(last row of triple t-2) + T(t-1) per lattice column; hl = the
  // last row of the previous triple.
  uint32_t Un[4], Uq[4], hln[4], hlq[4];
#pragma unroll
  for (int a = 0; a < 4; a++)
    Un[a] = Uq[a] = hln[a] = hlq[a] = 0u;
  uint32_t mprev[3] = {0u, 0u, 0u}, bprev = 0u, cmprev = 0u;

  // Pixel rows [pbeg, pend) of the run.
  const int pbeg = 3 * (ja - 2), pend = 3 * (ja + ntrip + 1);
  Pix *ring = lat_ring + (size_t)warp * kRingSlots * kStripStride<kLatCols>;
  StripRun r;
  r.X = kLatOut * sx;
  r.height = height;
  r.width = width;
  RowReader<Pix, kLatCols> reader(image, r, pbeg, pend - pbeg);
#pragma unroll
  for (int i = 0; i < kRingSlots - 1; i++) {
    reader.fetch(ring + i * kStripStride<kLatCols>);
    cp_async_commit();
  }

  uint32_t v[kLatCols];
  int slot_in = kRingSlots - 1, slot_now = 0;
  for (int t = 0; t < ntrip + 3; t++) {
    const int p0 = 3 * (ja - 2 + t);
    uint32_t Tn[4], Tq[4], mcur[3], cm = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      // Row p0 + k + kRingSlots - 1 goes out; row p0 + k has landed.
      __syncwarp();
      reader.fetch(ring + slot_in * kStripStride<kLatCols>);
      cp_async_commit();
      cp_async_wait<kRingSlots - 1>();
      __syncwarp();
      const Pix *slot = ring + slot_now * kStripStride<kLatCols>;
      slot_in = (slot_in + 1) % kRingSlots;
      slot_now = (slot_now + 1) % kRingSlots;
      if constexpr (k16) {
        const uint2 *src = reinterpret_cast<const uint2 *>(slot + kLatCols * lane);
#pragma unroll
        for (int i = 0; i < kLatCols / 4; i++) {
          const uint2 x = src[i];
          v[4 * i] = x.x & 0xFFFFu, v[4 * i + 1] = x.x >> 16;
          v[4 * i + 2] = x.y & 0xFFFFu, v[4 * i + 3] = x.y >> 16;
        }
      } else {
        const uint4 *src = reinterpret_cast<const uint4 *>(slot) + 3 * lane;
#pragma unroll
        for (int i = 0; i < kLatCols / 4; i++) {
          const uint4 x = src[i];
          v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
        }
      }
      uint32_t hn[4], hq[4];
      lat_row<Pix>(v, lane, hn, hq, &mcur[k]);
#pragma unroll
      for (int a = 0; a < 4; a++) {
        Tn[a] = k == 0 ? hn[a] : Tn[a] + hn[a];
        Tq[a] = k == 0 ? hq[a] : Tq[a] + hq[a];
      }
      if (k == 2) {
        // Masked centres of this row's lattice columns 2, 5, 8, 11: the
        // lattice row the next triple decides.
        const uint32_t m12 = mcur[2];
        cm = ((m12 >> 2) & 1u) | ((m12 >> 4) & 2u) | ((m12 >> 6) & 4u) | ((m12 >> 8) & 8u);
#pragma unroll
        for (int a = 0; a < 4; a++) {
          // Window rows p0 - 4 .. p0 + 2, centred on the previous triple's
          // last row (a lattice row).
          const uint32_t Wn = Un[a] + Tn[a], Wq = Uq[a] + Tq[a];
          Un[a] = hln[a] + Tn[a];
          Uq[a] = hlq[a] + Tq[a];
          hln[a] = hn[a];
          hlq[a] = hq[a];
          Tn[a] = Wn;
          Tq[a] = Wq;
        }
      }
    }
    if (t < 2) {
      cmprev = cm;
#pragma unroll
      for (int k = 0; k < 3; k++)
        mprev[k] = mcur[k];
      continue;  // warp-uniform: the windows are not yet whole
    }
    // Lattice row p0 - 1: four decisions by the lower bound (sf_lattice.cuh),
    // windows whose sums may be inexact taken as signal, masked centres set.
    uint32_t b4 = cmprev;
#pragma unroll
    for (int a = 0; a < 4; a++) {
      const uint32_t W = Tn[a];
      const uint32_t m = min(W >> kLatPS, (uint32_t)kLatN0);  // 49 pixels: m <= 49
      const uint32_t S = W & kLatMask;
      bool sig;
      if constexpr (k16) {
        // The reference's float test, exactly (sf_common.cuh stage0_u16).
        sig = stage0_u16((uint32_t)kLatN0 - m, S, Tq[a], P);
      } else {
        const uint2 c = tab[m];
        const unsigned long long L = (unsigned long long)Tq[a] * c.x;
        const unsigned long long Rr = (unsigned long long)S * ((S << kDec) + c.y);
        sig = (L > Rr) | (S >= kLatCap - 1u);  // (no branch)
      }
      b4 |= sig ? 1u << a : 0u;
    }
    // The bound bits at columns -1 (the lane before's 11), 2, 5, 8, 11.
    const uint32_t b5 = b4 << 1 | (__shfl_sync(0xffffffffu, b4, (lane + 31) & 31) >> 3 & 1u);
    if (t >= 3) {
      // The previous triple's rows p0 - 3 .. p0 - 1: the first two see the
      // lattice rows p0 - 4 and p0 - 1, the last only p0 - 1.
      const uint32_t bd01 = lut[bprev & b5], bd2 = lut[b5];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int r = p0 - 3 + k;
        const uint32_t bd = k < 2 ? bd01 : bd2;
        const uint32_t mk = mprev[k];
        const uint32_t c12 = bd & ~mk & inside;
        // Lane pairs: the first lane (odd) writes the pair's first two bytes,
        // the second the third.
        const uint32_t odd = __shfl_down_sync(0xffffffffu, c12, 1);
        if (writer && r < rb) {
          const size_t at = (size_t)r * bytes_per_row;
          if (first_of_pair) {
            if (pair_byte < bytes_per_row)
              fin[at + pair_byte] = (uint8_t)c12;
            if (pair_byte + 1 < bytes_per_row)
              fin[at + pair_byte + 1] = (uint8_t)((c12 >> 8) | (odd & 0xFu) << 4);
          } else if (pair_byte + 2 < bytes_per_row) {
            fin[at + pair_byte + 2] = (uint8_t)(c12 >> 4);
          }
        }
      }
    }
    bprev = b5;
    cmprev = cm;
#pragma unroll
    for (int k = 0; k < 3; k++)
      mprev[k] = mcur[k];
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// The exact check of the bound's candidates, on tiles of 8 rows x 28 columns.
//
//   lat_tiles   lists the tiles that hold a candidate (any order)
//   lat_verify  one warp per listed tile, persistent: the tile's 12 x 32
//               stage-0 windows (rows r0 - 2 .., columns c0 - 2 ..) from its
//               18 x 38 pixels, the erosion of its 8 x 28 pixels, and the
//               candidates that fail cleared from the mask
//
// A warp copies the next tile's pixels into shared memory (a TMA box where the
// frame allows) while it checks the current one, so the loads' latency is
// hidden behind the arithmetic. A lane a column, the column sums of 7 rows go
// to shared memory; then four rows of windows at a time, eight lanes a row, each
// lane decides four windows next to one another from ten column sums: the two
// bounds of sf_lattice.cuh, and the reference's sequence between them
// (sf_common.cuh). Rows without a window within 2 of a candidate are left out.
// The candidates, the decisions and the erosion are a row a lane. Tiles share
// mask words, so the clearing is an atomic AND; each candidate belongs to one
// tile, so the order does not matter. Bound by issue (64% of its rate, 820
// instructions a tile): 32 frames of 4362 x 4148 take 297 us, 16 of 16 bits 148, 4
// dense ones 621; with a lane a column for the windows too, each lane taking its
// column's needed ones in turn (11 rounds a tile, 12 lanes in them), and the
// erosion a row after another in every lane, 449, 250 and 967 us.
// ---------------------------------------------------------------------------
constexpr int kVerRows = 8;                  // output rows of a tile
constexpr int kVerTW = 28;                   // output columns of a tile
constexpr int kVerPR = kVerRows + 10;        // pixel rows
constexpr int kVerDR = kVerRows + 4;         // stage-0 rows
constexpr int kVerPC = 38;                   // pixel columns
constexpr int kVerPW = 44;                   // staged columns: 11 16-byte pieces
constexpr int kVerWarps = 4;
constexpr int kVerOcc = 6;                   // exact-check blocks an SM (a pixel buffer a warp)

__host__ __device__ inline int ver_ntx(int w) { return (w + kVerTW - 1) / kVerTW; }
__host__ __device__ inline int ver_nty(int h) { return (h + kVerRows - 1) / kVerRows; }

// Staged columns a pixel row (whole 16-byte pieces covering the 38 needed
// from a 16-byte boundary) and that boundary's alignment, in pixels: a TMA
// box row must be a multiple of 16 bytes and start on one.
template <typename Pix> struct VerPix;
template <> struct VerPix<uint32_t> {
  static constexpr int kPW = kVerPW, kAlign = 4;
};
template <> struct VerPix<uint16_t> {
  static constexpr int kPW = 48, kAlign = 8;
};

// One staged tile: 18 pixel rows (r0 - 5 .. r0 + 12) of kPW pixels from the
// aligned column xs, dense, as a TMA box lands in shared memory (128-byte
// aligned, the box load's destination rule).
template <typename Pix> struct alignas(128) TileBuf {
  Pix px[kVerPR][VerPix<Pix>::kPW];
};

template <typename Pix> struct alignas(128) VerWarp {
  TileBuf<Pix> pix;                      // staged pixels (the next tile's load goes out
                                         // once the current one's are read)
  uint64_t bar;                          // its TMA mbarrier
  uint32_t cw[2][kVerRows][2];           // the tile's candidate words, two tiles (s)
  alignas(16) uint2 vs[kVerDR][kVerPC + 2];  // column sums of 7 rows
  // Masked centres, a word a column (column i's at i + 1, so that a lane's four
  // are one load), bit d for stage-0 row d.
  alignas(16) uint32_t msk[kVerPC + 2];
  // The sums of squares' high words (32-bit frames, tiles with large counts).
  alignas(8) uint16_t vh[sizeof(Pix) == 4 ? kVerDR : 1][kVerPC + 2];
};

// The frames' 2-D tensor maps, boxes of one tile (kPW x 18 pixels), for the TMA
// staging of the exact check.
struct TileMaps {
  CUtensorMap map[kMaxBatch];
  unsigned long long mapped;  // bit f: frame f has a map (else its tiles are staged per lane)
  __device__ __forceinline__ bool has(int f) const { return (mapped >> f) & 1ull; }
};

template <typename Pix> __device__ __forceinline__ bool is_masked_px(uint32_t v) {
  return sizeof(Pix) == 2 ? v >= 0xFFFEu : v >= 0xFFFFFFFEu;
}

// The reference's decision for one window from exact sums, out of line: the
// callers reach it only between the two bounds.
__device__ __noinline__ bool lat_exact(uint32_t n, uint32_t S, uint32_t Q, const LaunchParams &P) {
  return stage0_u32(n, S, Q, P, P.root_lo, P.root_hi);
}

// The stage-0 bit (signal or masked; off the frame counts as set) of the
// window whose top-left staged pixel is (row, col) of a staged tile, with
// 64-bit sums, for tiles holding a pixel too large for the 32-bit ones. The
// staged tile holds pixels off the frame as masked, so they are skipped as
// the reference's clipped window skips them.
__device__ __noinline__ bool lat_wide(const uint32_t (*px)[kVerPW], int row, int col,
                                      const LaunchParams &P) {
  if (px[row + kLatK][col + kLatK] >= 0xFFFFFFFEu)
    return true;
  uint32_t n = 0;
  unsigned long long S = 0, Q = 0;
  for (int dy = 0; dy <= 2 * kLatK; dy++) {
#pragma unroll
    for (int dx = 0; dx <= 2 * kLatK; dx++) {
      const uint32_t v = px[row + dy][col + dx];
      if (v < 0xFFFFFFFEu) {
        n++;
        S += v;
        Q += (unsigned long long)v * v;
      }
    }
  }
  return stage0_u32(n, S, Q, P, P.root_lo, P.root_hi);
}

// Tiles of a tile row come in groups of 32 consecutive ones: 32 tiles of 28
// columns span 28 mask words (29 with the last tile's straddle), so lane l
// ORs word 28 g + l over the tile row's 8 rows and each lane tests its tile
// from two lanes' ORs. A warp takes a run of up to kTileRun groups (of any
// frames; fewer when a launch has too few groups to give every SM a few
// warps, so that a one-frame launch is not a few warps walking long runs):
// each group is a round trip to memory, so the run sets the kernel's length
// (a 64-frame launch: 131 us with runs of 32, 69 with 16, 45 with 8, 49 with
// 4, where the list's one counter starts to take the atomics in turn),
// keeps their ballots, and takes its list space with one atomic: the
// counter is shared by the whole launch, so fewer atomics contend less.
constexpr int kTileRun = 8;

__global__ void __launch_bounds__(256)
lat_tiles(const __grid_constant__ FramePtrs F, int nframes, int env_h, int env_w,
          const uint32_t *final_all, size_t words, uint32_t *__restrict__ list,
          uint32_t *__restrict__ counters, const __grid_constant__ FrameSpans S, int run) {
  previous_done();
  const int lane = threadIdx.x & 31;
  // Tile numbers are laid out over the batch's largest frame; each frame has
  // its own tile groups (S) and its own shape bounds its tiles.
  const int ntx = ver_ntx(env_w), nty = ver_nty(env_h);
  const uint32_t ntiles = (uint32_t)ntx * (uint32_t)nty;
  const uint32_t total = (uint32_t)S.start[nframes];
  const uint32_t g0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (uint32_t)run;
  if (g0 >= total)
    return;  // whole warp
  unsigned bal[kTileRun];
  uint32_t first[kTileRun];  // the tile number of each group's first tile
  uint32_t mine = 0, n = 0;
#pragma unroll
  for (int i = 0; i < kTileRun; i++) {
    const uint32_t g = g0 + i;
    bool any = false;
    first[i] = 0;
    if (i < run && g < total) {  // warp-uniform
      const int f = span_frame(S, nframes, (int)g);
      const uint32_t gf = g - (uint32_t)S.start[f];
      const uint32_t ty = fast_div(gf, S.by_row[f]), gx = gf - ty * S.by_row[f].d;
      first[i] = (uint32_t)f * ntiles + ty * (uint32_t)ntx + 32 * gx;
      const uint32_t *fin = final_all + (size_t)f * words;
      const int height = F.h[f], width = F.w[f];
      const int wpr = (width + 31) >> 5;
      const int wd = 28 * (int)gx + lane, r0 = (int)ty * kVerRows;
      uint32_t acc = 0;
      if (lane < 29 && wd < wpr) {
#pragma unroll
        for (int o = 0; o < kVerRows; o++)
          if (r0 + o < height)
            acc |= fin[(size_t)(r0 + o) * wpr + wd];
      }
      const int lw = (kVerTW * lane) >> 5, sh = (kVerTW * lane) & 31;
      const uint32_t lo = __shfl_sync(0xffffffffu, acc, lw);
      const uint32_t hi = __shfl_sync(0xffffffffu, acc, lw + 1);
      const int tx = 32 * (int)gx + lane;
      any = tx < ver_ntx(width) &&
            ((uint32_t)(((unsigned long long)hi << 32 | lo) >> sh) & ((1u << kVerTW) - 1u)) != 0u;
    }
    bal[i] = __ballot_sync(0xffffffffu, any);
    mine |= any ? 1u << i : 0u;
    n += (uint32_t)__popc(bal[i]);
  }
  if (n == 0)
    return;  // whole warp
  uint32_t base = 0;
  if (lane == 0)
    base = atomicAdd(counters + kCtrTiles, n);
  base = __shfl_sync(0xffffffffu, base, 0);
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < kTileRun; i++) {
    if ((mine >> i) & 1u)
      list[base + __popc(bal[i] & below)] = first[i] + lane;
    base += (uint32_t)__popc(bal[i]);
  }
}

// Copies a tile's pixel rows (r0 - 5 .. r0 + 12, the staged columns from xs)
// into pix (pieces off the frame are written as masked pixels), for frames
// without a tensor map. 16-bit frames come here only when 4 | width and they are
// 8-byte aligned.
template <typename Pix>
__device__ __forceinline__ void stage_pixels(Pix (*pix)[VerPix<Pix>::kPW], const Pix *image,
                                             int height, int width, int r0, int xs,
                                             int lane) {
  constexpr int kPW = VerPix<Pix>::kPW, kPieces = kPW / 4;
  if (width % 4 == 0 && reinterpret_cast<uintptr_t>(image) % (4 * sizeof(Pix)) == 0) {
    // Pieces of 4 pixels, each wholly inside the frame or wholly outside it.
    for (int k = lane; k < kVerPR * kPieces; k += 32) {
      const int r = k / kPieces, ch = k - r * kPieces;
      const int y = r0 - 5 + r, x = xs + 4 * ch;
      Pix *dst = &pix[r][4 * ch];
      if (y >= 0 && y < height && x >= 0 && x + 4 <= width)
        cp_async_piece<Pix>(dst, image + (size_t)y * width + x);
      else
        fill_piece_masked<Pix>(dst);
    }
  } else {
    for (int k = lane; k < kVerPR * kPW; k += 32) {
      const int r = k / kPW, c = k - r * kPW;
      const int y = r0 - 5 + r, x = xs + c;
      Pix *dst = &pix[r][c];
      if (y >= 0 && y < height && x >= 0 && x < width)
        cp_async4(dst, image + (size_t)y * width + x);
      else
        *dst = (Pix)~0u;
    }
  }
}

// The tile's pixels by one TMA box load of frame f's map at (xs, r0 - 5),
// issued by lane 0 once the warp is done with the buffer; it lands on bar.
template <typename Pix>
__device__ __forceinline__ void tma_stage(TileBuf<Pix> &buf, uint64_t *bar, const TileMaps &M,
                                          int f, int r0, int xs, int lane) {
  __syncwarp();
  if (lane == 0) {
    fence_proxy_async_smem();
    mbar_expect_tx(bar, (uint32_t)sizeof(buf.px));
    tma_load_2d(buf.px, &M.map[f], xs, r0 - 5, bar);
  }
}

// Waits for a TMA-staged tile (every lane, bounded; false in every lane if
// any lane's wait ran out) and, for a tile that reaches past the frame, turns
// the box's zero-filled pixels off the frame into masked ones, as the
// per-lane staging writes them.
template <typename Pix>
__device__ __forceinline__ bool tma_landed(TileBuf<Pix> &buf, uint64_t *bar, uint32_t parity,
                                           int height, int width, int r0, int xs, int lane) {
  constexpr int kPW = VerPix<Pix>::kPW;
  if (!__all_sync(0xffffffffu, mbar_wait(bar, parity)))
    return false;
  const int y0 = r0 - 5;
  if (y0 < 0 || y0 + kVerPR > height || xs < 0 || xs + kPW > width) {  // warp-uniform
    for (int k = lane; k < kVerPR * kPW; k += 32) {
      const int r = k / kPW, c = k - r * kPW;
      const int y = y0 + r, x = xs + c;
      if (y < 0 || y >= height || x < 0 || x >= width)
        buf.px[r][c] = (Pix)~0u;
    }
  }
  __syncwarp();
  return true;
}

// The tile origin of list entry e: frame, first output row and column.
struct TileAt {
  int f, r0, c0;
};
__device__ __forceinline__ TileAt tile_at(uint32_t e, uint32_t ntiles, int ntx,
                                          const FastDiv &by_ntiles, const FastDiv &by_ntx) {
  const uint32_t fu = fast_div(e, by_ntiles), t = e - fu * ntiles, tyu = fast_div(t, by_ntx);
  TileAt a;
  a.f = (int)fu;
  a.r0 = (int)tyu * kVerRows;
  a.c0 = (int)(t - tyu * (uint32_t)ntx) * kVerTW;
  return a;
}
// The staged columns' first column (aligned) for a tile starting at c0.
template <typename Pix> __device__ __forceinline__ int tile_xs(int c0) {
  return (c0 - 5) & ~(VerPix<Pix>::kAlign - 1);
}

template <typename Pix>
__device__ __forceinline__ void ver_stage(VerWarp<Pix> &sm, int s, uint32_t e, const FramePtrs &F,
                                          const TileMaps &M, uint32_t ntiles,
                                          int ntx, const FastDiv &by_ntiles,
                                          const FastDiv &by_ntx,
                                          const uint32_t *__restrict__ final_all,
                                          size_t words, int lane) {
  const TileAt a = tile_at(e, ntiles, ntx, by_ntiles, by_ntx);
  const int f = a.f, r0 = a.r0, c0 = a.c0;
  const int height = F.h[f], width = F.w[f];
  const int xs = tile_xs<Pix>(c0);
  __syncwarp();  // every lane is done with the pixel buffer
  if (M.has(f))
    tma_stage<Pix>(sm.pix, &sm.bar, M, f, r0, xs, lane);
  else
    stage_pixels<Pix>(sm.pix.px, reinterpret_cast<const Pix *>(F.image[f]), height, width, r0,
                      xs, lane);
  if (lane < 2 * kVerRows) {
    const int o = lane >> 1, wdx = (c0 >> 5) + (lane & 1);
    const int wpr = (width + 31) >> 5;
    uint32_t *dst = &sm.cw[s][o][lane & 1];
    if (r0 + o < height && wdx < wpr)
      cp_async4(dst, final_all + (size_t)f * words + (size_t)(r0 + o) * wpr + wdx);
    else
      *dst = 0u;
  }
}

// A lane decides four windows next to one another: stage-0 row d, columns 4j ..
// 4j + 3, of which only those of `need` matter. Their sums share the ten column
// sums they read; the result has bit c set where window c is signal. A window's
// masked count is clamped to its 49 pixels, which keeps the per-count tables in
// bounds whatever the sums.
constexpr int kVerGroup = 4;
static_assert(kVerDR * 32 / kVerGroup % 32 == 0, "whole rounds of groups over the lanes");

template <class Decide>
__device__ __forceinline__ void ver_windows(const uint2 *vs, Decide decide) {
  uint32_t n[kVerGroup + 6], q[kVerGroup + 6];
#pragma unroll
  for (int c = 0; c < (kVerGroup + 6) / 2; c++) {
    const uint4 x = reinterpret_cast<const uint4 *>(vs)[c];
    n[2 * c] = x.x, q[2 * c] = x.y, n[2 * c + 1] = x.z, q[2 * c + 1] = x.w;
  }
  uint32_t Wn = 0, Wq = 0;
#pragma unroll
  for (int c = 0; c < 7; c++) {
    Wn += n[c];
    Wq += q[c];
  }
#pragma unroll
  for (int c = 0; c < kVerGroup; c++) {
    if (c) {
      Wn = Wn - n[c - 1] + n[c + 6];
      Wq = Wq - q[c - 1] + q[c + 6];
    }
    decide(c, Wn, Wq);
  }
}

// 32-bit frames: the two bounds first; the needed windows between them (rare)
// by the reference's sequence. kClean: the tile holds no masked pixel.
template <bool kClean>
__device__ __forceinline__ uint32_t ver_group(const VerWarp<uint32_t> &sm, int d, int j,
                                              uint32_t need, const uint4 *tab,
                                              const LaunchParams &P) {
  uint32_t sig = 0, amb = 0;
  const uint4 t0 = tab[0];
  ver_windows(&sm.vs[d][kVerGroup * j], [&](int c, uint32_t Wn, uint32_t Wq) {
    const uint32_t S = kClean ? Wn : Wn & kLatMask;
    const uint4 t = kClean ? t0 : tab[min(Wn >> kLatPS, (uint32_t)kLatN0)];
    const unsigned long long L = (unsigned long long)Wq * t.x;
    const bool maybe = L > (unsigned long long)S * ((S << kDec) + t.y);
    const bool sure = L >= (unsigned long long)S * ((S << kDec) + t.z) + (2ull << kDec);
    sig |= sure ? 1u << c : 0u;
    amb |= (maybe & !sure) ? 1u << c : 0u;
  });
  amb &= need;
  if (amb) {
    ver_windows(&sm.vs[d][kVerGroup * j], [&](int c, uint32_t Wn, uint32_t Wq) {
      const uint32_t m = min(Wn >> kLatPS, (uint32_t)kLatN0);
      if ((amb >> c & 1u) && lat_exact((uint32_t)kLatN0 - m, Wn & kLatMask, Wq, P))
        sig |= 1u << c;
    });
  }
  return sig;
}

// 16-bit frames: the reference's float test, exactly, its factors {n, root} from
// the table.
template <bool kClean>
__device__ __forceinline__ uint32_t ver_group(const VerWarp<uint16_t> &sm, int d, int j, uint32_t,
                                              const uint4 *tab, const LaunchParams &P) {
  uint32_t sig = 0;
  const float gain = (float)P.gain, sigma_b = (float)P.sigma_b;
  const uint4 t0 = tab[0];
  ver_windows(&sm.vs[d][kVerGroup * j], [&](int c, uint32_t Wn, uint32_t Wq) {
    const uint32_t S = kClean ? Wn : Wn & kLatMask;
    const uint4 t = kClean ? t0 : tab[min(Wn >> kLatPS, (uint32_t)kLatN0)];
    sig |= stage0_float(__uint_as_float(t.x), __uint_as_float(t.y), S, Wq, gain, sigma_b) ? 1u << c
                                                                                         : 0u;
  });
  return sig;
}

// A tile that holds a valid pixel too large for the 32-bit sums but below
// kWidePixel: its column sums again, the masked count above a 28-bit sum and the
// sum of squares in 48 bits. (A launch of 4 dense frames of 4362 x 4148, whose
// tiles nearly all hold an overload, takes 621 us: 783 with the 32-bit sums taken
// first there too, 2136 summing each window's 49 pixels.)
constexpr uint32_t kWidePixel = 1u << 20;
constexpr int kWideCount = 28;
static_assert((2 * kLatK + 1) * (kWidePixel - 1) < (1u << kWideCount) &&
                  (2ull * kLatK + 1) * (kWidePixel - 1) * (kWidePixel - 1) < (1ull << 48),
              "a column's sums fit their fields");
// n Q below 2^53: the reference's own difference is exact, as the tests' 2 units
// between them need, and 2^8 n Q and S (2^8 S + c) stay below 2^64.
static_assert(49ull * 49ull * (kWidePixel - 1) * (kWidePixel - 1) < (1ull << 53),
              "a window's sums are exact in double");

// Returns the lane's largest valid pixel.
__device__ __noinline__ uint32_t ver_wide_columns(VerWarp<uint32_t> &sm, int off, int npass,
                                                  int lane) {
  uint32_t top = 0;
  for (int pass = 0; pass < npass; pass++) {
    const int i = 32 * pass + lane;
    if (i >= kVerPC)
      break;
    uint32_t u[kVerPR], masked = 0, cs = 0;  // (cs: count and sum)
    unsigned long long cq = 0;
#pragma unroll
    for (int r = 0; r < kVerPR; r++) {
      const uint32_t v = sm.pix.px[r][off + i];
      const bool m = is_masked_px<uint32_t>(v);
      masked |= m ? 1u << r : 0u;
      u[r] = m ? 0u : v;
      top = max(top, u[r]);
    }
#pragma unroll
    for (int r = 0; r < kVerPR; r++) {
      cs += u[r] + ((masked >> r & 1u) << kWideCount);
      cq += (unsigned long long)u[r] * u[r];
      if (r >= 2 * kLatK) {
        const int d = r - 2 * kLatK;
        sm.vs[d][i] = make_uint2(cs, (uint32_t)cq);
        sm.vh[d][i] = (uint16_t)(cq >> 32);
        cs -= u[d] + ((masked >> d & 1u) << kWideCount);
        cq -= (unsigned long long)u[d] * u[d];
      }
    }
    sm.msk[i + 1] = masked >> kLatK;  // (rows past the centres' are not looked at)
  }
  return top;
}

// ver_group from those sums: the same two bounds in 64 bits, then the reference's
// sequence.
__device__ __noinline__ uint32_t ver_wide_group(const VerWarp<uint32_t> &sm, int d, int j,
                                                uint32_t need, const uint4 *tab,
                                                const LaunchParams &P) {
  constexpr int kN = kVerGroup + 6;
  uint32_t n[kN], lo[kN], hi[kN];
#pragma unroll
  for (int c = 0; c < kN / 2; c++) {
    const uint4 x = reinterpret_cast<const uint4 *>(&sm.vs[d][kVerGroup * j])[c];
    const uint32_t h = reinterpret_cast<const uint32_t *>(&sm.vh[d][kVerGroup * j])[c];
    n[2 * c] = x.x, lo[2 * c] = x.y, hi[2 * c] = h & 0xFFFFu;
    n[2 * c + 1] = x.z, lo[2 * c + 1] = x.w, hi[2 * c + 1] = h >> 16;
  }
  uint32_t m = 0, S = 0, sig = 0;
  unsigned long long Q = 0;
#pragma unroll
  for (int c = 0; c < kN; c++) {
    m += n[c] >> kWideCount;
    S += n[c] & ((1u << kWideCount) - 1u);
    Q += (unsigned long long)hi[c] << 32 | lo[c];
    if (c >= 6) {
      const uint32_t mc = min(m, (uint32_t)kLatN0);
      const uint4 t = tab[mc];
      const unsigned long long L = Q * t.x, S8 = (unsigned long long)S << kDec;
      bool is = L >= S * (S8 + t.z) + (2ull << kDec);
      if (!is && (need >> (c - 6) & 1u) && L > S * (S8 + t.y))
        is = stage0_u32((uint32_t)kLatN0 - mc, S, Q, P, P.root_lo, P.root_hi);
      sig |= is ? 1u << (c - 6) : 0u;
      m -= n[c - 6] >> kWideCount;
      S -= n[c - 6] & ((1u << kWideCount) - 1u);
      Q -= (unsigned long long)hi[c - 6] << 32 | lo[c - 6];
    }
  }
  return sig;
}

template <int kOcc, typename Pix>
__global__ void __launch_bounds__(kVerWarps * 32, kOcc)
lat_verify(const __grid_constant__ FramePtrs F, const __grid_constant__ TileMaps M, int env_h,
           int env_w, const __grid_constant__ LaunchParams P,
           const __grid_constant__ StreamTables T, uint32_t *__restrict__ final_all, size_t words,
           const uint32_t *list, uint32_t *__restrict__ counters, FastDiv by_ntiles,
           FastDiv by_ntx) {
  previous_done();
  extern __shared__ __align__(128) unsigned char ver_smem_raw[];
  // The launch gives 128 bytes more than the layout needs: the tile buffers
  // start on a 128-byte boundary whatever the base's alignment.
  unsigned char *ver_smem = ver_smem_raw + ((128u - (smem_addr(ver_smem_raw) & 127u)) & 127u);
  uint4 *tab = reinterpret_cast<uint4 *>(ver_smem);
  constexpr bool k16 = sizeof(Pix) == 2;
  VerWarp<Pix> *warps = reinterpret_cast<VerWarp<Pix> *>(ver_smem + sizeof(uint4) * 64);
  for (int m = threadIdx.x; m <= kLatN0; m += blockDim.x)
    if constexpr (k16) {
      const int n = kLatN0 - m;  // (a NaN root: no test passes)
      tab[m] = make_uint4(__float_as_uint((float)n),
                          (uint32_t)n < P.min_local ? 0x7FFFFFFFu : __float_as_uint(P.rootf[n]),
                          0u, 0u);
    } else {
      tab[m] = make_uint4(T.nk[kLatN0 - m], T.clo[kLatN0 - m], T.chi[kLatN0 - m], 0u);
    }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  VerWarp<Pix> &sm = warps[warp];
  if (lane == 0) {
    mbar_init(&sm.bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  uint32_t parity = 0;  // the phase the next wait on bar waits for
  // Tile numbers are laid out over the batch's largest frame.
  const int ntx = ver_ntx(env_w);
  const uint32_t ntiles = (uint32_t)ntx * (uint32_t)ver_nty(env_h);
  const uint32_t narrow2 = T.narrow_max + 2u;
  const uint32_t count = counters[kCtrTiles];
  const uint32_t nw = gridDim.x * kVerWarps;
  uint32_t k = blockIdx.x * kVerWarps + warp;
  // List entries are read a tile before they are staged. A warp has one
  // pixel buffer: the next tile's load goes out as soon as this tile's pixels
  // have been read (after the column sums, or after the windows summed from
  // the pixels on a frame with very large counts), and runs under the rest of
  // this tile's check. The candidate words are staged into the other of two.
  uint32_t e = k < count ? list[k] : 0u;
  uint32_t e1 = k + nw < count ? list[k + nw] : 0u;
  if (k < count)
    ver_stage<Pix>(sm, 0, e, F, M, ntiles, ntx, by_ntiles, by_ntx, final_all, words,
                   lane);
  cp_async_commit();
  uint32_t e2 = 0u;
  // A TMA load not waited for.
  auto mapped = [&](uint32_t x) { return M.has((int)fast_div(x, by_ntiles)); };
  bool inflight = k < count && mapped(e);
  for (int s = 0; k < count; k += nw, s ^= 1, e = e1, e1 = e2) {
    e2 = k + 2 * nw < count ? list[k + 2 * nw] : 0u;
    cp_async_wait<0>();  // this tile's pieces have landed
    __syncwarp();
    const TileAt a = tile_at(e, ntiles, ntx, by_ntiles, by_ntx);
    const int f = a.f, r0 = a.r0, c0 = a.c0;
    const int height = F.h[f], width = F.w[f], wpr = (width + 31) >> 5;
    if (inflight) {
      inflight = false;
      if (!tma_landed<Pix>(sm.pix, &sm.bar, parity, height, width, r0,
                           tile_xs<Pix>(c0), lane)) {
        if (lane == 0)
          atomicOr(counters + kCtrFault, 1u);
        break;  // whole warp
      }
      parity ^= 1u;
    }
    // The next tile's load, once this tile's pixels have been read.
    auto stage_next = [&]() {
      if (k + nw < count) {
        ver_stage<Pix>(sm, s ^ 1, e1, F, M, ntiles, ntx, by_ntiles, by_ntx,
                       final_all, words, lane);
        inflight = mapped(e1);
      }
      cp_async_commit();
    };
    const int off = (c0 - 5) - tile_xs<Pix>(c0);
    const int w0 = c0 >> 5, sh = c0 & 31;
    // The tile's candidates, a row a lane (lanes 0-7).
    uint32_t cj = 0;
    if (lane < kVerRows)
      cj = (uint32_t)(((unsigned long long)sm.cw[s][lane][0] |
                       (unsigned long long)sm.cw[s][lane][1] << 32) >> sh) &
           ((1u << kVerTW) - 1u);
    // Columns B (pixel columns 32-37, stage-0 columns 26-31) matter only
    // when a candidate lies in the tile's last 6 columns.
    const bool late = __any_sync(0xffffffffu, (cj >> 22) != 0u);
    const int npass = late ? 2 : 1;
    // Pixel columns off + lane (A) and off + 32 + lane (B, lanes 0-5): the
    // masked centres, the largest valid pixel, and the column sums of 7
    // rows for the 12 stage-0 rows (exact in 32 bits unless the tile holds a
    // valid pixel at or above narrow_max, which the check below catches).
    // (A tile with a larger one leaves this for the wide sums at once.)
    uint32_t masked = 0;
    bool wide = false;
#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
      if (pass == npass)
        break;  // warp-uniform
      const bool on = pass == 0 || lane < kVerPC - 32;
      const int col = off + 32 * pass + (on ? lane : 0);
      uint32_t ns[kVerPR], q[kVerPR], mk = 0, mx = 0;
#pragma unroll
      for (int r = 0; r < kVerPR; r++) {
        const uint32_t v = sm.pix.px[r][col];
        if (!k16)
          mx = max(mx, v + 2u);
        ns[r] = is_masked_px<Pix>(v) ? (1u << kLatPS) : v;
      }
      if (!k16 && __any_sync(0xffffffffu, mx >= narrow2)) {
        wide = true;
        break;  // warp-uniform
      }
      if (!on)
        break;
#pragma unroll
      for (int r = 0; r < kVerPR; r++)
        q[r] = ns[r] * ns[r];
      // A valid pixel below narrow_max (2^14) leaves nothing of itself when
      // its count bit is shifted down; a 16-bit one may.
#pragma unroll
      for (int d = 0; d < kVerDR; d++)
        mk += k16 ? (ns[d + kLatK] >> kLatPS) << d : ns[d + kLatK] >> (kLatPS - d);
      sm.msk[32 * pass + lane + 1] = mk;
      uint32_t cn = 0, cq = 0;
#pragma unroll
      for (int r = 0; r < 2 * kLatK; r++) {
        cn += ns[r];
        cq += q[r];
      }
#pragma unroll
      for (int d = 0; d < kVerDR; d++) {
        cn += ns[d + 2 * kLatK];
        cq += q[d + 2 * kLatK];
        sm.vs[d][32 * pass + lane] = make_uint2(cn, cq);
        if (d == 0 || d == 7 || d == kVerDR - 1)
          masked |= cn;  // (these three cover the column)
        cn -= ns[d];
        cq -= q[d];
      }
    }
    __syncwarp();
    // 16-bit frames sum in 32 bits as the reference does: never wide.
    bool huge = false;
    if constexpr (!k16) {
      if (wide) {
        const uint32_t top = ver_wide_columns(sm, off, npass, lane);
        huge = __any_sync(0xffffffffu, top >= kWidePixel);
        __syncwarp();
      }
    }
    if (!huge)
      stage_next();  // the windows come from the column sums, not the pixels
    // The stage-0 positions within 2 of a candidate, lane d row d's (row r0 - 2
    // + d, bit = column c0 - 2 + bit): the rows' candidates d - 4 .. d (a lane
    // without a row so far up ORs itself again).
    uint32_t need = cj | __shfl_up_sync(0xffffffffu, cj, 1);
    need |= __shfl_up_sync(0xffffffffu, need, 2);
    need |= __shfl_up_sync(0xffffffffu, cj, 4);
    need = (need | need << 1) | (need | need << 1) << 2 | need << 4;
    const unsigned live = __ballot_sync(0xffffffffu, need != 0u);
    const bool clean = !wide && !__any_sync(0xffffffffu, (masked >> kLatPS) != 0u);
    // Rounds of four rows, a group of four windows a lane. A row's bit is set
    // where its window is signal, its centre masked, or neither needed.
    uint32_t D = 0xFFFFFFFFu;  // lane d: row d
#pragma unroll 1
    for (int d0 = 0; d0 < kVerDR; d0 += kVerGroup) {
      if (!(live >> d0 & ((1u << kVerGroup) - 1u)))
        continue;  // warp-uniform
      const int d = d0 + (lane >> 3), j = lane & 7;
      uint32_t nd = __shfl_sync(0xffffffffu, need, d) >> (kVerGroup * j) & 15u, sig;
      if (huge) {
        // 64-bit sums of each window's pixels (frames with very large counts).
        sig = 0;
        if constexpr (!k16)
          for (int c = 0; c < kVerGroup; c++)
            if (nd >> c & 1u)
              sig |= lat_wide(sm.pix.px, d, off + kVerGroup * j + c, P) ? 1u << c : 0u;
      } else if (clean) {
        sig = ver_group<true>(sm, d, j, nd, tab, P);
      } else {
        const uint4 m = *reinterpret_cast<const uint4 *>(&sm.msk[kVerGroup * j + kLatK + 1]);
        nd &= ~((m.x >> d & 1u) | (m.y >> d & 1u) << 1 | (m.z >> d & 1u) << 2 |
                (m.w >> d & 1u) << 3);
        if (!wide)
          sig = ver_group<false>(sm, d, j, nd, tab, P);
        else if constexpr (!k16)
          sig = ver_wide_group(sm, d, j, nd, tab, P);
      }
      uint32_t row = ((~nd | sig) & 15u) << (kVerGroup * j);
      row |= __shfl_xor_sync(0xffffffffu, row, 1);
      row |= __shfl_xor_sync(0xffffffffu, row, 2);
      row |= __shfl_xor_sync(0xffffffffu, row, 4);
      row = __shfl_sync(0xffffffffu, row, (8 * (lane - d0)) & 31);
      if (lane >= d0 && lane < d0 + kVerGroup)
        D = row;
    }
    if (huge)
      stage_next();
    __syncwarp();  // the next tile rewrites the shared rows
    // The exact erosion, lane o row o's; the candidates that fail leave the mask.
    uint32_t V = D & __shfl_down_sync(0xffffffffu, D, 1);
    V &= __shfl_down_sync(0xffffffffu, V, 2);
    V &= __shfl_down_sync(0xffffffffu, D, 4);
    uint32_t H = V & V >> 1;
    H &= H >> 2;
    H &= V >> 4;
    const uint32_t clear = cj & ~H;  // (cj is 0 in lanes without a row)
    if (clear) {
      const unsigned long long c64 = (unsigned long long)clear << sh;
      uint32_t *at = final_all + (size_t)f * words + (size_t)(r0 + lane) * wpr + w0;
      if ((uint32_t)c64)
        atomicAnd(at, ~(uint32_t)c64);
      if ((uint32_t)(c64 >> 32) && w0 + 1 < wpr)
        atomicAnd(at + 1, ~(uint32_t)(c64 >> 32));
    }
  }
  // After a fault: the load still in flight (bounded) before the buffer goes.
  if (inflight)
    (void)mbar_wait(&sm.bar, parity);
  cp_async_wait<0>();
}

// Adds 128 bytes for aligning the tile buffers (see the kernel).
template <typename Pix> constexpr size_t ver_smem_bytes() {
  return sizeof(uint4) * 64 + sizeof(VerWarp<Pix>) * kVerWarps + 128;
}
static_assert(sizeof(uint4) * 64 % 128 == 0, "the verify warps start 128-byte aligned");
static_assert((ver_smem_bytes<uint32_t>() + 1024) * kVerOcc <= 228 * 1024,
              "six exact-check blocks an SM");

int lat_slots() {
  static int slots = 0;
  if (!slots) {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, lat_stage01<kLatOcc, uint32_t>,
                                                  kLatWarps * 32, ring_bytes<uint32_t>());
    slots = std::max(1, per) * kLatWarps * device_sms();
  }
  return slots;
}

// Blocks an SM of a persistent kernel with `bytes` of dynamic shared memory,
// once per instantiation (the attribute set first).
template <class Kernel> cudaError_t persistent_blocks(Kernel k, size_t bytes, int *blocks) {
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  int per = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kVerWarps * 32, bytes);
  *blocks = std::max(1, per);
  return e;
}

// The launch's frames mapped for the TMA staging of tiles; a frame that cannot
// be (not 16-byte aligned, a row pitch that is not a multiple of 16 bytes, no
// driver entry point) has its tiles staged per lane.
template <typename Pix> void make_tile_maps(const FramePtrs &F, int nframes, TileMaps *M) {
  std::memset(M, 0, sizeof(*M));
  for (int f = 0; f < nframes; f++)
    if (encode_frame_map(&M->map[f], F.image[f], F.h[f], F.w[f], (int)sizeof(Pix),
                         VerPix<Pix>::kPW, kVerPR))
      M->mapped |= 1ull << f;
}

// Strips of a frame w wide (whole mask rows: the last strip reaches the end
// of the row's last word).
int lat_strips(int w) { return ((w + 31) / 32 * 32 + kLatOut - 1) / kLatOut; }

template <typename Pix>
cudaError_t lattice(const FramePtrs &F, int nframes, int h, int w, const LaunchParams &P,
                    const StreamTables &T, const StreamBuffers &b, int run_rows,
                    cudaStream_t stream) {
  // Each frame's strips x runs of run_rows rows, frame after frame.
  FrameSpans S;
  S.start[0] = 0;
  for (int f = 0; f < nframes; f++) {
    const int strips = lat_strips(F.w[f]);
    S.start[f + 1] = S.start[f] + strips * ((F.h[f] + run_rows - 1) / run_rows);
    S.by_row[f] = make_fastdiv((uint32_t)strips);
  }
  const size_t mask_bytes = b.words * sizeof(uint32_t);
  const unsigned lb = (unsigned)((S.start[nframes] + kLatWarps - 1) / kLatWarps);
  uint8_t *fin = reinterpret_cast<uint8_t *>(b.cand);
  lat_stage01<kLatOcc, Pix><<<lb, kLatWarps * 32, ring_bytes<Pix>(), stream>>>(
      F, nframes, S, run_rows, T, P, fin, mask_bytes, b.counters);
  static std::once_flag configured;
  static cudaError_t config_error = cudaSuccess;
  static int ver_blocks = 0;
  std::call_once(configured, [] {
    config_error = persistent_blocks(lat_verify<kVerOcc, Pix>, ver_smem_bytes<Pix>(),
                                     &ver_blocks);
  });
  if (config_error != cudaSuccess)
    return config_error;
  // Tile groups: each frame's tile rows x groups of 32 tiles.
  FrameSpans G;
  G.start[0] = 0;
  for (int f = 0; f < nframes; f++) {
    const int ngx = (ver_ntx(F.w[f]) + 31) / 32;
    G.start[f + 1] = G.start[f] + ver_nty(F.h[f]) * ngx;
    G.by_row[f] = make_fastdiv((uint32_t)ngx);
  }
  const long long tgroups = G.start[nframes];
  // Runs of kTileRun groups a warp, shorter when that would leave fewer than
  // 8 warps an SM (one frame: runs of 2).
  const int trun = (int)std::max(1ll, std::min((long long)kTileRun,
                                               tgroups / (8ll * device_sms())));
  const long long twarps = (tgroups + trun - 1) / trun;
  const unsigned tb = (unsigned)((twarps + 7) / 8);
  const size_t tiles = (size_t)ver_ntx(w) * (size_t)ver_nty(h);
  uint32_t *list = b.tiles;
  const FastDiv by_ntiles = make_fastdiv((uint32_t)tiles);
  const FastDiv by_ntx = make_fastdiv((uint32_t)ver_ntx(w));
  launch_after(lat_tiles, tb, 256, 0, stream, F, nframes, h, w, b.cand, b.words, list, b.counters,
               G, trun);
  TileMaps M;
  make_tile_maps<Pix>(F, nframes, &M);
  launch_after(lat_verify<kVerOcc, Pix>, ver_blocks * device_sms(), kVerWarps * 32,
               ver_smem_bytes<Pix>(), stream, F, M, h, w, P, T, b.cand, b.words, list, b.counters,
               by_ntiles, by_ntx);
  return cudaGetLastError();
}

} // namespace

bool encode_frame_map(CUtensorMap *map, const void *base, int h, int w, int bytes_per_pixel,
                      int box_w, int box_h) {
  // The driver's encoder, looked up once (no link against libcuda).
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }();
  const size_t pitch = (size_t)w * (size_t)bytes_per_pixel;
  if (!encode || !base || reinterpret_cast<uintptr_t>(base) % 16 != 0 || pitch % 16 != 0 ||
      h < 1 || w < 1 || (bytes_per_pixel != 2 && bytes_per_pixel != 4))
    return false;
  const cuuint64_t dims[2] = {(cuuint64_t)w, (cuuint64_t)h};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch};
  const cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
  const cuuint32_t step[2] = {1, 1};
  return encode(map,
                bytes_per_pixel == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32
                                     : CU_TENSOR_MAP_DATA_TYPE_UINT16,
                2, const_cast<void *>(base), dims, strides, box, step,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t lattice_tiles(int h, int w) { return (size_t)ver_ntx(w) * (size_t)ver_nty(h); }

// The run length for a launch whose tallest frame has h rows and whose frames
// have `strips` strips in all, unless run_rows is given (but see kShortRun), in whole triples of
// rows: the resident warps filled kLatWaves times over by runs of at least
// kLatLongRun rows (each reads 9 rows more than it writes), so that warps of
// unequal speed even out (32 frames of 4362 x 4148: 424 us, 447 with three times
// and 144 rows); else once, down to runs of kLatMinRunRows.
static int lat_run_rows(int h, long long strips, int run_rows) {
  const long long nruns = std::max(1ll, (long long)lat_slots() / std::max(1ll, strips));
  const int once = (int)((h + nruns - 1) / nruns);
  if (run_rows <= 0)
    run_rows = std::min(once, std::max(kLatLongRun, (once + kLatWaves - 1) / kLatWaves));
  else if (once < kShortRun)
    run_rows = std::min(run_rows, once);
  run_rows = std::max(run_rows, kLatMinRunRows);
  return (run_rows + 2) / 3 * 3;
}

LatticeGeometry lattice_geometry(int h, int w, int nframes, int run_rows) {
  LatticeGeometry g;
  g.nstrips = lat_strips(w);
  g.run_rows = lat_run_rows(h, (long long)nframes * g.nstrips, run_rows);
  g.nruns = (h + g.run_rows - 1) / g.run_rows;
  return g;
}

// The lattice pass's and the tile check's constants (sf_lattice.cu): a window
// of 49 pixels, its masked count above a 26-bit sum.
static void make_stream_tables(const LaunchParams &P, StreamTables *T) {
  constexpr int n0 = 49;
  // Exact 32-bit sums: the count and sum packed below 2^32, and the window's
  // sum of p^2 below 2^32 (p < sqrt(2^32 / n0) = 9362).
  const uint32_t by_pack = ((1u << 26) - 1u) / (uint32_t)n0;
  uint32_t by_sq = (uint32_t)std::floor(std::sqrt(4294967295.0 / n0));
  while ((uint64_t)by_sq * by_sq * (uint64_t)n0 > 0xFFFFFFFFull)
    by_sq--;
  T->narrow_max = std::min(by_pack, by_sq + 1);
  for (int n = 0; n <= kMaxN0; n++) {
    const bool testable = n >= 1 && (uint32_t)n >= P.min_local && n <= n0;
    // 2^8 (n - 1 + sigma_b r_n) bracketed from r_n's 2^-20 floor and ceiling.
    const uint64_t sb = P.sigma_b_int;
    const uint64_t lo = testable ? (sb * P.root_lo[n]) >> (kRootShift - kDec) : 0;
    const uint64_t hi =
        testable ? (sb * P.root_hi[n] + ((1ull << (kRootShift - kDec)) - 1)) >>
                       (kRootShift - kDec)
                 : 0;
    const uint64_t base = testable ? (uint64_t)(n - 1) << kDec : 0;
    T->clo[n] = (uint32_t)(base + lo);
    T->chi[n] = (uint32_t)(base + hi);
    // nk 0 makes every such window "surely not" (0 <= S (2^8 S + clo)).
    T->nk[n] = testable ? (uint32_t)n << kDec : 0u;
  }
}

cudaError_t launch_lattice(const FramePtrs &F, int nframes, int h, int w, int pixel_bytes,
                           const LaunchParams &P, const StreamBuffers &b, int run_rows,
                           cudaStream_t stream) {
  if (P.half != kLatK)
    return cudaErrorInvalidValue;
  StreamTables T;
  make_stream_tables(P, &T);
  long long strips = 0;
  for (int f = 0; f < nframes; f++)
    strips += lat_strips(F.w[f]);
  const int rr = lat_run_rows(h, strips, run_rows);
  return pixel_bytes == 2 ? lattice<uint16_t>(F, nframes, h, w, P, T, b, rr, stream)
                          : lattice<uint32_t>(F, nframes, h, w, P, T, b, rr, stream);
}

} // namespace sf
