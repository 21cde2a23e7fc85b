// The dispersion_extended threshold (the reference's algorithm,
// src/spots/dext.cc:53-222), for one frame or a batch of frames per launch
// sequence, of either pixel type, any kernel size, aligned or not:
//
//   ext_strip       stage 0 (the dispersion test) of every pixel and the
//                   erosion, one warp per strip and run of rows: the candidate
//                   mask, whose pixels with the masked ones are the reference's
//                   eroded mask
//   ext_decide      stage 2 (the Poisson test over the background) at each
//                   candidate: the strong-pixel mask, the passing pixels'
//                   results and the blocks' counts
//   scatter_pixels  the records, ascending (sf_groups.cuh)
//
// Each frame is thresholded alone: no sum, mask or list crosses frames, and no
// list of candidates is kept, so none can overflow.
//
// The stage-0 decision of 32-bit frames from exact window sums. The
// reference's test (dext.cc:99-109) is A > X in double, A = nQ - S^2 - g S (n -
// 1) and X = g S sigma_b r_n (r_n its double sqrt(2 (n - 1))). Writing c = g (n
// - 1 + sigma_b r_n), it is n Q > S (S + c). Per window count n the host gives
// integers clo <= 2^8 c <= chi and nk = 2^8 n (0 when n cannot be tested):
//   2^8 n Q <= S (2^8 S + clo)           =>  not signal
//   2^8 n Q >= S (2^8 S + chi) + 2^9     =>  signal
// both exact in 64-bit integers. With gain 1 and an integral sigma_b, A is
// exact in double and A >= X + 2 > RN(X) in the second case; with others clo
// and chi are a unit further out, S / 2^8 of margin against the reference's
// rounding of sums below 2^38 (under 2^-13). What lies between goes to the
// reference's own sequence (sf_common.cuh). 16-bit frames are decided by their
// float sequence everywhere.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "sf_common.cuh"
#include "sf_groups.cuh"
#include "sf_lattice.cuh"
#include "sf_stream.cuh"
#include "sf_strips.cuh"

namespace sf {
namespace {

// By window count n: nk, clo, chi above in 2^-8 units, and clo and chi rounded
// outwards to 2^-4 units; `big` is the sum of squares from which the 2^-4
// tests' products may leave 32 bits.
struct ExtTables {
  uint32_t nk[kMaxN0 + 1], clo[kMaxN0 + 1], chi[kMaxN0 + 1];
  uint32_t clo16[kMaxN0 + 1], chi16[kMaxN0 + 1];
  uint32_t big;
};

// The largest 2^8 c the 64-bit tests take: with S below 2^20 (sums of pixels
// below Cap), (S << 8) + chi stays in 32 bits.
constexpr double kMaxC8 = 2147483648.0;

// The reference's decision for one window of exact sums, out of line: reached
// only between the two bounds.
__device__ __noinline__ bool ext_exact(uint32_t n, unsigned long long S, unsigned long long Q,
                                         const LaunchParams &P) {
  return stage0_u32(n, S, Q, P, P.root_lo, P.root_hi);
}

// Pixels of 32-bit frames are kept up to kLargePixel in the ring. A column's sum
// of those of 2K + 1 rows stays below the count field, and n Q of a window below
// 2^53: with gain 1 and a whole sigma the reference's own difference is exact.
constexpr uint32_t kLargePixel = 1u << 20;
static_assert(9u * kLargePixel < (1u << kCountShift) &&
                  81ull * 81ull * kLargePixel * kLargePixel < (1ull << 53),
              "the sums of large pixels fit");

// A window's constants, of n valid pixels: the 2^-4 tests' {-nk,
// clo, chi - clo} and n, and the 2^-8 tests' {nk, clo, chi}; for 16-bit frames
// {n, rootf} as floats (rootf NaN, no test passes, below min_local).
struct ExtRow {
  uint4 a, b;
};

// A lane's 64-bit column sums, and by shuffles those of the K columns either side of
// its own, summed over the 2K + 1 columns around each of its own, in place.
template <int K, int C> __device__ __forceinline__ void wide_sums(unsigned long long v[C]) {
  unsigned long long e[C + 2 * K], h = 0;
#pragma unroll
  for (int c = 0; c < C; c++)
    e[K + c] = v[c];
#pragma unroll
  for (int k = 0; k < K; k++) {
    e[k] = __shfl_up_sync(0xffffffffu, v[C - K + k], 1);
    e[K + C + k] = __shfl_down_sync(0xffffffffu, v[k], 1);
  }
#pragma unroll
  for (int k = 0; k < 2 * K; k++)
    h += e[k];
#pragma unroll
  for (int c = 0; c < C; c++) {
    h += e[c + 2 * K];
    v[c] = h;
    h -= e[c];
  }
}

// The stage-0 bits of the windows centred on row y, columns cx ..: from 64-bit sums
// of the frame's pixels, for rows whose windows may hold a pixel too large for the
// strip's sums; a window off the frame is clipped as the reference's is. Masked
// centres, and those off the frame, are the caller's to set. (4 frames of 3262 x 3108
// with 2 million counts a pixel: 1.26 ms at kernel 2 and 2.37 at 4; 1.66 and 3.99
// where each lane read its neighbours' columns too, a pixel a load.)
template <int K, int C>
__device__ __noinline__ uint32_t ext_wide_row(const uint32_t *__restrict__ image, int height,
                                              int width, int y, int cx, const LaunchParams &P) {
  constexpr int kPacked = 48;  // valid pixels above their sum: 81 x 2^32 is below 2^39
  unsigned long long s[C], q[C];
#pragma unroll
  for (int c = 0; c < C; c++)
    s[c] = q[c] = 0ull;
  const bool pieces = cx >= 0 && cx + C <= width && width % 4 == 0 &&
                      reinterpret_cast<uintptr_t>(image) % 16 == 0;
  constexpr int kInFlight = C == kNarrowCols ? 2 * K + 1 : 1;  // rows (12 columns a lane spill)
#pragma unroll kInFlight
  for (int yy = max(0, y - K); yy <= min(height - 1, y + K); yy++) {
    const uint32_t *row = image + ((ptrdiff_t)yy * width + cx);
#pragma unroll
    for (int i = 0; i < C; i += 4) {
      uint4 x;
      if (pieces) {
        x = __ldg(reinterpret_cast<const uint4 *>(row + i));
      } else {
        auto at = [&](int c) {
          return cx + c >= 0 && cx + c < width ? __ldg(row + c) : 0xFFFFFFFFu;
        };
        x = make_uint4(at(i), at(i + 1), at(i + 2), at(i + 3));
      }
      const uint32_t v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const bool ok = v[c] < 0xFFFFFFFEu;
        s[i + c] += ok ? (1ull << kPacked) + v[c] : 0ull;
        q[i + c] += ok ? (unsigned long long)v[c] * v[c] : 0ull;
      }
    }
  }
  __syncwarp();
  wide_sums<K, C>(s);
  wide_sums<K, C>(q);
  uint32_t bits = 0;
#pragma unroll
  for (int c = 0; c < C; c++)
    bits |= ext_exact((uint32_t)(s[c] >> kPacked), s[c] & ((1ull << kPacked) - 1ull), q[c], P)
                ? 1u << c
                : 0u;
  return bits;
}

// The stage-0 bits of a lane's windows whose newest row is the ring's slot s, for rows whose windows may hold a pixel of Cap or more: the columns'
// sums again from the ring's rows, squares in 64 bits, and the 2^-8 tests in 64
// bits; by ext_wide_row where one of the warp's pixels is kLargePixel or more.
// (Two dense frames of 353 x 944 at kernel 4, every row of them so, take 80 us in all, 272 with every such row by
// ext_wide_row; 16 of 2162 x 2068 at kernel 2 take 0.97 ms.)
template <int K, int C>
__device__ __noinline__ uint32_t ext_large_row(const uint32_t *ring, int s, int lane,
                                               const ExtRow *tab, const LaunchParams &P,
                                               const uint32_t *image, int height, int width, int y,
                                               int cx) {
  using G = StripG<K>;
  uint32_t n[C + 2 * K], top = 0;
  unsigned long long q[C + 2 * K];
#pragma unroll
  for (int c = 0; c < C; c++)
    n[K + c] = 0u, q[K + c] = 0ull;
#pragma unroll 1
  for (int d = 0; d < G::W0; d++) {
    const uint4 *src = reinterpret_cast<const uint4 *>(ring + s * kStripStride<C> + C * lane);
#pragma unroll
    for (int i = 0; i < C / 4; i++) {
      const uint4 x = src[i];
      const uint32_t v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t u = (uint32_t)max((int)v[k], 0);
        top = max(top, u);
        n[K + 4 * i + k] += v[k];
        q[K + 4 * i + k] += (unsigned long long)u * u;
      }
    }
    s = s == 0 ? G::Slots - 1 : s - 1;
  }
  if (__any_sync(0xffffffffu, top >= kLargePixel))
    return ext_wide_row<K, C>(image, height, width, y, cx, P);
#pragma unroll
  for (int k = 0; k < K; k++) {
    n[k] = __shfl_up_sync(0xffffffffu, n[C + k], 1);
    q[k] = __shfl_up_sync(0xffffffffu, q[C + k], 1);
    n[K + C + k] = __shfl_down_sync(0xffffffffu, n[K + k], 1);
    q[K + C + k] = __shfl_down_sync(0xffffffffu, q[K + k], 1);
  }
  // With another gain or sigma it rounds, by far less than the 2 units between the
  // tests below this.
  const unsigned long long limit = P.int_ok ? ~0ull : 1ull << 42;
  uint32_t m = 0, S = 0, bits = 0;
  unsigned long long Q = 0;
#pragma unroll
  for (int j = 0; j < C + 2 * K; j++) {
    m -= masked_of(n[j]);
    S += n[j] & kSumMask;
    Q += q[j];
    if (j >= 2 * K) {
      const uint32_t masked = min(m, (uint32_t)G::N0);
      const uint4 t = tab[-(int)masked].b;
      const unsigned long long L = Q * t.x, S8 = (unsigned long long)S << 8;
      bool sig = L >= S * (S8 + t.z) + (2ull << 8);
      if (Q >= limit || (!sig && L > S * (S8 + t.y)))
        sig = ext_exact(G::N0 - masked, S, Q, P);
      bits |= sig ? 1u << (j - 2 * K) : 0u;
      m += masked_of(n[j - 2 * K]);
      S -= n[j - 2 * K] & kSumMask;
      Q -= q[j - 2 * K];
    }
  }
  return bits;
}

// The walk of sf_strips.cuh for stage 0, then the erosion (dext.cc:117-142):
// the rows' decision bits are kept for 2E + 1 rows and ANDed down the
// column, then across the lane's and its neighbours' columns. A warp row goes
// only as far as it must: the lower 2^-4 bound alone where no window of the
// row may be signal; both 2^-4 bounds; both 2^-8 bounds where a window lies
// between those or is too big for them; the reference's sequence between
// those; and 64-bit squares where a window may hold a pixel of Cap or more. Bound by
// issue and, at 10 to 13 warps an SM (registers), its latency: 51 instructions a
// pixel at 61% of the issue rate. 16 frames of 3262 x 3108 at kernel 4 take 372
// us, 425 with the decisions compared, selected and ORed (66 instructions), 556
// as 240-column strips with the windows' row sums carried in shared memory, the
// 64-bit rows and the ambiguous windows in passes of their own.
template <int K, typename Pix, int C>
__global__ void __launch_bounds__(kStripWarps * 32, StripG<K>::Occ)
ext_strip(const __grid_constant__ FramePtrs F, int nframes, const __grid_constant__ FrameSpans S,
          int run_rows, const __grid_constant__ ExtTables T,
          const __grid_constant__ LaunchParams P, uint8_t *__restrict__ cand_all,
          size_t mask_bytes) {
  previous_done();
  using G = StripG<K>;
  constexpr bool k16 = sizeof(Pix) == 2;
  constexpr int E = K - 1;
  extern __shared__ __align__(16) unsigned char ext_raw[];
  __shared__ ExtRow rows_tab[G::N0 + 1];  // by n
  ExtRow *tab = rows_tab + G::N0;  // by -m, m masked pixels of the window
  for (int n = threadIdx.x; n <= G::N0; n += blockDim.x) {
    if constexpr (k16) {
      const float root = (uint32_t)n < P.min_local ? __uint_as_float(0x7FFFFFFFu) : P.rootf[n];
      rows_tab[n].a = make_uint4(__float_as_uint((float)n), __float_as_uint(root), 0u, 0u);
      rows_tab[n].b = make_uint4(0u, 0u, 0u, 0u);
    } else {
      rows_tab[n].a =
          make_uint4(0u - (T.nk[n] >> 4), T.clo16[n], T.chi16[n] - T.clo16[n], (uint32_t)n);
      rows_tab[n].b = make_uint4(T.nk[n], T.clo[n], T.chi[n], 0u);
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  StripRun r;
  if (!strip_run<C>(F, nframes, S, run_rows, r))
    return;  // whole warp
  const Pix *image = reinterpret_cast<const Pix *>(F.image[r.frame]);
  const int rows = r.rb - r.ra + 2 * (K + E);
  Pix *ring = reinterpret_cast<Pix *>(ext_raw) + (size_t)warp * G::Slots * kStripStride<C>;
  RowReader<Pix, C> reader(image, r, r.ra - E - K, rows);
  auto after = [&](int s) { return s + 1 == G::Slots ? 0 : s + 1; };
#pragma unroll
  for (int i = 0; i < G::Ahead; i++) {
    reader.fetch(ring + i * kStripStride<C>);
    cp_async_commit();
  }
  uint32_t Vn[C], Vq[C];
#pragma unroll
  for (int c = 0; c < C; c++)
    Vn[c] = Vq[c] = 0u;
  const float gain = (float)P.gain, sigma_b = (float)P.sigma_b;
  uint8_t *out_row = cand_all + (size_t)r.frame * mask_bytes + (size_t)r.ra * r.bytes_per_row +
                     r.pair_byte;
  const int bytes_left = r.bytes_per_row - r.pair_byte;
  // The last 2E + 1 rows' decision bits and the last E + 1 rows' masked bits,
  // a bit a column in 16-bit halves, the newest lowest.
  uint32_t dec[4] = {0u, 0u, 0u, 0u}, msk[2] = {0u, 0u};
  int large = 0;
  int s_cur = 0;  // the current row's slot
  for (int i = 0; i < rows; i++) {
    __syncwarp();  // every lane is done with the slot that is filled next
    const int s_in = s_cur + G::Ahead < G::Slots ? s_cur + G::Ahead : s_cur + G::Ahead - G::Slots;
    reader.fetch(ring + s_in * kStripStride<C>);
    cp_async_commit();
    cp_async_wait<G::Ahead>();
    __syncwarp();
    {
      uint32_t v[C], o[C];
      read_row<Pix, C, kLargePixel, true>(ring + s_cur * kStripStride<C>, lane, v);
      if (i >= G::W0) {  // warp-uniform
        read_row<Pix, C, kLargePixel, false>(ring + after(s_in) * kStripStride<C>, lane, o);
      } else {
#pragma unroll
        for (int c = 0; c < C; c++)
          o[c] = 0u;
      }
      add_rows<C>(Vn, Vq, v, o);
      if constexpr (!k16) {
        // Rows left whose windows may hold a pixel too large for these sums (they
        // wrap, and are right again when it has left them).
        int top = 0;
#pragma unroll
        for (int c = 0; c < C; c++)
          top = max(top, (int)v[c]);
        large = __any_sync(0xffffffffu, top >= (int)G::Cap) ? G::W0 : large - 1;
      }
    }
    if (i >= 2 * K) {  // warp-uniform: the windows are whole
      uint32_t hn[C], hq[C];
      window_sums<K, C>(Vn, hn);
      window_sums<K, C>(Vq, hq);
      uint32_t any_masked = 0;
#pragma unroll
      for (int c = 0; c < C; c++)
        any_masked |= hn[c];
      // Warp rows whose windows hold no masked pixel (most) take the whole
      // window's constants; the others look each window's count up.
      const bool uniform = !__any_sync(0xffffffffu, any_masked >> kCountShift) && large <= 0;
      uint32_t sig = 0, masked_at = 0;
      if (!uniform) {
        uint32_t v[C];
        const int s_mid = s_cur >= K ? s_cur - K : s_cur + G::Slots - K;
        read_row<Pix, C, kLargePixel, false>(ring + s_mid * kStripStride<C>, lane, v);
        masked_at = sign_bits<C>([&](int c) { return v[c]; });
      }
      if constexpr (k16) {
        if (uniform) {
          const uint4 t = tab[0].a;
          const float m = __uint_as_float(t.x), root = __uint_as_float(t.y);
#pragma unroll
          for (int c = 0; c < C; c++)
            sig |= stage0_float(m, root, hn[c], hq[c], gain, sigma_b) ? 1u << c : 0u;
        } else {
#pragma unroll
          for (int c = 0; c < C; c++) {
            const uint4 t = tab[masked_of(hn[c])].a;
            sig |= stage0_float(__uint_as_float(t.x), __uint_as_float(t.y), hn[c] & kSumMask, hq[c],
                             gain, sigma_b)
                       ? 1u << c
                       : 0u;
          }
        }
      } else if (large > 0) {  // warp-uniform
        sig = ext_large_row<K, C>(reinterpret_cast<const uint32_t *>(ring), s_cur, lane, tab, P,
                               reinterpret_cast<const uint32_t *>(image), r.height, r.width,
                               r.ra - E + i - 2 * K, r.cx);
      } else {
        // A row with a window too big for the 2^-4 bounds takes the 2^-8 ones at
        // once; else the lower 2^-4 bound, and the upper where it leaves any.
        // (Signs gathered by shifts: four instructions a window for the lower bound,
        // seven compared, selected and ORed.)
        uint32_t most = 0;
#pragma unroll
        for (int c = 0; c < C; c++)
          most = max(most, hq[c]);
        bool finer = __any_sync(0xffffffffu, most >= T.big);
        if (!finer) {
          const uint4 t0 = tab[0].a;
          // The lower bound's difference (and what the upper adds to it).
          auto plain = [&](int c) { return hq[c] * t0.x + hn[c] * ((hn[c] << 4) + t0.y); };
          auto looked_up = [&](int c, bool upper) {
            const uint4 t = tab[masked_of(hn[c])].a;
            const uint32_t s = hn[c] & kSumMask;
            return hq[c] * t.x + s * ((s << 4) + t.y) + (upper ? s * t.z + 31u : 0u);
          };
          const uint32_t maybe =
              uniform ? sign_bits<C>(plain) : sign_bits<C>([&](int c) { return looked_up(c, false); });
          sig = maybe;
          if (__any_sync(0xffffffffu, maybe != 0u)) {
            const uint32_t sure =
                uniform ? sign_bits<C>([&](int c) { return plain(c) + hn[c] * t0.z + 31u; })
                        : sign_bits<C>([&](int c) { return looked_up(c, true); });
            sig = sure;
            finer = __any_sync(0xffffffffu, (maybe & ~sure) != 0u);
          }
        }
        if (finer) {
          uint32_t between = 0;
          sig = 0;
#pragma unroll
          for (int c = 0; c < C; c++) {
            const uint4 t = tab[masked_of(hn[c])].b;
            const uint32_t s = hn[c] & kSumMask;
            const unsigned long long L = (unsigned long long)hq[c] * t.x;
            const bool above = L > (unsigned long long)s * ((s << 8) + t.y);
            const bool over = L >= (unsigned long long)s * ((s << 8) + t.z) + (2ull << 8);
            sig |= over ? 1u << c : 0u;
            between |= above & !over ? 1u << c : 0u;
          }
          if (__any_sync(0xffffffffu, between != 0u)) {
#pragma unroll
            for (int c = 0; c < C; c++) {
              if ((between >> c) & 1u) {
                if (ext_exact(G::N0 + masked_of(hn[c]), hn[c] & kSumMask, hq[c], P))
                  sig |= 1u << c;
              }
            }
          }
        }
      }
      // Row d = ra - E + i - 2K: signal or masked; then the erosion of row d - E.
#pragma unroll
      for (int k = 3; k > 0; k--)
        dec[k] = __funnelshift_l(dec[k - 1], dec[k], 16);
      dec[0] = dec[0] << 16 | sig | masked_at;
      msk[1] = __funnelshift_l(msk[0], msk[1], 16);
      msk[0] = msk[0] << 16 | masked_at;
      if (i >= 2 * K + 2 * E) {  // warp-uniform
        uint32_t col = dec[0];
#pragma unroll
        for (int k = 1; k <= 2 * E; k++)
          col &= k & 1 ? dec[k >> 1] >> 16 : dec[k >> 1];
        col &= (1u << C) - 1u;
        const uint32_t left = __shfl_up_sync(0xffffffffu, col, 1);
        const uint32_t right = __shfl_down_sync(0xffffffffu, col, 1);
        const uint32_t all = left >> (C - E) | col << E | right << (C + E);
        uint32_t kept = all;
#pragma unroll
        for (int k = 1; k <= 2 * E; k++)
          kept &= all >> k;
        const uint32_t mrow = E & 1 ? msk[E >> 1] >> 16 : msk[E >> 1];
        write_bits<C>(r, out_row, bytes_left, kept & ~mrow & r.inside);
        out_row += r.bytes_per_row;
      }
    }
    s_cur = after(s_cur);
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// Stage 2 (dext.cc:151-222): a candidate's background is the valid pixels
// outside the eroded mask (the candidates and the masked pixels) in its clipped
// (2K + 5)-square window.
// ---------------------------------------------------------------------------

// One warp's chunk: the background's {count, sum} over the window's rows by
// output row and column, the pixels of the output rows, and the run's strong
// words and counts so far.
struct ExtWarp {
  uint2 col[kBandRows][32];
  uint32_t px[kBandRows][32];
  uint32_t strong[kBandRows * kRunWords];
  uint32_t passed[kBandRows];
};

// A window's background one pixel after another, in 64 bits, for chunks that
// hold a pixel of 2^24 or more.
template <typename Pix>
__device__ __noinline__ void ext_wide_window(const Pix *image, const uint32_t *cand, int height,
                                             int width, int half, int y, int x, uint32_t *n_out,
                                             unsigned long long *S_out) {
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5;
  uint32_t n = 0;
  unsigned long long S = 0;
  for (int yy = max(0, y - half); yy <= min(height - 1, y + half); yy++)
    for (int xx = max(0, x - half); xx <= min(width - 1, x + half); xx++) {
      const uint32_t v = __ldg(image + (size_t)yy * width + xx);
      if (v < Traits<Pix>::kMasked &&
          (cand[(size_t)yy * wpr + (xx >> 5)] >> (xx & 31) & 1u) == 0u) {
        n++;
        S += v;
      }
    }
  *n_out = n;
  *S_out = S;
}

constexpr int kListItems = 256;  // runs listed at a time
constexpr int kListAhead = 4;    // their words read together
constexpr uint32_t kHeavyRun = 48;  // candidates of a run that is taken early

// A warp takes a run of a band at a time (128 columns x 8 rows, a word a lane)
// and its candidates in chunks: from the leftmost column with one left, the NC
// columns whose windows 32 columns cover, for all 8 rows (a spot's candidates
// are about 7 x 7). The chunk's pixels are read once, a lane a column, added up
// over the window's rows into shared memory; then its candidates are spread
// over the lanes, each adding up its window's columns for the test. A block
// first lists the runs of its bands that hold a candidate, four a warp on
// their way at once; its warps then take them in turn, those with many candidates
// first, so that they even out. Bound by issue: 32 frames of 4362 x 4148 (174
// thousand candidates each) take 266 us, 290 with the runs taken in order, the
// empty ones among them, each read when its turn came (one frame 19 and 22). A
// window a candidate, four lanes each, took 568 us, chunks of one row 427, and
// tests row by row, only the row's candidates' lanes busy, 553.
template <int K, typename Pix>
__global__ void __launch_bounds__(kScanT, 4)
ext_decide(const __grid_constant__ FramePtrs F, const __grid_constant__ LaunchParams P,
           const uint32_t *__restrict__ cand_all, uint32_t *__restrict__ bits_all, size_t words,
           Kept kept, uint32_t *__restrict__ block_sums, uint32_t *__restrict__ cand_sums) {
  previous_done();
  constexpr int K2 = K + 2, W2 = 2 * K2 + 1, NC = 32 - 2 * K2, ROWS = kBandRows + 2 * K2;
  __shared__ ExtWarp s_warps[kScanT / 32];
  __shared__ uint32_t s_count[2], s_heavy, s_light, s_next;
  __shared__ uint16_t s_items[kListItems];
  ExtWarp &sm = s_warps[threadIdx.x >> 5];
  const int f = blockIdx.y, lane = threadIdx.x & 31;
  const Pix *image = reinterpret_cast<const Pix *>(F.image[f]);
  const int height = F.h[f], width = F.w[f];
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5, rpr = (uint32_t)runs_per_row(width);
  const uint32_t lane_bit = 1u << lane;
  const uint32_t *cand = cand_all + (size_t)f * words;
  uint32_t *bits = bits_all + (size_t)f * words;
  uint2 *res = kept.res + (size_t)f * kept.stride;
  if (threadIdx.x < 2)
    s_count[threadIdx.x] = 0u;
  __syncthreads();  // (a block without rows comes to no other barrier before the counts)
  int row_lo, row_hi;
  band_share(height, &row_lo, &row_hi);
  const uint32_t items = (uint32_t)((row_hi - row_lo + kBandRows - 1) / kBandRows) * rpr;
  const int lr = lane / kRunWords, lc = lane % kRunWords;  // this lane's row and word of a run
  uint32_t count = 0, total = 0;
  for (uint32_t base = 0; base < items; base += kListItems) {
    // The runs that hold a candidate, those with many from the list's front and
    // the others from its back; the rest have no strong pixel.
    const uint32_t chunk = min(items - base, (uint32_t)kListItems);
    if (threadIdx.x == 0)
      s_heavy = s_light = s_next = 0u;
    __syncthreads();
    for (uint32_t i0 = threadIdx.x >> 5; i0 < chunk; i0 += kListAhead * (kScanT / 32)) {
      uint32_t w[kListAhead];
      size_t at[kListAhead];
#pragma unroll
      for (int u = 0; u < kListAhead; u++) {
        const uint32_t i = i0 + u * (kScanT / 32), band = (base + i) / rpr,
                       run = base + i - band * rpr;
        const int y = row_lo + (int)band * kBandRows + lr;
        const bool in = i < chunk && y < row_hi && run * kRunWords + lc < wpr;
        at[u] = in ? (size_t)y * wpr + run * kRunWords + lc : ~(size_t)0;
        w[u] = in ? __ldg(cand + at[u]) : 0u;
      }
#pragma unroll
      for (int u = 0; u < kListAhead; u++) {
        const uint32_t n = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(w[u]));
        total += n;  // (the same in every lane)
        if (n == 0u) {
          if (at[u] != ~(size_t)0)
            bits[at[u]] = 0u;
        } else if (lane == 0) {
          const uint32_t place = n >= kHeavyRun ? atomicAdd(&s_heavy, 1u)
                                                : kListItems - 1u - atomicAdd(&s_light, 1u);
          s_items[place] = (uint16_t)(i0 + u * (kScanT / 32));
        }
      }
    }
    __syncthreads();
    const uint32_t heavy = s_heavy, listed = heavy + s_light;
    for (;;) {
      uint32_t item = 0;
      if (lane == 0)
        item = atomicAdd(&s_next, 1u);
      item = __shfl_sync(0xffffffffu, item, 0);
      if (item >= listed)
        break;  // whole warp
      item = base + s_items[item < heavy ? item : kListItems - 1u - (item - heavy)];
      const uint32_t band = item / rpr, run = item - band * rpr;
      const int y0 = row_lo + (int)band * kBandRows, xr = (int)run * kRunWords * 32;
      const bool in = y0 + lr < row_hi && run * kRunWords + lc < wpr;
      const size_t wi = (size_t)(y0 + lr) * wpr + run * kRunWords + lc;
      uint32_t left = in ? __ldg(cand + wi) : 0u;  // this lane's candidates not yet decided
      sm.strong[lane] = 0u;
      if (lane < kBandRows)
        sm.passed[lane] = 0u;
      for (;;) {
        // The leftmost column with a candidate left.
        uint32_t any = left;
        any |= __shfl_xor_sync(0xffffffffu, any, 4);
        any |= __shfl_xor_sync(0xffffffffu, any, 8);
        any |= __shfl_xor_sync(0xffffffffu, any, 16);
        const unsigned live = __ballot_sync(0xffffffffu, any != 0u) & 0xFu;
        if (!live)
          break;  // whole warp
        const int c0 = __ffs(live) - 1, s = __ffs(__shfl_sync(0xffffffffu, any, c0)) - 1;
        const int x0 = xr + 32 * c0 + s;
        const unsigned long long span = (unsigned long long)((1u << NC) - 1u) << s;
        left &= lc == c0 ? ~(uint32_t)span : lc == c0 + 1 ? ~(uint32_t)(span >> 32) : ~0u;
        // The chunk's pixels start at (xl, yt); lane d holds the 32 mask bits over row d.
        const int xl = x0 - K2, yt = y0 - K2;
        uint32_t er_row = 0, v[ROWS];
        if (xl >= 0 && xl + 32 <= width && yt >= 0 && yt + ROWS <= height) {  // warp-uniform
          if (lane < ROWS) {
            const uint32_t *cw = cand + (uint32_t)(yt + lane) * wpr + (uint32_t)(xl >> 5);
            er_row = __funnelshift_r(__ldg(cw), __ldg(cw + ((xl & 31) != 0 ? 1 : 0)), xl & 31);
          }
          const Pix *at = image + (size_t)yt * width + (xl + lane);
#pragma unroll
          for (int d = 0; d < ROWS; d++) {
            v[d] = (uint32_t)__ldg(at);
            at += width;
          }
        } else {
          if (lane < ROWS && yt + lane >= 0 && yt + lane < height) {
            const uint32_t *row = cand + (size_t)(yt + lane) * wpr;
            const int w0 = xl >> 5;  // (-1 left of the frame)
            const uint32_t a = w0 >= 0 ? __ldg(row + w0) : 0u;
            const uint32_t b = w0 + 1 < (int)wpr ? __ldg(row + w0 + 1) : 0u;
            er_row = __funnelshift_r(a, b, xl & 31);
          }
          const int x = xl + lane;
#pragma unroll
          for (int d = 0; d < ROWS; d++) {
            const bool inside = x >= 0 && x < width && yt + d >= 0 && yt + d < height;
            v[d] = inside ? (uint32_t)__ldg(image + (size_t)(yt + d) * width + x)
                          : Traits<Pix>::kMasked;
          }
        }
        // Row r's candidates of the chunk, in lane r (columns past the run are
        // the next one's), and the candidates before them.
        uint32_t mine = __shfl_sync(0xffffffffu, er_row, (lane + K2) & 31) >> K2;
        mine &= lane < kBandRows ? (1u << NC) - 1u : 0u;
        if (x0 + NC > xr + 32 * kRunWords)
          mine &= (1u << (xr + 32 * kRunWords - x0)) - 1u;
        const uint32_t incl = warp_inclusive((uint32_t)__popc(mine), lane);
        const uint32_t ncand = __shfl_sync(0xffffffffu, incl, 31);
        // The background over the window's rows, by column.
        uint32_t most = 0;
        {
          uint32_t n = 0, sum = 0;
#pragma unroll
          for (int d = 0; d < ROWS; d++) {
            const bool ok = (v[d] < Traits<Pix>::kMasked) &
                            ((__shfl_sync(0xffffffffu, er_row, d) & lane_bit) == 0u);
            if (d >= K2 && d < K2 + kBandRows)
              sm.px[d - K2][lane] = v[d];
            v[d] = ok ? v[d] : Traits<Pix>::kMasked;  // background or not, from here on
            n += ok ? 1u : 0u;
            sum += ok ? v[d] : 0u;
            most |= ok ? v[d] : 0u;
            if (d >= W2 - 1) {
              sm.col[d - (W2 - 1)][lane] = make_uint2(n, sum);
              const bool was = v[d - (W2 - 1)] < Traits<Pix>::kMasked;
              n -= was ? 1u : 0u;
              sum -= was ? v[d - (W2 - 1)] : 0u;
            }
          }
        }
        const bool wide = sizeof(Pix) == 4 && __any_sync(0xffffffffu, most >= 1u << 24);
        __syncwarp();
        for (uint32_t q0 = 0; q0 < ncand; q0 += 32) {  // warp-uniform
          const uint32_t q = q0 + lane;
          int r = 0;
#pragma unroll
          for (int k = 4; k; k >>= 1)
            r += __shfl_sync(0xffffffffu, incl, r + k - 1) <= q ? k : 0;
          r &= 7;
          const uint32_t row_bits = __shfl_sync(0xffffffffu, mine, r);
          const uint32_t first = __shfl_sync(0xffffffffu, incl, r) - (uint32_t)__popc(row_bits);
          bool ok = q < ncand;
          const int j = ok ? select_bit(row_bits, q - first) : 0;
          uint32_t n = 0, s32 = 0;
#pragma unroll
          for (int k = 0; k < W2; k++) {
            const uint2 c = sm.col[r][j + k];
            n += c.x;
            s32 += c.y;
          }
          unsigned long long S = s32;
          if (sizeof(Pix) == 4 && wide && ok)
            ext_wide_window(image, cand, height, width, K2, y0 + r, x0 + j, &n, &S);
          float mean = 0.0f;
          if (ok) {
            const uint32_t p = sm.px[r][j + K2];
            // dext.cc:205: only pixels above the global threshold are tested.
            ok = (uint64_t)p >= P.p_min;
            if (ok) {
              if constexpr (sizeof(Pix) == 2)
                ok = stage2_u16(p, n, (uint32_t)S, P, &mean);
              else
                ok = stage2_u32(p, n, S, P, &mean);
            }
          }
          // This row's passing candidates in these lanes, and before them.
          const unsigned pass = __ballot_sync(0xffffffffu, ok);
          const int from = max((int)first - (int)q0, 0);
          const uint32_t before = sm.passed[r];
          const uint32_t at = before + (uint32_t)__popc(pass & (lane_bit - 1u) & (~0u << from));
          if (ok) {
            if (at < kept.keep)
              res[((size_t)(y0 + r) * rpr + run) * kept.keep + at] =
                  make_uint2(__float_as_uint(mean), n);
            const int b = x0 + j - xr;
            atomicOr(&sm.strong[r * kRunWords + (b >> 5)], 1u << (b & 31));
          }
          __syncwarp();
          if (ok)
            atomicMax(&sm.passed[r], at + 1u);
          count += ok ? 1u : 0u;
          __syncwarp();
        }
        __syncwarp();  // the next chunk rewrites the shared sums
      }
      if (in)
        bits[wi] = sm.strong[lane];
      __syncwarp();
    }
    __syncthreads();
  }
  count = __reduce_add_sync(0xffffffffu, count);
  if (lane == 0) {
    atomicAdd(&s_count[0], count);
    atomicAdd(&s_count[1], total);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    block_sums[(size_t)f * gridDim.x + blockIdx.x] = s_count[0];
    cand_sums[(size_t)f * gridDim.x + blockIdx.x] = s_count[1];
  }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------

bool testable(const LaunchParams &P, int n, int n0) {
  return n >= 1 && (uint32_t)n >= P.min_local && n <= n0;
}

// c = g (n - 1 + sigma_b r_n) as integers in 2^-8 units below and above it.
// With gain 1 and an integral sigma_b from r_n's 2^-20 brackets, exactly; else
// from the double product, a unit outwards.
void bracket_c(const LaunchParams &P, int n, double *lo, double *hi) {
  if (P.int_ok) {
    const int shift = kRootShift - 8;
    const uint64_t sb = P.sigma_b_int, base = (uint64_t)(n - 1) << 8;
    *lo = (double)(base + ((sb * P.root_lo[n]) >> shift));
    *hi = (double)(base + ((sb * P.root_hi[n] + ((1ull << shift) - 1)) >> shift));
  } else {
    const double c = 256.0 * P.gain * (n - 1 + P.sigma_b * P.root[n]);
    *lo = std::max(0.0, std::floor(c) - 1.0);
    *hi = std::ceil(c) + 1.0;
  }
}

ExtTables make_ext_tables(const LaunchParams &P) {
  ExtTables T;
  const int n0 = (2 * P.half + 1) * (2 * P.half + 1);
  T.big = P.half == 2 ? StripG<2>::Big : P.half == 3 ? StripG<3>::Big : StripG<4>::Big;
  for (int n = 0; n <= kMaxN0; n++) {
    double lo = 0.0, hi = 0.0;
    if (testable(P, n, n0))
      bracket_c(P, n, &lo, &hi);
    T.clo[n] = (uint32_t)lo;
    T.chi[n] = (uint32_t)hi;
    T.clo16[n] = T.clo[n] >> 4;
    T.chi16[n] = (T.chi[n] + 15u) >> 4;
    // nk 0 makes every such window "surely not" (0 <= S (2^8 S + clo)).
    T.nk[n] = testable(P, n, n0) ? (uint32_t)n << 8 : 0u;
    if (T.chi16[n] >= kMaxC16)
      T.big = 0;  // constants too large for the 32-bit tests: every window is big
  }
  return T;
}

// Whether stage 0 and the erosion take the lattice (sf_lattice.cu): kernel 3,3,
// 32-bit frames at gain 1 with integral sigmas, or 16-bit ones where 4 | width
// and they are 8-byte aligned. Spots cover a few percent of such frames, and
// the lattice decides a ninth of the windows and the tiles that hold a
// candidate: 32 frames of 4362 x 4148 take 0.95 ms so and 1.38 ms on strips.
// Launches of up to kStripPixels take strips, narrow ones that size (sf_strips.cuh):
// there the lattice's two more launches cost more than they save. In a captured graph,
// us on the lattice and on strips: one frame of 1065 x 1030 35 and 29, 2 of 1024 x 1024
// 37 and 35, 3 and 4 of them 37 and 37, 39 and 41, one of 2162 x 2068 39 and 39, of 2400
// x 2400 43 and 46; the last two with a tenth of the pixels masked 45 and 39, 51 and 49,
// with a fiftieth overloaded 109 and 103, 133 and 135, 16-bit 36 and 37, 39 and 41. Frames
// with few large pixels (1 in 2000) would be better off on the lattice from 2 million
// pixels on (39 and 49, at one of 2162 x 2068 47 and 61): a strip's whole row is summed
// again for one.
constexpr long long kStripPixels = 5000000;
bool lattice_path(const FramePtrs &F, int nframes, int pixel_bytes, const LaunchParams &P) {
  if (P.half != 3 || P.algorithm != SF_DISPERSION_EXTENDED)
    return false;
  long long pixels = 0;
  for (int f = 0; f < nframes; f++)
    pixels += (long long)F.h[f] * F.w[f];
  if (pixels <= kStripPixels)
    return false;
  if (pixel_bytes == 4)
    return P.int_ok != 0;
  for (int f = 0; f < nframes; f++)
    if (F.w[f] % 4 != 0 || reinterpret_cast<uintptr_t>(F.image[f]) % 8 != 0)
      return false;
  return true;
}

template <int K, typename Pix, int C> cudaError_t ext_slots(int *slots_out) {
  using G = StripG<K>;
  constexpr size_t smem = strip_smem<K, Pix, C>();
  static_assert(sizeof(Pix) == 2 ||
                    (smem + sizeof(ExtRow) * (G::N0 + 1) + 1024) * G::Occ <= 228 * 1024,
                "the blocks an SM that the kernel is built for");
  static std::once_flag configured;
  static cudaError_t config_error = cudaSuccess;
  static int slots = 0;
  std::call_once(configured, [] {
    config_error = cudaFuncSetAttribute(ext_strip<K, Pix, C>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per = 0;
    if (config_error == cudaSuccess)
      config_error = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ext_strip<K, Pix, C>,
                                                                   kStripWarps * 32, smem);
    slots = std::max(1, per) * kStripWarps * device_sms();
  });
  *slots_out = slots;
  return config_error;
}

template <int K, typename Pix, int C>
cudaError_t launch_strips(const FramePtrs &F, int nframes, const LaunchParams &P,
                          const StreamBuffers &b, int run_rows, cudaStream_t stream) {
  int slots = 0;
  const cudaError_t e = ext_slots<K, Pix, C>(&slots);
  if (e != cudaSuccess)
    return e;
  FrameSpans S;
  run_rows = strip_spans<C>(F, nframes, slots, run_rows, &S);
  const unsigned blocks = (unsigned)((S.start[nframes] + kStripWarps - 1) / kStripWarps);
  ext_strip<K, Pix, C><<<blocks, kStripWarps * 32, strip_smem<K, Pix, C>(), stream>>>(
      F, nframes, S, run_rows, make_ext_tables(P), P, reinterpret_cast<uint8_t *>(b.cand),
      b.words * sizeof(uint32_t));
  return cudaSuccess;
}

template <int K, typename Pix>
cudaError_t launch_ext(const FramePtrs &F, int nframes, int h, int w, const LaunchParams &P,
                       const StreamBuffers &b, int run_rows, cudaStream_t stream,
                       const StreamMarks *marks) {
  const bool lattice = lattice_path(F, nframes, (int)sizeof(Pix), P);
  cudaError_t e;
  if (lattice) {
    e = launch_lattice(F, nframes, h, w, (int)sizeof(Pix), P, b, run_rows, stream);
    if (e != cudaSuccess)
      return e;
  } else {
    int slots = 0;
    if ((e = ext_slots<K, Pix, kWideCols>(&slots)) != cudaSuccess)
      return e;
    e = narrow_strips(F, nframes, slots)
            ? launch_strips<K, Pix, kNarrowCols>(F, nframes, P, b, run_rows, stream)
            : launch_strips<K, Pix, kWideCols>(F, nframes, P, b, run_rows, stream);
    if (e != cudaSuccess)
      return e;
  }
  if (marks)
    cudaEventRecord(marks->stage01, stream);
  const dim3 grid = band_grid(nframes, h, w);
  const Kept kept = make_kept(b, h, w);
  launch_after(ext_decide<K, Pix>, grid, kScanT, 0, stream, F, P, b.cand, b.bits, b.words, kept,
               b.block_sums, b.cand_sums);
  if (marks)
    cudaEventRecord(marks->stage2, stream);
  launch_after(scatter_pixels<Pix, true>, grid, kScanT, 0, stream, F, b.bits, b.words, b.cand,
               K + 2, kept, P.min_local, b.block_sums, b.cand_sums, b.cand_limit,
               lattice ? b.counters + kCtrFault : nullptr, b.out, b.out_stride, b.capacity,
               b.count_out, b.prefix);
  if (marks)
    cudaEventRecord(marks->order, stream);
  return cudaGetLastError();
}

} // namespace

int device_sms() {
  static int cached = 0;
  if (cached)
    return cached;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      sms <= 0)
    return 152;  // not cached: asked again once a device answers
  cached = sms;
  return cached;
}

bool streaming_path(const LaunchParams &P, int pixel_bytes) {
  if (pixel_bytes == 2)
    return true;
  if (!(P.gain >= 0.0 && P.sigma_b >= 0.0 && P.sigma_s >= 0.0))
    return false;
  double lo, hi;
  bracket_c(P, kMaxN0, &lo, &hi);
  return hi < kMaxC8;
}

cudaError_t launch_extended(const FramePtrs &F, int nframes, int h, int w, int pixel_bytes,
                            const LaunchParams &P, const StreamBuffers &b, int run_rows,
                            cudaStream_t stream, const StreamMarks *marks) {
  if (nframes < 1 || nframes > kMaxBatch || P.algorithm != SF_DISPERSION_EXTENDED ||
      !streaming_path(P, pixel_bytes))
    return cudaErrorInvalidValue;
  if (marks)
    cudaEventRecord(marks->start, stream);
  auto launch = [&](auto k) {
    constexpr int K = decltype(k)::value;
    return pixel_bytes == 2 ? launch_ext<K, uint16_t>(F, nframes, h, w, P, b, run_rows, stream, marks)
                            : launch_ext<K, uint32_t>(F, nframes, h, w, P, b, run_rows, stream, marks);
  };
  switch (P.half) {
  case 2:
    return launch(std::integral_constant<int, 2>());
  case 3:
    return launch(std::integral_constant<int, 3>());
  case 4:
    return launch(std::integral_constant<int, 4>());
  default:
    return cudaErrorInvalidValue;
  }
}

template <int K> cudaError_t default_run_rows(const FramePtrs &F, int nframes, int *rows) {
  int slots = 0;
  cudaError_t e = ext_slots<K, uint32_t, kWideCols>(&slots);
  if (e != cudaSuccess)
    return e;
  FrameSpans S;
  if (!narrow_strips(F, nframes, slots)) {
    *rows = strip_spans<kWideCols>(F, nframes, slots, 0, &S);
  } else if ((e = ext_slots<K, uint32_t, kNarrowCols>(&slots)) == cudaSuccess) {
    *rows = strip_spans<kNarrowCols>(F, nframes, slots, 0, &S);
  }
  return e;
}

int stream_default_run_rows(const LaunchParams &P, int h, int w, int nframes) {
  FramePtrs F = {};
  nframes = std::min(nframes, kMaxBatch);
  for (int f = 0; f < nframes; f++)
    F.h[f] = h, F.w[f] = w;
  if (lattice_path(F, nframes, 4, P))
    return lattice_geometry(h, w, nframes, 0).run_rows;
  int rows = kMinRunRows;
  if ((P.half == 2   ? default_run_rows<2>(F, nframes, &rows)
       : P.half == 3 ? default_run_rows<3>(F, nframes, &rows)
                     : default_run_rows<4>(F, nframes, &rows)) != cudaSuccess)
    cudaGetLastError();
  return rows;
}

} // namespace sf
