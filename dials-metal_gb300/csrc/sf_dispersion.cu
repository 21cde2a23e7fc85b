// The plain dispersion threshold (SF_DISPERSION) for frames of either pixel
// type: a valid pixel above the global threshold is strong when its clipped
// (2K + 1)-square window passes the dispersion test of stage 0 and
// (n p - S) > sigma_s sqrt(gain S n).
//
//   disp_strip    every pixel's window, one warp per strip and run of rows: a
//                 mask that holds every strong pixel and few others
//   disp_decide   each set pixel decided from its window's full sums by the
//                 reference's sequence; the failures leave the mask, which is
//                 then the strong-pixel mask, and the blocks count theirs
//   scatter_pixels  the mask's pixels as records, ascending, each at its place
//                 from the counts (and, when asked for, each word's place)
//
// No list of candidates is kept between the passes (the records' sums are
// taken again from the frame), so no frame can overflow one: a frame where
// every pixel is a candidate is decided like any other.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "sf_common.cuh"
#include "sf_groups.cuh"
#include "sf_scan.cuh"
#include "sf_stream.cuh"
#include "sf_strips.cuh"

namespace sf {
namespace {

// The filters' constants for a window of n valid pixels, rounded down: nk =
// 16 n (0 when n cannot be tested), clo <= 16 c where the dispersion test is n
// Q - S (S + c) > 0 but for rounding, and kk <= sigma_s^2 gain n.
constexpr uint32_t kDispMaxKK = 3640;  // keeps S kk below 2^31 for S <= 81 x 7281
constexpr int kDispMaxD = 46340;       // d^2 + d below 2^31, and not below S kk
static_assert((uint64_t)kDispMaxKK * 81u * 7281u <= (uint64_t)kDispMaxD * (kDispMaxD + 1) - 1u &&
                  (uint64_t)kDispMaxD * (kDispMaxD + 1) < (1ull << 31),
              "both sides of the second filter fit, and the largest d passes");
struct DispTables {
  uint32_t nk[kMaxN0 + 1], clo[kMaxN0 + 1], kk[kMaxN0 + 1];
};

// The second test of a window of n valid 16-bit pixels with sum S and of its
// centre pixel p: the reference's float sequence.
__device__ __forceinline__ bool disp_float2(uint32_t p, uint32_t n, uint32_t S,
                                            const LaunchParams &P) {
  const float m = __uint2float_rn(n), s = __uint2float_rn(S), v = __uint2float_rn(p);
  return __fsub_rn(__fmul_rn(m, v), s) >
         __fmul_rn((float)P.sigma_s, __fsqrt_rn(__fmul_rn(__fmul_rn((float)P.gain, s), m)));
}

// The walk of sf_strips.cuh: a lane adds each row to its column sums as it
// enters the window, subtracts it as it leaves, and reads it once more as the
// centre row; a window is 2K + 1 column sums.
// Bound by issue: 39 instructions a pixel at 66% of the issue rate. 16 frames of
// 3262 x 3108 took 4.57 ms as 32 x 32 tiles (each pixel's window summed in
// 64 bits from shared memory, the halo staged 2.6 times over), and take 0.37 ms
// here: 271 us in this kernel (344 with both tests compared, selected and ORed,
// 437 with branches around their halves), 79 and 30 in the two below.
template <int K, typename Pix, int C>
__global__ void __launch_bounds__(kStripWarps * 32, StripG<K>::Occ)
disp_strip(const __grid_constant__ FramePtrs F, int nframes, const __grid_constant__ FrameSpans S,
           int run_rows, const __grid_constant__ DispTables T,
           const __grid_constant__ LaunchParams P, uint8_t *__restrict__ mask_all,
           size_t mask_bytes) {
  previous_done();
  using G = StripG<K>;
  extern __shared__ __align__(16) unsigned char disp_raw[];
  __shared__ uint4 rows_tab[G::N0 + 1];  // by n: -nk, clo, kk
  const uint4 *tab = rows_tab + G::N0;   // by -m, m masked pixels of the window
  for (int n = threadIdx.x; n <= G::N0; n += blockDim.x)
    rows_tab[n] = make_uint4(0u - T.nk[n], T.clo[n], T.kk[n], 0u);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  StripRun r;
  if (!strip_run<C>(F, nframes, S, run_rows, r))
    return;  // whole warp
  const Pix *image = reinterpret_cast<const Pix *>(F.image[r.frame]);
  const int rows = r.rb - r.ra + 2 * K;
  Pix *ring = reinterpret_cast<Pix *>(disp_raw) + (size_t)warp * G::Slots * kStripStride<C>;
  RowReader<Pix, C> reader(image, r, r.ra - K, rows);
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
  const uint4 whole = tab[0];
  uint8_t *out_row = mask_all + (size_t)r.frame * mask_bytes + (size_t)r.ra * r.bytes_per_row +
                     r.pair_byte;
  const int bytes_left = r.bytes_per_row - r.pair_byte;
  int s_cur = 0;  // the current row's slot
  for (int i = 0; i < rows; i++) {
    __syncwarp();  // every lane is done with the slot that is filled next
    const int s_in = s_cur + G::Ahead < G::Slots ? s_cur + G::Ahead : s_cur + G::Ahead - G::Slots;
    reader.fetch(ring + s_in * kStripStride<C>);
    cp_async_commit();
    cp_async_wait<G::Ahead>();
    __syncwarp();
    uint32_t v[C], o[C];
    read_row<Pix, C, G::Cap, true>(ring + s_cur * kStripStride<C>, lane, v);
    if (i >= G::W0) {  // warp-uniform
      read_row<Pix, C, G::Cap, false>(ring + after(s_in) * kStripStride<C>, lane, o);
    } else {
#pragma unroll
      for (int c = 0; c < C; c++)
        o[c] = 0u;
    }
    add_rows<C>(Vn, Vq, v, o);
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
      const bool uniform = !__any_sync(0xffffffffu, any_masked >> kCountShift);
      // The lower bound of the dispersion test, by the sign of its difference
      // (sf_strips.cuh); a window too big for it passes.
      uint32_t out = 0;
      if constexpr (sizeof(Pix) == 2) {
        // (The reference's float test itself.)
        if (uniform) {
#pragma unroll
          for (int c = 0; c < C; c++)
            out |= stage0_u16(G::N0, hn[c], hq[c], P) ? 1u << c : 0u;
        } else {
#pragma unroll
          for (int c = 0; c < C; c++) {
            out |= stage0_u16(G::N0 + masked_of(hn[c]), hn[c] & kSumMask, hq[c], P) ? 1u << c : 0u;
          }
        }
      } else {
        out = uniform ? sign_bits<C>([&](int c) {
          return hq[c] * whole.x + hn[c] * ((hn[c] << 4) + whole.y);
        })
                      : sign_bits<C>([&](int c) {
                          const uint4 t = tab[masked_of(hn[c])];
                          const uint32_t s = hn[c] & kSumMask;
                          return hq[c] * t.x + s * ((s << 4) + t.y);
                        });
        uint32_t most = 0;
#pragma unroll
        for (int c = 0; c < C; c++)
          most = max(most, hq[c]);
        if (__any_sync(0xffffffffu, most >= G::Big)) {
#pragma unroll
          for (int c = 0; c < C; c++)
            out |= hq[c] >= G::Big ? 1u << c : 0u;
        }
      }
      out &= r.inside;
      if (__any_sync(0xffffffffu, out != 0u)) {
        const int s_mid = s_cur >= K ? s_cur - K : s_cur + G::Slots - K;
        read_row<Pix, C, G::Cap, false>(ring + s_mid * kStripStride<C>, lane, v);
        uint32_t out2 = 0, masked_at = 0;
        if (!uniform)
          masked_at = sign_bits<C>([&](int c) { return v[c]; });
        if constexpr (sizeof(Pix) == 2) {
#pragma unroll
          for (int c = 0; c < C; c++) {
            const uint32_t n = G::N0 + (uniform ? 0 : masked_of(hn[c]));
            out2 |= disp_float2(v[c], n, hn[c] & kSumMask, P) ? 1u << c : 0u;
          }
        } else {
          // d = n p - S against sqrt(kk S): d falls and kk S rises with S, so a
          // saturated sum, at most the true one, passes wherever the true one
          // does. d^2 + d covers the rounding of the reference's right side (under
          // half a unit in d, and kk is a unit low), and a d of kDispMaxD or more
          // passes whatever S is.
          auto below = [&](int c, uint32_t n, uint32_t s, uint32_t kk) {
            const uint32_t e = (uint32_t)max(min((int)(n * v[c]) - (int)s, kDispMaxD), 0);
            return s * kk - (e * e + e);
          };
          out2 = uniform ? sign_bits<C>([&](int c) { return below(c, G::N0, hn[c], whole.z); })
                         : sign_bits<C>([&](int c) {
                             const int m = masked_of(hn[c]);
                             return below(c, G::N0 + m, hn[c] & kSumMask, tab[m].z);
                           });
          int most = 0;
#pragma unroll
          for (int c = 0; c < C; c++)
            most = max(most, (int)v[c]);
          if (__any_sync(0xffffffffu, most >= (int)G::Cap)) {
            // A saturated pixel's own test is left to the next pass.
#pragma unroll
            for (int c = 0; c < C; c++)
              out2 |= (int)v[c] >= (int)G::Cap ? 1u << c : 0u;
          }
        }
        out2 &= ~masked_at;
        out &= out2;
      }
      write_bits<C>(r, out_row, bytes_left, out);
      out_row += r.bytes_per_row;
    }
    s_cur = after(s_cur);
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// The candidates, four lanes each.
// ---------------------------------------------------------------------------

// The sums of the clipped window around (x, y), a quarter of its rows by each
// of the four lanes `sub`, added up across them: all four return them. A
// pixel a load, all of a lane's in flight at once (whole 16-byte pieces read
// half as many pixels again and had each one's column to check). Windows of
// pixels below 7282 (or 16-bit ones, whose squares the reference sums modulo
// 2^32) fit 32-bit sums; a window with a larger pixel is summed again.
template <int K, typename Pix>
__device__ __forceinline__ void disp_window(const Pix *__restrict__ image, int height, int width,
                                            bool live, int sub, int y, int x, uint32_t *n_out,
                                            unsigned long long *S_out,
                                            unsigned long long *Q_out) {
  constexpr int W0 = 2 * K + 1, ROWS = (W0 + 3) / 4;
  uint32_t n = 0, s32 = 0, q32 = 0, most = 0;
  const bool inner = x >= K && x + K < width && y >= K && y + K < height;
  if (live && inner) {
    const Pix *at = image + (size_t)(y - K + sub) * width + (x - K);
    uint32_t v[ROWS][W0];
#pragma unroll
    for (int k = 0; k < ROWS; k++)
#pragma unroll
      for (int c = 0; c < W0; c++)
        v[k][c] = sub + 4 * k < W0 ? (uint32_t)__ldg(at + (size_t)(4 * k) * width + c)
                                   : Traits<Pix>::kMasked;
#pragma unroll
    for (int k = 0; k < ROWS; k++)
#pragma unroll
      for (int c = 0; c < W0; c++) {
        const bool ok = v[k][c] < Traits<Pix>::kMasked;
        const uint32_t u = ok ? v[k][c] : 0u;
        n += ok ? 1u : 0u;
        s32 += u;
        q32 += u * u;
        most = max(most, u);
      }
  }
  const bool again = live && (!inner || (sizeof(Pix) == 4 && most > 7281u));
  unsigned long long S = s32, Q = q32;
  if (__any_sync(0xffffffffu, again)) {
    // The four lanes of a candidate go together.
    const bool all = __any_sync(0xFu << ((threadIdx.x & 31) & ~3), again);
    if (live && all) {
      n = 0;
      S = Q = 0;
      const int xlo = max(0, x - K), xhi = min(width - 1, x + K);
      for (int yy = max(0, y - K) + sub; yy <= min(height - 1, y + K); yy += 4)
        for (int xx = xlo; xx <= xhi; xx++) {
          const uint32_t v = __ldg(image + (size_t)yy * width + xx);
          if (v < Traits<Pix>::kMasked) {
            n++;
            S += v;
            Q += (unsigned long long)v * v;
          }
        }
    }
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    n += __shfl_xor_sync(0xffffffffu, n, o);
    S += __shfl_xor_sync(0xffffffffu, S, o);
    Q += __shfl_xor_sync(0xffffffffu, Q, o);
  }
  *n_out = n;
  *S_out = S;
  *Q_out = Q;
}

// (m p - s) > sigma_s sqrt(gain s m) and the mean, in double as the
// reference's other 32-bit tests: out of line, reached near ties.
__device__ __noinline__ bool disp_double(uint32_t p, uint32_t n, unsigned long long S,
                                         const LaunchParams &P) {
  const double m = (double)n, s = __ull2double_rn(S);
  return __dsub_rn(__dmul_rn(m, (double)p), s) >
         __dmul_rn(P.sigma_s, __dsqrt_rn(__dmul_rn(__dmul_rn(P.gain, s), m)));
}

// Both tests of a valid pixel p from its window's full sums.
template <typename Pix>
__device__ __forceinline__ bool disp_strong(uint32_t p, uint32_t n, unsigned long long S,
                                            unsigned long long Q, const LaunchParams &P) {
  if ((uint64_t)p < P.p_min)
    return false;
  if constexpr (sizeof(Pix) == 2) {
    return stage0_u16(n, (uint32_t)S, (uint32_t)Q, P) &&
           disp_float2(p, n, (uint32_t)S, P);
  } else {
    if (!stage0_u32(n, S, Q, P, P.root_lo, P.root_hi))
      return false;
    if (P.int_ok && S < (1ull << 24)) {
      // d against r = sigma_s sqrt(S n) < 2^26: further than 1 apart, the
      // rounding of the double sequence cannot matter.
      const long long d = (long long)n * (long long)p - (long long)S;
      if (d <= 0)
        return false;
      if (d >= (1ll << 30))
        return true;
      const long long D = d * d, R = (long long)P.sigma_s2_int * (long long)S * (long long)n;
      if (D > R + 2 * d)
        return true;
      if (D + 2 * d + 1 < R)
        return false;
    }
    return disp_double(p, n, S, P);
  }
}

// The windows' sums of a lane's four columns from its own column sums and those of
// the K columns either side: its neighbours', and at the run's ends the halo's (lane
// j < K holds that of the run's j-th column before, lane K + j of its j-th after).
template <int K>
__device__ __forceinline__ void run_windows(const unsigned long long col[4],
                                            unsigned long long halo, int lane,
                                            unsigned long long win[4]) {
  unsigned long long e[4 + 2 * K];
#pragma unroll
  for (int c = 0; c < 4; c++)
    e[K + c] = col[c];
#pragma unroll
  for (int k = 0; k < K; k++) {
    const unsigned long long l = __shfl_up_sync(0xffffffffu, col[4 - K + k], 1),
                             hl = __shfl_sync(0xffffffffu, halo, k),
                             r = __shfl_down_sync(0xffffffffu, col[k], 1),
                             hr = __shfl_sync(0xffffffffu, halo, K + k);
    e[k] = lane == 0 ? hl : l;
    e[K + 4 + k] = lane == 31 ? hr : r;
  }
  win[0] = 0ull;
#pragma unroll
  for (int k = 0; k <= 2 * K; k++)
    win[0] += e[k];
#pragma unroll
  for (int c = 1; c < 4; c++)
    win[c] = win[c - 1] + e[c + 2 * K] - e[c - 1];
}

// One run's candidates decided by the whole warp, four columns a lane (`cand` the
// lane's four bits): every window's sums, from the columns' sums over its rows.
// Returns the lane's passing bits and fills their results.
constexpr int kPackedN = 48;  // a sum's valid pixels above it: 81 x 2^32 is below 2^39
template <int K, typename Pix>
__device__ __forceinline__ uint32_t disp_dense_run(const Pix *__restrict__ image, int height,
                                                   int width, int y, int x0, uint32_t cand,
                                                   const LaunchParams &P, uint2 *mine) {
  const int lane = threadIdx.x & 31, x = x0 + 4 * lane;
  const int xh = lane < K ? x0 - K + lane : x0 + 128 + (lane - K);  // the halo column, lanes < 2K
  const bool has_halo = lane < 2 * K && xh >= 0 && xh < width;
  unsigned long long s[4] = {0, 0, 0, 0}, q[4] = {0, 0, 0, 0}, hs = 0, hq = 0;
  uint32_t centre[4] = {0, 0, 0, 0};
  auto add = [](uint32_t v, unsigned long long &sum, unsigned long long &sq) {
    const bool ok = v < Traits<Pix>::kMasked;
    sum += ok ? (1ull << kPackedN) + v : 0ull;
    sq += ok ? (unsigned long long)v * v : 0ull;
  };
#pragma unroll 3
  for (int d = -K; d <= K; d++) {
    const bool in = y + d >= 0 && y + d < height;  // warp-uniform
    const Pix *row = image + (ptrdiff_t)(y + d) * width;
    uint32_t v[4];
#pragma unroll
    for (int c = 0; c < 4; c++)
      v[c] = in && x + c < width ? (uint32_t)__ldg(row + x + c) : Traits<Pix>::kMasked;
    const uint32_t vh = in && has_halo ? (uint32_t)__ldg(row + xh) : Traits<Pix>::kMasked;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      add(v[c], s[c], q[c]);
      centre[c] = d == 0 ? v[c] : centre[c];
    }
    add(vh, hs, hq);
  }
  unsigned long long ws[4], wq[4];
  run_windows<K>(s, hs, lane, ws);
  run_windows<K>(q, hq, lane, wq);
  uint32_t pass = 0;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const uint32_t n = (uint32_t)(ws[c] >> kPackedN);
    const unsigned long long S = ws[c] & ((1ull << kPackedN) - 1ull);
    if ((cand >> c & 1u) && disp_strong<Pix>(centre[c], n, S, wq[c], P)) {
      pass |= 1u << c;
      mine[c] = make_uint2(__float_as_uint(window_mean<Pix>(n, S, P.min_local)), n);
    }
  }
  return pass;
}

// Whether a group of runs that holds `all` candidates is taken run by run, all
// windows of a run at once, instead of candidate by candidate. (Frames whose
// background reaches the strips' saturation are candidates everywhere: 4 of 3262 x
// 3108 with 15,000 counts a pixel take 0.63 ms so at kernel 3 and 4.03 the other
// way; with a third of the pixels strong 0.87 and 1.30; with a fifth 1.13 and 0.90,
// where the line of 40 leaves them.) Those groups come after the warp's others: the
// call in their midst cost frames without any 1%.
constexpr uint32_t kDenseRun = 40;  // candidates a run of 128 pixels
__device__ __forceinline__ bool dense_group(uint32_t all, uint32_t run0, uint32_t end) {
  return all >= kDenseRun * min(32u, end - run0);
}

// The dense groups of a warp (its groups start at first, first + kScanT, ..): as
// disp_decide's own loop. Returns the number of passing pixels.
template <int K, typename Pix>
__device__ __noinline__ uint32_t disp_dense_groups(const Pix *__restrict__ image, int height,
                                                   int width, uint32_t first, uint32_t end,
                                                   const LaunchParams &P, uint32_t *bits,
                                                   const Kept &kept, uint2 *res_all) {
  const int lane = threadIdx.x & 31, shift = (lane & 7) * 4;
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5, rpr = (uint32_t)runs_per_row(width);
  uint32_t count = 0;
  for (uint32_t run0 = first; run0 < end; run0 += kScanT) {
    const LaneRun r = load_run(bits, run0 + lane, end, rpr, wpr);
    if (!dense_group(__reduce_add_sync(0xffffffffu, run_pixels(r)), run0, end))
      continue;  // whole warp
    uint2 *res = res_all + (size_t)run0 * kept.keep;
    const uint32_t places = group_places(kept, run0, end);
    uint32_t passed = 0;
    for (uint32_t run = run0; run < min(end, run0 + 32u); run++) {
      // The run's word of this lane's columns.
      const uint32_t y = run / rpr, word = (run - y * rpr) * kRunWords + (uint32_t)(lane >> 3);
      uint32_t *at_word = bits + (size_t)y * wpr + word;
      const uint32_t w = word < wpr ? *at_word : 0u;
      if (!__any_sync(0xffffffffu, w != 0u))
        continue;  // whole warp
      uint2 mine[4];
      const uint32_t pass = disp_dense_run<K, Pix>(
          image, height, width, (int)y, (int)((run - y * rpr) * kRunWords * 32u),
          w >> shift & 15u, P, mine);
      const uint32_t upto = warp_inclusive((uint32_t)__popc(pass), lane);
      uint32_t at = passed + upto - (uint32_t)__popc(pass);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (pass >> c & 1u) {
          if (at < places)
            res[at] = mine[c];
          at++;
        }
      }
      passed += __shfl_sync(0xffffffffu, upto, 31);
      uint32_t left = pass << shift;
      left |= __shfl_xor_sync(0xffffffffu, left, 1);
      left |= __shfl_xor_sync(0xffffffffu, left, 2);
      left |= __shfl_xor_sync(0xffffffffu, left, 4);
      if ((lane & 7) == 0 && left != w)
        *at_word = left;
    }
    count += passed;
  }
  return count;
}

template <int K, typename Pix>
__global__ void __launch_bounds__(kScanT, 4)
disp_decide(const __grid_constant__ FramePtrs F, const __grid_constant__ LaunchParams P,
            uint32_t *__restrict__ bits_all, size_t words, Kept kept,
            uint32_t *__restrict__ block_sums) {
  previous_done();
  __shared__ uint32_t s_clear[kScanT / 32][32 * kRunWords];
  const int f = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Pix *image = reinterpret_cast<const Pix *>(F.image[f]);
  const int height = F.h[f], width = F.w[f];
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5, rpr = (uint32_t)runs_per_row(width);
  uint32_t *bits = bits_all + (size_t)f * words;
  int row_lo, row_hi;
  band_share(height, &row_lo, &row_hi);
  const uint32_t first = (uint32_t)row_lo * rpr + (uint32_t)warp * 32u;
  const uint32_t end = (uint32_t)row_hi * rpr;
  uint32_t count = 0;
  bool dense = false;  // a group is left for disp_dense_groups
  for (uint32_t run0 = first; run0 < end; run0 += kScanT) {
    const LaneRun r = load_run(bits, run0 + lane, end, rpr, wpr);
    const uint32_t incl = warp_inclusive(run_pixels(r), lane);
    const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
    if (dense_group(all, run0, end)) {
      dense = true;
      continue;  // whole warp
    }
    if (all == 0)
      continue;  // whole warp
#pragma unroll
    for (int k = 0; k < kRunWords; k++)
      s_clear[warp][kRunWords * lane + k] = 0u;
    __syncwarp();
    uint2 *res = kept.res + (size_t)f * kept.stride + (size_t)run0 * kept.keep;
    uint32_t passed = 0;  // of these runs so far
    visit_pixels<4>(r, incl, lane,
                    [&](bool live, uint32_t, uint32_t, int owner, int k, int bit, int y, int x) {
                      uint32_t n;
                      unsigned long long S, Q;
                      disp_window<K, Pix>(image, height, width, live, lane & 3, y, x, &n, &S, &Q);
                      const bool mine = live && (lane & 3) == 0;
                      const bool ok =
                          mine && disp_strong<Pix>(
                                      (uint32_t)__ldg(image + (size_t)y * width + x), n, S, Q, P);
                      const unsigned pass = __ballot_sync(0xffffffffu, ok);
                      const uint32_t at = passed + __popc(pass & ((1u << lane) - 1u));
                      if (ok && at < group_places(kept, run0, end))
                        res[at] =
                            make_uint2(__float_as_uint(window_mean<Pix>(n, S, P.min_local)), n);
                      if (mine && !ok)
                        atomicOr(&s_clear[warp][kRunWords * owner + k], 1u << bit);
                      passed += (uint32_t)__popc(pass);
                    });
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kRunWords; k++) {
      const uint32_t clear = s_clear[warp][kRunWords * lane + k];
      if (clear)
        bits[(size_t)r.y * wpr + r.word + k] = r.w[k] & ~clear;
    }
    __syncwarp();
    count += lane == 0 ? passed : 0u;
  }
  if (dense) {  // whole warp
    const uint32_t passed =
        disp_dense_groups<K, Pix>(image, height, width, first, end, P, bits, kept,
                                  kept.res + (size_t)f * kept.stride);
    count += lane == 0 ? passed : 0u;
  }
  uint32_t total;
  (void)block_exclusive_scan(count, &total);
  if (threadIdx.x == 0)
    block_sums[(size_t)f * gridDim.x + blockIdx.x] = total;
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------

DispTables make_disp_tables(const LaunchParams &P) {
  DispTables T;
  const int n0 = (2 * P.half + 1) * (2 * P.half + 1);
  // One unit below the floor: the reference's rounding of its own sums (below
  // 2^31 where a window is filtered by these) moves the tests by less.
  auto floored = [](double x, uint32_t most) {
    const double v = std::floor(x) - 1.0;
    return v <= 0.0 ? 0u : v >= (double)most ? most : (uint32_t)v;
  };
  for (int n = 0; n <= kMaxN0; n++) {
    const bool testable = n >= 1 && (uint32_t)n >= P.min_local && n <= n0;
    T.nk[n] = testable ? 16u * (uint32_t)n : 0u;
    T.clo[n] =
        testable ? floored(16.0 * P.gain * (n - 1 + P.sigma_b * P.root[n]), kMaxC16) : 0u;
    T.kk[n] = testable ? floored(P.sigma_s * P.sigma_s * P.gain * n, kDispMaxKK) : 0u;
  }
  return T;
}

template <int K, typename Pix, int C> cudaError_t disp_slots(int *slots_out) {
  using G = StripG<K>;
  constexpr size_t smem = strip_smem<K, Pix, C>();
  static_assert(sizeof(Pix) == 2 || (smem + sizeof(uint4) * (G::N0 + 1) + 1024) * G::Occ <=
                                        228 * 1024,
                "the blocks an SM that the kernel is built for");
  static std::once_flag configured;
  static cudaError_t config_error = cudaSuccess;
  static int slots = 0;
  std::call_once(configured, [] {
    config_error = cudaFuncSetAttribute(disp_strip<K, Pix, C>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per = 0;
    if (config_error == cudaSuccess)
      config_error = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, disp_strip<K, Pix, C>,
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
  const cudaError_t e = disp_slots<K, Pix, C>(&slots);
  if (e != cudaSuccess)
    return e;
  FrameSpans S;
  run_rows = strip_spans<C>(F, nframes, slots, run_rows, &S);
  const unsigned blocks = (unsigned)((S.start[nframes] + kStripWarps - 1) / kStripWarps);
  disp_strip<K, Pix, C><<<blocks, kStripWarps * 32, strip_smem<K, Pix, C>(), stream>>>(
      F, nframes, S, run_rows, make_disp_tables(P), P, reinterpret_cast<uint8_t *>(b.bits),
      b.words * sizeof(uint32_t));
  return cudaSuccess;
}

template <int K, typename Pix>
cudaError_t launch_disp(const FramePtrs &F, int nframes, int h, int w, const LaunchParams &P,
                        const StreamBuffers &b, int run_rows, cudaStream_t stream,
                        const StreamMarks *marks) {
  int slots = 0;
  cudaError_t e = disp_slots<K, Pix, kWideCols>(&slots);
  if (e == cudaSuccess)
    e = narrow_strips(F, nframes, slots)
            ? launch_strips<K, Pix, kNarrowCols>(F, nframes, P, b, run_rows, stream)
            : launch_strips<K, Pix, kWideCols>(F, nframes, P, b, run_rows, stream);
  if (e != cudaSuccess)
    return e;
  if (marks)
    cudaEventRecord(marks->stage01, stream);
  const dim3 grid = band_grid(nframes, h, w);
  const Kept kept = make_kept(b, h, w);
  launch_after(disp_decide<K, Pix>, grid, kScanT, 0, stream, F, P, b.bits, b.words, kept,
               b.block_sums);
  if (marks)
    cudaEventRecord(marks->stage2, stream);
  launch_after(scatter_pixels<Pix, false>, grid, kScanT, 0, stream, F, b.bits, b.words, nullptr, K,
               kept, P.min_local, b.block_sums, nullptr, 0u, nullptr, b.out, b.out_stride,
               b.capacity, b.count_out, b.prefix);
  if (marks)
    cudaEventRecord(marks->order, stream);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_dispersion(const FramePtrs &F, int nframes, int h, int w, int pixel_bytes,
                              const LaunchParams &P, const StreamBuffers &b, int run_rows,
                              cudaStream_t stream, const StreamMarks *marks) {
  if (nframes < 1 || nframes > kMaxBatch || P.algorithm != SF_DISPERSION ||
      !streaming_path(P, pixel_bytes))
    return cudaErrorInvalidValue;
  if (marks)
    cudaEventRecord(marks->start, stream);
  auto launch = [&](auto k) {
    constexpr int K = decltype(k)::value;
    return pixel_bytes == 2 ? launch_disp<K, uint16_t>(F, nframes, h, w, P, b, run_rows, stream, marks)
                            : launch_disp<K, uint32_t>(F, nframes, h, w, P, b, run_rows, stream, marks);
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

} // namespace sf
