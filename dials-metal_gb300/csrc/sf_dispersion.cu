// The plain dispersion threshold (SF_DISPERSION) for frames of either pixel
// type: a valid pixel above the global threshold is strong when its clipped
// (2K + 1)-square window passes the dispersion test of stage 0 and
// (n p - S) > sigma_s sqrt(gain S n).
//
//   disp_strip    every pixel's window, one warp per 360-column strip and run
//                 of rows: a mask that holds every strong pixel and few others
//   disp_decide   each set pixel decided from its window's full sums by the
//                 reference's sequence; the failures leave the mask, which is
//                 then the strong-pixel mask, and the blocks count theirs
//   disp_scatter  the mask's pixels as records, ascending, each at its place
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
#include "sf_order.cuh"
#include "sf_scan.cuh"
#include "sf_stream.cuh"
#include "sf_strips.cuh"

namespace sf {
namespace {

constexpr int kDispCols = 12;                       // columns a lane owns
constexpr int kDispOut = kDispCols * 30;            // lanes 1-30 write; 0 and 31 are their halos
constexpr int kDispWarps = 2;                       // warps a block
constexpr int kDispStride = kDispCols * 32;         // pixels a staged row
constexpr int kDispMinRun = 8;                      // shortest run of output rows
constexpr int kDispLongRun = 64;                    // shortest for the sake of even waves
constexpr int kDispWaves = 4;
// A window's masked count above its sum: 81 << 25 and 81 x 65533 both fit.
constexpr uint32_t kDispPS = 25;
constexpr uint32_t kDispMask = (1u << kDispPS) - 1u;

template <int K> struct DispG {
  static constexpr int W0 = 2 * K + 1;
  static constexpr int N0 = W0 * W0;
  // Rows in flight ahead of the current one, the staged rows (from the one
  // leaving the window to the last in flight) and the blocks an SM that those
  // of 32-bit frames leave room for. One row's arithmetic takes longer than a
  // load, so few rows ahead and more warps.
  static constexpr int Ahead = K == 4 ? 1 : 2;
  static constexpr int Slots = W0 + Ahead + 1;
  static constexpr int Occ = K == 2 ? 8 : K == 3 ? 7 : 6;
  // Valid 32-bit pixels saturate at Cap, so that a window's sum of squares
  // stays below 2^32, and a window whose sum of squares reaches Big passes the
  // first filter. Below Big it holds no saturated pixel, its sum is at most
  // sqrt(N0 Big) = 2^13.5, and the filter's products stay below 2^32.
  static constexpr uint32_t Cap = K == 2 ? 13107 : K == 3 ? 9362 : 7281;
  static constexpr uint32_t Big = (1u << 27) / N0;
  static_assert((unsigned long long)Cap * Cap * N0 < (1ull << 32) && Cap * Cap >= Big,
                "exact squares, and a saturated pixel makes its window big");
};

// The filters' constants for a window of n valid pixels, rounded down: nk =
// 16 n (0 when n cannot be tested), clo <= 16 c where the dispersion test is n
// Q - S (S + c) > 0 but for rounding, and kk <= sigma_s^2 gain n.
constexpr uint32_t kDispMaxC = 1u << 17;  // keeps 16 S^2 + S clo below 2^32 for S <= 2^13.5
constexpr uint32_t kDispMaxKK = 7200;     // keeps S kk below 65535 x 65536 for S <= 81 x 7281
struct DispTables {
  uint32_t nk[kMaxN0 + 1], clo[kMaxN0 + 1], kk[kMaxN0 + 1];
};

template <int K, typename Pix>
constexpr size_t disp_smem() {
  return (size_t)kDispWarps * DispG<K>::Slots * kDispStride * sizeof(Pix);
}

__device__ __forceinline__ bool disp_aligned(const void *image, int width, int bytes) {
  return width % 4 == 0 && reinterpret_cast<uintptr_t>(image) % (4 * bytes) == 0;
}

// A valid pixel's value, or a lone count bit for a masked one (whose square
// wraps to 0).
template <int K, typename Pix> __device__ __forceinline__ uint32_t disp_pack(uint32_t v) {
  if (sizeof(Pix) == 2)
    return v >= 0xFFFEu ? 1u << kDispPS : v;
  return v >= 0xFFFFFFFEu ? 1u << kDispPS : min(v, DispG<K>::Cap);
}

// A lane's 12 staged pixels, packed. 32-bit rows are packed in place when
// they arrive (kRaw reads them first), 16-bit rows whenever they are read.
template <int K, typename Pix, bool kRaw>
__device__ __forceinline__ void disp_read(Pix *slot, int lane, uint32_t v[kDispCols]) {
  if constexpr (sizeof(Pix) == 2) {
    const uint2 *src = reinterpret_cast<const uint2 *>(slot + kDispCols * lane);
#pragma unroll
    for (int i = 0; i < kDispCols / 4; i++) {
      const uint2 x = src[i];
      v[4 * i] = disp_pack<K, Pix>(x.x & 0xFFFFu), v[4 * i + 1] = disp_pack<K, Pix>(x.x >> 16);
      v[4 * i + 2] = disp_pack<K, Pix>(x.y & 0xFFFFu), v[4 * i + 3] = disp_pack<K, Pix>(x.y >> 16);
    }
  } else {
    uint4 *src = reinterpret_cast<uint4 *>(slot + kDispCols * lane);
#pragma unroll
    for (int i = 0; i < kDispCols / 4; i++) {
      uint4 x = src[i];
      if (kRaw) {
        x.x = disp_pack<K, Pix>(x.x), x.y = disp_pack<K, Pix>(x.y);
        x.z = disp_pack<K, Pix>(x.z), x.w = disp_pack<K, Pix>(x.w);
        src[i] = x;
      }
      v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
    }
  }
}

// The tests of one window of n valid pixels with sum S and sum of squares Q,
// and of its centre pixel p (packed): false only where the reference's are.
template <int K, typename Pix>
__device__ __forceinline__ bool disp_maybe0(uint32_t n, uint32_t S, uint32_t Q, uint32_t nk,
                                            uint32_t clo, const LaunchParams &P) {
  if constexpr (sizeof(Pix) == 2)
    return stage0_u16(n, S, Q, P);  // the reference's float test itself
  // (Bitwise: branches around the halves took the kernel from 344 to 437 us.)
  return (Q >= DispG<K>::Big) | (Q * nk > S * ((S << 4) + clo));
}
template <int K, typename Pix>
__device__ __forceinline__ bool disp_maybe2(uint32_t p, uint32_t n, uint32_t S, uint32_t kk,
                                            const LaunchParams &P) {
  if constexpr (sizeof(Pix) == 2) {
    const float m = __uint2float_rn(n), s = __uint2float_rn(S), v = __uint2float_rn(p);
    return __fsub_rn(__fmul_rn(m, v), s) >
           __fmul_rn((float)P.sigma_s, __fsqrt_rn(__fmul_rn(__fmul_rn((float)P.gain, s), m)));
  }
  // d = n p - S against sqrt(kk S): d falls and kk S rises with S, so a
  // saturated sum, at most the true one, passes wherever the true one does.
  // d^2 + d covers the rounding of the reference's right side (under half a
  // unit in d), and d beyond 65535 passes whatever S is.
  const int d = (int)(n * p) - (int)S;
  const uint32_t e = (uint32_t)min(d, 65535);
  return (p >= DispG<K>::Cap) | ((d > 0) & (e * e + e >= S * kk));
}

// One warp walks down a strip of 360 output columns for a run of rows. Lane l
// owns 12 columns; lanes 0 and 31 hold the columns on either side of the strip
// that the others' windows reach into. Each pixel row is staged in shared
// memory by cp.async three rows ahead and stays there until it leaves the
// window: the lane adds the row to its 12 column sums as it enters, subtracts
// it as it leaves, and reads it once more as the centre row. A window is 2K +
// 1 column sums; the K beyond either end of a lane's columns come by shuffles.
// Bound by issue: 50 instructions a pixel at 70% of the issue rate. 16 frames of
// 3262 x 3108 took 4.57 ms as 32 x 32 tiles (each pixel's window summed in
// 64 bits from shared memory, the halo staged 2.6 times over), and take 0.44 ms
// here: 344 us in this kernel, 70 and 30 in the two below.
template <int K, typename Pix>
__global__ void __launch_bounds__(kDispWarps * 32, DispG<K>::Occ)
disp_strip(const __grid_constant__ FramePtrs F, int nframes, const __grid_constant__ FrameSpans S,
           int run_rows, const __grid_constant__ DispTables T,
           const __grid_constant__ LaunchParams P, uint8_t *__restrict__ mask_all,
           size_t mask_bytes) {
  using G = DispG<K>;
  extern __shared__ __align__(16) unsigned char disp_raw[];
  __shared__ uint4 tab[G::N0 + 1];  // by masked count m: nk, clo, kk of n = N0 - m
  for (int m = threadIdx.x; m <= G::N0; m += blockDim.x)
    tab[m] = make_uint4(T.nk[G::N0 - m], T.clo[G::N0 - m], T.kk[G::N0 - m], 0u);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gw = blockIdx.x * kDispWarps + warp;
  if (gw >= S.start[nframes])
    return;  // whole warp
  const int f = span_frame(S, nframes, gw);
  const uint32_t local = (uint32_t)(gw - S.start[f]);
  const int ry = (int)fast_div(local, S.by_row[f]);
  const int sx = (int)(local - (uint32_t)ry * S.by_row[f].d);
  const int height = F.h[f], width = F.w[f];
  const Pix *image = reinterpret_cast<const Pix *>(F.image[f]);
  const bool aligned = disp_aligned(image, width, sizeof(Pix));
  const int bytes_per_row = ((width + 31) >> 5) * 4;
  uint8_t *mask = mask_all + (size_t)f * mask_bytes;
  const int X = kDispOut * sx, cx = X + kDispCols * (lane - 1);
  const bool writer = lane >= 1 && lane <= 30, first_of_pair = (lane & 1) != 0;
  const int pair_byte = (X + 24 * ((lane - 1) >> 1)) >> 3;
  const uint32_t inside12 =
      (cx < 0 || cx >= width) ? 0u
                              : (cx + kDispCols <= width ? 0xFFFu : ((1u << (width - cx)) - 1u));
  const int ra = ry * run_rows, rb = min(height, ra + run_rows);
  const int pbeg = ra - K, rows = rb - ra + 2 * K;
  Pix *ring = reinterpret_cast<Pix *>(disp_raw) + (size_t)warp * G::Slots * kDispStride;

  // Row pbeg + i into its slot: pieces of 4 pixels where the frame's rows are
  // whole aligned pieces, else a pixel at a time. Bit u of `inside`: this
  // lane's u-th piece or pixel of a row lies in the frame.
  const int x0 = X - kDispCols;  // the staged row's first column
  uint32_t inside = 0;
#pragma unroll
  for (int u = 0; u < kDispCols; u++) {
    const int c = aligned ? x0 + 4 * lane + 128 * u : x0 + lane + 32 * u;
    inside |= (aligned ? u < 3 && c >= 0 && c + 4 <= width : c >= 0 && c < width) ? 1u << u : 0u;
  }
  const Pix *next_row = image + (ptrdiff_t)pbeg * width + x0 + (aligned ? 4 * lane : lane);
  int next_p = pbeg;
  const int pend = min(height, pbeg + rows);
  auto fetch = [&](Pix *slot) {
    const uint32_t in = next_p >= 0 && next_p < pend ? inside : 0u;
    if (aligned) {
      Pix *dst = slot + 4 * lane;
#pragma unroll
      for (int u = 0; u < 3; u++) {
        if ((in >> u) & 1u)
          cp_async_piece<Pix>(dst + 128 * u, next_row + 128 * u);
        else
          fill_piece_masked<Pix>(dst + 128 * u);
      }
    } else {
      Pix *dst = slot + lane;
#pragma unroll
      for (int u = 0; u < kDispCols; u++) {
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
  };
  auto after = [&](int s) { return s + 1 == G::Slots ? 0 : s + 1; };
#pragma unroll
  for (int i = 0; i < G::Ahead; i++) {
    fetch(ring + i * kDispStride);
    cp_async_commit();
  }
  uint32_t Vn[kDispCols], Vq[kDispCols];
#pragma unroll
  for (int c = 0; c < kDispCols; c++)
    Vn[c] = Vq[c] = 0u;
  const uint4 whole = tab[0];
  uint8_t *out_row = mask + (size_t)ra * bytes_per_row + pair_byte;
  const int bytes_left = bytes_per_row - pair_byte;
  // Slots of the row in flight, the current, the centre and the leaving row.
  int s_in = G::Ahead, s_cur = 0, s_mid = G::Slots - K, s_old = G::Slots - G::W0;
  for (int i = 0; i < rows; i++) {
    __syncwarp();  // every lane is done with the slot that is filled next
    fetch(ring + s_in * kDispStride);
    cp_async_commit();
    cp_async_wait<G::Ahead>();
    __syncwarp();
    uint32_t v[kDispCols], o[kDispCols];
    disp_read<K, Pix, true>(ring + s_cur * kDispStride, lane, v);
    if (i >= G::W0) {  // warp-uniform
      disp_read<K, Pix, false>(ring + s_old * kDispStride, lane, o);
    } else {
#pragma unroll
      for (int c = 0; c < kDispCols; c++)
        o[c] = 0u;
    }
#pragma unroll
    for (int c = 0; c < kDispCols; c++) {
      Vn[c] += v[c] - o[c];
      Vq[c] += v[c] * v[c] - o[c] * o[c];
    }
    if (i >= 2 * K) {  // warp-uniform: the windows are whole
      // The column sums from K columns before this lane's to K after them.
      uint32_t en[kDispCols + 2 * K], eq[kDispCols + 2 * K];
#pragma unroll
      for (int c = 0; c < kDispCols; c++)
        en[K + c] = Vn[c], eq[K + c] = Vq[c];
#pragma unroll
      for (int k = 0; k < K; k++) {
        en[k] = __shfl_up_sync(0xffffffffu, Vn[kDispCols - K + k], 1);
        eq[k] = __shfl_up_sync(0xffffffffu, Vq[kDispCols - K + k], 1);
        en[K + kDispCols + k] = __shfl_down_sync(0xffffffffu, Vn[k], 1);
        eq[K + kDispCols + k] = __shfl_down_sync(0xffffffffu, Vq[k], 1);
      }
      uint32_t hn[kDispCols], hq[kDispCols];
      hn[0] = hq[0] = 0u;
#pragma unroll
      for (int k = 0; k < G::W0; k++)
        hn[0] += en[k], hq[0] += eq[k];
      uint32_t any_masked = hn[0];
#pragma unroll
      for (int c = 1; c < kDispCols; c++) {
        hn[c] = hn[c - 1] + en[c + 2 * K] - en[c - 1];
        hq[c] = hq[c - 1] + eq[c + 2 * K] - eq[c - 1];
        any_masked |= hn[c];
      }
      // Warp rows whose windows hold no masked pixel (most) take the whole
      // window's constants; the others look each window's count up.
      const bool uniform = !__any_sync(0xffffffffu, any_masked >> kDispPS);
      uint32_t out = 0;
      if (uniform) {
#pragma unroll
        for (int c = 0; c < kDispCols; c++)
          out |= disp_maybe0<K, Pix>(G::N0, hn[c], hq[c], whole.x, whole.y, P) ? 1u << c : 0u;
      } else {
#pragma unroll
        for (int c = 0; c < kDispCols; c++) {
          const uint32_t m = min(hn[c] >> kDispPS, (uint32_t)G::N0);
          const uint4 t = tab[m];
          out |= disp_maybe0<K, Pix>(G::N0 - m, hn[c] & kDispMask, hq[c], t.x, t.y, P) ? 1u << c
                                                                                     : 0u;
        }
      }
      out &= inside12;
      if (__any_sync(0xffffffffu, out != 0u)) {
        disp_read<K, Pix, false>(ring + s_mid * kDispStride, lane, v);
        uint32_t out2 = 0;
#pragma unroll
        for (int c = 0; c < kDispCols; c++) {
          uint32_t n = G::N0, kk = whole.z, W = hn[c];
          bool valid = true;
          if (!uniform) {
            const uint32_t m = min(W >> kDispPS, (uint32_t)G::N0);
            n -= m;
            kk = tab[m].z;
            W &= kDispMask;
            valid = v[c] < (1u << kDispPS);
          }
          out2 |= valid & disp_maybe2<K, Pix>(v[c], n, W, kk, P) ? 1u << c : 0u;
        }
        out &= out2;
      }
      // Lane pairs: the first lane (odd) writes the pair's first two bytes,
      // the second the third.
      const uint32_t next = __shfl_down_sync(0xffffffffu, out, 1);
      if (writer) {
        if (first_of_pair) {
          if (bytes_left > 0)
            out_row[0] = (uint8_t)out;
          if (bytes_left > 1)
            out_row[1] = (uint8_t)((out >> 8) | (next & 0xFu) << 4);
        } else if (bytes_left > 2) {
          out_row[2] = (uint8_t)(out >> 4);
        }
      }
      out_row += bytes_per_row;
    }
    s_in = after(s_in);
    s_cur = after(s_cur);
    s_mid = after(s_mid);
    s_old = after(s_old);
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
           disp_maybe2<2, Pix>(p, n, (uint32_t)S, 0u, P);  // the float test itself
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

// The window's mean as the records hold it: float(RN_double(S / n)) is
// RN_float(S / n) for S below 2^24 (sf_common.cuh), and 16-bit frames divide in
// float.
template <typename Pix>
__device__ __forceinline__ float disp_mean(uint32_t n, unsigned long long S) {
  return sizeof(Pix) == 2 || S < (1ull << 24)
             ? __fdiv_rn(__uint2float_rn((uint32_t)S), __uint2float_rn(n))
             : __double2float_rn(__ddiv_rn(__ull2double_rn(S), (double)n));
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

// The two kernels below give a warp groups of 128 mask words, kWordsPer
// consecutive ones a lane: about 15 candidates on frames of spots, enough for
// whole rounds of eight (groups of 32 words took 1.8 times the time), and
// few enough that a small frame's spread over the GPU.
constexpr int kWordsPer = 4;
constexpr int kGroupWords = 32 * kWordsPer;
constexpr int kDispPass = kScanT * kWordsPer;

// A lane's words of the group at `base` of n (zeros past the end).
__device__ __forceinline__ void group_words(const uint32_t *bits, size_t base, size_t n, int lane,
                                            uint32_t w[kWordsPer]) {
#pragma unroll
  for (int k = 0; k < kWordsPer; k++) {
    const size_t i = base + (size_t)kWordsPer * lane + k;
    w[k] = i < n ? bits[i] : 0u;
  }
}
__device__ __forceinline__ uint32_t group_pixels(const uint32_t w[kWordsPer]) {
  uint32_t c = 0;
#pragma unroll
  for (int k = 0; k < kWordsPer; k++)
    c += (uint32_t)__popc(w[k]);
  return c;
}

// The set pixels of a group (lane l's words w, incl the inclusive prefix of
// their counts over the lanes), in order, 32 / kLanes at a time with kLanes
// lanes each: visit(live, q, word, bit, y, x), q the pixel's place among them
// and word its word's place in the group. The whole warp calls it.
template <int kLanes, class Visit>
__device__ __forceinline__ void visit_pixels(const uint32_t w[kWordsPer], uint32_t incl,
                                             uint32_t first, uint32_t wpr, int lane,
                                             Visit visit) {
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t excl = incl - group_pixels(w);
  for (uint32_t q0 = 0; q0 < total; q0 += 32 / kLanes) {  // warp-uniform
    const uint32_t q = q0 + lane / kLanes;
    const bool live = q < total;
    int owner = 0;
#pragma unroll
    for (int s = 16; s; s >>= 1)
      owner += __shfl_sync(0xffffffffu, incl, owner + s - 1) <= q ? s : 0;
    owner &= 31;
    uint32_t k = q - __shfl_sync(0xffffffffu, excl, owner), word = 0;
    int j = 0;
#pragma unroll
    for (int i = 0; i < kWordsPer; i++) {
      const uint32_t x = __shfl_sync(0xffffffffu, w[i], owner), c = (uint32_t)__popc(x);
      word = j == i ? x : word;
      if (j == i && i + 1 < kWordsPer && k >= c) {
        k -= c;
        j = i + 1;
      }
    }
    const int bit = live ? select_bit(word, k) : 0;
    const int at = owner * kWordsPer + j;
    const uint32_t wi = first + at, y = wi / wpr;
    visit(live, q, at, bit, (int)y, (int)((wi - y * wpr) * 32u) + bit);
  }
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

// This block's share [lo, hi) of n mask words, in whole passes.
__device__ __forceinline__ void disp_share(size_t n, size_t *lo, size_t *hi) {
  const size_t passes = (n + kDispPass - 1) / kDispPass;
  const size_t share = (passes + gridDim.x - 1) / gridDim.x * kDispPass;
  *lo = min(n, (size_t)blockIdx.x * share);
  *hi = min(n, *lo + share);
}

// Results kept between the two kernels: a group of 128 words of a frame has
// `keep` places, the passing pixels' backgrounds and populations in order. A
// group with more than that has its windows summed again (keep 0: all have).
struct DispKept {
  uint2 *res;
  uint32_t stride, keep;  // places a frame, and a group
};
template <int K, typename Pix>
__global__ void __launch_bounds__(kScanT)
disp_decide(const __grid_constant__ FramePtrs F, const __grid_constant__ LaunchParams P,
            uint32_t *__restrict__ bits_all, size_t words, DispKept kept,
            uint32_t *__restrict__ block_sums) {
  __shared__ uint32_t s_clear[kScanT / 32][kGroupWords];
  const int f = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Pix *image = reinterpret_cast<const Pix *>(F.image[f]);
  const int height = F.h[f], width = F.w[f];
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5;
  uint32_t *bits = bits_all + (size_t)f * words;
  size_t lo, hi;
  disp_share(frame_words(F, f), &lo, &hi);
  uint32_t count = 0;
  for (size_t base = lo + (size_t)warp * kGroupWords; base < hi; base += kDispPass) {
    uint32_t w[kWordsPer];
    group_words(bits, base, hi, lane, w);
    const uint32_t incl = warp_inclusive(group_pixels(w), lane);
    if (__shfl_sync(0xffffffffu, incl, 31) == 0)
      continue;  // whole warp
#pragma unroll
    for (int k = 0; k < kWordsPer; k++)
      s_clear[warp][kWordsPer * lane + k] = 0u;
    __syncwarp();
    uint2 *res = kept.res + (size_t)f * kept.stride + base / kGroupWords * kept.keep;
    uint32_t passed = 0;  // of this group so far
    visit_pixels<4>(w, incl, (uint32_t)base, wpr, lane,
                    [&](bool live, uint32_t, int word, int bit, int y, int x) {
                      uint32_t n;
                      unsigned long long S, Q;
                      disp_window<K, Pix>(image, height, width, live, lane & 3, y, x, &n, &S, &Q);
                      const bool mine = live && (lane & 3) == 0;
                      const bool ok =
                          mine && disp_strong<Pix>(
                                      (uint32_t)__ldg(image + (size_t)y * width + x), n, S, Q, P);
                      const unsigned pass = __ballot_sync(0xffffffffu, ok);
                      const uint32_t at = passed + __popc(pass & ((1u << lane) - 1u));
                      if (ok && at < kept.keep)
                        res[at] = make_uint2(__float_as_uint(disp_mean<Pix>(n, S)), n);
                      if (mine && !ok)
                        atomicOr(&s_clear[warp][word], 1u << bit);
                      passed += (uint32_t)__popc(pass);
                    });
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kWordsPer; k++) {
      const uint32_t clear = s_clear[warp][kWordsPer * lane + k];
      if (clear)
        bits[base + (size_t)kWordsPer * lane + k] = w[k] & ~clear;
    }
    __syncwarp();
    count += lane == 0 ? passed : 0u;
  }
  uint32_t total;
  (void)block_exclusive_scan(count, &total);
  if (threadIdx.x == 0)
    block_sums[(size_t)f * gridDim.x + blockIdx.x] = total;
}

template <int K, typename Pix>
__global__ void __launch_bounds__(kScanT)
disp_scatter(const __grid_constant__ FramePtrs F, const uint32_t *__restrict__ bits_all,
             size_t words, DispKept kept, const uint32_t *__restrict__ block_sums,
             sf_signal_pixel *__restrict__ out_all, size_t out_stride, uint32_t capacity,
             uint32_t *__restrict__ count_out, uint32_t *__restrict__ prefix_all) {
  const int f = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Pix *image = reinterpret_cast<const Pix *>(F.image[f]);
  const int height = F.h[f], width = F.w[f];
  const uint32_t wpr = ((uint32_t)width + 31u) >> 5;
  const uint32_t *bits = bits_all + (size_t)f * words;
  sf_signal_pixel *out = out_all + (size_t)f * out_stride;
  uint32_t total;
  uint32_t run = block_base(block_sums, &total);
  if (blockIdx.x == 0 && threadIdx.x == 0)
    count_out[f] = total;
  __shared__ uint32_t s_warp[kScanT / 32];
  auto put = [&](uint32_t at, int y, int x, float background, uint32_t n) {
    if (at >= capacity)
      return;
    sf_signal_pixel rec;
    rec.index = (uint32_t)y * (uint32_t)width + (uint32_t)x;
    rec.value = (uint32_t)__ldg(image + rec.index);
    rec.background = background;
    rec.population = (uint16_t)n;
    rec.reserved = 0;
    out[at] = rec;
  };
  size_t lo, hi;
  disp_share(frame_words(F, f), &lo, &hi);
  for (size_t pass = lo; pass < hi; pass += kDispPass) {  // block-uniform
    const size_t base = pass + (size_t)warp * kGroupWords;
    uint32_t w[kWordsPer];
    group_words(bits, base, hi, lane, w);
    const uint32_t incl = warp_inclusive(group_pixels(w), lane);
    const uint32_t mine = __shfl_sync(0xffffffffu, incl, 31);
    __syncthreads();  // the last pass's sums have been read
    if (lane == 0)
      s_warp[warp] = mine;
    __syncthreads();
    uint32_t pos = run;
#pragma unroll
    for (int k = 0; k < kScanT / 32; k++) {
      pos += k < warp ? s_warp[k] : 0u;
      run += s_warp[k];
    }
    if (!prefix_all && mine == 0)
      continue;  // warp-uniform, and the barriers above are reached again
    const bool held = mine <= kept.keep;
    const uint2 *res = kept.res + (size_t)f * kept.stride + base / kGroupWords * kept.keep;
    if (prefix_all) {
      uint32_t at = pos + incl - group_pixels(w);
#pragma unroll
      for (int k = 0; k < kWordsPer; k++) {
        const size_t i = base + (size_t)kWordsPer * lane + k;
        if (i < hi)
          prefix_all[(size_t)f * words + i] = at;
        at += (uint32_t)__popc(w[k]);
      }
    }
    if (held)
      visit_pixels<1>(w, incl, (uint32_t)base, wpr, lane,
                      [&](bool live, uint32_t q, int, int, int y, int x) {
                        if (live) {
                          const uint2 b = __ldg(res + q);
                          put(pos + q, y, x, __uint_as_float(b.x), b.y);
                        }
                      });
    else
      visit_pixels<4>(w, incl, (uint32_t)base, wpr, lane,
                      [&](bool live, uint32_t q, int, int, int y, int x) {
                        uint32_t n;
                        unsigned long long S, Q;
                        disp_window<K, Pix>(image, height, width, live, lane & 3, y, x, &n, &S,
                                            &Q);
                        if (live && (lane & 3) == 0)
                          put(pos + q, y, x, disp_mean<Pix>(n, S), n);
                      });
  }
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
        testable ? floored(16.0 * P.gain * (n - 1 + P.sigma_b * P.root[n]), kDispMaxC) : 0u;
    T.kk[n] = testable ? floored(P.sigma_s * P.sigma_s * P.gain * n, kDispMaxKK) : 0u;
  }
  return T;
}

template <int K, typename Pix>
cudaError_t launch_disp(const FramePtrs &F, int nframes, const LaunchParams &P,
                        const StreamBuffers &b, int run_rows, cudaStream_t stream,
                        const StreamMarks *marks) {
  using G = DispG<K>;
  constexpr size_t smem = disp_smem<K, Pix>();
  static std::once_flag configured;
  static cudaError_t config_error = cudaSuccess;
  static int slots = 0;
  std::call_once(configured, [] {
    config_error = cudaFuncSetAttribute(disp_strip<K, Pix>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per = 0;
    if (config_error == cudaSuccess)
      config_error = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, disp_strip<K, Pix>,
                                                                   kDispWarps * 32, smem);
    slots = std::max(1, per) * kDispWarps * device_sms();
  });
  if (config_error != cudaSuccess)
    return config_error;
  static_assert(sizeof(Pix) == 2 || (smem + sizeof(uint4) * (G::N0 + 1) + 1024) * G::Occ <=
                                        228 * 1024,
                "the blocks an SM that the kernel is built for");
  // Runs that fill the resident warps kDispWaves times over, so that warps of
  // unequal cost even out (one wave left 36% of the warps' time idle), as
  // long as a run's rows stay kDispLongRun or more (each run reads 2K rows
  // more than it writes); else once, down to runs of kDispMinRun.
  long long strips = 0;
  int tallest = 0;
  auto strips_of = [](int w) { return ((w + 31) / 32 * 32 + kDispOut - 1) / kDispOut; };
  for (int f = 0; f < nframes; f++) {
    strips += strips_of(F.w[f]);
    tallest = std::max(tallest, F.h[f]);
  }
  if (run_rows <= 0) {
    const long long runs = std::max(1ll, slots / strips);
    const int once = (int)((tallest + runs - 1) / runs);
    run_rows = std::min(once, std::max(kDispLongRun, (once + kDispWaves - 1) / kDispWaves));
  }
  run_rows = std::max(run_rows, kDispMinRun);
  FrameSpans S;
  S.start[0] = 0;
  for (int f = 0; f < nframes; f++) {
    S.start[f + 1] = S.start[f] + strips_of(F.w[f]) * ((F.h[f] + run_rows - 1) / run_rows);
    S.by_row[f] = make_fastdiv((uint32_t)strips_of(F.w[f]));
  }
  const unsigned blocks = (unsigned)((S.start[nframes] + kDispWarps - 1) / kDispWarps);
  disp_strip<K, Pix><<<blocks, kDispWarps * 32, smem, stream>>>(
      F, nframes, S, run_rows, make_disp_tables(P), P, reinterpret_cast<uint8_t *>(b.bits),
      b.words * sizeof(uint32_t));
  if (marks)
    cudaEventRecord(marks->stage01, stream);
  const size_t passes = (b.words + kDispPass - 1) / kDispPass;
  const dim3 og((unsigned)std::min(passes, (size_t)(stream_order_blocks() / nframes)),
                (unsigned)nframes);
  const size_t groups = (b.words + kGroupWords - 1) / kGroupWords;
  const DispKept kept = {b.res, b.cand_cap, (uint32_t)(b.cand_cap / groups)};
  disp_decide<K, Pix><<<og, kScanT, 0, stream>>>(F, P, b.bits, b.words, kept, b.block_sums);
  if (marks)
    cudaEventRecord(marks->stage2, stream);
  disp_scatter<K, Pix><<<og, kScanT, 0, stream>>>(F, b.bits, b.words, kept, b.block_sums, b.out,
                                                  b.out_stride, b.capacity, b.count_out,
                                                  b.prefix);
  if (marks)
    cudaEventRecord(marks->order, stream);
  return cudaGetLastError();
}

}  // namespace

bool dispersion_path(const LaunchParams &P, int pixel_bytes) {
  if (P.algorithm != SF_DISPERSION)
    return false;
  // 32-bit windows are filtered by bounds that need a right side of at least
  // zero; 16-bit ones are tested by the reference's sequence itself.
  return pixel_bytes == 2 || (P.gain >= 0.0 && P.sigma_b >= 0.0 && P.sigma_s >= 0.0);
}

cudaError_t launch_dispersion(const FramePtrs &F, int nframes, int pixel_bytes,
                              const LaunchParams &P, const StreamBuffers &b, int run_rows,
                              cudaStream_t stream, const StreamMarks *marks) {
  if (nframes < 1 || nframes > kMaxBatch || !dispersion_path(P, pixel_bytes))
    return cudaErrorInvalidValue;
  if (marks)
    cudaEventRecord(marks->start, stream);
  auto launch = [&](auto k) {
    constexpr int K = decltype(k)::value;
    return pixel_bytes == 2 ? launch_disp<K, uint16_t>(F, nframes, P, b, run_rows, stream, marks)
                            : launch_disp<K, uint32_t>(F, nframes, P, b, run_rows, stream, marks);
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
