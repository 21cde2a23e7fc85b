// Internal interface of the lattice path (sf_lattice.cu).
//
// The stage-0 decision from exact 32-bit window sums. With gain 1 and an
// integral sigma_b the reference's test (src/spots/dext.cc:99-109) is
// A > RN(X), A = nQ - S(S + n - 1) exact in double and X = S sigma_b r_n
// (r_n the reference's double sqrt(2 (n - 1))). Writing c = n - 1 +
// sigma_b r_n, A - X = nQ - S(S + c). Per window count n the host gives two
// integers in 2^-8 units, clo <= 2^8 c <= chi (from the 2^-20 brackets of
// r_n), and nk = 2^8 n (0 when n cannot be tested):
//   2^8 n Q <= S (2^8 S + clo)           =>  A <= X: not signal
//   2^8 n Q >= S (2^8 S + chi) + 2^9     =>  A >= X + 2 > RN(X): signal
// both exact in 64-bit integers. The thin band between goes to the exact
// decision of sf_common.cuh. The packed sums (the window's masked-pixel count above
// a 26-bit sum) and the 32-bit sum of squares hold while every valid pixel is below
// narrow_max; a tile holding a larger valid pixel is decided in 64 bits.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "sf_common.cuh"
#include "sf_stream.cuh"

namespace sf {

// The launch's counter words.
enum {
  kCtrTiles = 0,  // tiles listed for the exact check
  kCtrFault = 1,  // a bounded device wait ran out (the launch's lists are void)
  kCounterWords = 2
};

constexpr int kDec = 8;  // fixed-point bits of clo / chi

struct StreamTables {
  uint32_t narrow_max;  // valid pixels at or above this take the 64-bit path
  uint32_t nk[kMaxN0 + 1], clo[kMaxN0 + 1], chi[kMaxN0 + 1];
};

// The lattice pass for kernel 3,3 (sf_lattice.cu): strips of 360 output
// columns (one warp each) by runs of run_rows rows, a multiple of 3.
constexpr int kLatMinRunRows = 9, kLatLongRun = 96, kLatWaves = 5;
struct LatticeGeometry {
  int nstrips, nruns, run_rows;
};
// run_rows 0: the default geometry.
LatticeGeometry lattice_geometry(int h, int w, int nframes, int run_rows);
// Stage 0 and the erosion for kernel 3,3: the lattice bound, then the exact
// check of its candidates; writes the candidate masks b.cand (the reference's
// eroded masks but for the masked pixels). pixel_bytes 4 (32-bit frames) or 2
// (16-bit frames: 4 | w, 8-byte aligned).
cudaError_t launch_lattice(const FramePtrs &frames, int nframes, int h, int w, int pixel_bytes,
                           const LaunchParams &P, const StreamBuffers &b, int run_rows,
                           cudaStream_t stream);

} // namespace sf
