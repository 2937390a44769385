// bits.cuh -- tests on a double's bits.  A double comparison, minimum or maximum takes a
// slot of the FP64 pipe (64 cycles per warp and quarter SM on GB300); these do not.
#pragma once
#include "snap.cuh"

namespace fmf {

// the bits, by a move the compiler does not see through (it turns sign and zero tests of a
// reinterpreted double back into comparisons)
__device__ __forceinline__ long long raw(double x) {
  long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
}
constexpr long long kOneBits = 0x3ff0000000000000ll;  // 1.0
constexpr long long kInfBits = 0x7ff0000000000000ll;

// the magnitude bits shifted up: 0 for +0 and -0 only
__device__ __forceinline__ unsigned long long mag(double x) {
  return (unsigned long long)raw(x) << 1;
}
__device__ __forceinline__ bool is_nan(double x) { return mag(x) > ((unsigned long long)kInfBits << 1); }
__device__ __forceinline__ bool finite_bits(long long b) { return ((b >> 52) & 0x7ff) != 0x7ff; }
// x >= 0 (true for -0; differs from the comparison for NaN only)
__device__ __forceinline__ bool nonneg(double x) {
  const long long b = raw(x);
  return b >= 0 || (b << 1) == 0;
}
// fmax(fmin(p, 1), 0): NaN gives 1, as fmin does; -0 gives 0
__device__ __forceinline__ double clip01(double p) {
  const long long b = raw(p);
  if (b > kOneBits || is_nan(p)) return 1.0;
  return b < 0 ? 0.0 : p;
}
// the snap of phi outside the band
__device__ __forceinline__ double snap01(double p, const Snap& s) { return snapped(p, raw(p), s); }

// The point of this thread in a plane of w points a row (from (0, 0); may be past the
// ends); blockIdx.z is the plane.  A warp takes 8 x 4 points, so that of the warps that
// skip their arithmetic where all their points are flat fewer meet an interface than of
// rows of 32 (one of 10 cells normal to x: 2 in 16 columns of warps, not 1.3 in 4).  A
// block takes 32 x 4 or 32 x 8 points, which share their rows in the L1, or (one row of
// blocks) the next of the plane's warps: on small grids, where the ragged last columns of
// blocks are a large part.  A step of 32x32x16: 421 us with the first, 410 with the second;
// fmf_dev_csf_fused on 128x64x256: 353 and 411.
struct Tile {
  int x, y;
};
__device__ __forceinline__ Tile warp_tile(int w) {
  const int v = (int)threadIdx.x >> 5, l = (int)threadIdx.x & 31;
  if (gridDim.y > 1)
    return {(int)blockIdx.x * 32 + (v & 3) * 8 + (l & 7),
            (int)(blockIdx.y * (blockDim.x >> 5)) + (v >> 2) * 4 + (l >> 3)};
  const int n = (int)(blockIdx.x * (blockDim.x >> 5)) + v, nx = (w + 7) >> 3, ty = n / nx;
  return {(n - ty * nx) * 8 + (l & 7), ty * 4 + (l >> 3)};
}
inline dim3 tile_grid(int w, int h, int planes, int block) {
  const int rows = block / 32;
  if ((long)w * h * planes >= 1L << 17 && h > rows)
    return dim3((unsigned)((w + 31) / 32), (unsigned)((h + rows - 1) / rows), (unsigned)planes);
  const long warps = (long)((w + 7) / 8) * ((h + 3) / 4);
  return dim3((unsigned)((warps + rows - 1) / rows), 1, (unsigned)planes);
}

}  // namespace fmf
