// fused_mthinc.cu -- the vertex gradients (cal_grad_p2a.f), MTHINC fluxes
// (solphi_mthinc1.f) and snap (solphi_mthinc3.f:61-120) for the fused step; the rest of
// the transport is in k_transport.cu.
//
// Away from the interface phi is exactly 0 or 1 (solphi_mthinc3's snap), and there
// these kernels' FP64 operations give zeros or the value they were given: a warp
// whose points are all such takes that result from the bits of what it read and does
// no arithmetic.  The FP64 pipe, 64 cycles per warp instruction, bounds every kernel
// here otherwise.
//
// Fluxes: two kernels instead of one thread per cell on the full 0..n+1 range:
//   k_classify: every cell forms its normal from the 8 vertex gradients; cells
//     outside the interface band write their truncated upwind fluxes at once,
//     band cells are appended to a compact list;
//   k_band: one thread per band cell (list entry) runs the 10 Newton steps and
//     writes the swept-volume fluxes.
// A warp then carries band cells only, instead of idling on the bulk cells that
// share its x-run.  The sigmoid derivative uses 1/cosh^2(a) = 4 s (1 - s) with
// s = 1/(1 + exp(-2a)) (same function, one exp per Gauss point).
//
// Face ownership: a face is written by its donor cell (u>0: the west cell, u<0:
// the east cell) or left zero; cells write their east/north/top face when u>=0
// and their west/south/bottom face when u<0, so every face in 0..n of every
// interior row gets exactly one writer (solphi_mthinc1.f:121-130 zeroes first;
// faces nobody donates through hold the zero written by k_classify's owner).
#include <cmath>
#include <cstring>

#include "../../include/fmf_capi.h"
#include "bits.cuh"
#include "fused.cuh"
#include "recip.cuh"

namespace fmf {
namespace fused {

namespace {
struct MC {
  double gp1, gp2, lim, bet, dt, dxi, dyi, dzi;
  double lim2lo, lim2hi;  // lim^2 (1 -/+ 1e-12)
  double dtdx, dtdy, dtdz;  // dt dxinv etc.
  Snap snap;                // with eps_trunc
};
// the constants of solphi_mthinc1.f and solphi_mthinc3.f (dt = 0 for the latter)
MC make_mc(double dxinv, double dyinv, double dzinv, double dt, double bet) {
  MC m;
  const double dx = 1.0 / dxinv, dy = 1.0 / dyinv, dz = 1.0 / dzinv;
  m.gp1 = -0.5 / std::sqrt(3.0);
  m.gp2 = 0.5 / std::sqrt(3.0);
  const double dcellinv = 1.0 / std::sqrt((dx * dx + dy * dy + dz * dz) / 3.0);
  const double ch = std::cosh(-bet * 1.5);
  m.lim = bet / (2.0 * (ch * ch)) * dcellinv;
  m.lim2lo = m.lim * m.lim * (1.0 - 1.0e-12);
  m.lim2hi = m.lim * m.lim * (1.0 + 1.0e-12);
  m.snap = make_snap(0.5 * (std::tanh(-bet * 2.5) + 1.0));
  m.bet = bet;
  m.dt = dt;
  m.dxi = dxinv;
  m.dyi = dyinv;
  m.dzi = dzinv;
  m.dtdx = dt * dxinv;
  m.dtdy = dt * dyinv;
  m.dtdz = dt * dzinv;
  return m;
}

// The 8 vertex gradients around a cell, and whether any of them is not 0
struct G8 {
  double v[8];
  __device__ __forceinline__ unsigned long long load(const double* __restrict__ p, long c, long X, long Y, long Z) {
    v[0] = __ldg(p + c - X - Y - Z);
    v[1] = __ldg(p + c - Y - Z);
    v[2] = __ldg(p + c - X - Z);
    v[3] = __ldg(p + c - Z);
    v[4] = __ldg(p + c - X - Y);
    v[5] = __ldg(p + c - Y);
    v[6] = __ldg(p + c - X);
    v[7] = __ldg(p + c);
    unsigned long long z = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) z |= mag(v[t]);
    return z;
  }
  __device__ __forceinline__ double mean() const {
    return (v[0] + v[1] + v[2] + v[3] + v[4] + v[5] + v[6] + v[7]) * 0.125;
  }
};
// The band test sqrt(q2) <= lim of the reference for the squared norm q2 of the mean
// gradient: decided on q2 against lim^2 where q2 is clearly on one side (compared as
// bit patterns: all three are non-negative), with the square root only within 1e-12 of
// it.  q2 is rounded operation by operation, as the adjoint's record of the snap does.
__device__ __forceinline__ bool outside_band(const G8& gx, const G8& gy, const G8& gz, const MC& m) {
  const double x = gx.mean(), y = gy.mean(), z = gz.mean();
  const double q2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
  const long long qb = raw(q2);
  return qb < raw(m.lim2lo) ? true
                                             : (qb > raw(m.lim2hi) ? false : sqrt(q2) <= m.lim);
}

__device__ __forceinline__ double avg8(const double* __restrict__ p, long c, long X, long Y, long Z) {
  return (__ldg(p + c - X - Y - Z) + __ldg(p + c - Y - Z) + __ldg(p + c - X - Z) + __ldg(p + c - Z) +
          __ldg(p + c - X - Y) + __ldg(p + c - Y) + __ldg(p + c - X) + __ldg(p + c)) *
         0.125;
}

__device__ __forceinline__ double ex(double x) { return exp(x); }
__device__ __forceinline__ float ex(float x) { return expf(fminf(x, 80.0f)); }

// 1/(1+e) for e >= 0: the division-free reciprocal in double (an overflowed e gives
// exactly 0, as the quotient does; NaN stays NaN), the quotient in float
__device__ __forceinline__ double inv1p(double e) {
  const double a = 1.0 + e;
  return (__double2hiint(a) == 0x7ff00000 && __double2loint(a) == 0) ? 0.0 : recip_nr(a);
}
__device__ __forceinline__ float inv1p(float e) { return 1.0f / (1.0f + e); }

// The sum over the 8 Gauss points t of w/(1+exp(m2b (a_t + d))) (m2b = -2 bet) and,
// optionally, the sum of s(1-s) (1-s = e/(1+e), exact in relative terms for any
// a_t), with exp(m2b (a_t + d)) factorised: a_t = x + y + z over the Gauss
// offsets of the three axes, so exp(m2b a_t) = X Y Z of per-axis factors (E_t,
// gexp8) and only exp(m2b d) changes with d.  Every factor is bounded by the
// normal's unit length times the Gauss offsets; where exp(m2b d) overflows or
// underflows, so does the unfactorised exponential.  Six exponentials per cell
// and one per Newton step instead of eight per step.
template <class R>
__device__ __forceinline__ R sig8f(const R* E, R w, R ed, R* sd) {
  R s = 0, q = 0;
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const R e = E[t] * ed;
    const R r = inv1p(e);
    s += r;
    if (sizeof(R) == 8 && r == (R)0) continue;  // an overflowed e: no 0 times infinity
    if (sd) q += e * r * r;
  }
  if (sd) *sd = q;
  return w * s;
}
// E_t over the 8 Gauss points, x fastest, then y, then z: factors X1 X2, Y1 Y2, Z1 Z2
template <class R>
__device__ __forceinline__ void gexp8(R* E, R X1, R X2, R Y1, R Y2, R Z1, R Z2) {
  const R a = X1 * Y1, b = X2 * Y1, c = X1 * Y2, d = X2 * Y2;
  E[0] = a * Z1;
  E[1] = b * Z1;
  E[2] = c * Z1;
  E[3] = d * Z1;
  E[4] = a * Z2;
  E[5] = b * Z2;
  E[6] = c * Z2;
  E[7] = d * Z2;
}
// (at 256x128x128: 199 us, 178 with five blocks per SM, 151 with warps of 8 x 4 and the
// fluxes and sign tests below)
__global__ void __launch_bounds__(256, 5) k_classify(Grid g, MC m, const double* __restrict__ phi,
                                                  const double* __restrict__ gx, const double* __restrict__ gy,
                                                  const double* __restrict__ gz, const double* __restrict__ u,
                                                  const double* __restrict__ v, const double* __restrict__ w,
                                                  double* __restrict__ fx, double* __restrict__ fy,
                                                  double* __restrict__ fz, int* __restrict__ list,
                                                  int* __restrict__ count) {
  after_previous();
  const Tile T = warp_tile(g.ni + 2);
  const int i = T.x, j = T.y, k = (int)blockIdx.z;
  if (i > g.ni + 1 || j > g.nj + 1) return;
  const long X = 1, Y = g.sy, Z = g.sz;
  const long c = g.at(i, j, k);
  G8 ax, ay, az;
  const bool graded = (ax.load(gx, c, X, Y, Z) | ay.load(gy, c, X, Y, Z) | az.load(gz, c, X, Y, Z)) != 0;
  const double uw = __ldg(u + c - X), ue = __ldg(u + c), vs = __ldg(v + c - Y), vn = __ldg(v + c),
               wb = __ldg(w + c - Z), wt = __ldg(w + c);
  const unsigned warp = __activemask();
  const bool band = __any_sync(warp, graded) && !outside_band(ax, ay, az, m);
  if (band) {
    const int slot = atomicAdd(count, 1);
    list[slot] = (int)c;
  }
  const double phi00 = band ? 0.0 : snap01(__ldg(phi + c), m.snap);
  // owned faces: east/north/top when the velocity there is >= 0 (this cell donates or
  // the flux is zero), west/south/bottom when < 0; band cells leave the donated
  // faces to k_band but still zero the owned faces they do not donate through.
  // Fluxes are v phi dt/dx with phi dt/dx formed first.
  // One product per axis, of the velocity that donates, and a second where a lane donates
  // both ways, formed by the whole warp (stores under their lanes' signs alone: products
  // under them were issued per set of lanes, 15 slots of the FP64 pipe for 3 products).
  const long long pb = raw(phi00);
  double pdx = 0.0, pdy = 0.0, pdz = 0.0;
  // (a velocity that is not finite has a flux that is not, where phi is 0 as well)
  auto size = [](double x) { return __double2hiint(x) & 0x7fffffff; };
  const int fastest = max(max(max(size(uw), size(ue)), max(size(vs), size(vn))), max(size(wb), size(wt)));
  const bool filled = __any_sync(warp, pb != 0 || fastest >= 0x7ff00000);
  if (filled) {
    if (__any_sync(warp, pb != 0 && pb != kOneBits)) {
      pdx = phi00 * m.dtdx;
      pdy = phi00 * m.dtdy;
      pdz = phi00 * m.dtdz;
    } else if (pb != 0) {
      pdx = m.dtdx;
      pdy = m.dtdy;
      pdz = m.dtdz;
    }
  }
  const bool e_ = nonneg(ue), w_ = nonneg(uw), n_ = nonneg(vn), s_ = nonneg(vs), t_ = nonneg(wt), b_ = nonneg(wb);
  const bool two_x = __any_sync(warp, e_ && !w_), two_y = __any_sync(warp, n_ && !s_), two_z = __any_sync(warp, t_ && !b_);
  double xe = 0.0, xw = 0.0, yn = 0.0, ys = 0.0, zt = 0.0, zb = 0.0;
  if (filled) {
    xe = xw = (e_ ? ue : uw) * pdx;
    yn = ys = (n_ ? vn : vs) * pdy;
    zt = zb = (t_ ? wt : wb) * pdz;
    if (two_x) xw = uw * pdx;
    if (two_y) ys = vs * pdy;
    if (two_z) zb = wb * pdz;
  }
  if (e_) fx[c] = xe;
  if (!w_) fx[c - X] = xw;
  if (n_) fy[c] = yn;
  if (!s_) fy[c - Y] = ys;
  if (t_) fz[c] = zt;
  if (!b_) fz[c - Z] = zb;
  // west/south/bottom faces of the first cells with no in-range donor stay zero
  if (i == 0 && w_) fx[c - X] = 0.0;
  if (j == 0 && s_) fy[c - Y] = 0.0;
  if (k == 0 && b_) fz[c - Z] = 0.0;
  if (i == g.ni + 1 && !e_) fx[c] = 0.0;
  if (j == g.nj + 1 && !n_) fy[c] = 0.0;
  if (k == g.nk + 1 && !t_) fz[c] = 0.0;
}

// The ten Newton steps on the offset itself.  R = float: the mixed-precision step (normal,
// band test and the fluxes' storage stay double; the Newton solve and the Gauss-point
// integrals run in float with the exponent argument clamped to the float range and the
// Newton regularisation 1e-99 raised to 1e-30).  R = double: FP64 outside the steepnesses
// of k_band below (band_in_y).
template <class R>
__global__ void __launch_bounds__(128) k_band_ten(Grid g, MC m, const double* __restrict__ phi,
                                              const double* __restrict__ gx, const double* __restrict__ gy,
                                              const double* __restrict__ gz, const double* __restrict__ u,
                                              const double* __restrict__ v, const double* __restrict__ w,
                                              double* __restrict__ fx, double* __restrict__ fy,
                                              double* __restrict__ fz, const int* __restrict__ list,
                                              const int* __restrict__ count, double* __restrict__ newton,
                                              long cap) {
  after_previous();
  const int n = *count;
  const long X = 1, Y = g.sy, Z = g.sz;
  const R m2b = (R)(-2.0 * m.bet), gp1 = (R)m.gp1, gp2 = (R)m.gp2, bet = (R)m.bet, dtt = (R)m.dt;
  const R reg = sizeof(R) == 8 ? (R)1.0e-99 : (R)1.0e-30;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const long c = list[e];
    double nx = avg8(gx, c, X, Y, Z), ny = avg8(gy, c, X, Y, Z), nz = avg8(gz, c, X, Y, Z);
    const double q00 = sqrt(nx * nx + ny * ny + nz * nz);
    const double coef = 1.0 / q00;
    const R rnx = (R)(nx * coef), rny = (R)(ny * coef), rnz = (R)(nz * coef);
    // per-axis factors exp(m2b n gp) of the centred Gauss points
    const R X1 = ex(m2b * rnx * gp1), X2 = ex(m2b * rnx * gp2), Y1 = ex(m2b * rny * gp1),
            Y2 = ex(m2b * rny * gp2), Z1 = ex(m2b * rnz * gp1), Z2 = ex(m2b * rnz * gp2);
    R E[8];
    gexp8<R>(E, X1, X2, Y1, Y2, Z1, Z2);
    const R ph = (R)__ldg(phi + c);
    R ddd = 0, step = 0;
#pragma unroll 1
    for (int it = 0; it < 10; ++it) {
      R sd;
      const R f = sig8f<R>(E, (R)0.125, ex(m2b * ddd), &sd) - ph;
      // df = 0.5 bet sum 0.125/cosh^2 = 0.5 bet * 0.125 * 4 * sum s(1-s)
      const R df = (R)0.25 * bet * sd;
      step = sizeof(R) == 8 ? (R)((double)(f * df) * recip_nr((double)(df * df + reg))) : f * df / (df * df + reg);
      const R dn = ddd - step;
      // once d no longer changes, every remaining iteration recomputes the same
      // f, df and step: stopping here is the ten-step result bit for bit.  In
      // float the iterate can dither in its last bit instead; there a step below
      // float precision ends the loop.
      if (dn == ddd) break;
      ddd = dn;
      if (sizeof(R) == 4 && fabs((double)step) <= 1.0e-7 * (1.0 + fabs((double)ddd))) break;
    }
    if (newton) {
      newton[e] = (double)ddd;
      newton[cap + e] = (double)step;
    }
    const double uw = __ldg(u + c - X), ue = __ldg(u + c), vs = __ldg(v + c - Y), vn = __ldg(v + c),
                 wb = __ldg(w + c - Z), wt = __ldg(w + c);
    const R edf = ex(m2b * ddd);  // exp(m2b d) at the offset found
    auto side = [&](double vel, double dinv, int axis, bool minus, double* out) {
      const R vd = (R)vel * dtt * (R)dinv;
      const R st = minus ? (R)-0.5 : (R)0.5 - vd, en = minus ? (R)-0.5 - vd : (R)0.5;
      const R g1 = (st + en) * (R)0.5 + (-st + en) * gp1, g2 = (st + en) * (R)0.5 + (-st + en) * gp2;
      // the flux axis takes the swept interval's Gauss points, the others the centred ones
      R Eb[8];
      if (axis == 0) gexp8<R>(Eb, ex(m2b * rnx * g1), ex(m2b * rnx * g2), Y1, Y2, Z1, Z2);
      else if (axis == 1) gexp8<R>(Eb, X1, X2, ex(m2b * rny * g1), ex(m2b * rny * g2), Z1, Z2);
      else gexp8<R>(Eb, X1, X2, Y1, Y2, ex(m2b * rnz * g1), ex(m2b * rnz * g2));
      *out = (double)sig8f<R>(Eb, (R)0.125 * vd, edf, nullptr);
    };
    if (uw < 0.0) side(uw, m.dxi, 0, true, fx + c - X);
    if (ue > 0.0) side(ue, m.dxi, 0, false, fx + c);
    if (vs < 0.0) side(vs, m.dyi, 1, true, fy + c - Y);
    if (vn > 0.0) side(vn, m.dyi, 1, false, fy + c);
    if (wb < 0.0) side(wb, m.dzi, 2, true, fz + c - Z);
    if (wt > 0.0) side(wt, m.dzi, 2, false, fz + c);
  }
}
// FP64 band cells, bound by the FP64 pipe: 10 Newton steps per warp in nearly all (a cell
// with phi near 0 or 1 takes them, at about 1/(2 bet) each, and may not have converged),
// then the fluxes.
//  * The centred Gauss points come in pairs of opposite signs, so with E + 1/E = k and
//    y = exp(m2b d) a pair's sum of sigmoids is (2 + k y)/(1 + k y + y^2) and its sum of
//    s (1 - s) is y (k + 4 y + k y^2)/(1 + k y + y^2)^2: four reciprocals per step instead
//    of eight.  On the swept axis the factors F1, F2 take the two other axes' pairs with
//    F y in the place of y.
//  * The iteration runs in y, which is all the fluxes need of the offset: a step of d
//    multiplies y by exp(-m2b step).
//  * A step below 1e-9 (1 + |d|) is the last: Newton's error squares per step and leaves
//    the root to rounding, where the ten steps of solphi_mthinc1.f dither.
//  * The exponentials have small arguments: exp16 below.
//  * One pass per axis for the faces of both sides: lanes of unlike velocity share it.
// 1.57 -> 0.96 ms at 512x256x256, 317 -> 182 us at 128x64x64, 63 -> 45 at 32x32x16 (the last
// of these 616 -> 543 us of the couette 256x128x128).
// Sixteenths: exp(k/16), k = -64 .. 64, formed on the host.
struct Exp16 {
  double t[129];
};
// exp(z) = exp(k/16) exp(r), k the integer nearest 16 z, |r| <= 1/32, the second factor by
// its Taylor polynomial (the term after z^7/7! is below 3e-17 of the sum); |z| > 4 and NaN:
// exp itself
__device__ __forceinline__ double exp16(const Exp16& T, double z) {
  if (!(mag(z) <= mag(4.0))) return exp(z);
  const double s = fma(z, 16.0, 6755399441055744.0);  // 1.5 * 2^52: the sum's low bits are k
  const int k = __double2loint(s);
  const double r = fma(s - 6755399441055744.0, -0.0625, z);
  double p = fma(r, 1.0 / 5040.0, 1.0 / 720.0);
  p = fma(p, r, 1.0 / 120.0);
  p = fma(p, r, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  const double e = T.t[k + 64];
  return fma(p * r, e, e);
}
// 1/D for D >= 1 (an overflowed D gives exactly 0; NaN stays NaN)
__device__ __forceinline__ double recip_ge1(double d) {
  return (__double2hiint(d) == 0x7ff00000 && __double2loint(d) == 0) ? 0.0 : recip_h(d);
}
__global__ void __launch_bounds__(64) k_band(Grid g, MC m, __grid_constant__ const Exp16 T,
                                             const double* __restrict__ phi, const double* __restrict__ gx,
                                             const double* __restrict__ gy, const double* __restrict__ gz,
                                             const double* __restrict__ u, const double* __restrict__ v,
                                             const double* __restrict__ w, double* __restrict__ fx,
                                             double* __restrict__ fy, double* __restrict__ fz,
                                             const int* __restrict__ list, const int* __restrict__ count,
                                             double* __restrict__ newton, long cap) {
  after_previous();
  const int n = *count;
  const long X = 1, Y = g.sy, Z = g.sz;
  const double m2b = -2.0 * m.bet;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const long c = list[e];
    const double nx = avg8(gx, c, X, Y, Z), ny = avg8(gy, c, X, Y, Z), nz = avg8(gz, c, X, Y, Z);
    const double coef = m2b * rsqrt_h(fma(nz, nz, fma(ny, ny, nx * nx)));
    const double b[3] = {nx * coef, ny * coef, nz * coef};  // m2b times the unit normal
    // per axis exp(b gp) of the two centred Gauss points (gp1 = -gp2)
    const double X2 = exp16(T, b[0] * m.gp2), Y2 = exp16(T, b[1] * m.gp2), Z2 = exp16(T, b[2] * m.gp2);
    const double X1 = recip_h(X2), Y1 = recip_h(Y2), Z1 = recip_h(Z2);
    // k = E + 1/E of the pairs: same and opposite signs on the two axes other than x, y, z
    const double yz = Y2 * Z2, yzi = Y1 * Z1, yoz = Y2 * Z1, zoy = Y1 * Z2;
    const double kx0 = yz + yzi, kx1 = yoz + zoy;
    const double ky0 = fma(X2, Z2, X1 * Z1), ky1 = fma(X2, Z1, X1 * Z2);
    const double kz0 = fma(X2, Y2, X1 * Y1), kz1 = fma(X2, Y1, X1 * Y2);
    const double ph = __ldg(phi + c);
    double y = 1.0, ddd = 0.0, step = 0.0;
    {
      const double kk[4] = {fma(X2, yz, X1 * yzi), fma(X1, yz, X2 * yzi), fma(X2, yoz, X1 * zoy), fma(X1, yoz, X2 * zoy)};
#pragma unroll 1
      for (int it = 0; it < 10; ++it) {
        const double y2 = y * y, y4 = 4.0 * y2;
        double s = 0.0, q = 0.0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const double ky = kk[t] * y, r = recip_ge1(fma(y, y, 1.0 + ky));
          s = fma(2.0 + ky, r, s);
          q = fma(fma(ky, y2 * r, (ky + y4) * r), r, q);  // y^2 r <= 1: no overflow
        }
        // df = 0.5 bet sum 0.125/cosh^2 = 0.5 bet * 0.125 * 4 * sum s(1-s)
        const double f = fma(s, 0.125, -ph), df = 0.25 * m.bet * q;
        step = f * df * recip_h(fma(df, df, 1.0e-99));
        ddd -= step;
        if (mag(step) == 0) break;
        y *= exp16(T, -m2b * step);
        if (mag(y) > mag(1.0e150) && !is_nan(y)) y = 1.0e150;  // y^2 stays finite
        if (mag(step) <= mag(fma(fabs(ddd), 1.0e-9, 1.0e-9))) {
          step = 0.0;  // converged: the next step is rounding
          break;
        }
      }
    }
    if (newton) {
      newton[e] = ddd;
      newton[cap + e] = step;
    }
    const double uw = __ldg(u + c - X), ue = __ldg(u + c), vs = __ldg(v + c - Y), vn = __ldg(v + c),
                 wb = __ldg(w + c - Z), wt = __ldg(w + c);
    // the fluxes along an axis with b, k0, k1 through the low face (west, south, bottom) where
    // its velocity is negative and the high one where its is positive: the Gauss points of the
    // swept interval lie |vd| (1/2 + gp) inside the face, the high face's mirrored (-b).  One
    // pass for the lanes that donate, through either, and another where one does through both.
    auto axis = [&](double lo, double hi, double dtd, double bb, double k0, double k1, double* flo, double* fhi) {
      const bool dl = raw(lo) < 0 && mag(lo) != 0, dh = raw(hi) > 0;
      bool high = dh, on = dl || dh;
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
        if (on) {
          const double vd = (high ? hi : lo) * dtd, bs = high ? -bb : bb, av = fabs(vd);
          double s = 0.0;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const double f = y * exp16(T, bs * fma(av, 0.5 + (t ? m.gp2 : m.gp1), -0.5));
            const double a = k0 * f, d = k1 * f;
            s = fma(2.0 + a, recip_ge1(fma(f, f, 1.0 + a)), s);
            s = fma(2.0 + d, recip_ge1(fma(f, f, 1.0 + d)), s);
          }
          *(high ? fhi : flo) = 0.125 * vd * s;
        }
        on = dl && dh;
        high = false;
        if (!__any_sync(__activemask(), on)) break;
      }
    };
    axis(uw, ue, m.dtdx, b[0], kx0, kx1, fx + c - X, fx + c);
    axis(vs, vn, m.dtdy, b[1], ky0, ky1, fy + c - Y, fy + c);
    axis(wb, wt, m.dtdz, b[2], kz0, kz1, fz + c - Z, fz + c);
  }
}
// n arguments: spread over [-5, 5] (exp16 hands over to exp at 4), and the same moved to an
// odd thirty-second, where k turns, give or take a few units in the last place
__global__ void k_check_exp16(__grid_constant__ const Exp16 T, long n, unsigned long long* worst) {
  unsigned long long m = 0;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    double z = -5.0 + 10.0 * ((double)t + 0.5) / (double)n;
    if (t & 1) {
      z = (2.0 * rint(16.0 * z - 0.5) + 1.0) * 0.03125;
      z = __longlong_as_double(__double_as_longlong(z) + (t / 2) % 7 - 3);
    }
    const double q = exp(z);
    m = max(m, (unsigned long long)__double_as_longlong(fabs(exp16(T, z) - q) / q));
  }
  atomicMax(worst, m);
}
// cal_grad_p2a.f:46-60 for the fused step: the vertex gradient at (i+1/2, j+1/2,
// k+1/2), i, j, k in -2..n+2, from the 8 surrounding points.  Per (i, j) corner the sum s and difference
// d of the two k planes; with ta = s(+,+) - s(0,0) and tb = s(+,0) - s(0,+) the x sum is
// ta + tb, the y sum ta - tb and the z sum the four differences: 18 FP64 operations per
// point instead of the reference's 27, none in a warp whose points are all flat.
// NEAR1 (phin before its snap, for the band test alone): eight values within 64 units in
// the last place below 1 count as flat.  There phin is 1 but for the roundings of
// solphi_mthinc2.  What that drops is a gradient of at most 2^-47 dxinv per vertex, 7e-13 of
// the band test's limit at bet = 2, 1e-10 at 4, 1e-5 at 8 and more than all of it at 12; but
// a cell is one of the eight values of each of its vertices, so a cell whose test that can
// turn is itself within 64 units of 1, and snapped or not it stays there: phin changes by
// 7.1e-15 at most, whatever bet > 0 is.
template <bool NEAR1>
__global__ void __launch_bounds__(128) k_vertex_grad(Grid g, double cx, double cy, double cz,
                                                     const double* __restrict__ q, double* __restrict__ qx,
                                                     double* __restrict__ qy, double* __restrict__ qz) {
  after_previous();
  const Tile T = warp_tile(g.ni + 5);
  if (T.x >= g.ni + 5 || T.y >= g.nj + 5) return;
  const long X = 1, Y = g.sy, Z = g.sz;
  const long c = g.at(T.x - 2, T.y - 2, (int)blockIdx.z - 2);
  const double q000 = __ldg(q + c), qp00 = __ldg(q + c + X), q0p0 = __ldg(q + c + Y), qpp0 = __ldg(q + c + X + Y),
               q00p = __ldg(q + c + Z), qp0p = __ldg(q + c + X + Z), q0pp = __ldg(q + c + Y + Z),
               qppp = __ldg(q + c + X + Y + Z);
  const long long r = raw(q000);
  auto df = [&](double x) { return (unsigned long long)(raw(x) ^ r); };
  bool flat = (df(qp00) | df(q0p0) | df(qpp0) | df(q00p) | df(qp0p) | df(q0pp) | df(qppp)) == 0 && finite_bits(r);
  if (NEAR1) {
    auto below = [&](double x) { return (unsigned long long)(kOneBits - raw(x)); };
    flat = flat || (below(q000) | below(qp00) | below(q0p0) | below(qpp0) | below(q00p) | below(qp0p) | below(q0pp) |
                    below(qppp)) < 64;
  }
  double gx = 0.0, gy = 0.0, gz = 0.0;
  if (!flat) {
    const double s00 = q000 + q00p, sp0 = qp00 + qp0p, s0p = q0p0 + q0pp, spp = qpp0 + qppp;
    const double ta = spp - s00, tb = sp0 - s0p;
    gx = (ta + tb) * cx;
    gy = (ta - tb) * cy;
    gz = ((q00p - q000) + (qp0p - qp00) + ((q0pp - q0p0) + (qppp - qpp0))) * cz;
  }
  qx[c] = gx;
  qy[c] = gy;
  qz[c] = gz;
}

// solphi_mthinc3.f:61-120: the snap over 0..n+1 of cells outside the band (by the vertex
// gradients of phin) and the clip of the interior, in one pass (each touches its point
// alone).
__global__ void __launch_bounds__(256) k_snap(Grid g, MC m, const double* __restrict__ gx,
                                              const double* __restrict__ gy, const double* __restrict__ gz,
                                              double* __restrict__ phin) {
  after_previous();
  const Tile T = warp_tile(g.ni + 2);
  const int i = T.x, j = T.y, k = (int)blockIdx.z;
  if (i > g.ni + 1 || j > g.nj + 1) return;
  const long X = 1, Y = g.sy, Z = g.sz;
  const long c = g.at(i, j, k);
  G8 ax, ay, az;
  const bool graded = (ax.load(gx, c, X, Y, Z) | ay.load(gy, c, X, Y, Z) | az.load(gz, c, X, Y, Z)) != 0;
  double p = phin[c];
  if (!__any_sync(__activemask(), graded) || outside_band(ax, ay, az, m)) p = snap01(p, m.snap);
  if (i >= 1 && i <= g.ni && j >= 1 && j <= g.nj && k >= 1 && k <= g.nk) p = clip01(p);
  phin[c] = p;
}
}  // namespace

void vertex_gradient(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, const double* q,
                     double* qx, double* qy, double* qz, bool near1) {
  const dim3 gr = tile_grid(g.ni + 5, g.nj + 5, g.nk + 5, 128);
  if (near1)
    chain(s, gr, 128, k_vertex_grad<true>)(g, 0.25 * dxinv, 0.25 * dyinv, 0.25 * dzinv, q, qx, qy, qz);
  else
    chain(s, gr, 128, k_vertex_grad<false>)(g, 0.25 * dxinv, 0.25 * dyinv, 0.25 * dzinv, q, qx, qy, qz);
  count_launch();
}

void mthinc_snap(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double bet,
                 const double* gx, const double* gy, const double* gz, double* phin) {
  const dim3 gr = tile_grid(g.ni + 2, g.nj + 2, g.nk + 2, 256);
  chain(s, gr, 256, k_snap)(g, make_mc(dxinv, dyinv, dzinv, 0.0, bet), gx, gy, gz, phin);
  count_launch();
}

static const Exp16& exp16_table() {
  static const Exp16 table = [] {
    Exp16 e;
    for (int k = -64; k <= 64; ++k) e.t[k + 64] = std::exp(k / 16.0);
    return e;
  }();
  return table;
}

// Up to bet = 4 the ten Newton steps converge or approach their root from one side, and
// either form gives the reference's fluxes to rounding.  Beyond, cells with phi near 0 or 1
// overshoot into the flat tail, where the tenth iterate multiplies every rounding.  Largest
// difference of phi from the oracle after a step, 786 432 cells of random phi, the ten
// steps on the offset itself and k_band's form: 7.8e-16 and 7.8e-16 at 4, 3.8e-11 and
// 1.3e-10 at 6, 9.3e-11 and 3.2e-9 at 8, 1.5e-8 and 2.4e-6 at 12 (cells beyond 1e-13: 64
// and 100, 260 and 476, 833 and 276 128).  The fluxes of a couette 128x64x64 at 4.01 take 586
// us in the former, 379 in the latter.  bet <= 0 (a profile the wrong way round) takes the
// former as well.
bool band_in_y(double bet) { return bet > 0.0 && bet <= 4.0; }

void mthinc_fluxes(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double dt, double bet,
                   const double* phi, const double* gx, const double* gy, const double* gz, const double* u,
                   const double* v, const double* w, double* fx, double* fy, double* fz, int* list, int* count,
                   bool fp32, double* newton) {
  const MC m = make_mc(dxinv, dyinv, dzinv, dt, bet);
  FMF_CUDA(cudaMemsetAsync(count, 0, sizeof(int), s));
  chain(s, tile_grid(g.ni + 2, g.nj + 2, g.nk + 2, 256), 256, k_classify)(g, m, phi, gx, gy, gz, u, v, w, fx, fy, fz, list, count);
  const long cap = (long)(g.ni + 2) * (g.nj + 2) * (g.nk + 2);
  if (fp32)
    chain(s, 152 * 8, 128, k_band_ten<float>)(g, m, phi, gx, gy, gz, u, v, w, fx, fy, fz, list, count, newton, cap);
  else if (!band_in_y(bet))
    chain(s, 152 * 8, 128, k_band_ten<double>)(g, m, phi, gx, gy, gz, u, v, w, fx, fy, fz, list, count, newton, cap);
  else
    chain(s, 152 * 16, 64, k_band)(g, m, exp16_table(), phi, gx, gy, gz, u, v, w, fx, fy, fz, list, count, newton, cap);
  count_launch(2);
}

int check_exp16(long n, double* max_rel_err) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, sizeof(unsigned long long)) != cudaSuccess) return FMF_ERR_NOMEM;
  cudaMemset(d, 0, sizeof(unsigned long long));
  k_check_exp16<<<152 * 4, 256>>>(exp16_table(), n, d);
  count_launch();
  unsigned long long h = 0;
  const cudaError_t e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess || cudaGetLastError() != cudaSuccess) return FMF_ERR_CUDA;
  std::memcpy(max_rel_err, &h, sizeof(double));
  return FMF_OK;
}

}  // namespace fused
}  // namespace fmf

// The short exponential of the band kernel against exp.  Verification support; no
// counterpart in the reference.
extern "C" int fmf_check_exponential(long long n, double* max_rel_err) {
  return max_rel_err && n > 0 ? fmf::fused::check_exp16((long)n, max_rel_err) : FMF_ERR_ARG;
}
