// fused_visc.cu -- the implicit viscous solve of the fused step (solu_sor4.f with
// the coefficients of cal_arith_coef_vis.f / cal_harm_coef_vis.f).
//
// The 45 coefficient arrays are products of six viscosities and constant grid
// factors (cal_arith_coef_vis.f:211-231): for u at (i+1/2,j,k) the x-viscosities
// are the cell values mu(i), mu(i+1) and the y/z ones are edge means shared with
// the neighbours.  k_edges stores the three edge means once per step (the same
// 4-cell sums, in the same order, as the reference) and k_src_ab, per component,
// A = 0.5/(rho00*D) and B = src/D with D = 1/dt + 0.5*a_p/rho00, so a point update
// of solu_sor4.f:150-170 becomes q_new = A*visn + B with visn the 14-neighbour sum.
// Colours are processed in their independent pairs (1,2) (3,4) (5,6) (7,8): two
// colours that differ in every index parity never read each other, so one launch
// per pair gives the sequential result.  The wall/halo refresh after every second
// colour (bndu + bnd_periodic of the swept component, solu_sor4.f:176-180) is one
// kernel (k_refresh; three ordered plane kernels on grids under 8 cells a side) after a
// component's first pair and done by the sweep itself after the others.
//
// The mixed-precision step solves the same system by one step of iterative
// refinement: the residual of the first sweep is formed in FP64 at u, then the
// sweeps run in FP32 on the correction d = un - u (FP32 storage and arithmetic),
// and un = u + d is formed in FP64 at the end.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "bits.cuh"
#include "df64.cuh"
#include "fused.cuh"
#include "recip.cuh"
#include "refresh.cuh"

namespace fmf {
namespace fused {

namespace {
struct VP {
  double dxi, dyi, dzi, dtinv, dx2, dy2, dz2, dxy, dxz, dyz;
  int harmonic;
};

// whether five doubles have the same bits
__device__ __forceinline__ bool same_bits(double a, double b, double c, double d, double e) {
  const long long r = raw(a);
  return ((raw(b) ^ r) | (raw(c) ^ r) | (raw(d) ^ r) |
          (raw(e) ^ r)) == 0;
}
__device__ __forceinline__ double mean4(double a, double b, double c, double d, int harm) {
  if (!harm) return 0.25 * (a + b + c + d);
  return 4.0 / (1.0 / a + 1.0 / b + 1.0 / c + 1.0 / d);
}

// Edge viscosities over i,j,k in 0..n, then A/B per component over the interior.
// f[0..2] non-null: FP32 copies of the three edge arrays as well.
struct F3 {
  float* f[3];
};
// Where the seven viscosities are equal bits their arithmetic means are that value (2a
// is exact, 3a within one unit of a's last place, so 3a + a rounds to 4a), and a warp of
// such points takes it without the arithmetic.  Threads over the flattened (i, j) plane.
__global__ void __launch_bounds__(128) k_edges(Grid g, VP p, const double* __restrict__ mu, double* __restrict__ exy,
                                               double* __restrict__ exz, double* __restrict__ eyz, F3 f, int* count) {
  after_previous();
  if (count && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x) == 0) *count = 0;  // k_src_ab adds to it
  const Tile T = warp_tile(g.ni + 1);
  const int i = T.x, j = T.y, k = (int)blockIdx.z;
  if (i > g.ni || j > g.nj) return;
  const long X = 1, Y = g.sy, Z = g.sz;
  const long c = g.at(i, j, k);
  const double m0 = __ldg(mu + c), mx = __ldg(mu + c + X), my = __ldg(mu + c + Y), mz = __ldg(mu + c + Z),
               mxy = __ldg(mu + c + X + Y), mxz = __ldg(mu + c + X + Z), myz = __ldg(mu + c + Y + Z);
  const bool flat = same_bits(m0, mx, my, mz, mxy) && same_bits(m0, mxz, myz, m0, m0) && !p.harmonic;
  double a = m0, b = m0, d = m0;
  if (__any_sync(__activemask(), !flat)) {
    a = mean4(m0, mx, my, mxy, p.harmonic);
    b = mean4(m0, mx, mz, mxz, p.harmonic);
    d = mean4(m0, my, mz, myz, p.harmonic);
  }
  exy[c] = a;
  exz[c] = b;
  eyz[c] = d;
  if (f.f[0]) {
    f.f[0][c] = df::d2f(a);
    f.f[1][c] = df::d2f(b);
    f.f[2][c] = df::d2f(d);
  }
}

// cal_srcu.f:53-137 fused with the update factors: src is formed in registers and
// only A = 0.5/(rho00*D), B = src/D are stored, and the pressure gradient of
// cal_grad_prs.f is taken from phat = 2 p - po.  With T = 1/(rho00/dt + a_p/2) these are
// A = T/2 and B = (rho00*(explicit terms) - prs + vis/2)*T.
struct SrcIn {
  const double *u, *v, *w, *rho, *rhon, *adv[3], *advo[3], *phat, *vis[3], *fst[3], *fstn[3];
  double grvb, grvp;
};
// Outputs: FP64 A and B per component, or (k_src_ab_e) FP32 A and the FP64 first-sweep
// residual R = A*visn(u) + B - u rounded to FP32 (the right-hand side of the
// correction sweeps of the mixed-precision solve).
struct ABOut {
  double *a[3], *b[3];
  float *af[3], *rf[3];
};
// the grid factors in the arithmetic type of a viscous sum, converted on the host (a
// conversion in a kernel takes an FP64-pipe slot)
template <class T>
struct Fac {
  T dx2, dy2, dz2, dxy, dxz, dyz;
  Fac() = default;
  explicit Fac(const VP& p)
      : dx2((T)p.dx2), dy2((T)p.dy2), dz2((T)p.dz2), dxy((T)p.dxy), dxz((T)p.dxz), dyz((T)p.dyz) {}
};
template <int COMP, class T>
__device__ __forceinline__ T visn_at(const Grid& g, const Fac<T>& p, long c, const T* __restrict__ mu,
                                     const T* __restrict__ exy, const T* __restrict__ exz,
                                     const T* __restrict__ eyz, const T* un, const T* vn, const T* wn);
// FP64 (the FP64 step).  With s = the sum of the four densities (4 rho00), T's
// denominator doubled is 1/A = s/(2 dt) + a_p, one reciprocal (recip_h), and
// B = A (s (explicit terms)/2 - 2 prs + vis), the constants folded on the host: 70 FP64
// operations per cell against 84 and 6 for the gradient's own kernel.  Where the
// densities and viscosities a point reads are one fluid's own (hd: its A per component,
// from the host), a warp of such points skips the denominators: 31 operations.
struct SrcK {
  double hdt;                      // 1/(2 dt)
  double dx2, dy2, dz2;            // dxinv^2 ...
  double tx2, ty2, tz2;            // 2 dxinv^2 ...
  double px, py, pz;               // -2 dxinv ...
  double hg[3];                    // half the body force per component
  long long rb[2], mb[2];          // the two fluids' density and viscosity, as bits
  double s[2], a[2][3];            // 4 rho and A of each
  unsigned char* fluid;            // FlatFluid's bytes and count, or null
  int* count;
};
__global__ void __launch_bounds__(256) k_src_ab(Grid g, SrcK K, SrcIn in, const double* __restrict__ mu,
                                                const double* __restrict__ exy, const double* __restrict__ exz,
                                                const double* __restrict__ eyz, ABOut out) {
  after_previous();
  const Tile T = warp_tile(g.ni);
  const int i = 1 + T.x, j = 1 + T.y, k = 1 + (int)blockIdx.z;
  const bool here = i <= g.ni && j <= g.nj;  // (the count below takes every thread)
  const long X = 1, Y = g.sy, Z = g.sz;
  const long c = here ? g.at(i, j, k) : g.at(1, 1, k);
  auto L = [&](const double* a, long o) { return __ldg(a + c + o); };
  const double r0 = L(in.rho, 0), rx = L(in.rho, X), ry = L(in.rho, Y), rz = L(in.rho, Z);
  const double n0 = L(in.rhon, 0), nx = L(in.rhon, X), ny = L(in.rhon, Y), nz = L(in.rhon, Z);
  const double m0 = L(mu, 0), mx = L(mu, X), my = L(mu, Y), mz = L(mu, Z);
  const double xy0 = L(exy, 0), xyx = L(exy, -X), xyy = L(exy, -Y), xz0 = L(exz, 0), xzx = L(exz, -X),
               xzz = L(exz, -Z), yz0 = L(eyz, 0), yzy = L(eyz, -Y), yzz = L(eyz, -Z);
  const long long rb = raw(r0), mb = raw(m0);
  const bool flat = same_bits(r0, rx, ry, rz, n0) && same_bits(r0, nx, ny, nz, r0) && same_bits(m0, mx, my, mz, xy0) &&
                    same_bits(m0, xyx, xyy, xz0, xzx) && same_bits(m0, xzz, yz0, yzy, yzz);
  const int f = flat && rb == K.rb[0] && mb == K.mb[0] ? 0 : (flat && rb == K.rb[1] && mb == K.mb[1] ? 1 : -1);
  if (K.fluid) {
    if (here) K.fluid[c] = (unsigned char)(f < 0 ? 2 : f);
    const int flats = __syncthreads_count(here && f >= 0);
    if (threadIdx.x == 0 && flats) atomicAdd(K.count, flats);
  }
  if (!here) return;
  double su, sv, sw, Au, Av, Aw;
  if (__any_sync(__activemask(), f < 0)) {
    const double s0 = r0 + n0;
    su = s0 + (rx + nx);
    sv = s0 + (ry + ny);
    sw = s0 + (rz + nz);
    Au = recip_h(fma(K.dz2, xzz + xz0, fma(K.dy2, xyy + xy0, fma(K.tx2, m0 + mx, su * K.hdt))));
    Av = recip_h(fma(K.dz2, yzz + yz0, fma(K.ty2, m0 + my, fma(K.dx2, xyx + xy0, sv * K.hdt))));
    Aw = recip_h(fma(K.tz2, m0 + mz, fma(K.dy2, yzy + yz0, fma(K.dx2, xzx + xz0, sw * K.hdt))));
  } else {
    su = sv = sw = f ? K.s[1] : K.s[0];
    Au = f ? K.a[1][0] : K.a[0][0];
    Av = f ? K.a[1][1] : K.a[0][1];
    Aw = f ? K.a[1][2] : K.a[0][2];
  }
  const double p0 = L(in.phat, 0);
  // B = A (s (vel/dt - 1.5 adv + 0.5 (advo + fst + fstn) + grav)/2 - 2 prs + vis)
  auto store = [&](int q, const double* vel, double s, double A, double pd, double pk) {
    const double t = (L(in.fst[q], 0) + L(in.fstn[q], 0)) + L(in.advo[q], 0);
    const double e = fma(t, 0.25, fma(L(in.adv[q], 0), -0.75, fma(L(vel, 0), K.hdt, K.hg[q])));
    out.a[q][c] = A;
    out.b[q][c] = A * fma(pd, pk, fma(s, e, L(in.vis[q], 0)));
  };
  store(0, in.u, su, Au, L(in.phat, X) - p0, K.px);
  if (j <= g.nj - 1) store(1, in.v, sv, Av, L(in.phat, Y) - p0, K.py);
  store(2, in.w, sw, Aw, L(in.phat, Z) - p0, K.pz);
}

// The mixed-precision step's factors: A and B in FP32-pair arithmetic (each double read
// split into a pair, A and B rounded to doubles once) and from them the first-sweep
// residual R = A visn(u) + B - u in FP64.  The viscous sum visn reads 20 doubles for about
// 25 operations; in pairs as well the kernel measured 10.2 ms against 9.7 for an all-FP64
// kernel at 512x256x256 (the splits cost more than the FP64 operations they replace); in
// this form, 6.7 ms.  (The FP64-accurate step took A and B alone from here; k_src_ab is
// faster now: 1.9 ms against 3.6.)  The momentum-factor denominator is
// grouped as dz2 (e(-Z) + e(0)) + dy2 (e(-Y) + e(0)) + 2 dx2 (mu(0) + mu(X)) (and
// likewise per component), the same sum.
struct VPS {
  df::D dtinv, dx2, dy2, dz2, dx2x2, dy2x2, dz2x2, grvb, grvp;
};
struct FlatE {
  const float2* pairs;
  unsigned char* fluid;
  int* count;
  long long rb[2], mb[2];
};
// T = 1/(rho00/dt + a_p/2), a_p = ka (sum of two) + kb (..) + kc (..)
__device__ __forceinline__ df::D diag_e(const VPS& p, df::D r, df::D ka, df::D a, df::D kb, df::D b, df::D kc, df::D c) {
  using namespace df;
  const D ap = add(add(mul(ka, a), mul(kb, b)), mul(kc, c));
  return div(D{1.0f, 0.0f}, add(mul(r, p.dtinv), scale(ap, 0.5f)));
}
// FlatFluid's pairs: what the general branch below forms where every density and viscosity
// it reads is fluid f's
__global__ void k_flat_pairs(VPS p, Fluids fl, float2* __restrict__ out) {
  after_previous();
  using namespace df;
  const int f = (int)threadIdx.x;
  if (f > 1) return;
  const D R = split_double(f ? fl.rhog : fl.rhol), M = split_double(f ? fl.rmug : fl.rmul);
  const D R2 = add(R, R), M2 = add(M, M), r = scale(add(R2, R2), 0.25f);
  const D T[3] = {diag_e(p, r, p.dz2, M2, p.dy2, M2, p.dx2x2, M2), diag_e(p, r, p.dz2, M2, p.dy2x2, M2, p.dx2, M2),
                  diag_e(p, r, p.dz2x2, M2, p.dy2, M2, p.dx2, M2)};
  out[4 * f] = make_float2(r.h, r.l);
  for (int q = 0; q < 3; ++q) out[4 * f + 1 + q] = make_float2(T[q].h, T[q].l);
}
// FE.pairs: a warp whose points are each in one fluid takes rho00 and T from there.  Bound
// by the FP64 pipe (78 operations per cell, 80 % busy).  At 256x128x128 872 us with the 80
// registers it would take, 777 with 64 (four blocks per SM), 734 with the floats rounded by
// integer operations (df::d2f) and the pairs of the pure fluids, 651 with one copy of the
// sums after both branches and six blocks per SM (five 685, seven 718).
__global__ void __launch_bounds__(256, 6) k_src_ab_e(Grid g, VPS p, VP pv, Fac<double> pd, SrcIn in, FlatE FE,
                                                  const double* __restrict__ mu,
                                                  const double* __restrict__ exy, const double* __restrict__ exz,
                                                  const double* __restrict__ eyz, ABOut out) {
  after_previous();
  using namespace df;
  const Tile tile = warp_tile(g.ni);
  const int i = 1 + tile.x, j = 1 + tile.y, k = 1 + (int)blockIdx.z;
  const bool here = i <= g.ni && j <= g.nj;  // (the count below takes every thread)
  const long X = 1, Y = g.sy, Z = g.sz;
  const long c = here ? g.at(i, j, k) : g.at(1, 1, k);
  int f = 2;
  {
    auto V = [&](const double* a, long o) { return __ldg(a + c + o); };
    const double r0 = V(in.rho, 0), m0 = V(mu, 0);
    const long long rb = raw(r0), mb = raw(m0);
    const bool flat =
        same_bits(r0, V(in.rho, X), V(in.rho, Y), V(in.rho, Z), V(in.rhon, 0)) &&
        same_bits(r0, V(in.rhon, X), V(in.rhon, Y), V(in.rhon, Z), r0) &&
        same_bits(m0, V(mu, X), V(mu, Y), V(mu, Z), V(exy, 0)) &&
        same_bits(m0, V(exy, -X), V(exy, -Y), V(exz, 0), V(exz, -X)) &&
        same_bits(m0, V(exz, -Z), V(eyz, 0), V(eyz, -Y), V(eyz, -Z));
    if (flat && rb == FE.rb[1] && mb == FE.mb[1]) f = 1;
    if (flat && rb == FE.rb[0] && mb == FE.mb[0]) f = 0;
  }
  if (FE.fluid) {
    if (here) FE.fluid[c] = (unsigned char)f;
    const int flats = __syncthreads_count(here && f != 2);
    if (threadIdx.x == 0 && flats) atomicAdd(FE.count, flats);
  }
  if (!here) return;
  auto L = [&](const double* a, long o) { return split_double(__ldg(a + c + o)); };
  // rho00 * src; the pressure gradient as cal_grad_prs rounds it
  const double p0 = __ldg(in.phat + c);
  auto rsrc = [&](int q, const double* vel, D r, D grav, long S, double di) {
    const D prs = split_double(__dmul_rn(__dsub_rn(__ldg(in.phat + c + S), p0), di));
    D t = sub(mul(L(vel, 0), p.dtinv), mulf(L(in.adv[q], 0), 1.5f));
    t = add(t, scale(add(add(L(in.advo[q], 0), L(in.fst[q], 0)), L(in.fstn[q], 0)), 0.5f));
    t = add(t, grav);
    return add(sub(mul(r, t), prs), scale(L(in.vis[q], 0), 0.5f));
  };
  // A = T/2, B = rs T; A and R = A visn + B - u (FP64) as floats (T.h is the nearest float
  // of the pair T)
  auto store = [&](int q, D T, D rs, double vn, const double* vel) {
    const double A = to_double(scale(T, 0.5f)), B = to_double(mul(rs, T));
    out.af[q][c] = 0.5f * T.h;
    out.rf[q][c] = d2f(A * vn + B - __ldg(vel + c));
  };
  const D zero{0.0f, 0.0f};
  D ru, rv, rw, Tu, Tv, Tw;  // rho00 and T of the components
  if (__any_sync(__activemask(), f == 2)) {
    const D r0n0 = add(L(in.rho, 0), L(in.rhon, 0)), mu0 = L(mu, 0);
    ru = scale(add(r0n0, add(L(in.rho, X), L(in.rhon, X))), 0.25f);
    rv = scale(add(r0n0, add(L(in.rho, Y), L(in.rhon, Y))), 0.25f);
    rw = scale(add(r0n0, add(L(in.rho, Z), L(in.rhon, Z))), 0.25f);
    Tu = diag_e(p, ru, p.dz2, add(L(exz, -Z), L(exz, 0)), p.dy2, add(L(exy, -Y), L(exy, 0)), p.dx2x2, add(mu0, L(mu, X)));
    Tv = diag_e(p, rv, p.dz2, add(L(eyz, -Z), L(eyz, 0)), p.dy2x2, add(mu0, L(mu, Y)), p.dx2, add(L(exy, -X), L(exy, 0)));
    Tw = diag_e(p, rw, p.dz2x2, add(mu0, L(mu, Z)), p.dy2, add(L(eyz, -Y), L(eyz, 0)), p.dx2, add(L(exz, -X), L(exz, 0)));
  } else {
    auto P = [&](int q) {
      const float2 t = __ldg(FE.pairs + 4 * f + q);
      return D{t.x, t.y};
    };
    ru = rv = rw = P(0);
    Tu = P(1);
    Tv = P(2);
    Tw = P(3);
  }
  store(0, Tu, rsrc(0, in.u, ru, p.grvb, X, pv.dxi),
        visn_at<0, double>(g, pd, c, mu, exy, exz, eyz, in.u, in.v, in.w), in.u);
  if (j <= g.nj - 1)
    store(1, Tv, rsrc(1, in.v, rv, p.grvp, Y, pv.dyi),
          visn_at<1, double>(g, pd, c, mu, exy, exz, eyz, in.u, in.v, in.w), in.v);
  store(2, Tw, rsrc(2, in.w, rw, zero, Z, pv.dzi),
        visn_at<2, double>(g, pd, c, mu, exy, exz, eyz, in.u, in.v, in.w), in.w);
}

// The explicit viscous term 2 div(mu S) of main.f90:538-541 (calsij, cal_arith_tau,
// cal_div_tensor) for the interior u, v, w points, which are all the step reads.
// k_stress forms six stresses over i, j, k in 0..n+1 (the points the interior divergence
// reads) straight from u, v, w and mu, each without its constant factor:
//   t_xx = mu du (tau_xx = 2 mu du dxinv),
//   t_xy = (sum of 4 mu) (du_y + (dyinv/dxinv)^-1 dv_x) (tau_xy = t_xy dyinv / 4), ...
// and k_div_stress takes their divergence on the interior with the factors folded into
// its own: 26 + 18 FP64 operations per cell against 33 + 21; where the viscosities are
// equal bits, their sum is 4 mu exactly (see k_edges) and the first 18.  The strain never
// goes through memory.
// (sk, optional: the six strain components of calsij.f:28-139 at the same points,
// kept by the adjoint's record of the step)
struct StressK {
  double dxi, dyi, dzi;
  double rxy, rxz, ryz;        // dxinv/dyinv, dxinv/dzinv, dyinv/dzinv
  double xx, yy, zz;           // 2 dxinv^2 ...
  double qyy, qzz, qxy, qxz, qyz;  // dyinv^2/4, dzinv^2/4, dxinv dyinv/4, dxinv dzinv/4, dyinv dzinv/4
};
__global__ void __launch_bounds__(128) k_stress(Grid g, StressK K, const double* __restrict__ u,
                                                const double* __restrict__ v, const double* __restrict__ w,
                                                const double* __restrict__ mu, double* __restrict__ tau,
                                                double* __restrict__ sk) {
  after_previous();
  const int W = g.ni + 2;
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= W * (g.nj + 2)) return;
  const int j = t / W, i = t - j * W, k = (int)blockIdx.y;
  const long X = 1, Y = g.sy, Z = g.sz, n = g.n;
  const long c = g.at(i, j, k);
  const double m0 = __ldg(mu + c), mx = __ldg(mu + c + X), my = __ldg(mu + c + Y), mz = __ldg(mu + c + Z),
               mxy = __ldg(mu + c + X + Y), mxz = __ldg(mu + c + X + Z), myz = __ldg(mu + c + Y + Z);
  const double u0 = __ldg(u + c), v0 = __ldg(v + c), w0 = __ldg(w + c);
  const double dux = u0 - __ldg(u + c - X), dvy = v0 - __ldg(v + c - Y), dwz = w0 - __ldg(w + c - Z);
  const double duy = __ldg(u + c + Y) - u0, dvx = __ldg(v + c + X) - v0, duz = __ldg(u + c + Z) - u0,
               dwx = __ldg(w + c + X) - w0, dvz = __ldg(v + c + Z) - v0, dwy = __ldg(w + c + Y) - w0;
  const bool flat = same_bits(m0, mx, my, mz, mxy) && same_bits(m0, mxz, myz, m0, m0);
  double sxy, sxz, syz;
  if (__any_sync(__activemask(), !flat)) {
    const double mx0 = m0 + mx, my0 = m0 + my;
    sxy = mx0 + (my + mxy);
    sxz = mx0 + (mz + mxz);
    syz = my0 + (mz + myz);
  } else {
    sxy = sxz = syz = 4.0 * m0;
  }
  tau[c] = dux * m0;
  tau[c + n] = dvy * m0;
  tau[c + 2 * n] = dwz * m0;
  tau[c + 3 * n] = fma(dvx, K.rxy, duy) * sxy;
  tau[c + 4 * n] = fma(dwx, K.rxz, duz) * sxz;
  tau[c + 5 * n] = fma(dwy, K.ryz, dvz) * syz;
  if (sk) {
    sk[c] = dux * K.dxi;
    sk[c + n] = dvy * K.dyi;
    sk[c + 2 * n] = dwz * K.dzi;
    sk[c + 3 * n] = (duy * K.dyi + dvx * K.dxi) * 0.5;
    sk[c + 4 * n] = (duz * K.dzi + dwx * K.dxi) * 0.5;
    sk[c + 5 * n] = (dvz * K.dzi + dwy * K.dyi) * 0.5;
  }
}
__global__ void __launch_bounds__(256) k_div_stress(Grid g, StressK K, const double* __restrict__ t,
                                                    double* __restrict__ vu, double* __restrict__ vv,
                                                    double* __restrict__ vw) {
  after_previous();
  const int i = 1 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int j = 1 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  const int k = 1 + (int)blockIdx.z;
  if (i > g.ni || j > g.nj) return;
  const long X = 1, Y = g.sy, Z = g.sz, n = g.n;
  const long c = g.at(i, j, k);
  const double* t1 = t;
  const double* t2 = t + n;
  const double* t3 = t + 2 * n;
  const double* t4 = t + 3 * n;
  const double* t5 = t + 4 * n;
  const double* t6 = t + 5 * n;
  const double a4 = __ldg(t4 + c), a5 = __ldg(t5 + c), a6 = __ldg(t6 + c);
  vu[c] = (__ldg(t1 + c + X) - __ldg(t1 + c)) * K.xx + (a4 - __ldg(t4 + c - Y)) * K.qyy + (a5 - __ldg(t5 + c - Z)) * K.qzz;
  vv[c] = (a4 - __ldg(t4 + c - X)) * K.qxy + (__ldg(t2 + c + Y) - __ldg(t2 + c)) * K.yy + (a6 - __ldg(t6 + c - Z)) * K.qzz;
  vw[c] = (a5 - __ldg(t5 + c - X)) * K.qxz + (a6 - __ldg(t6 + c - Y)) * K.qyz + (__ldg(t3 + c + Z) - __ldg(t3 + c)) * K.zz;
}

// The FP64-accurate and mixed-precision steps: the stresses themselves and their
// divergence in FP32-pair arithmetic (each double read split into a pair, each output
// rounded to a double once).  Bound by the integer and FP32 pipes, the conversions
// (df::split_double, to_double) in front: at 256x128x128 207 + 129 us with every double
// read split where it is read, 129 + 67 as below.
// With sk (the adjoint's record of a mixed-precision step) the strain components
// are written as well, in FP64 as k_stress forms them.
struct VPT {
  df::D dxi2, dyi2, dzi2, hx, hy, hz, dxi, dyi, dzi;  // 2 dxi, ..., dxi/4, ..., dxi, ...
  double dxd, dyd, dzd;                               // dxi, dyi, dzi (the strain in FP64)
};
// uvw: the split pairs of u, v, w (those of the WENO5 stage), field f at uvw[f n ..]; tau is
// stored as the split pairs of the doubles the stresses round to, which is what
// k_div_stress_e reads: 15 + 12 fewer conversions per cell.
__global__ void __launch_bounds__(256) k_stress_e(Grid g, VPT p, const float2* __restrict__ uvw,
                                                  const double* __restrict__ u, const double* __restrict__ v,
                                                  const double* __restrict__ w, const double* __restrict__ mu,
                                                  float2* __restrict__ tau, double* __restrict__ sk) {
  after_previous();
  using namespace df;
  const Tile T = warp_tile(g.ni + 2);
  const int i = T.x, j = T.y, k = (int)blockIdx.z;
  if (i > g.ni + 1 || j > g.nj + 1) return;
  const long X = 1, Y = g.sy, Z = g.sz, n = g.n;
  const long c = g.at(i, j, k);
  const double d0 = __ldg(mu + c), dx = __ldg(mu + c + X), dy = __ldg(mu + c + Y), dz = __ldg(mu + c + Z),
               dxy = __ldg(mu + c + X + Y), dxz = __ldg(mu + c + X + Z), dyz = __ldg(mu + c + Y + Z);
  auto L = [&](int f, long o) {
    const float2 q = __ldg(uvw + f * n + c + o);
    return D{q.x, q.y};
  };
  auto put = [&](int q, D t) {
    const D r = split_double(to_double(t));
    tau[q * n + c] = make_float2(r.h, r.l);
  };
  const D m0 = split_double(d0), u0 = L(0, 0), v0 = L(1, 0), w0 = L(2, 0);
  D sxy, sxz, syz;  // the sums of four viscosities
  if (__any_sync(__activemask(), !(same_bits(d0, dx, dy, dz, dxy) && same_bits(d0, dxz, dyz, d0, d0)))) {
    const D mx = split_double(dx), my = split_double(dy), mz = split_double(dz);
    sxy = add(add(m0, mx), add(my, split_double(dxy)));
    sxz = add(add(m0, mx), add(mz, split_double(dxz)));
    syz = add(add(m0, my), add(mz, split_double(dyz)));
  } else {
    const D two = add(m0, m0);
    sxy = sxz = syz = add(two, two);
  }
  put(0, mul(mul(sub(u0, L(0, -X)), m0), p.dxi2));
  put(1, mul(mul(sub(v0, L(1, -Y)), m0), p.dyi2));
  put(2, mul(mul(sub(w0, L(2, -Z)), m0), p.dzi2));
  put(3, mul(add(mul(sub(L(0, Y), u0), p.hy), mul(sub(L(1, X), v0), p.hx)), sxy));
  put(4, mul(add(mul(sub(L(0, Z), u0), p.hz), mul(sub(L(2, X), w0), p.hx)), sxz));
  put(5, mul(add(mul(sub(L(1, Z), v0), p.hz), mul(sub(L(2, Y), w0), p.hy)), syz));
  if (sk) {
    const double dxi = p.dxd, dyi = p.dyd, dzi = p.dzd;
    const double ud = __ldg(u + c), vd = __ldg(v + c), wd = __ldg(w + c);
    sk[c] = (ud - __ldg(u + c - X)) * dxi;
    sk[c + n] = (vd - __ldg(v + c - Y)) * dyi;
    sk[c + 2 * n] = (wd - __ldg(w + c - Z)) * dzi;
    sk[c + 3 * n] = ((__ldg(u + c + Y) - ud) * dyi + (__ldg(v + c + X) - vd) * dxi) * 0.5;
    sk[c + 4 * n] = ((__ldg(u + c + Z) - ud) * dzi + (__ldg(w + c + X) - wd) * dxi) * 0.5;
    sk[c + 5 * n] = ((__ldg(v + c + Z) - vd) * dzi + (__ldg(w + c + Y) - wd) * dyi) * 0.5;
  }
}
__global__ void __launch_bounds__(256) k_div_stress_e(Grid g, VPT p, const float2* __restrict__ t,
                                                      double* __restrict__ vu, double* __restrict__ vv,
                                                      double* __restrict__ vw) {
  after_previous();
  using namespace df;
  const int i = 1 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int j = 1 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  const int k = 1 + (int)blockIdx.z;
  if (i > g.ni || j > g.nj) return;
  const long X = 1, Y = g.sy, Z = g.sz, n = g.n;
  const long c = g.at(i, j, k);
  auto L = [&](int q, long o) {
    const float2 r = __ldg(t + q * n + c + o);
    return D{r.x, r.y};
  };
  const D a4 = L(3, 0), a5 = L(4, 0), a6 = L(5, 0);
  vu[c] = to_double(add(add(mul(sub(L(0, X), L(0, 0)), p.dxi), mul(sub(a4, L(3, -Y)), p.dyi)),
                        mul(sub(a5, L(4, -Z)), p.dzi)));
  vv[c] = to_double(add(add(mul(sub(a4, L(3, -X)), p.dxi), mul(sub(L(1, Y), L(1, 0)), p.dyi)),
                        mul(sub(a6, L(5, -Z)), p.dzi)));
  vw[c] = to_double(add(add(mul(sub(a5, L(4, -X)), p.dxi), mul(sub(a6, L(5, -Y)), p.dyi)),
                        mul(sub(L(2, Z), L(2, 0)), p.dzi)));
}

// visn of component COMP at point c (solu_sor4.f:150-170 without the A/B factors)
template <int COMP, class T, class M>
__device__ __forceinline__ T visn_of(const Grid& g, const Fac<T>& p, long c, M coef, const T* un, const T* vn,
                                     const T* wn) {
  const long X = 1, Y = g.sy, Z = g.sz;
  const T dx2 = p.dx2, dy2 = p.dy2, dz2 = p.dz2, dxy = p.dxy, dxz = p.dxz, dyz = p.dyz;
  auto U = [&](long o) { return un[c + o]; };
  auto V = [&](long o) { return vn[c + o]; };
  auto W = [&](long o) { return wn[c + o]; };
  constexpr int mu = 0, exy = 1, exz = 2, eyz = 3;
  if (COMP == 0) {
    const T ym = coef(exy, -Y), yp = coef(exy, 0), zm = coef(exz, -Z), zp = coef(exz, 0);
    return dz2 * (zm * U(-Z) + zp * U(Z)) + dy2 * (ym * U(-Y) + yp * U(Y)) +
           (T)2 * dx2 * (coef(mu, 0) * U(-X) + coef(mu, X) * U(X)) + dxy * (ym * (V(-Y) - V(X - Y)) + yp * (V(X) - V(0))) +
           dxz * (zm * (W(-Z) - W(X - Z)) + zp * (W(X) - W(0)));
  } else if (COMP == 1) {
    const T xm = coef(exy, -X), xp = coef(exy, 0), zm = coef(eyz, -Z), zp = coef(eyz, 0);
    return dz2 * (zm * V(-Z) + zp * V(Z)) + (T)2 * dy2 * (coef(mu, 0) * V(-Y) + coef(mu, Y) * V(Y)) +
           dx2 * (xm * V(-X) + xp * V(X)) + dxy * (xm * (U(-X) - U(-X + Y)) + xp * (U(Y) - U(0))) +
           dyz * (zm * (W(-Z) - W(Y - Z)) + zp * (W(Y) - W(0)));
  } else {
    const T xm = coef(exz, -X), xp = coef(exz, 0), ym = coef(eyz, -Y), yp = coef(eyz, 0);
    return (T)2 * dz2 * (coef(mu, 0) * W(-Z) + coef(mu, Z) * W(Z)) + dy2 * (ym * W(-Y) + yp * W(Y)) +
           dx2 * (xm * W(-X) + xp * W(X)) + dxz * (xm * (U(-X) - U(-X + Z)) + xp * (U(Z) - U(0))) +
           dyz * (ym * (V(-Y) - V(-Y + Z)) + yp * (V(Z) - V(0)));
  }
}
template <int COMP, class T>
__device__ __forceinline__ T visn_at(const Grid& g, const Fac<T>& p, long c, const T* __restrict__ mu,
                                     const T* __restrict__ exy, const T* __restrict__ exz,
                                     const T* __restrict__ eyz, const T* un, const T* vn, const T* wn) {
  auto coef = [&](int a, long o) { return __ldg((a == 0 ? mu : (a == 1 ? exy : (a == 2 ? exz : eyz))) + c + o); };
  return visn_of<COMP, T>(g, p, c, coef, un, vn, wn);
}

// --- the colour-pair sweeps ----------------------------------------------------------
// visn of component COMP in the sweeps.  FP64: with S the component's own axis and, per
// transverse axis T with its edge viscosity e and field F,
//   e(-T) (q(-T) + r (F(-T) - F(S-T))) + e(0) (q(T) + r (F(S) - F(0))),  r = dSinv/dTinv,
// times dTinv^2: 17 operations, as visn_at's 19 in another grouping.  FP32: visn_at.
template <class T>
struct SweepK;
template <>
struct SweepK<double> {
  double own, t1, t2, r1, r2;  // 2 dSinv^2, dTinv^2 and r of the two transverse axes
  const unsigned char* fluid;  // FlatFluid's bytes and count; per fluid A mu times own, t1, t2
  const int* count;
  int enough;
  double fo[2], f1[2], f2[2];
  SweepK(const VP& p, int comp, const FlatFluid& flat = FlatFluid()) {
    const double d[3] = {p.dxi, p.dyi, p.dzi};
    const double s = d[comp], a = d[comp == 0 ? 1 : 0], b = d[comp == 2 ? 1 : 2];
    own = 2.0 * s * s;
    t1 = a * a;
    t2 = b * b;
    r1 = s / a;
    r2 = s / b;
    fluid = flat.fluid;
    count = flat.count;
    enough = flat.enough;
    for (int f = 0; f < 2; ++f) {
      fo[f] = flat.a[f][comp] * flat.mu[f] * own;
      f1[f] = flat.a[f][comp] * flat.mu[f] * t1;
      f2[f] = flat.a[f][comp] * flat.mu[f] * t2;
    }
  }
};
template <>
struct SweepK<float> {
  Fac<float> f;
  const unsigned char* fluid;
  const int* count;
  int enough;
  float mu[2];
  SweepK(const VP& p, int, const FlatFluid& flat = FlatFluid())
      : f(p), fluid(flat.fluid), count(flat.count), enough(flat.enough), mu{(float)flat.mu[0], (float)flat.mu[1]} {}
};
// A visn + B of a point in fluid f alone, in FP32: the same operations, the viscosities
// not read
template <int COMP>
__device__ __forceinline__ float flat_sweep(std::true_type, const Grid& g, const SweepK<float>& K, long c, bool f,
                                            const float* A, float B, const float* un, const float* vn,
                                            const float* wn) {
  const float m = f ? K.mu[1] : K.mu[0];
  const float visn = visn_of<COMP, float>(g, K.f, c, [&](int, long) { return m; }, un, vn, wn);
  return __ldg(A + c) * visn + B;
}
// A visn + B of a point in fluid f alone (A, mu and the edge viscosities constant): 16
// operations and 16 values read, not 20 and 23
template <int COMP>
__device__ __forceinline__ double flat_sweep(std::true_type, const Grid& g, const SweepK<double>& K, long c, bool f, const double*, double B,
                                             const double* un, const double* vn, const double* wn) {
  const long X = 1, Y = g.sy, Z = g.sz;
  const long S = COMP == 0 ? X : (COMP == 1 ? Y : Z), T1 = COMP == 0 ? Y : X, T2 = COMP == 2 ? Y : Z;
  const double *q = (COMP == 0 ? un : (COMP == 1 ? vn : wn)) + c, *p1 = (COMP == 0 ? vn : un) + c,
               *p2 = (COMP == 2 ? vn : wn) + c;
  const double a = fma(K.r1, (p1[S] - p1[0]) + (p1[-T1] - p1[S - T1]), q[T1] + q[-T1]);
  const double b = fma(K.r2, (p2[S] - p2[0]) + (p2[-T2] - p2[S - T2]), q[T2] + q[-T2]);
  return fma(f ? K.fo[1] : K.fo[0], q[S] + q[-S], fma(f ? K.f1[1] : K.f1[0], a, fma(f ? K.f2[1] : K.f2[0], b, B)));
}
template <int COMP>
__device__ __forceinline__ double visn_sweep(const Grid& g, const SweepK<double>& K, long c, const double* __restrict__ mu,
                                             const double* __restrict__ exy, const double* __restrict__ exz,
                                             const double* __restrict__ eyz, const double* un, const double* vn,
                                             const double* wn) {
  const long X = 1, Y = g.sy, Z = g.sz;
  const long S = COMP == 0 ? X : (COMP == 1 ? Y : Z), T1 = COMP == 0 ? Y : X, T2 = COMP == 2 ? Y : Z;
  const double *q = (COMP == 0 ? un : (COMP == 1 ? vn : wn)) + c, *f1 = (COMP == 0 ? vn : un) + c,
               *f2 = (COMP == 2 ? vn : wn) + c;
  const double *e1 = (COMP == 2 ? exz : exy) + c, *e2 = (COMP == 0 ? exz : eyz) + c;
  const double a = fma(__ldg(e1), fma(K.r1, f1[S] - f1[0], q[T1]),
                       __ldg(e1 - T1) * fma(K.r1, f1[-T1] - f1[S - T1], q[-T1]));
  const double b = fma(__ldg(e2), fma(K.r2, f2[S] - f2[0], q[T2]),
                       __ldg(e2 - T2) * fma(K.r2, f2[-T2] - f2[S - T2], q[-T2]));
  const double o = fma(__ldg(mu + c + S), q[S], __ldg(mu + c) * q[-S]);
  return fma(K.own, o, fma(K.t1, a, K.t2 * b));
}
template <int COMP>
__device__ __forceinline__ float visn_sweep(const Grid& g, const SweepK<float>& K, long c, const float* __restrict__ mu,
                                            const float* __restrict__ exy, const float* __restrict__ exz,
                                            const float* __restrict__ eyz, const float* un, const float* vn,
                                            const float* wn) {
  return visn_at<COMP, float>(g, K.f, c, mu, exy, exz, eyz, un, vn, wn);
}

// The ghost points that one updated point of the swept component fills (refresh below,
// seen from the source): its x and z images (the plain periodic copy)
// and, next to a wall, the wall rows of its column with their images.  ni, nj, nk >= 8.
struct Ghosts64 {
  double uwall;
  const double* wc;
};
template <int COMP>
__device__ __noinline__ void fill_ghosts(const Grid& g, const Ghosts64& G, double* q, int i, int j, int k, double v) {
  const int NI = g.ni, NJ = g.nj, NK = g.nk;
  const int ix = i <= 3 ? i + NI : (i >= NI - 2 ? i - NI : i), kx = k <= 3 ? k + NK : (k >= NK - 2 ? k - NK : k);
  auto put = [&](int jj, double x, bool base) {
    if (base) q[g.at(i, jj, k)] = x;
    if (ix != i) q[g.at(ix, jj, k)] = x;
    if (kx != k) {
      q[g.at(i, jj, kx)] = x;
      if (ix != i) q[g.at(ix, jj, kx)] = x;
    }
  };
  put(j, v, false);
  if (COMP == 1) {  // v(-m) = -v(m), m = 1, 2; v(nj+m) = -v(nj-m), m = 1..3
    if (j <= 2) put(-j, -v, true);
    if (j >= NJ - 3) put(2 * NJ - j, -v, true);
  } else if (j == 1 || j == NJ) {
    const int side = j == 1 ? 0 : 1, t = side ? 1 : -1;
    const double* wc = G.wc + (((long)side * (NK + 6) + (k + 2)) * (NI + 6) + (i + 2)) * 2;
    const double c2 = wc[1];
    const double x1 = COMP == 0 ? fma(c2, v, wc[0] * (side ? G.uwall : -G.uwall)) : c2 * v;
    const double x2 = 2.0 * x1 - v;
    put(j + t, x1, true);
    put(j + 2 * t, x2, true);
    put(j + 3 * t, 2.0 * x2 - x1, true);
  }
}
// the same on the mixed step's corrections, each with its constant
struct Ghosts32 {
  const float *gw, *gx, *gz;
};
constexpr int kGW = 12, kGH = 24;
__device__ __forceinline__ long wall_slot(const Grid& g, int side, int k, int i) {
  return (((long)side * (g.nk + 6) + (k + 2)) * (g.ni + 6) + (i + 2));
}
__device__ __forceinline__ int gslot(int d, int N, int sh) { return d <= 0 ? d + 2 : d - N + 2 - sh; }
template <int COMP>
__device__ __noinline__ void fill_ghosts(const Grid& g, const Ghosts32& G, float* q, int i, int j, int k, float v) {
  const int NI = g.ni, NJ = g.nj, NK = g.nk;
  constexpr int xb = COMP == 0 ? 0 : 6 * COMP + 6, zb = 6 * COMP;
  const int ix = i <= 3 ? i + NI : (i >= NI - 2 ? i - NI : i), kx = k <= 3 ? k + NK : (k >= NK - 2 ? k - NK : k);
  auto gz = [&](int ii, int jj) {
    return __ldg(G.gz + ((long)(jj + 2) * (NI + 6) + (ii + 2)) * kGH + zb + gslot(kx, NK, 0));
  };
  auto put = [&](int jj, float x, bool base) {
    if (base) q[g.at(i, jj, k)] = x;
    if (kx != k) q[g.at(i, jj, kx)] = x + gz(i, jj);
    if (ix != i) {
      const float y = x + __ldg(G.gx + ((long)(k + 2) * (NJ + 6) + (jj + 2)) * kGH + xb + gslot(ix, NI, 0));
      q[g.at(ix, jj, k)] = y;
      if (kx != k) q[g.at(ix, jj, kx)] = y + gz(ix, jj);
    }
  };
  put(j, v, false);
  if (COMP == 1) {
    const float* c0 = G.gw + wall_slot(g, 0, k, i) * kGW + 4;
    const float* c1 = G.gw + wall_slot(g, 1, k, i) * kGW + 4;
    if (j <= 2) put(-j, -v + __ldg(c0 + j), true);
    if (j >= NJ - 3 && j < NJ) put(2 * NJ - j, -v + __ldg(c1 + NJ - j), true);
  } else if (j == 1 || j == NJ) {
    const int side = j == 1 ? 0 : 1, t = side ? 1 : -1;
    const float* c = G.gw + wall_slot(g, side, k, i) * kGW;
    const float* h = c + (COMP == 0 ? 1 : 8);
    const float x1 = __ldg(c) * v + __ldg(h), x2 = 2.f * x1 - v + __ldg(h + 1), x3 = 2.f * x2 - x1 + __ldg(h + 2);
    put(j + t, x1, true);
    put(j + 2 * t, x2, true);
    put(j + 3 * t, x3, true);
  }
}

// One colour pair of one component, whose first colour has parities (pi, pj, pk); the
// second has all three flipped.  Thread (a, b) of a colour's (i, j) plane takes kz points
// of its column, of both colours (BOTH) or of the one blockIdx.z says.
// T = double: the FP64 step, q_new = A*visn(q) + B on the velocity itself.
// T = float: the mixed-precision step, d_new = A*visn(d) + R on the correction
// d = un - u (R is the FP64 first-sweep residual; see refine_prep).
// GHOSTS: the ghost points of the swept component are refreshed by the points they come
// from.  The other points of the pair do not read them: an image has its source's
// colour, and a wall row is read by its own column's point alone, before that writes it.
// part[block] = (first) or += the block's sum of (q_new - q)^2.
// The FP64 sweep is bound by the FP64 pipe (20 operations per point and 0.4 for its sum;
// visn_at's grouping and a shuffle tree per warp took 25): 431 -> 340 us per pair with its
// refresh at 512x256x256, 12.9 -> 7.6 at 32x32x16.
// FLAT (FlatFluid; from 2^21 cells): a warp both of whose colours' points are in one fluid
// takes flat_sweep, for one byte per point read a plane ahead; both colours take the same
// branch, so that their loads are in flight together (a branch each: 4 % slower where half
// the rows are flat).  An iteration of the drop: 4070 -> 3350 us at 512x256x256, 654 -> 590
// at 256x128x128.  With an interface normal to x (86 % of the cells flat, half of the warps)
// it would be 652 -> 664: hence nine tenths as the share that switches it on.  Warps of 8 x 4
// points here read more lines: 756.
template <int COMP, class T, class G, bool GHOSTS, bool BOTH, bool FLAT>
__global__ void __launch_bounds__(128) k_pair(Grid g, SweepK<T> K, int pi, int pj, int pk, int kz,
                                              const T* __restrict__ mu, const T* __restrict__ exy,
                                              const T* __restrict__ exz, const T* __restrict__ eyz,
                                              const T* __restrict__ A, const T* __restrict__ B, T* un, T* vn, T* wn,
                                              G gh, double* __restrict__ part, int first) {
  after_previous();
  __shared__ T sh[128];
  const int jmax = COMP == 1 ? g.nj - 1 : g.nj;
  T* q = COMP == 0 ? un : (COMP == 1 ? vn : wn);
  T e = 0;
  const int t = (int)(threadIdx.y * blockDim.x + threadIdx.x);
  const int a = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int rows = (g.nj / 2 + (int)blockDim.y - 1) / (int)blockDim.y;
  const int b = (int)(blockIdx.y % rows) * blockDim.y + threadIdx.y;
  const int k0 = (int)(blockIdx.y / rows) * kz, k1 = min(g.nk / 2, k0 + kz);
  double* o = part + ((long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  const double before = t == 0 && !first ? *o : 0.0;  // in flight while the points are
  // FLAT: the bytes of the next plane's points in flight while this plane's are swept
  int fluid[2] = {2, 2};
  bool use = false;
  if constexpr (FLAT) use = __ldg(K.count) >= K.enough;
  auto fluid_at = [&](int kk, bool h) {
    if constexpr (FLAT) {
      if (!use) return 2;
      const int i = (h ? 3 - pi : pi) + 2 * a, j = (h ? 3 - pj : pj) + 2 * b, k = (h ? 3 - pk : pk) + 2 * kk;
      return kk < k1 && i <= g.ni && j <= jmax ? (int)__ldg(K.fluid + g.at(i, j, k)) : 0;
    } else {
      return 2;
    }
  };
  if (FLAT) {
    fluid[0] = fluid_at(k0, BOTH ? false : blockIdx.z != 0);
    if (BOTH) fluid[1] = fluid_at(k0, true);
  }
#pragma unroll 1
  for (int kk = k0; kk < k1; ++kk) {
    bool mixed = !FLAT, second[2] = {false, false};
    if (FLAT) {
#pragma unroll
      for (int hh = 0; hh < (BOTH ? 2 : 1); ++hh) {
        mixed = mixed || fluid[hh] == 2;
        second[hh] = fluid[hh] == 1;
        fluid[hh] = fluid_at(kk + 1, BOTH ? hh != 0 : blockIdx.z != 0);
      }
      mixed = __any_sync(0xffffffffu, mixed);
    }
    auto colours = [&](auto flat) {
#pragma unroll
      for (int hh = 0; hh < (BOTH ? 2 : 1); ++hh) {
        const bool h = BOTH ? hh != 0 : blockIdx.z != 0;
        const int i = (h ? 3 - pi : pi) + 2 * a, j = (h ? 3 - pj : pj) + 2 * b, k = (h ? 3 - pk : pk) + 2 * kk;
        if (i > g.ni || j > jmax) continue;
        const long c = g.at(i, j, k);
        T qn;
        if constexpr (flat.value) {
          qn = flat_sweep<COMP>(flat, g, K, c, second[hh], A, __ldg(B + c), un, vn, wn);
        } else {
          const T visn = visn_sweep<COMP>(g, K, c, mu, exy, exz, eyz, un, vn, wn);
          qn = __ldg(A + c) * visn + __ldg(B + c);
        }
        const T d = qn - q[c];
        q[c] = qn;
        if (GHOSTS && (i <= 3 || i >= g.ni - 2 || j <= 3 || j >= g.nj - 3 || k <= 3 || k >= g.nk - 2))
          fill_ghosts<COMP>(g, gh, q, i, j, k, qn);
        e += d * d;
      }
    };
    if constexpr (FLAT) {
      if (mixed) colours(std::false_type());
      else colours(std::true_type());
    } else {
      colours(std::false_type());
    }
  }
  // the block's sum: one warp adds the others' values before the tree, which costs 8 FP64
  // operations per block and not 5 per warp
  const int nt = (int)(blockDim.x * blockDim.y);
  sh[t] = e;
  __syncthreads();
  if (t >= 32) return;
  for (int w = 32; w < nt; w += 32) e += sh[w + t];
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if (t == 0) *o = before + (double)e;
}

// --- wall/halo refresh: bndu(un,vn,wn) then bnd_periodic(swept component) ----------
// k_wall_coef: Navier-slip coefficients c1, c2 per wall point (bndu.f:39-45), constant
// during the solve (phi, l1, l2 do not change).  Layout wc[side][k+2][i+2][2].
__global__ void __launch_bounds__(256) k_wall_coef(Grid g, double dy, const double* __restrict__ l1,
                                                   const double* __restrict__ l2, const double* __restrict__ phi,
                                                   double* __restrict__ wc) {
  after_previous();
  const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int kk = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (i > g.ni + 3 || kk > 2 * (g.nk + 6) - 3) return;
  const int side = kk >= g.nk + 4 ? 1 : 0;
  const int k = side ? kk - (g.nk + 6) : kk;
  const int jw = side ? g.nj : 1;
  const double pa = (phi[g.at(i, jw, k)] + phi[g.at((i + 1) % (g.ni + 3), jw, k)]) / 2.0;
  const double i1 = pa / l1[g.at(i, jw, k)], i2 = (1.0 - pa) / l2[g.at(i, jw, k)];
  const double ls = 1.0 / (i1 + i2);
  const long o = (((long)side * (g.nk + 6) + (k + 2)) * (g.ni + 6) + (i + 2)) * 2;
  wc[o] = (2.0 * dy) / (2.0 * ls + dy);
  wc[o + 1] = (2.0 * ls - dy) / (2.0 * ls + dy);
}
// The three refresh kernels issue every load of a thread before its first store: in
// each of them the points written and the points read are disjoint (ghost rows are
// written from interior rows; halo copies read rows the same kernel never writes),
// so this is the sequential result with one memory round trip per thread.
__global__ void __launch_bounds__(256) k_wall(Grid g, double uwall, const double* __restrict__ wc,
                                              double* __restrict__ uk, double* __restrict__ vk,
                                              double* __restrict__ wk) {
  after_previous();
  const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int kk = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (i > g.ni + 3 || kk > 2 * (g.nk + 6) - 3) return;
  const int side = kk >= g.nk + 4 ? 1 : 0;
  const int k = side ? kk - (g.nk + 6) : kk;
  const int NJ = g.nj;
  const long o = (((long)side * (g.nk + 6) + (k + 2)) * (g.ni + 6) + (i + 2)) * 2;
  const double c1 = wc[o], c2 = wc[o + 1];
  const long Y = g.sy;
  if (!side) {
    const long c = g.at(i, 1, k);
    const double u1 = uk[c], v1 = vk[c], v2 = vk[c + Y], w1 = wk[c];
    const double u0 = fma(c2, u1, c1 * (-uwall));  // one contraction, the same in k_refresh
    const double um1 = 2.0 * u0 - u1;
    uk[c - Y] = u0;
    uk[c - 2 * Y] = um1;
    uk[c - 3 * Y] = 2.0 * um1 - u0;
    vk[c - 3 * Y] = -v2;
    vk[c - 2 * Y] = -v1;
    vk[c - Y] = 0.0;
    const double w0 = c2 * w1;
    const double wm1 = 2.0 * w0 - w1;
    wk[c - Y] = w0;
    wk[c - 2 * Y] = wm1;
    wk[c - 3 * Y] = 2.0 * wm1 - w0;
  } else {
    const long c = g.at(i, NJ, k);
    const double u1 = uk[c], w1 = wk[c];
    const double vm1 = vk[c - Y], vm2 = vk[c - 2 * Y], vm3 = vk[c - 3 * Y];
    const double u0 = fma(c2, u1, c1 * uwall);
    const double up2 = 2.0 * u0 - u1;
    uk[c + Y] = u0;
    uk[c + 2 * Y] = up2;
    uk[c + 3 * Y] = 2.0 * up2 - u0;
    vk[c] = 0.0;
    vk[c + Y] = -vm1;
    vk[c + 2 * Y] = -vm2;
    vk[c + 3 * Y] = -vm3;
    const double w0 = c2 * w1;
    const double wp2 = 2.0 * w0 - w1;
    wk[c + Y] = w0;
    wk[c + 2 * Y] = wp2;
    wk[c + 3 * Y] = 2.0 * wp2 - w0;
  }
}
// x halos of all three components.  Bit c of `normal` set: component c gets the
// plain periodic copy (bnd_periodic applied after bndu overwrites bndu's halos);
// clear: bndu's copy, which for u is shifted by one (bndu.f:107-109).
__global__ void __launch_bounds__(256) k_halo_x(Grid g, int normal, double* __restrict__ uk,
                                                double* __restrict__ vk, double* __restrict__ wk) {
  after_previous();
  const int j = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int k = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (j > g.nj + 3 || k > g.nk + 3) return;
  const int NI = g.ni;
  const long r = g.at(0, j, k);
  double* q[3] = {uk, vk, wk};
  const bool shifted = !(normal & 1);
  // sources of the destinations -2, -1, 0, ni+1, ni+2, ni+3 (offsets from r);
  // bndu's u: u(0)=u(ni+1), u(-1)=u(ni), u(-2)=u(ni-1), u(ni+1) untouched
  double t[3][6];
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    const double* a = q[cmp];
    const int sh = (cmp == 0 && shifted) ? 1 : 0;
    t[cmp][0] = a[r + NI - 2 + sh];
    t[cmp][1] = a[r + NI - 1 + sh];
    t[cmp][2] = a[r + NI + sh];
    t[cmp][3] = sh ? 0.0 : a[r + 1];
    t[cmp][4] = a[r + 2];
    t[cmp][5] = a[r + 3];
  }
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    double* a = q[cmp];
    a[r - 2] = t[cmp][0];
    a[r - 1] = t[cmp][1];
    a[r] = t[cmp][2];
    if (!(cmp == 0 && shifted)) a[r + NI + 1] = t[cmp][3];
    a[r + NI + 2] = t[cmp][4];
    a[r + NI + 3] = t[cmp][5];
  }
}
// z halos; for w bndu's copy is shifted by one (bndu.f:144-146).
__global__ void __launch_bounds__(256) k_halo_z(Grid g, int normal, double* __restrict__ uk,
                                                double* __restrict__ vk, double* __restrict__ wk) {
  after_previous();
  const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int j = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (i > g.ni + 3 || j > g.nj + 3) return;
  const int NK = g.nk;
  const long Z = g.sz;
  const long r = g.at(i, j, 0);
  double* q[3] = {uk, vk, wk};
  const bool shifted = !(normal & 4);
  // bndu's w: w(0)=w(nk+1), w(-1)=w(nk), w(-2)=w(nk-1), w(nk+1) untouched
  double t[3][6];
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    const double* a = q[cmp];
    const int sh = (cmp == 2 && shifted) ? 1 : 0;
    t[cmp][0] = a[r + (NK - 2 + sh) * Z];
    t[cmp][1] = a[r + (NK - 1 + sh) * Z];
    t[cmp][2] = a[r + (NK + sh) * Z];
    t[cmp][3] = sh ? 0.0 : a[r + Z];
    t[cmp][4] = a[r + 2 * Z];
    t[cmp][5] = a[r + 3 * Z];
  }
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    double* a = q[cmp];
    a[r - 2 * Z] = t[cmp][0];
    a[r - Z] = t[cmp][1];
    a[r] = t[cmp][2];
    if (!(cmp == 2 && shifted)) a[r + (NK + 1) * Z] = t[cmp][3];
    a[r + (NK + 2) * Z] = t[cmp][4];
    a[r + (NK + 3) * Z] = t[cmp][5];
  }
}
// k_halo_x for ni >= 8 with 8 lanes per (j, k, component): lanes 0-2 write the low
// ghosts -2..0, lanes 3-5 the high ghosts ni+1..ni+3, each from its interior source
// (none of which the kernel writes).  A warp then reads and writes a few contiguous
// runs instead of 32 rows, and the work spreads over every SM.
__global__ void __launch_bounds__(256) k_halo_x8(Grid g, int normal, double* __restrict__ uk,
                                                 double* __restrict__ vk, double* __restrict__ wk) {
  after_previous();
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int m = (int)(t & 7);
  const long task = t >> 3;
  const long JK = (long)(g.nj + 6) * (g.nk + 6);
  if (m >= 6 || task >= 3 * JK) return;
  const int cmp = (int)(task / JK);
  const int rem = (int)(task % JK);
  double* a = cmp == 0 ? uk : (cmp == 1 ? vk : wk);
  const bool sh = cmp == 0 && !(normal & 1);  // bndu's u: u(-2..0) = u(ni-1..ni+1), u(ni+1) kept
  const long r = g.at(0, -2 + rem % (g.nj + 6), -2 + rem / (g.nj + 6));
  if (m < 3) {
    a[r + m - 2] = a[r + g.ni - 2 + m + (sh ? 1 : 0)];
  } else if (!(sh && m == 3)) {
    a[r + g.ni + m - 2] = a[r + m - 2];
  }
}
// k_wall, k_halo_x and k_halo_z in one pass (ni, nj, nk >= 8).  Composed, the three
// give every refreshed point as a function of points none of them writes: a ghost
// column (x or z destination) holds its source column's values, its wall rows
// included, and the wall rows of a column are the extrapolation of its source
// column's interior rows with that column's coefficients.  So the threads write
// their points in any order.  Blocks [0, nbW): the wall rows of every column, one
// thread per (column, wall); [nbW, nbW + nbX): the other rows of the x-ghost
// columns, one thread per (j, k, component) for its six ghost slots; the rest: the
// other rows of the z-ghost planes over the columns that are not x destinations,
// one thread per (i, j, component).  A thread reads all its sources before writing.
// (refresh: thread t of one of the three regions)
__device__ __forceinline__ void refresh(const Grid& g, int normal, const Ghosts64& G, double* uk, double* vk, double* wk,
                                        int region, long t) {
  const double uwall = G.uwall;
  const double* __restrict__ wc = G.wc;
  const int shu = !(normal & 1), shw = !(normal & 4);  // bndu's shifted copies: u along x, w along z
  const int NI = g.ni, NJ = g.nj, NK = g.nk;
  const long Y = g.sy;
  if (region == 0) {
    const int W = NI + 6;
    if (t >= 2L * W * (NK + 6)) return;
    const int i = (int)(t % W) - 2;
    const int kk = (int)(t / W);
    const int side = kk >= NK + 6 ? 1 : 0;
    const int k = kk - side * (NK + 6) - 2;
    const int jw = side ? NJ : 1;
    auto wco = [&](int ci, int ck) { return (((long)side * (NK + 6) + (ck + 2)) * W + (ci + 2)) * 2; };
    // u from its source column
    const int iu = halo_src(i, NI, shu), ku = halo_src(k, NK, 0);
    const long ou = wco(iu, ku);
    const double u1 = uk[g.at(iu, jw, ku)];
    // v, w
    const int iv = halo_src(i, NI, 0), kv = halo_src(k, NK, 0);
    const int iw = halo_src(i, NI, 0), kw = halo_src(k, NK, shw);
    const double w1 = wk[g.at(iw, jw, kw)];
    const double c2w = wc[wco(iw, kw) + 1];
    const long cv = g.at(iv, jw, kv);
    double va, vb, vc = 0.0;
    if (!side) {
      va = vk[cv];
      vb = vk[cv + Y];
    } else {
      va = vk[cv - Y];
      vb = vk[cv - 2 * Y];
      vc = vk[cv - 3 * Y];
    }
    const double c1 = wc[ou], c2 = wc[ou + 1];
    const long c = g.at(i, jw, k);
    const long t1 = side ? Y : -Y;
    const double u0 = fma(c2, u1, c1 * (side ? uwall : -uwall));  // as k_wall
    const double um = 2.0 * u0 - u1;
    uk[c + t1] = u0;
    uk[c + 2 * t1] = um;
    uk[c + 3 * t1] = 2.0 * um - u0;
    const double w0 = c2w * w1;
    const double wm = 2.0 * w0 - w1;
    wk[c + t1] = w0;
    wk[c + 2 * t1] = wm;
    wk[c + 3 * t1] = 2.0 * wm - w0;
    if (!side) {  // v(0) = 0, v(-1) = -v(1), v(-2) = -v(2)
      vk[c - 3 * Y] = -vb;
      vk[c - 2 * Y] = -va;
      vk[c - Y] = 0.0;
    } else {  // v(nj) = 0, v(nj+m) = -v(nj-m)
      vk[c] = 0.0;
      vk[c + Y] = -va;
      vk[c + 2 * Y] = -vb;
      vk[c + 3 * Y] = -vc;
    }
    return;
  }
  if (region == 1) {
    const long task = t;
    if (task >= 3L * NJ * (NK + 6)) return;
    const int cmp = (int)(task / ((long)NJ * (NK + 6)));
    const int rem = (int)(task % ((long)NJ * (NK + 6)));
    const int j = 1 + rem % NJ, k = -2 + rem / NJ;
    if (cmp == 1 && j == NJ) return;  // a wall row of v
    const int sx = cmp == 0 ? shu : 0, sz = cmp == 2 ? shw : 0;
    const int ks = halo_src(k, NK, sz);
    double* a = cmp == 0 ? uk : (cmp == 1 ? vk : wk);
    double v[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const int d = halo_dest(m, NI, sx);
      v[m] = d == kNoHalo ? 0.0 : a[g.at(halo_src(d, NI, sx), j, ks)];
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const int d = halo_dest(m, NI, sx);
      if (d != kNoHalo) a[g.at(d, j, k)] = v[m];
    }
    return;
  }
  const int i = 1 + (int)(t % (NI + 1));
  const long r = t / (NI + 1);
  const int j = 1 + (int)(r % NJ);
  const int cmp = (int)(r / NJ);
  if (cmp >= 3 || (cmp == 1 && j == NJ)) return;
  const int sx = cmp == 0 ? shu : 0, sz = cmp == 2 ? shw : 0;
  if (halo_src(i, NI, sx) != i) return;  // an x-ghost column: done above
  double* a = cmp == 0 ? uk : (cmp == 1 ? vk : wk);
  double v[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const int d = halo_dest(m, NK, sz);
    v[m] = d == kNoHalo ? 0.0 : a[g.at(i, j, halo_src(d, NK, sz))];
  }
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const int d = halo_dest(m, NK, sz);
    if (d != kNoHalo) a[g.at(i, j, d)] = v[m];
  }
}
// --- mixed precision: FP32 sweeps on the correction d = un - u ---------------------
// During the solve un = u + d holds at every point, halos and wall ghosts included:
// d starts at zero (un = u, main.f90:605-607) and every operation on un has an
// exact counterpart on d.  A sweep q_new = A*visn(q) + B becomes d_new = A*visn(d) + R
// with R = A*visn(u) + B - u; each wall/halo operation dst = f(src) is affine with
// fixed coefficients, so it becomes d_dst = f_lin(d_src) + gamma_dst with
// gamma_dst = f(u_src) - u_dst, formed once per step in FP64 from u.
//
// Wall constants per (side, k, i), 12 floats: c2, gamma_u[3], gamma_v[4], gamma_w[3], pad.
// x-halo constants per (j, k) and z-halo constants per (i, j), 24 floats: the six
// destinations of the plain copy of u, v, w and the five of bndu's shifted copy
// (u in x: slots 6..10, v 12..17, w 18..23; z: u 0..5, v 6..11, w 12..17, shifted w 18..22).

__global__ void __launch_bounds__(256) k_gamma_wall(Grid g, double uwall, const double* __restrict__ wc,
                                                    const double* __restrict__ u, const double* __restrict__ v,
                                                    const double* __restrict__ w, float* __restrict__ gw) {
  after_previous();
  const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int kk = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (i > g.ni + 3 || kk > 2 * (g.nk + 6) - 3) return;
  const int side = kk >= g.nk + 4 ? 1 : 0;
  const int k = side ? kk - (g.nk + 6) : kk;
  const long o = wall_slot(g, side, k, i);
  const double c1 = wc[2 * o], c2 = wc[2 * o + 1];
  const long Y = g.sy;
  const long c = g.at(i, side ? g.nj : 1, k);
  const long t = side ? Y : -Y;  // towards the ghost rows
  float* G = gw + o * kGW;
  // u, w: q(g1) = K + c2 q(c), q(g2) = 2 q(g1) - q(c), q(g3) = 2 q(g2) - q(g1)
  auto lin = [&](const double* q, double K, float* out) {
    const double q1 = q[c], g1 = q[c + t], g2 = q[c + 2 * t], g3 = q[c + 3 * t];
    out[0] = (float)(K + c2 * q1 - g1);
    out[1] = (float)(2.0 * g1 - q1 - g2);
    out[2] = (float)(2.0 * g2 - g1 - g3);
  };
  G[0] = (float)c2;
  lin(u, side ? c1 * uwall : c1 * (-uwall), G + 1);
  lin(w, 0.0, G + 8);
  if (!side) {  // v(0) = 0, v(-1) = -v(1), v(-2) = -v(2)
    G[4] = (float)(-v[c - Y]);
    G[5] = (float)(-v[c] - v[c - 2 * Y]);
    G[6] = (float)(-v[c + Y] - v[c - 3 * Y]);
    G[7] = 0.f;
  } else {  // v(nj) = 0, v(nj+m) = -v(nj-m), m = 1..3
    G[4] = (float)(-v[c]);
    G[5] = (float)(-v[c - Y] - v[c + Y]);
    G[6] = (float)(-v[c - 2 * Y] - v[c + 2 * Y]);
    G[7] = (float)(-v[c - 3 * Y] - v[c + 3 * Y]);
  }
  G[11] = 0.f;
}
__global__ void __launch_bounds__(256) k_gamma_x(Grid g, const double* __restrict__ u, const double* __restrict__ v,
                                                 const double* __restrict__ w, float* __restrict__ gx) {
  after_previous();
  const int j = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int k = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (j > g.nj + 3 || k > g.nk + 3) return;
  const int NI = g.ni;
  const long r = g.at(0, j, k);
  float* G = gx + ((long)(k + 2) * (g.nj + 6) + (j + 2)) * kGH;
  const int dst[6] = {-2, -1, 0, NI + 1, NI + 2, NI + 3};
  const int src[6] = {NI - 2, NI - 1, NI, 1, 2, 3};
  const double* q[3] = {u, v, w};
  const int base[3] = {0, 12, 18};
  for (int cmp = 0; cmp < 3; ++cmp)
    for (int t = 0; t < 6; ++t) G[base[cmp] + t] = (float)(q[cmp][r + src[t]] - q[cmp][r + dst[t]]);
  // bndu's u: destinations -2, -1, 0, ni+2, ni+3 from ni-1, ni, ni+1, 2, 3
  const int sd[5] = {-2, -1, 0, NI + 2, NI + 3};
  const int ss[5] = {NI - 1, NI, NI + 1, 2, 3};
  for (int t = 0; t < 5; ++t) G[6 + t] = (float)(u[r + ss[t]] - u[r + sd[t]]);
  G[11] = 0.f;
}
__global__ void __launch_bounds__(256) k_gamma_z(Grid g, const double* __restrict__ u, const double* __restrict__ v,
                                                 const double* __restrict__ w, float* __restrict__ gz) {
  after_previous();
  const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int j = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (i > g.ni + 3 || j > g.nj + 3) return;
  const int NK = g.nk;
  const long Z = g.sz;
  const long r = g.at(i, j, 0);
  float* G = gz + ((long)(j + 2) * (g.ni + 6) + (i + 2)) * kGH;
  const int dst[6] = {-2, -1, 0, NK + 1, NK + 2, NK + 3};
  const int src[6] = {NK - 2, NK - 1, NK, 1, 2, 3};
  const double* q[3] = {u, v, w};
  for (int cmp = 0; cmp < 3; ++cmp)
    for (int t = 0; t < 6; ++t) G[6 * cmp + t] = (float)(q[cmp][r + src[t] * Z] - q[cmp][r + dst[t] * Z]);
  const int sd[5] = {-2, -1, 0, NK + 2, NK + 3};
  const int ss[5] = {NK - 1, NK, NK + 1, 2, 3};
  for (int t = 0; t < 5; ++t) G[18 + t] = (float)(w[r + ss[t] * Z] - w[r + sd[t] * Z]);
  G[23] = 0.f;
}

// k_wall on the corrections
__global__ void __launch_bounds__(256) k_wall_d(Grid g, const float* __restrict__ gw, float* __restrict__ du,
                                                float* __restrict__ dv, float* __restrict__ dw) {
  after_previous();
  const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int kk = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (i > g.ni + 3 || kk > 2 * (g.nk + 6) - 3) return;
  const int side = kk >= g.nk + 4 ? 1 : 0;
  const int k = side ? kk - (g.nk + 6) : kk;
  const float4* G4 = reinterpret_cast<const float4*>(gw + wall_slot(g, side, k, i) * kGW);
  const float4 a = __ldg(G4), b = __ldg(G4 + 1), e = __ldg(G4 + 2);
  const float c2 = a.x;
  const long Y = g.sy;
  const long c = g.at(i, side ? g.nj : 1, k);
  const long t = side ? Y : -Y;
  const float u1 = du[c], w1 = dw[c];
  float v1, v2, v3;
  if (!side) {
    v1 = dv[c];
    v2 = dv[c + Y];
    v3 = 0.f;
  } else {
    v1 = dv[c - Y];
    v2 = dv[c - 2 * Y];
    v3 = dv[c - 3 * Y];
  }
  const float ug1 = c2 * u1 + a.y, ug2 = 2.f * ug1 - u1 + a.z, ug3 = 2.f * ug2 - ug1 + a.w;
  du[c + t] = ug1;
  du[c + 2 * t] = ug2;
  du[c + 3 * t] = ug3;
  const float wg1 = c2 * w1 + e.x, wg2 = 2.f * wg1 - w1 + e.y, wg3 = 2.f * wg2 - wg1 + e.z;
  dw[c + t] = wg1;
  dw[c + 2 * t] = wg2;
  dw[c + 3 * t] = wg3;
  if (!side) {
    dv[c - Y] = b.x;
    dv[c - 2 * Y] = -v1 + b.y;
    dv[c - 3 * Y] = -v2 + b.z;
  } else {
    dv[c] = b.x;
    dv[c + Y] = -v1 + b.y;
    dv[c + 2 * Y] = -v2 + b.z;
    dv[c + 3 * Y] = -v3 + b.w;
  }
}
// k_halo_x on the corrections
__global__ void __launch_bounds__(256) k_halo_x_d(Grid g, int normal, const float* __restrict__ gx,
                                                  float* __restrict__ du, float* __restrict__ dv,
                                                  float* __restrict__ dw) {
  after_previous();
  const int j = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int k = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (j > g.nj + 3 || k > g.nk + 3) return;
  const int NI = g.ni;
  const long r = g.at(0, j, k);
  const float* G = gx + ((long)(k + 2) * (g.nj + 6) + (j + 2)) * kGH;
  float* q[3] = {du, dv, dw};
  const bool shifted = !(normal & 1);
  float t[3][6];
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    const float* a = q[cmp];
    const int sh = (cmp == 0 && shifted) ? 1 : 0;
    t[cmp][0] = a[r + NI - 2 + sh];
    t[cmp][1] = a[r + NI - 1 + sh];
    t[cmp][2] = a[r + NI + sh];
    t[cmp][3] = sh ? 0.f : a[r + 1];
    t[cmp][4] = a[r + 2];
    t[cmp][5] = a[r + 3];
  }
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    float* a = q[cmp];
    if (cmp == 0 && shifted) {
      const float* s = G + 6;
      a[r - 2] = t[0][0] + __ldg(s);
      a[r - 1] = t[0][1] + __ldg(s + 1);
      a[r] = t[0][2] + __ldg(s + 2);
      a[r + NI + 2] = t[0][4] + __ldg(s + 3);
      a[r + NI + 3] = t[0][5] + __ldg(s + 4);
    } else {
      const float* s = G + (cmp == 0 ? 0 : (cmp == 1 ? 12 : 18));
      a[r - 2] = t[cmp][0] + __ldg(s);
      a[r - 1] = t[cmp][1] + __ldg(s + 1);
      a[r] = t[cmp][2] + __ldg(s + 2);
      a[r + NI + 1] = t[cmp][3] + __ldg(s + 3);
      a[r + NI + 2] = t[cmp][4] + __ldg(s + 4);
      a[r + NI + 3] = t[cmp][5] + __ldg(s + 5);
    }
  }
}
// k_halo_z on the corrections
__global__ void __launch_bounds__(256) k_halo_z_d(Grid g, int normal, const float* __restrict__ gz,
                                                  float* __restrict__ du, float* __restrict__ dv,
                                                  float* __restrict__ dw) {
  after_previous();
  const int i = -2 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int j = -2 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (i > g.ni + 3 || j > g.nj + 3) return;
  const int NK = g.nk;
  const long Z = g.sz;
  const long r = g.at(i, j, 0);
  const float* G = gz + ((long)(j + 2) * (g.ni + 6) + (i + 2)) * kGH;
  float* q[3] = {du, dv, dw};
  const bool shifted = !(normal & 4);
  float t[3][6];
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    const float* a = q[cmp];
    const int sh = (cmp == 2 && shifted) ? 1 : 0;
    t[cmp][0] = a[r + (NK - 2 + sh) * Z];
    t[cmp][1] = a[r + (NK - 1 + sh) * Z];
    t[cmp][2] = a[r + (NK + sh) * Z];
    t[cmp][3] = sh ? 0.f : a[r + Z];
    t[cmp][4] = a[r + 2 * Z];
    t[cmp][5] = a[r + 3 * Z];
  }
#pragma unroll
  for (int cmp = 0; cmp < 3; ++cmp) {
    float* a = q[cmp];
    if (cmp == 2 && shifted) {
      const float* s = G + 18;
      a[r - 2 * Z] = t[2][0] + __ldg(s);
      a[r - Z] = t[2][1] + __ldg(s + 1);
      a[r] = t[2][2] + __ldg(s + 2);
      a[r + (NK + 2) * Z] = t[2][4] + __ldg(s + 3);
      a[r + (NK + 3) * Z] = t[2][5] + __ldg(s + 4);
    } else {
      const float* s = G + 6 * cmp;
      a[r - 2 * Z] = t[cmp][0] + __ldg(s);
      a[r - Z] = t[cmp][1] + __ldg(s + 1);
      a[r] = t[cmp][2] + __ldg(s + 2);
      a[r + (NK + 1) * Z] = t[cmp][3] + __ldg(s + 3);
      a[r + (NK + 2) * Z] = t[cmp][4] + __ldg(s + 4);
      a[r + (NK + 3) * Z] = t[cmp][5] + __ldg(s + 5);
    }
  }
}
// k_wall_d, k_halo_x_d and k_halo_z_d in one pass (ni, nj, nk >= 8), composed as
// k_refresh composes their FP64 counterparts, with the per-point constants added
// in the same order (wall extrapolation of the source column, then + the x
// constant of the source plane's row, then + the z constant of the final column's
// row), so the result is bit for bit that of the three kernels.  Blocks [0, nbW):
// the wall rows of every column, one thread per (column, wall); [nbW, nbW + nbX):
// the other rows of the x-ghost columns, one thread per (j, k, component);
// the rest: the other rows of the z-ghost planes of the columns that are not x
// destinations, one thread per (i, j, component).
__device__ __forceinline__ void refresh(const Grid& g, int normal, const Ghosts32& G, float* du, float* dv, float* dw,
                                        int region, long t, int only = -1) {
  const float *__restrict__ gw = G.gw, *__restrict__ gx = G.gx, *__restrict__ gz = G.gz;
  const int shu = !(normal & 1), shw = !(normal & 4);
  const int NI = g.ni, NJ = g.nj, NK = g.nk;
  // constant slots: x (per (k, j)): u 0, shifted u 6, v 12, w 18; z (per (j, i)): u 0,
  // v 6, w 12, shifted w 18
  auto xb = [&](int cmp) { return cmp == 0 ? (shu ? 6 : 0) : 6 * cmp + 6; };
  auto zb = [&](int cmp) { return cmp == 2 ? (shw ? 18 : 12) : 6 * cmp; };
  auto GX = [&](int j, int k, int slot) { return __ldg(gx + ((long)(k + 2) * (NJ + 6) + (j + 2)) * kGH + slot); };
  auto GZ = [&](int i, int j, int slot) { return __ldg(gz + ((long)(j + 2) * (NI + 6) + (i + 2)) * kGH + slot); };
  if (region == 0) {
    const int W = NI + 6;
    if (t >= 2L * W * (NK + 6)) return;
    const int i = (int)(t % W) - 2;
    const int kk = (int)(t / W);
    const int side = kk >= NK + 6 ? 1 : 0;
    const int k = kk - side * (NK + 6) - 2;
    const int jw = side ? NJ : 1, tj = side ? 1 : -1;
    // value of ghost row j of this column from the source column's value v
    auto compose = [&](float v, int cmp, int is, int ks, int j) {
      if (is != i) v = v + GX(j, ks, xb(cmp) + gslot(i, NI, cmp == 0 ? shu : 0));
      if (ks != k) v = v + GZ(i, j, zb(cmp) + gslot(k, NK, cmp == 2 ? shw : 0));
      return v;
    };
    // u and w: q(g1) = c2 q1 + G1, q(g2) = 2 q(g1) - q1 + G2, q(g3) = 2 q(g2) - q(g1) + G3
#pragma unroll
    for (int cmp = 0; cmp < 3; cmp += 2) {
      if (only >= 0 && cmp != only) continue;
      const int is = halo_src(i, NI, cmp == 0 ? shu : 0), ks = halo_src(k, NK, cmp == 2 ? shw : 0);
      const float4* G4 = reinterpret_cast<const float4*>(gw + wall_slot(g, side, ks, is) * kGW);
      const float4 a = __ldg(G4), e = __ldg(G4 + 2);
      float* q = cmp == 0 ? du : dw;
      const float q1 = q[g.at(is, jw, ks)];
      const float c2 = a.x;
      const float h1 = cmp == 0 ? a.y : e.x, h2 = cmp == 0 ? a.z : e.y, h3 = cmp == 0 ? a.w : e.z;
      const float g1 = c2 * q1 + h1, g2 = 2.f * g1 - q1 + h2, g3 = 2.f * g2 - g1 + h3;
      q[g.at(i, jw + tj, k)] = compose(g1, cmp, is, ks, jw + tj);
      q[g.at(i, jw + 2 * tj, k)] = compose(g2, cmp, is, ks, jw + 2 * tj);
      q[g.at(i, jw + 3 * tj, k)] = compose(g3, cmp, is, ks, jw + 3 * tj);
    }
    if (only < 0 || only == 1) {
      const int is = halo_src(i, NI, 0), ks = halo_src(k, NK, 0);
      const float4 bb = __ldg(reinterpret_cast<const float4*>(gw + wall_slot(g, side, ks, is) * kGW) + 1);
      const long c = g.at(is, jw, ks);
      const long Y = g.sy;
      if (!side) {  // v(0), v(-1), v(-2)
        const float v1 = dv[c], v2 = dv[c + Y];
        dv[g.at(i, 0, k)] = compose(bb.x, 1, is, ks, 0);
        dv[g.at(i, -1, k)] = compose(-v1 + bb.y, 1, is, ks, -1);
        dv[g.at(i, -2, k)] = compose(-v2 + bb.z, 1, is, ks, -2);
      } else {  // v(nj), v(nj+1..nj+3)
        const float v1 = dv[c - Y], v2 = dv[c - 2 * Y], v3 = dv[c - 3 * Y];
        dv[g.at(i, NJ, k)] = compose(bb.x, 1, is, ks, NJ);
        dv[g.at(i, NJ + 1, k)] = compose(-v1 + bb.y, 1, is, ks, NJ + 1);
        dv[g.at(i, NJ + 2, k)] = compose(-v2 + bb.z, 1, is, ks, NJ + 2);
        dv[g.at(i, NJ + 3, k)] = compose(-v3 + bb.w, 1, is, ks, NJ + 3);
      }
    }
    return;
  }
  if (region == 1) {
    const long task = t;
    if (task >= (only >= 0 ? 1L : 3L) * NJ * (NK + 6)) return;
    const int cmp = only >= 0 ? only : (int)(task / ((long)NJ * (NK + 6)));
    const int rem = (int)(task % ((long)NJ * (NK + 6)));
    const int j = 1 + rem % NJ, k = -2 + rem / NJ;
    if (cmp == 1 && j == NJ) return;  // a wall row of v
    const int sx = cmp == 0 ? shu : 0, sz = cmp == 2 ? shw : 0;
    const int ks = halo_src(k, NK, sz);
    float* a = cmp == 0 ? du : (cmp == 1 ? dv : dw);
    float v[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const int d = halo_dest(m, NI, sx);
      if (d == kNoHalo) {
        v[m] = 0.f;
        continue;
      }
      v[m] = a[g.at(halo_src(d, NI, sx), j, ks)] + GX(j, ks, xb(cmp) + gslot(d, NI, sx));
      if (ks != k) v[m] = v[m] + GZ(d, j, zb(cmp) + gslot(k, NK, sz));
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const int d = halo_dest(m, NI, sx);
      if (d != kNoHalo) a[g.at(d, j, k)] = v[m];
    }
    return;
  }
  const int i = 1 + (int)(t % (NI + 1));
  const long r = t / (NI + 1);
  const int j = 1 + (int)(r % NJ);
  const int cmp = only >= 0 ? only : (int)(r / NJ);
  if (only >= 0 && r >= NJ) return;
  if (cmp >= 3 || (cmp == 1 && j == NJ)) return;
  const int sx = cmp == 0 ? shu : 0, sz = cmp == 2 ? shw : 0;
  if (halo_src(i, NI, sx) != i) return;  // an x-ghost column: done above
  float* a = cmp == 0 ? du : (cmp == 1 ? dv : dw);
  float v[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const int d = halo_dest(m, NK, sz);
    v[m] = d == kNoHalo ? 0.f : a[g.at(i, j, halo_src(d, NK, sz))] + GZ(i, j, zb(cmp) + gslot(d, NK, sz));
  }
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const int d = halo_dest(m, NK, sz);
    if (d != kNoHalo) a[g.at(i, j, d)] = v[m];
  }
}
// threads of the three regions: the wall rows, the x-ghost columns, the z-ghost planes
__host__ __device__ __forceinline__ long refresh_tasks(const Grid& g, int region) {
  return region == 0 ? 2L * (g.ni + 6) * (g.nk + 6) : (region == 1 ? 3L * g.nj * (g.nk + 6) : 3L * (g.ni + 1) * g.nj);
}
// (the FP32 corrections' refresh of one component only)
__global__ void __launch_bounds__(256) k_refresh_one(Grid g, int comp, Ghosts32 gh, float* du, float* dv, float* dw,
                                                     int nbW, int nbX) {
  after_previous();
  const int b = (int)blockIdx.x, region = b < nbW ? 0 : (b < nbW + nbX ? 1 : 2);
  refresh(g, 1 << comp, gh, du, dv, dw, region,
          (long)(b - (region > 0 ? nbW : 0) - (region > 1 ? nbX : 0)) * 256 + threadIdx.x, comp);
}
template <class T, class G>
__global__ void __launch_bounds__(256) k_refresh(Grid g, int normal, G gh, T* uk, T* vk, T* wk, int nbW, int nbX) {
  after_previous();
  const int b = (int)blockIdx.x, region = b < nbW ? 0 : (b < nbW + nbX ? 1 : 2);
  refresh(g, normal, gh, uk, vk, wk, region, (long)(b - (region > 0 ? nbW : 0) - (region > 1 ? nbX : 0)) * 256 + threadIdx.x);
}

// The whole viscous solve of a small grid in one launch: a cluster of 16 blocks runs outer
// iterations (sweeps and refreshes as sweep_all orders them, a cluster barrier between
// them) until the stop rule of solu_sor4.f:130,291-293 ends it (SorLoop), and logs it.
// A phase costs about 2.3 us for its barrier, its stores' way to L2 and the next loads'
// back, and the sweep's arithmetic on 16 SMs; a launch costs 4, and the rule's loop two
// more and a conditional node per iteration.  A step, us (launches -> cluster): FP64
// 32x16x16 436 -> 367, 32x32x16 459 -> 407, 64x32x16 482 -> 489 (16 SMs' FP64 pipes are
// full); mixed 32x32x16 467 -> 413, 64x32x16 484 -> 436, 64x32x32 526 -> 531: hence the two
// limits.
constexpr int kClusterBlocks = 16, kClusterThreads = 512;
constexpr long kClusterCells64 = 1L << 14, kClusterCells32 = 1L << 15;
template <class T>
struct SolveK {
  SweepK<T> k[3];
  const T *mu, *exy, *exz, *eyz, *A[3], *B[3];
  T *un, *vn, *wn;
};
template <int COMP, bool GHOSTS, class T, class G>
__device__ __forceinline__ T cluster_pair(const Grid& g, const SolveK<T>& K, const G& gh, int pi, int pj, int pk,
                                          int me) {
  const int lw = 31 - __clz(g.ni / 2), lj = 31 - __clz(g.nj / 2), half = (g.ni / 2) * (g.nj / 2) * (g.nk / 2);
  const int jmax = COMP == 1 ? g.nj - 1 : g.nj;
  T* q = COMP == 0 ? K.un : (COMP == 1 ? K.vn : K.wn);
  T e = 0;
#pragma unroll 1
  for (int p = me; p < 2 * half; p += kClusterBlocks * kClusterThreads) {
    const bool h = p >= half;
    const int r = h ? p - half : p;
    const int i = (h ? 3 - pi : pi) + 2 * (r & (g.ni / 2 - 1)), j = (h ? 3 - pj : pj) + 2 * ((r >> lw) & (g.nj / 2 - 1)),
              k = (h ? 3 - pk : pk) + 2 * (r >> (lw + lj));
    if (j > jmax) continue;
    const long c = g.at(i, j, k);
    const T visn = visn_sweep<COMP>(g, K.k[COMP], c, K.mu, K.exy, K.exz, K.eyz, K.un, K.vn, K.wn);
    const T qn = __ldg(K.A[COMP] + c) * visn + __ldg(K.B[COMP] + c);
    const T d = qn - q[c];
    q[c] = qn;
    if (GHOSTS && (i <= 3 || i >= g.ni - 2 || j <= 3 || j >= g.nj - 3 || k <= 3 || k >= g.nk - 2))
      fill_ghosts<COMP>(g, gh, q, i, j, k, qn);
    e += d * d;
  }
  return e;
}
// A thread's sum over the sweeps, which k_pair's blocks add up in double: in FP32 with the
// roundings of the additions kept (a conversion per sweep would take the FP64 pipe)
__device__ __forceinline__ void sweep_sum(double& s, double e) { s += e; }
__device__ __forceinline__ void sweep_sum(df::D& s, float e) {
  const df::D t = df::two_sum(s.h, e);
  s = df::D{t.h, df::fadd(s.l, t.l)};
}
__device__ __forceinline__ double sum_of(double s) { return s; }
__device__ __forceinline__ double sum_of(df::D s) { return (double)s.h + (double)s.l; }
template <class T>
using SweepSum = typename std::conditional<std::is_same<T, double>::value, double, df::D>::type;
template <int COMP, class T, class G, class Sync>
__device__ __forceinline__ void cluster_component(const Grid& g, const SolveK<T>& K, const G& gh, int me, SweepSum<T>& e,
                                                  Sync sync) {
  sweep_sum(e, cluster_pair<COMP, false>(g, K, gh, 1, 1, 1, me));
  sync();
  for (int region = 0; region < 3; ++region)
    for (long t = me; t < refresh_tasks(g, region); t += kClusterBlocks * kClusterThreads)
      refresh(g, 1 << COMP, gh, K.un, K.vn, K.wn, region, t);
  sync();
  sweep_sum(e, cluster_pair<COMP, true>(g, K, gh, 1, 1, 2, me));
  sync();
  sweep_sum(e, cluster_pair<COMP, true>(g, K, gh, 1, 2, 1, me));
  sync();
  sweep_sum(e, cluster_pair<COMP, true>(g, K, gh, 2, 1, 1, me));
  sync();
}
template <class T, class G>
__global__ void __launch_bounds__(kClusterThreads) k_solve_cluster(Grid g, SolveK<T> K, G gh, SorLoop* L, int* log) {
  after_previous();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double parts[kClusterBlocks], warps[kClusterThreads / 32];
  __shared__ int verdict;
  // tasks by warps, a warp of every block in turn: few tasks spread over all 16 SMs
  const int t = (int)threadIdx.x, me = ((t >> 5) * kClusterBlocks + (int)cl.block_rank()) * 32 + (t & 31);
  auto sync = [&] { cl.sync(); };
  const double tol = L->tol, cells = L->cells;
  const int mx = min(max(L->maxit, 1), kSorMax);
  double err0 = 0.0;
  for (int it = 1;; ++it) {
    SweepSum<T> e{};
    cluster_component<0>(g, K, gh, me, e, sync);
    cluster_component<1>(g, K, gh, me, e, sync);
    cluster_component<2>(g, K, gh, me, e, sync);
    // every block gets every block's sum and applies the rule to the same total
    double s = sum_of(e);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((t & 31) == 0) warps[t >> 5] = s;
    __syncthreads();
    if (t < 32) {
      s = t < kClusterThreads / 32 ? warps[t] : 0.0;
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (t < kClusterBlocks) *cl.map_shared_rank(&parts[cl.block_rank()], t) = s;
    }
    cl.sync();
    if (t < 32) {
      s = t < kClusterBlocks ? parts[t] : 0.0;
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (t == 0) {
        int entry = it;
        bool done = it >= mx;
        if (!isfinite(s)) {
          entry |= kSorNonfinite;
          done = true;
        } else {
          const double err = sqrt(s / cells) + 1.0e-99;
          if (it == 1) err0 = err;
          if (err / err0 <= tol)
            done = true;
          else if (done)
            entry |= kSorCapped;
        }
        verdict = done ? entry : 0;
      }
    }
    __syncthreads();
    if (verdict) break;
  }
  if (me == 0) {
    if (L->nlog < kSorLog) log[L->nlog] = verdict;
    L->nlog += 1;
  }
}
__global__ void k_to_float(long n, const double* __restrict__ a, float* __restrict__ b) {
  after_previous();
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
    b[t] = (float)a[t];
}
// un = u + du, vn = v + dv, wn = w + dw at every point
__global__ void k_refine_finish(long n, const double* __restrict__ u, const double* __restrict__ v,
                                const double* __restrict__ w, const float* __restrict__ du,
                                const float* __restrict__ dv, const float* __restrict__ dw, double* __restrict__ un,
                                double* __restrict__ vn, double* __restrict__ wn) {
  after_previous();
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    un[t] = u[t] + (double)du[t];
    vn[t] = v[t] + (double)dv[t];
    wn[t] = w[t] + (double)dw[t];
  }
}

__global__ void __launch_bounds__(1024) k_sum_parts2(const double* part, long n, double* out) {
  after_previous();
  __shared__ double sh[32];
  double a = 0.0;
  for (long t = threadIdx.x; t < n; t += 1024) a += part[t];
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  a = sh[threadIdx.x];
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  if (threadIdx.x == 0) out[0] = a;
}

}  // namespace

// The one-pass refresh kernels where the grid allows them, unless FMF_REFRESH_ORDERED
// is set in the environment (then the ordered plane kernels, which give the same
// values: the tests compare the two).
bool one_pass_refresh(const Grid& g) {
  static const bool ordered = std::getenv("FMF_REFRESH_ORDERED") != nullptr;
  return !ordered && refresh_one_pass(g.ni, g.nj, g.nk);
}

namespace {
VP make_vp(double dxinv, double dyinv, double dzinv, double dt, int harmonic) {
  VP p;
  p.dxi = dxinv;
  p.dyi = dyinv;
  p.dzi = dzinv;
  p.dtinv = dt > 0.0 ? 1.0 / dt : 0.0;
  p.dx2 = dxinv * dxinv;
  p.dy2 = dyinv * dyinv;
  p.dz2 = dzinv * dzinv;
  p.dxy = dxinv * dyinv;
  p.dxz = dxinv * dzinv;
  p.dyz = dyinv * dzinv;
  p.harmonic = harmonic;
  return p;
}
const dim3 kB(32, 8, 1);
dim3 wall_grid(const Grid& g) { return dim3((g.ni + 6 + 31) / 32, (2 * (g.nk + 6) + 7) / 8); }
dim3 xh_grid(const Grid& g) { return dim3((g.nj + 6 + 31) / 32, (g.nk + 6 + 7) / 8); }
dim3 zh_grid(const Grid& g) { return dim3((g.ni + 6 + 31) / 32, (g.nj + 6 + 7) / 8); }
struct PairShape {
  dim3 grid, block;
  int kz;
  bool both, ghosts, flat;
};
// The split of a colour pair's points, by what bounds the sweep at each size.  Small grids:
// the launch and one warp's chain, so two-warp blocks and one point per thread, the two
// colours apart.  FP64 beyond: the FP64 pipe, with both colours in a thread for the rows
// they share and, on the largest, 4 planes per thread (fewer sums and partials).  FP32:
// memory, so both colours together once the fields leave L2, and beyond the ghosts
// refreshed apart, the swept component's alone (the sweep's own scattered writes cost it
// more there than the launches).  One outer iteration, us, as
// (block, both or split, planes): FP64 32x32x16 (64, s, 1) 92, (64, b, 1) 115; 128x64x64
// (64, s, 1) 162, (64, b, 1) 147, (128, b, 4) 224; 256x128x128 (64, b, 1) 677, (128, b, 4)
// 655; 512x256x256 4267, 4086.  FP32, g: with the ghosts: 128x64x64 (64, s, 1) g 122,
// (64, b, 1) g 131, (64, b, 1) 154; 256x64x64 g 152, (128, b, 1) g 145, (64, b, 1) 159;
// 256x128x64 (FLAT, a drop) g 224, (64, b, 1) 205; 256x128x128 (64, s, 1) 342, (64, b, 1)
// 311, (128, b, 2) 319, g 358; 512x256x256 1779, 1661, 1606, g 1696.
PairShape pair_shape(const Grid& g, bool fp64) {
  PairShape p;
  const long n = g.cells();
  p.both = n >= (fp64 ? 1L << 18 : 1L << 20);
  p.kz = fp64 && n >= 1L << 21 ? 4 : (!fp64 && n >= 1L << 23 ? 2 : 1);
  p.ghosts = fp64 || n < 1L << 21;
  const int nt = n >= (fp64 ? 1L << 21 : 1L << 23) || (!fp64 && p.both && p.ghosts) ? 128 : 64;
  p.flat = flat_sweeps(g);
  const int bx = std::min(32, g.ni / 2), by = nt / bx;
  p.block = dim3((unsigned)bx, (unsigned)by);
  const int rows = (g.nj / 2 + by - 1) / by, planes = (g.nk / 2 + p.kz - 1) / p.kz;
  p.grid = dim3((unsigned)((g.ni / 2 + bx - 1) / bx), (unsigned)((long)rows * planes), p.both ? 1 : 2);
  return p;
}
// first colour of each pair (solu_sor4.f:94-120): (1,1,1) (1,1,2) (1,2,1) (2,1,1)
const int kPi[4] = {1, 1, 1, 2}, kPj[4] = {1, 1, 2, 1}, kPk[4] = {1, 2, 1, 1};

VPS make_vps(const VP& p, double grvb, double grvp) {
  using df::split_double;
  VPS ps;
  ps.dtinv = split_double(p.dtinv);
  ps.dx2 = split_double(p.dx2);
  ps.dy2 = split_double(p.dy2);
  ps.dz2 = split_double(p.dz2);
  ps.dx2x2 = split_double(2.0 * p.dx2);
  ps.dy2x2 = split_double(2.0 * p.dy2);
  ps.dz2x2 = split_double(2.0 * p.dz2);
  ps.grvb = split_double(grvb);
  ps.grvp = split_double(grvp);
  return ps;
}

// A of component t in a fluid of density r and viscosity m
double fluid_a(const VP& p, double r, double m, int t) {
  const double xx = 2.0 * m * p.dx2, yy = 2.0 * m * p.dy2, zz = 2.0 * m * p.dz2;
  return 1.0 / (2.0 * r * p.dtinv + (t == 0 ? 2.0 * xx : xx) + (t == 1 ? 2.0 * yy : yy) + (t == 2 ? 2.0 * zz : zz));
}

// k_edges, k_src_ab or (REFINE) k_src_ab_e, k_wall_coef
template <bool REFINE>
void src_prep(cudaStream_t s, const Grid& g, const VP& p, const double* u, const double* v, const double* w,
              const double* const* adv, const double* const* advo, const double* phat,
              const double* const* vis, const double* const* fst, const double* const* fstn, double grvb,
              double grvp, const Fluids& fl, const double* mu, const double* rho, const double* rhon, double* const* E,
              F3 ef, ABOut out, const double* l1, const double* l2, const double* phi, double dy, double* wallc,
              const FlatFluid& flat = FlatFluid()) {
  SrcIn in;
  in.u = u;
  in.v = v;
  in.w = w;
  in.rho = rho;
  in.rhon = rhon;
  for (int q = 0; q < 3; ++q) {
    in.adv[q] = adv[q];
    in.advo[q] = advo[q];
    in.vis[q] = vis[q];
    in.fst[q] = fst[q];
    in.fstn[q] = fstn[q];
  }
  in.phat = phat;
  in.grvb = grvb;
  in.grvp = grvp;
  chain(s, tile_grid(g.ni + 1, g.nj + 1, g.nk + 1, 128), 128, k_edges)(
      g, p, mu, E[0], E[1], E[2], ef, flat.count);
  if (REFINE) {
    FlatE FE;
    FE.pairs = flat.pairs;
    FE.fluid = flat.fluid;
    FE.count = flat.count;
    const double rf[2] = {fl.rhol, fl.rhog}, mf[2] = {fl.rmul, fl.rmug};
    for (int q = 0; q < 2; ++q) {
      std::memcpy(&FE.rb[q], &rf[q], sizeof(double));
      std::memcpy(&FE.mb[q], &mf[q], sizeof(double));
    }
    chain(s, tile_grid(g.ni, g.nj, g.nk, 256), 256, k_src_ab_e)(g, make_vps(p, grvb, grvp), p, Fac<double>(p), in, FE,
                                                                mu, E[0], E[1], E[2], out);
  } else {
    SrcK K;
    K.hdt = 0.5 * p.dtinv;
    K.dx2 = p.dx2;
    K.dy2 = p.dy2;
    K.dz2 = p.dz2;
    K.tx2 = 2.0 * p.dx2;
    K.ty2 = 2.0 * p.dy2;
    K.tz2 = 2.0 * p.dz2;
    K.px = -2.0 * p.dxi;
    K.py = -2.0 * p.dyi;
    K.pz = -2.0 * p.dzi;
    K.hg[0] = 0.5 * grvb;
    K.hg[1] = 0.5 * grvp;
    K.hg[2] = 0.0;
    const double rf[2] = {fl.rhol, fl.rhog}, mf[2] = {fl.rmul, fl.rmug};
    for (int q = 0; q < 2; ++q) {
      std::memcpy(&K.rb[q], &rf[q], sizeof(double));
      std::memcpy(&K.mb[q], &mf[q], sizeof(double));
      K.s[q] = 4.0 * rf[q];
      for (int t = 0; t < 3; ++t) K.a[q][t] = fluid_a(p, rf[q], mf[q], t);
    }
    K.fluid = flat.fluid;
    K.count = flat.count;
    chain(s, tile_grid(g.ni, g.nj, g.nk, 256), 256, k_src_ab)(g, K, in, mu, E[0], E[1], E[2], out);
  }
  chain(s, wall_grid(g), kB, k_wall_coef)(g, dy, l1, l2, phi, wallc);
  count_launch(3);
}

// The colour-pair sweeps of one outer iteration: per component 4 pairs, each followed
// by the wall/halo refresh; then the residual sum into errsum[0].  The refresh after a
// component's first pair moves its ghosts from bndu's copies to the plain periodic ones
// (and the previous component's back), so it runs in full; after the other three only
// the swept component's ghosts change, and the points write them (GHOSTS) where the grid
// allows the one-pass refresh.
template <class T, class G, class HaloFn>
void sweep_all(cudaStream_t s, const Grid& g, const VP& p, const T* mu, const T* exy, const T* exz, const T* eyz,
               T* const* A, T* const* B, T* un, T* vn, T* wn, const G& gh, double* part, double* errsum, HaloFn halo,
               const FlatFluid& flat = FlatFluid(), const std::function<void(int, int)>& before = nullptr) {
  const PairShape sp = pair_shape(g, sizeof(T) == 8);
  const bool fill = one_pass_refresh(g) && sp.ghosts;
  for (int comp = 0; comp < 3; ++comp) {
    const SweepK<T> K(p, comp, flat);
    for (int pr = 0; pr < 4; ++pr) {
      if (before) before(comp, pr);
      auto run = [&](auto fn) {
        chain(s, sp.grid, sp.block, fn)(g, K, kPi[pr], kPj[pr], kPk[pr], sp.kz, mu, exy, exz, eyz, A[comp], B[comp], un,
                                        vn, wn, gh, part, comp == 0 && pr == 0);
        count_launch();
      };
      const bool own = fill && pr > 0;
      auto pair = [&](auto ghosts, auto both, auto fl) {
        if (comp == 0) run(k_pair<0, T, G, ghosts.value, both.value, fl.value>);
        else if (comp == 1) run(k_pair<1, T, G, ghosts.value, both.value, fl.value>);
        else run(k_pair<2, T, G, ghosts.value, both.value, fl.value>);
      };
      constexpr std::true_type yes;
      constexpr std::false_type no;
      auto kinds = [&](auto fl) {  // (FLAT's sizes have both colours in a thread)
        if (own && sp.both) pair(yes, yes, fl);
        else if (sp.both) pair(no, yes, fl);
        else if constexpr (!fl.value) own ? pair(yes, no, fl) : pair(no, no, fl);
      };
      sp.flat && flat.fluid ? kinds(yes) : kinds(no);
      if (!own) halo(1 << comp, pr == 0);
    }
  }
  if (!errsum) return;
  chain(s, 1, 1024, k_sum_parts2)(part, (long)sp.grid.x * sp.grid.y * sp.grid.z, errsum);
  count_launch();
}
}  // namespace

void src_visc_prep(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double dt, int harmonic,
                   double grvb, double grvp, const double* u, const double* v, const double* w,
                   const double* const* adv, const double* const* advo, const double* phat,
                   const double* const* vis, const double* const* fst, const double* const* fstn, const Fluids& fl,
                   const double* mu, const double* rho, const double* rhon, double* const* E, double* const* AB, const double* l1,
                   const double* l2, const double* phi, double dy, double* wallc, const FlatFluid& flat) {
  ABOut out{};
  for (int q = 0; q < 3; ++q) {
    out.a[q] = AB[2 * q];
    out.b[q] = AB[2 * q + 1];
  }
  src_prep<false>(s, g, make_vp(dxinv, dyinv, dzinv, dt, harmonic), u, v, w, adv, advo, phat, vis, fst, fstn, grvb,
                  grvp, fl, mu, rho, rhon, E, F3{{nullptr, nullptr, nullptr}}, out, l1, l2, phi, dy, wallc, flat);
}

// (below, a plane's loads no longer hide the bytes': 64x64x64 119 us without, 124 with)
bool flat_sweeps(const Grid& g) { return g.cells() >= 1L << 21; }
FlatFluid make_flat(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double dt,
                    const Fluids& fl, unsigned char* bytes, bool mixed) {
  FlatFluid f;
  if (!bytes) return f;
  const VP p = make_vp(dxinv, dyinv, dzinv, dt, 0);
  if (mixed) {
    float2* pairs = (float2*)(bytes + g.n + 8);  // (g.n is a multiple of 8)
    chain(s, 1, 32, k_flat_pairs)(make_vps(p, 0.0, 0.0), fl, pairs);
    count_launch();
    f.pairs = pairs;
  }
  if (!flat_sweeps(g)) return f;
  f.fluid = bytes;
  f.count = (int*)(bytes + g.n);
  f.enough = (int)(g.cells() - g.cells() / 10);
  f.mu[0] = fl.rmul;
  f.mu[1] = fl.rmug;
  for (int t = 0; t < 3; ++t) {
    f.a[0][t] = fluid_a(p, fl.rhol, fl.rmul, t);
    f.a[1][t] = fluid_a(p, fl.rhog, fl.rmug, t);
  }
  return f;
}

void wall_coef(cudaStream_t s, const Grid& g, double dy, const double* l1, const double* l2, const double* phi,
               double* wallc) {
  chain(s, wall_grid(g), kB, k_wall_coef)(g, dy, l1, l2, phi, wallc);
  count_launch();
}

void explicit_viscous(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, const double* u,
                      const double* v, const double* w, const double* mu, double* tau, double* const* vis,
                      double* sk, const float2* uvw) {
  if (uvw) {
    using df::split_double;
    VPT p;
    p.dxd = dxinv;
    p.dyd = dyinv;
    p.dzd = dzinv;
    p.dxi2 = split_double(2.0 * dxinv);
    p.dyi2 = split_double(2.0 * dyinv);
    p.dzi2 = split_double(2.0 * dzinv);
    p.hx = split_double(0.25 * dxinv);
    p.hy = split_double(0.25 * dyinv);
    p.hz = split_double(0.25 * dzinv);
    p.dxi = split_double(dxinv);
    p.dyi = split_double(dyinv);
    p.dzi = split_double(dzinv);
    float2* tp = (float2*)tau;
    chain(s, tile_grid(g.ni + 2, g.nj + 2, g.nk + 2, 256), 256, k_stress_e)(g, p, uvw, u, v, w, mu, tp, sk);
    chain(s, dim3((g.ni + 31) / 32, (g.nj + 7) / 8, g.nk), kB, k_div_stress_e)(g, p, tp, vis[0], vis[1], vis[2]);
    count_launch(2);
    return;
  }
  const StressK K{dxinv, dyinv, dzinv, dxinv / dyinv, dxinv / dzinv, dyinv / dzinv, 2.0 * dxinv * dxinv,
                  2.0 * dyinv * dyinv, 2.0 * dzinv * dzinv, 0.25 * dyinv * dyinv, 0.25 * dzinv * dzinv,
                  0.25 * dxinv * dyinv, 0.25 * dxinv * dzinv, 0.25 * dyinv * dzinv};
  chain(s, dim3((unsigned)(((long)(g.ni + 2) * (g.nj + 2) + 127) / 128), (unsigned)(g.nk + 2)), 128, k_stress)(
      g, K, u, v, w, mu, tau, sk);
  chain(s, dim3((g.ni + 31) / 32, (g.nj + 7) / 8, g.nk), kB, k_div_stress)(g, K, tau, vis[0], vis[1], vis[2]);
  count_launch(2);
}

void wall_halo(cudaStream_t s, const Grid& g, int normal, double uwall, const double* wallc, double* un, double* vn,
               double* wn) {
  if (one_pass_refresh(g)) {
    const long tw = refresh_tasks(g, 0), tx = refresh_tasks(g, 1), tz = refresh_tasks(g, 2);
    const int nbW = (int)((tw + 255) / 256), nbX = (int)((tx + 255) / 256), nbZ = (int)((tz + 255) / 256);
    chain(s, nbW + nbX + nbZ, 256, k_refresh<double, Ghosts64>)(g, normal, Ghosts64{uwall, wallc}, un, vn, wn, nbW, nbX);
    count_launch();
    return;
  }
  chain(s, wall_grid(g), kB, k_wall)(g, uwall, wallc, un, vn, wn);
  if (g.ni >= 8)
    chain(s, (unsigned)((24L * (g.nj + 6) * (g.nk + 6) + 255) / 256), 256, k_halo_x8)(g, normal, un, vn, wn);
  else
    chain(s, xh_grid(g), kB, k_halo_x)(g, normal, un, vn, wn);
  chain(s, zh_grid(g), kB, k_halo_z)(g, normal, un, vn, wn);
  count_launch(3);
}

void sor_iteration(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, int harmonic,
                   const double* mu, double* const* E, double* const* AB, double uwall, const double* wallc,
                   double* un, double* vn, double* wn, double* part, double* errsum, const FlatFluid& flat,
                   const std::function<void(int, int)>& before) {
  double* const A[3] = {AB[0], AB[2], AB[4]};
  double* const B[3] = {AB[1], AB[3], AB[5]};
  sweep_all<double>(s, g, make_vp(dxinv, dyinv, dzinv, 0.0, harmonic), mu, E[0], E[1], E[2], A, B, un, vn, wn,
                    Ghosts64{uwall, wallc}, part, errsum,
                    [&](int normal, bool) { wall_halo(s, g, normal, uwall, wallc, un, vn, wn); }, flat, before);
}

__global__ void k_sor_rule(SorLoop* L, double tol, int maxit, double cells) {
  after_previous();
  L->tol = tol;
  L->maxit = maxit;
  L->cells = cells;
  L->nlog = 0;
}
void sor_rule(cudaStream_t s, SorLoop* L, double tol, int maxit, double cells) {
  chain(s, 1, 1, k_sor_rule)(L, tol, maxit, cells);
  count_launch();
}
// whether a cluster of 16 blocks of the kernel fits this device (asked once per device)
template <class T, class G>
static bool cluster_fits() {
  static thread_local int cached_dev = -1;
  static thread_local bool cached = false;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev == cached_dev) return cached;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = kClusterBlocks;
  cfg.blockDim = kClusterThreads;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kClusterBlocks;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int n = 0;
  cached = cudaFuncSetAttribute(k_solve_cluster<T, G>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
           cudaOccupancyMaxActiveClusters(&n, k_solve_cluster<T, G>, &cfg) == cudaSuccess && n > 0;
  cudaGetLastError();  // a device without such clusters takes the separate launches
  cached_dev = dev;
  return cached;
}
template <class T, class G>
static void solve_cluster(cudaStream_t s, const Grid& g, const SolveK<T>& K, const G& gh, SorLoop* L, int* log) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = kClusterBlocks;
  cfg.blockDim = kClusterThreads;
  cfg.stream = s;
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kClusterBlocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as chain
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  FMF_CUDA(cudaLaunchKernelEx(&cfg, k_solve_cluster<T, G>, g, K, gh, L, log));
  count_launch();
}
bool solve_small_supported(const Grid& g, bool fp64) {
  if (!one_pass_refresh(g) || g.cells() > (fp64 ? kClusterCells64 : kClusterCells32)) return false;
  return fp64 ? cluster_fits<double, Ghosts64>() : cluster_fits<float, Ghosts32>();
}
void solve_small(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, const double* mu,
                 double* const* E, double* const* AB, double uwall, const double* wallc, double* un, double* vn,
                 double* wn, SorLoop* L, int* log) {
  const VP p = make_vp(dxinv, dyinv, dzinv, 0.0, 0);
  const SolveK<double> K{{{p, 0}, {p, 1}, {p, 2}}, mu, E[0], E[1], E[2], {AB[0], AB[2], AB[4]}, {AB[1], AB[3], AB[5]},
                         un, vn, wn};
  solve_cluster(s, g, K, Ghosts64{uwall, wallc}, L, log);
}
void solve_small_refine(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, const RefineBufs& rb,
                        SorLoop* L, int* log) {
  const VP p = make_vp(dxinv, dyinv, dzinv, 0.0, 0);
  const SolveK<float> K{{{p, 0}, {p, 1}, {p, 2}}, rb.mu, rb.e[0], rb.e[1], rb.e[2], {rb.a[0], rb.a[1], rb.a[2]},
                        {rb.r[0], rb.r[1], rb.r[2]}, rb.d[0], rb.d[1], rb.d[2]};
  solve_cluster(s, g, K, Ghosts32{rb.gw, rb.gx, rb.gz}, L, log);
}

long refine_floats(const Grid& g, int part) {
  switch (part) {
    case 0: return 2L * (g.nk + 6) * (g.ni + 6) * kGW;
    case 1: return (long)(g.nj + 6) * (g.nk + 6) * kGH;
    default: return (long)(g.ni + 6) * (g.nj + 6) * kGH;
  }
}

void refine_prep(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double dt, int harmonic,
                 double grvb, double grvp, const double* u, const double* v, const double* w,
                 const double* const* adv, const double* const* advo, const double* phat,
                 const double* const* vis, const double* const* fst, const double* const* fstn, const Fluids& fl,
                 const double* mu, const double* rho, const double* rhon, double* const* E, const double* l1, const double* l2,
                 const double* phi, double dy, double uwall, double* wallc, const RefineBufs& rb,
                 const FlatFluid& flat) {
  ABOut out{};
  for (int q = 0; q < 3; ++q) {
    out.af[q] = rb.a[q];
    out.rf[q] = rb.r[q];
  }
  // A and B in FP32 pairs, the residual in FP64 (k_src_ab_e)
  src_prep<true>(s, g, make_vp(dxinv, dyinv, dzinv, dt, harmonic), u, v, w, adv, advo, phat, vis, fst, fstn, grvb,
                 grvp, fl, mu, rho, rhon, E, F3{{rb.e[0], rb.e[1], rb.e[2]}}, out, l1, l2, phi, dy, wallc, flat);
  chain(s, 4 * 152, 256, k_to_float)(g.n, mu, rb.mu);
  chain(s, wall_grid(g), kB, k_gamma_wall)(g, uwall, wallc, u, v, w, rb.gw);
  chain(s, xh_grid(g), kB, k_gamma_x)(g, u, v, w, rb.gx);
  chain(s, zh_grid(g), kB, k_gamma_z)(g, u, v, w, rb.gz);
  count_launch(4);
  for (int q = 0; q < 3; ++q) FMF_CUDA(cudaMemsetAsync(rb.d[q], 0, sizeof(float) * g.n, s));
}

void sor_iteration_refine(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv,
                          const RefineBufs& rb, double* part, double* errsum, const FlatFluid& flat) {
  float *du = rb.d[0], *dv = rb.d[1], *dw = rb.d[2];
  sweep_all<float>(
      s, g, make_vp(dxinv, dyinv, dzinv, 0.0, 0), rb.mu, rb.e[0], rb.e[1], rb.e[2], rb.a, rb.r, du, dv, dw,
      Ghosts32{rb.gw, rb.gx, rb.gz}, part, errsum,
      [&](int normal, bool first) {
        if (one_pass_refresh(g) && !first) {  // the swept component's ghosts alone change
          const int nbW = (int)((refresh_tasks(g, 0) + 255) / 256), nbX = (int)((refresh_tasks(g, 1) / 3 + 255) / 256),
                    nbZ = (int)((refresh_tasks(g, 2) / 3 + 255) / 256);
          chain(s, nbW + nbX + nbZ, 256, k_refresh_one)(g, normal >> 1, Ghosts32{rb.gw, rb.gx, rb.gz}, du, dv, dw, nbW,
                                                        nbX);
          count_launch();
          return;
        }
        if (one_pass_refresh(g)) {
          const long tw = refresh_tasks(g, 0), tx = refresh_tasks(g, 1), tz = refresh_tasks(g, 2);
          const int nbW = (int)((tw + 255) / 256), nbX = (int)((tx + 255) / 256), nbZ = (int)((tz + 255) / 256);
          chain(s, nbW + nbX + nbZ, 256, k_refresh<float, Ghosts32>)(g, normal, Ghosts32{rb.gw, rb.gx, rb.gz}, du, dv, dw,
                                                                     nbW, nbX);
          count_launch();
          return;
        }
        chain(s, wall_grid(g), kB, k_wall_d)(g, rb.gw, du, dv, dw);
        chain(s, xh_grid(g), kB, k_halo_x_d)(g, normal, rb.gx, du, dv, dw);
        chain(s, zh_grid(g), kB, k_halo_z_d)(g, normal, rb.gz, du, dv, dw);
        count_launch(3);
      },
      flat);
}

void refine_finish(cudaStream_t s, const Grid& g, const double* u, const double* v, const double* w,
                   const RefineBufs& rb, double* un, double* vn, double* wn) {
  chain(s, 4 * 152, 256, k_refine_finish)(g.n, u, v, w, rb.d[0], rb.d[1], rb.d[2], un, vn, wn);
  count_launch();
}

long sor_parts(const Grid& g) {
  const dim3 a = pair_shape(g, true).grid, b = pair_shape(g, false).grid;
  return std::max((long)a.x * a.y * a.z, (long)b.x * b.y * b.z);
}

}  // namespace fused
}  // namespace fmf
