// fused_csf.cu -- CSF surface-tension force of one volume-fraction field in one
// pass (main.f90:548-567: cal_grad_p2a, calrn x4, calrkap, cal_grad_p2uvw, calfst).
//
// Per interior cell the force on the u, v, w faces is
//   f_u = -(2 sigma/(rho_l+rho_g)) * kappa_u * (phi(i+1)-phi(i))/dx   (calfst.f:40-42)
// with kappa_u the divergence of the unit normal over the u control volume
// (calrkap.f:45-98), built from four families of normals (calrn.f:45-87):
//   npp at cell centres  = N(mean of the 8 vertex gradients around the cell),
//   n12 at (i+1/2,j+1/2,k) = N(mean of vertex gradients k-1/2, k+1/2),
//   n13 at (i+1/2,j,k+1/2) = N(mean over j-1/2, j+1/2),
//   n23 at (i,j+1/2,k+1/2) = N(mean over i-1/2, i+1/2),
// N(v) = v/(|v| + 1e-30*|dxinv|) and vertex gradients from cal_grad_p2a.f:46-60.
//
// FP64 (the FP64 and the FP64-accurate step): three kernels over the whole grid, k_csf_grad (the vertex
// gradients G), k_csf_normals (the four families) and k_csf_force, with G and the nine
// normal components used in device memory (12 n doubles of workspace).
//
// FP32 (R = float, the mixed-precision step) and FP32 pairs (R = Pr: fmf_dev_csf_fused in
// FMF_FP64E, which needs no workspace; in the step the three kernels are faster, 203
// against 245 us for a drop at 256x128x128): one kernel, k_csf.  A block owns a 32 x 8 tile of (i,j) columns and
// marches over a chunk of k planes; each phi plane is converted once into a
// shared-memory ring of three planes.  Vertex gradients G of planes k, k+1 and the
// normals of planes k-1..k+1 live in shared memory; H(k+1) = G(k)+G(k+1) gives both
// n12(k+1) and, summed over the four surrounding (i,j), npp(k+1).  Each normal is
// formed once per block, and the forces are widened or rounded to double on the store.
#include <algorithm>
#include <type_traits>

#include "../../include/fmf_capi.h"
#include "bits.cuh"
#include "df64.cuh"
#include "fused.cuh"
#include "recip.cuh"

namespace fmf {
namespace fused {

namespace {
constexpr int TX = 32, TY = 8;
constexpr int GX = TX + 2, GY = TY + 2;  // G and H region: i in [I0-1, I0+TX], j in [J0-1, J0+TY]
constexpr int NX = TX + 1, NY = TY + 1;  // normal regions
constexpr int GP = GX * GY, NP = NX * NY;
constexpr int QX = GX + 1, QY = GY + 1;  // staged phi plane: i in [I0-1, I0+TX+1], j in [J0-1, J0+TY+1]
constexpr int QP = QX * QY;

// FP32 pair (df64.cuh) with the arithmetic operators the kernel's template uses
struct Pr {
  df::D v;
  Pr() = default;
  __host__ __device__ Pr(df::D d) : v(d) {}
  __host__ __device__ explicit Pr(double q) : v(df::split_double(q)) {}
  __device__ explicit operator double() const { return df::to_double(v); }
};
__host__ __device__ __forceinline__ Pr operator+(Pr a, Pr b) { return df::add(a.v, b.v); }
__host__ __device__ __forceinline__ Pr operator-(Pr a, Pr b) { return df::sub(a.v, b.v); }
__host__ __device__ __forceinline__ Pr operator*(Pr a, Pr b) { return df::mul(a.v, b.v); }
__host__ __device__ __forceinline__ Pr operator-(Pr a) { return df::neg(a.v); }

// bits: whether a and b differ, whether a vector is 0 (either sign), whether a is finite
__device__ __forceinline__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }
__device__ __forceinline__ bool differ(Pr a, Pr b) { return differ(a.v.h, b.v.h) || differ(a.v.l, b.v.l); }
__device__ __forceinline__ bool finite(float a) { return (__float_as_uint(a) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool finite(Pr a) { return finite(a.v.h) && finite(a.v.l); }
__device__ __forceinline__ bool nonzero(float a) { return (__float_as_uint(a) << 1) != 0; }
__device__ __forceinline__ bool nonzero(Pr a) { return nonzero(a.v.h) || nonzero(a.v.l); }
__device__ __forceinline__ float zero(float) { return 0.0f; }
__device__ __forceinline__ Pr zero(Pr) { return df::D{0.0f, 0.0f}; }

template <class R>
struct CsfP {
  R dxi, dyi, dzi, gx, gy, gz, vs2, vs8;  // vs2 = 2 vs, vs8 = 8 vs
  R fx, fy, fz;                           // -(2 sigma/(rho_l + rho_g)) dxinv etc. (calfst.f:40-42)
};

template <class R>
struct Smem {
  R G[2][3][GP];    // vertex gradients, two planes (ring)
  R H[3][GP];       // G(k) + G(k+1)
  R pp[2][3][NP];   // npp, planes k and k+1 (ring); region i in [I0, I0+TX], j in [J0, J0+TY]
  R a12[2][2][NP];  // n12 (x, y), planes k and k+1; region i in [I0-1, I0+TX-1], j in [J0-1, J0+TY-1]
  R a13[2][2][NP];  // n13 (x, z), planes k-1 and k; same region
  R a23[2][2][NP];  // n23 (y, z), planes k-1 and k; same region
  R Q[3][QP];       // staged phi planes, slot = plane % 3
};

// N(v) = v/(|v| + vs).  Callers pass v scaled by 1/c (a sum instead of a mean) with
// vs scaled by 1/c: N(c w) = w/(|w| + vs/c).
// FP32: where |v| < 1e-15 the squares would leave the normal range, so numerator
// and denominator are both scaled by 2^64 first (an exact power-of-two scaling).
__device__ __forceinline__ void unit_of(float x, float y, float z, float vs, float* o) {
  float s = x * x + y * y + z * z;
  if (s < 1.0e-30f) {
    const float c = 18446744073709551616.0f;  // 2^64
    x *= c;
    y *= c;
    z *= c;
    vs *= c;
    s = x * x + y * y + z * z;
  }
  const float inv = 1.0f / (sqrtf(s) + vs);
  o[0] = x * inv;
  o[1] = y * inv;
  o[2] = z * inv;
}

// FP32 pairs.  Where |v| is below about 2^-50 the squares approach float's normal
// range, so v and vs are scaled by 2^64 first (exact; N is unchanged); a sum of
// squares below 2^-126 after that counts as 0 (|v| + vs = vs).
__device__ __forceinline__ void unit_of(Pr x, Pr y, Pr z, Pr vs, Pr* o) {
  using namespace df;
  D X = x.v, Y = y.v, Z = z.v, V = vs.v;
  D s = add(add(sqr(X), sqr(Y)), sqr(Z));
  if (s.h < 0x1p-100f) {
    const float c = 0x1p64f;
    X = scale(X, c);
    Y = scale(Y, c);
    Z = scale(Z, c);
    V = scale(V, c);
    s = add(add(sqr(X), sqr(Y)), sqr(Z));
  }
  const float big = fmul(V.h, 1.0e12f);
  D inv;
  if (s.h > fmul(big, big))
    inv = rsqrt(s);
  else if (fexp(s.h) == 0)
    inv = div(D{1.0f, 0.0f}, V);
  else
    inv = div(D{1.0f, 0.0f}, add(mul(s, rsqrt(s)), V));
  o[0] = mul(X, inv);
  o[1] = mul(Y, inv);
  o[2] = mul(Z, inv);
}

// a warp of zero vectors takes the zeros without the reciprocal
template <class R>
__device__ __forceinline__ void unit(R x, R y, R z, R vs, R* o) {
  if (__any_sync(__activemask(), nonzero(x) || nonzero(y) || nonzero(z)))
    unit_of(x, y, z, vs, o);
  else
    o[0] = o[1] = o[2] = zero(x);
}

// vertex gradient at (i+1/2, j+1/2, k+1/2) from two staged planes (Qa = plane k, Qb =
// plane k+1)
template <class R>
__device__ void grad_staged(const CsfP<R>& p, const R* Qa, const R* Qb, R (*G)[GP]) {
  for (int e = threadIdx.x; e < GP; e += blockDim.x) {
    const int a = e % GX, b = e / GX;
    const int c = b * QX + a;
    const R q000 = Qa[c], qp00 = Qa[c + 1], q0p0 = Qa[c + QX], qpp0 = Qa[c + QX + 1];
    const R q00p = Qb[c], qp0p = Qb[c + 1], q0pp = Qb[c + QX], qppp = Qb[c + QX + 1];
    // a warp of flat points stores the zeros that the sums would give
    const bool varies = !finite(q000) || differ(q000, qp00) || differ(q000, q0p0) || differ(q000, qpp0) ||
                        differ(q000, q00p) || differ(q000, qp0p) || differ(q000, q0pp) || differ(q000, qppp);
    if (!__any_sync(__activemask(), varies)) {
      G[0][e] = G[1][e] = G[2][e] = zero(q000);
      continue;
    }
    if constexpr (std::is_same<R, Pr>::value) {
      // the FP64 path's sums and differences of the two planes (15 pair additions)
      const R s00 = q000 + q00p, sp0 = qp00 + qp0p, s0p = q0p0 + q0pp, spp = qpp0 + qppp;
      const R d00 = q00p - q000, dp0 = qp0p - qp00, d0p = q0pp - q0p0, dpp = qppp - qpp0;
      const R ta = spp - s00, tb = sp0 - s0p;
      G[0][e] = (ta + tb) * p.gx;
      G[1][e] = (ta - tb) * p.gy;
      G[2][e] = ((d00 + dp0) + (d0p + dpp)) * p.gz;
    } else {
      G[0][e] = (-q000 + qp00 - q0p0 + qpp0 - q00p + qp0p - q0pp + qppp) * p.gx;
      G[1][e] = (-q000 - qp00 + q0p0 + qpp0 - q00p - qp0p + q0pp + qppp) * p.gy;
      G[2][e] = (-q000 - qp00 - q0p0 - qpp0 + q00p + qp0p + q0pp + qppp) * p.gz;
    }
  }
}
// phi plane k (i in [I0-1, I0+TX+1], j in [J0-1, J0+TY+1]) into Q, converted to R
template <class R>
__device__ void stage_plane(const Grid& g, const double* __restrict__ phi, int I0, int J0, int k, R* Q) {
  for (int e = threadIdx.x; e < QP; e += blockDim.x) {
    const int a = e % QX, b = e / QX;
    Q[e] = (R)__ldg(phi + g.at(I0 - 1 + a, J0 - 1 + b, k));
  }
}
// n13 and n23 of plane k from G(k) (slot gk) into ring slot s
template <class R>
__device__ void side_normals(const CsfP<R>& p, Smem<R>& S, int gk, int s) {
  for (int e = threadIdx.x; e < NP; e += blockDim.x) {
    const int a = e % NX, b = e / NX;  // normal point (I0-1+a, J0-1+b)
    const int ga = a, gb = b;          // same point in the G region (offset -1,-1)
    const int c0 = gb * GX + ga;
    R o[3];
    // n13(i,j): mean of G(i, j-1) and G(i, j) (the sum, with 2 vs)
    const int cm = (gb - 1) * GX + ga;
    if (gb >= 1) {
      unit(S.G[gk][0][cm] + S.G[gk][0][c0], S.G[gk][1][cm] + S.G[gk][1][c0], S.G[gk][2][cm] + S.G[gk][2][c0], p.vs2,
           o);
      S.a13[s][0][e] = o[0];
      S.a13[s][1][e] = o[2];
    }
    // n23(i,j): mean of G(i-1, j) and G(i, j)
    if (ga >= 1) {
      const int cw = gb * GX + ga - 1;
      unit(S.G[gk][0][cw] + S.G[gk][0][c0], S.G[gk][1][cw] + S.G[gk][1][c0], S.G[gk][2][cw] + S.G[gk][2][c0], p.vs2,
           o);
      S.a23[s][0][e] = o[1];
      S.a23[s][1][e] = o[2];
    }
  }
}
// H = G(gk) + G(gk1); then npp (slot s) and n12 (slot s) of the plane of G(gk1)
template <class R>
__device__ void centre_normals(const CsfP<R>& p, Smem<R>& S, int gk, int gk1, int s) {
  for (int e = threadIdx.x; e < GP; e += blockDim.x)
    for (int q = 0; q < 3; ++q) S.H[q][e] = S.G[gk][q][e] + S.G[gk1][q][e];
  __syncthreads();
  for (int e = threadIdx.x; e < NP; e += blockDim.x) {
    const int a = e % NX, b = e / NX;
    R o[3];
    // npp at (I0+a, J0+b): H over (i-1..i, j-1..j) = G region (a..a+1, b..b+1), the
    // sum of the 8 vertex gradients with 8 vs
    const int h00 = b * GX + a, h10 = h00 + 1, h01 = h00 + GX, h11 = h01 + 1;
    unit(S.H[0][h00] + S.H[0][h10] + S.H[0][h01] + S.H[0][h11], S.H[1][h00] + S.H[1][h10] + S.H[1][h01] + S.H[1][h11],
         S.H[2][h00] + S.H[2][h10] + S.H[2][h01] + S.H[2][h11], p.vs8, o);
    S.pp[s][0][e] = o[0];
    S.pp[s][1][e] = o[1];
    S.pp[s][2][e] = o[2];
    // n12 at (I0-1+a, J0-1+b): H at the same point
    unit(S.H[0][h00], S.H[1][h00], S.H[2][h00], p.vs2, o);
    S.a12[s][0][e] = o[0];
    S.a12[s][1][e] = o[1];
  }
}

template <class R>
__global__ void __launch_bounds__(256) k_csf(Grid g, CsfP<R> p, int kchunk, const double* __restrict__ phi,
                                             double* __restrict__ fu, double* __restrict__ fv,
                                             double* __restrict__ fw, const int* __restrict__ skip) {
  after_previous();
  if (skip && *skip) return;  // the whole block leaves before any barrier
  extern __shared__ double smraw[];
  Smem<R>& S = *reinterpret_cast<Smem<R>*>(smraw);
  const int I0 = 1 + blockIdx.x * TX, J0 = 1 + blockIdx.y * TY;
  const int kb = 1 + blockIdx.z * kchunk, ke = min(g.nk, kb + kchunk - 1);
  int gA = 0, gB = 1;  // G slots: gA holds plane k, gB the next
  int sp = 0;          // pp/n12 slot of plane k
  int sm = 0;          // n13/n23 slot of plane k-1
  // warm-up: G(kb-1) -> gB, G(kb) -> gA; n13/n23(kb-1) from gB; npp/n12(kb) from both
  for (int q = kb - 1; q <= kb + 1; ++q) stage_plane(g, phi, I0, J0, q, S.Q[q % 3]);
  __syncthreads();
  grad_staged(p, S.Q[(kb - 1) % 3], S.Q[kb % 3], S.G[gB]);
  grad_staged(p, S.Q[kb % 3], S.Q[(kb + 1) % 3], S.G[gA]);
  __syncthreads();
  side_normals(p, S, gB, sm);
  centre_normals(p, S, gB, gA, sp);
  __syncthreads();
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int i = I0 + tx, j = J0 + ty;
  for (int k = kb; k <= ke; ++k) {
    // G(k+1) -> gB; n13/n23(k) from gA; npp/n12(k+1)
    stage_plane(g, phi, I0, J0, k + 2, S.Q[(k + 2) % 3]);  // the slot of plane k-1, unused from here on
    __syncthreads();
    grad_staged(p, S.Q[(k + 1) % 3], S.Q[(k + 2) % 3], S.G[gB]);
    __syncthreads();
    side_normals(p, S, gA, sm ^ 1);
    centre_normals(p, S, gA, gB, sp ^ 1);
    __syncthreads();
    if (i <= g.ni && j <= g.nj) {
      const long c = g.at(i, j, k);
      const int e = ty * NX + tx;            // npp point (i, j)
      const int f = (ty + 1) * NX + tx + 1;  // n12/n13/n23 point (i, j)
      const int cq = (ty + 1) * QX + tx + 1;
      const R* Qk = S.Q[k % 3];
      const R ph = Qk[cq], px = Qk[cq + 1], py = Qk[cq + QX], pz = S.Q[(k + 1) % 3][cq];
      const bool varies = !finite(ph) || differ(ph, px) || differ(ph, py) || differ(ph, pz);
      if (__any_sync(__activemask(), varies)) {
        const R ku = (S.pp[sp][0][e + 1] - S.pp[sp][0][e]) * p.dxi + (S.a12[sp][1][f] - S.a12[sp][1][f - NX]) * p.dyi +
                     (S.a13[sm ^ 1][1][f] - S.a13[sm][1][f]) * p.dzi;
        const R kv = (S.a12[sp][0][f] - S.a12[sp][0][f - 1]) * p.dxi + (S.pp[sp][1][e + NX] - S.pp[sp][1][e]) * p.dyi +
                     (S.a23[sm ^ 1][1][f] - S.a23[sm][1][f]) * p.dzi;
        const R kw = (S.a13[sm ^ 1][0][f] - S.a13[sm ^ 1][0][f - 1]) * p.dxi +
                     (S.a23[sm ^ 1][0][f] - S.a23[sm ^ 1][0][f - NX]) * p.dyi + (S.pp[sp ^ 1][2][e] - S.pp[sp][2][e]) * p.dzi;
        fu[c] = (double)(ku * (px - ph) * p.fx);
        fv[c] = (double)(kv * (py - ph) * p.fy);
        fw[c] = (double)(kw * (pz - ph) * p.fz);
      } else {
        fu[c] = fv[c] = fw[c] = 0.0;
      }
    }
    __syncthreads();
    gA ^= 1;
    gB ^= 1;
    sp ^= 1;
    sm ^= 1;
  }
}

// k planes per block.  A block of c planes costs about c + 1 plane passes (the
// first plane's gradients and side normals are formed twice), and blocks run in
// waves of (SMs x resident blocks per SM); the chunk minimises waves x (c + 1)
// over 4 <= c <= nk (nk itself on small grids), so the last wave is not left
// mostly empty.  Occupancy and SM count are queried once per kernel and device.
int csf_chunk(const Grid& g, const void* fn, size_t smem) {
  static thread_local const void* cached_fn = nullptr;
  static thread_local int cached_dev = -1, cached_cap = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (fn != cached_fn || dev != cached_dev) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, smem);
    cached_fn = fn;
    cached_dev = dev;
    cached_cap = std::max(1, sms * per_sm);
  }
  if (g.nk < 16) return g.nk;
  const long tiles = (long)(g.ni / TX) * (g.nj / TY);
  int best = 16;
  long best_cost = -1;
  for (int c = 4; c <= g.nk; ++c) {
    const long blocks = tiles * ((g.nk + c - 1) / c);
    const long cost = ((blocks + cached_cap - 1) / cached_cap) * (c + 1);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = c;
    }
  }
  return best;
}

template <class R>
void launch_csf(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double rhol, double rhog,
                double sigma, const double* phi, double* fu, double* fv, double* fw, const int* skip) {
  CsfP<R> p;
  p.dxi = (R)dxinv;
  p.dyi = (R)dyinv;
  p.dzi = (R)dzinv;
  p.gx = (R)(0.25 * dxinv);
  p.gy = (R)(0.25 * dyinv);
  p.gz = (R)(0.25 * dzinv);
  const double vs = std::sqrt(dxinv * dxinv + dyinv * dyinv + dzinv * dzinv) * 1.0e-30;
  p.vs2 = (R)(2.0 * vs);
  p.vs8 = (R)(8.0 * vs);
  const double st = 2.0 * sigma / (rhol + rhog);
  p.fx = (R)(-st * dxinv);
  p.fy = (R)(-st * dyinv);
  p.fz = (R)(-st * dzinv);
  const size_t smem = sizeof(Smem<R>);
  cudaFuncSetAttribute(k_csf<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int kchunk = csf_chunk(g, (const void*)k_csf<R>, smem);
  dim3 gr((unsigned)(g.ni / TX), (unsigned)(g.nj / TY), (unsigned)((g.nk + kchunk - 1) / kchunk));
  chain(s, gr, 256, k_csf<R>, smem)(g, p, kchunk, phi, fu, fv, fw, skip);
  count_launch();
}

// ---- FP64 ------------------------------------------------------------------------
// Bound by the FP64 pipe (64 cycles per warp instruction and quarter SM), so the three
// kernels trade device memory for operations: each vertex gradient and each normal is
// formed once (one tiled kernel formed 1.4 and 1.25 of each, with five barriers per
// plane), the sums the families share are formed once, and warps whose points all lie
// where phi is constant store the zeros that the arithmetic would give without doing
// it: away from the interface phi is exactly 0 or 1 (solphi_mthinc3's snap).  At
// 512x256x256 (sessile drop) 11.9 -> 1.2 ms, at 256x128x128 1.59 -> 0.30, at 128x64x256
// with a profile that varies nearly everywhere 0.92 -> 0.33, at 32x32x16 0.068 -> 0.017.
struct CsfD {
  double gx, gy, gz;      // 0.25 dxinv ...
  double dxi, dyi, dzi;
  double vs2, vs8;        // 2 vs, 8 vs
  double big2, big8;      // (1e12 vs2)^2, (1e12 vs8)^2
  double fx, fy, fz;      // -(2 sigma/(rho_l + rho_g)) dxinv etc. (calfst.f:40-42)
};
// 1/(sqrt(s) + vs) for s = |v|^2.  Where |v| exceeds vs by more than 1e12 the relative
// correction vs/|v| is below 1e-12 and 1/|v| is used (the comparisons are on the bit
// patterns: all are non-negative); s = 0 gives 0 (the components it multiplies are 0 or
// their squares underflowed), other small s the exact expression.
__device__ __forceinline__ double inv_norm(double s, double vs, double big) {
  if (raw(s) > raw(big)) return rsqrt_h(s);
  return mag(s) == 0 ? 0.0 : 1.0 / (sqrt(s) + vs);
}

// G at (i+1/2, j+1/2, k+1/2) for i, j, k in -1..n+1 into G[0..2] (n apart); threads
// over the flattened (i, j) plane so that every warp is full
__global__ void __launch_bounds__(128) k_csf_grad(Grid g, CsfD p, const double* __restrict__ phi,
                                                  double* __restrict__ G, const int* __restrict__ skip) {
  after_previous();
  if (skip && *skip) return;
  const Tile T = warp_tile(g.ni + 3);
  if (T.x >= g.ni + 3 || T.y >= g.nj + 3) return;
  const long X = 1, Y = g.sy, Z = g.sz, n = g.n;
  const long c = g.at(T.x - 1, T.y - 1, (int)blockIdx.z - 1);
  const double q000 = __ldg(phi + c), qp00 = __ldg(phi + c + X), q0p0 = __ldg(phi + c + Y),
               qpp0 = __ldg(phi + c + X + Y), q00p = __ldg(phi + c + Z), qp0p = __ldg(phi + c + X + Z),
               q0pp = __ldg(phi + c + Y + Z), qppp = __ldg(phi + c + X + Y + Z);
  // all eight equal in every bit and finite: the gradient is 0
  const long long r = raw(q000);
  auto df = [&](double x) { return (unsigned long long)(raw(x) ^ r); };
  const bool varies = (df(qp00) | df(q0p0) | df(qpp0) | df(q00p) | df(qp0p) | df(q0pp) | df(qppp)) != 0 ||
                      !finite_bits(r);
  if (!__any_sync(__activemask(), varies)) {
    G[c] = 0.0;
    G[c + n] = 0.0;
    G[c + 2 * n] = 0.0;
    return;
  }
  // per (i, j) corner the sum and the difference of the two k planes; with
  // ta = s(+,+) - s(0,0) and tb = s(+,0) - s(0,+), the x sum is ta + tb, the y sum ta - tb
  // and the z sum the four differences (18 operations instead of 24)
  const double s00 = q000 + q00p, sp0 = qp00 + qp0p, s0p = q0p0 + q0pp, spp = qpp0 + qppp;
  const double d00 = q00p - q000, dp0 = qp0p - qp00, d0p = q0pp - q0p0, dpp = qppp - qpp0;
  const double ta = spp - s00, tb = sp0 - s0p;
  G[c] = (ta + tb) * p.gx;
  G[c + n] = (ta - tb) * p.gy;
  G[c + 2 * n] = ((d00 + dp0) + (d0p + dpp)) * p.gz;
}

// The normals at i, j, k in 0..n+1 from G, arrays n apart: npp in pp; n12 (x, y) and the
// x of n13 in n12; the z of n13 and n23 (y, z) in nside.  A thread walks m planes of its (i, j)
// column: P, the sum of G over the four vertices around the column, and G itself are
// kept from plane to plane, so the means take 18 additions per point.
__global__ void __launch_bounds__(128) k_csf_normals(Grid g, CsfD p, int m, const double* __restrict__ G,
                                                     double* __restrict__ pp, double* __restrict__ n12,
                                                     double* __restrict__ nside, const int* __restrict__ skip) {
  after_previous();
  if (skip && *skip) return;
  const Tile T = warp_tile(g.ni + 2);
  const int a = T.x, b = T.y;
  if (a >= g.ni + 2 || b >= g.nj + 2) return;
  const long X = 1, Y = g.sy, Z = g.sz, n = g.n;
  const int k0 = (int)blockIdx.z * m, k1 = min(g.nk + 2, k0 + m);
  long c = g.at(a, b, k0 - 1);  // the plane below the first
  double g0[3], P0[3];
  unsigned long long any0 = 0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double* Gq = G + q * n + c;
    const double gc = __ldg(Gq), gx = __ldg(Gq - X), gy = __ldg(Gq - Y), gxy = __ldg(Gq - X - Y);
    any0 |= mag(gc) | mag(gx) | mag(gy) | mag(gxy);
    g0[q] = gc;
    P0[q] = (gx + gc) + (gxy + gy);
  }
  c += Z;
#pragma unroll 1
  for (int k = k0; k < k1; ++k, c += Z) {
    double gc[3], gx[3], gy[3], gxy[3];
    unsigned long long any1 = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double* Gq = G + q * n + c;
      gc[q] = __ldg(Gq);
      gx[q] = __ldg(Gq - X);
      gy[q] = __ldg(Gq - Y);
      gxy[q] = __ldg(Gq - X - Y);
      any1 |= mag(gc[q]) | mag(gx[q]) | mag(gy[q]) | mag(gxy[q]);
    }
    if (!__any_sync(__activemask(), (any0 | any1) != 0)) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        pp[c + q * n] = 0.0;
        n12[c + q * n] = 0.0;
        nside[c + q * n] = 0.0;
        g0[q] = 0.0;
        P0[q] = 0.0;
      }
      any0 = 0;
      continue;
    }
    double sx[3], sy[3], P[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      sx[q] = gx[q] + gc[q];
      sy[q] = gy[q] + gc[q];
      P[q] = sx[q] + (gxy[q] + gy[q]);
    }
    auto norm = [&](double x, double y, double z, double vs, double big) {
      return inv_norm(fma(z, z, fma(y, y, x * x)), vs, big);
    };
    {  // npp: the 8 vertices around the cell, with 8 vs
      const double x = P0[0] + P[0], y = P0[1] + P[1], z = P0[2] + P[2], r = norm(x, y, z, p.vs8, p.big8);
      pp[c] = x * r;
      pp[c + n] = y * r;
      pp[c + 2 * n] = z * r;
    }
    {  // n12: G of this plane and the one below
      const double x = g0[0] + gc[0], y = g0[1] + gc[1], z = g0[2] + gc[2], r = norm(x, y, z, p.vs2, p.big2);
      n12[c] = x * r;
      n12[c + n] = y * r;
    }
    {  // n13: G(j-1) and G(j)
      const double r = norm(sy[0], sy[1], sy[2], p.vs2, p.big2);
      n12[c + 2 * n] = sy[0] * r;
      nside[c] = sy[2] * r;
    }
    {  // n23: G(i-1) and G(i)
      const double r = norm(sx[0], sx[1], sx[2], p.vs2, p.big2);
      nside[c + n] = sx[1] * r;
      nside[c + 2 * n] = sx[2] * r;
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      g0[q] = gc[q];
      P0[q] = P[q];
    }
    any0 = any1;
  }
}

// the curvatures (calrkap.f:45-98) and the force on the interior u, v, w points; where
// phi does not differ from its three upper neighbours the force is 0
__global__ void __launch_bounds__(256) k_csf_force(Grid g, CsfD p, const double* __restrict__ phi,
                                                   const double* __restrict__ pp, const double* __restrict__ n12,
                                                   const double* __restrict__ nside, double* __restrict__ fu,
                                                   double* __restrict__ fv, double* __restrict__ fw,
                                                   const int* __restrict__ skip) {
  after_previous();
  if (skip && *skip) return;
  const Tile T = warp_tile(g.ni);
  const int i = 1 + T.x, j = 1 + T.y;
  if (i > g.ni || j > g.nj) return;
  const long X = 1, Y = g.sy, Z = g.sz, n = g.n;
  const long c = g.at(i, j, 1 + (int)blockIdx.z);
  const double ph = __ldg(phi + c), px = __ldg(phi + c + X), py = __ldg(phi + c + Y), pz = __ldg(phi + c + Z);
  const long long r = raw(ph);
  const bool varies = ((raw(px) ^ r) | (raw(py) ^ r) |
                       (raw(pz) ^ r)) != 0 || !finite_bits(r);
  if (!__any_sync(__activemask(), varies)) {
    fu[c] = 0.0;
    fv[c] = 0.0;
    fw[c] = 0.0;
    return;
  }
  const double *ax = n12, *ay = n12 + n, *bx = n12 + 2 * n, *bz = nside, *ey = nside + n, *ez = nside + 2 * n;
  const double ku = (__ldg(pp + c + X) - __ldg(pp + c)) * p.dxi + (__ldg(ay + c) - __ldg(ay + c - Y)) * p.dyi +
                    (__ldg(bz + c) - __ldg(bz + c - Z)) * p.dzi;
  const double kv = (__ldg(ax + c) - __ldg(ax + c - X)) * p.dxi + (__ldg(pp + n + c + Y) - __ldg(pp + n + c)) * p.dyi +
                    (__ldg(ez + c) - __ldg(ez + c - Z)) * p.dzi;
  const double kw = (__ldg(bx + c) - __ldg(bx + c - X)) * p.dxi + (__ldg(ey + c) - __ldg(ey + c - Y)) * p.dyi +
                    (__ldg(pp + 2 * n + c + Z) - __ldg(pp + 2 * n + c)) * p.dzi;
  fu[c] = ku * (px - ph) * p.fx;
  fv[c] = kv * (py - ph) * p.fy;
  fw[c] = kw * (pz - ph) * p.fz;
}

void csf_fp64(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double rhol, double rhog,
              double sigma, const double* phi, double* fu, double* fv, double* fw, double* const* work,
              const int* skip) {
  CsfD p;
  p.dxi = dxinv;
  p.dyi = dyinv;
  p.dzi = dzinv;
  p.gx = 0.25 * dxinv;
  p.gy = 0.25 * dyinv;
  p.gz = 0.25 * dzinv;
  const double vs = std::sqrt(dxinv * dxinv + dyinv * dyinv + dzinv * dzinv) * 1.0e-30;
  p.vs2 = 2.0 * vs;
  p.vs8 = 8.0 * vs;
  p.big2 = p.vs2 * 1.0e12 * (p.vs2 * 1.0e12);
  p.big8 = p.vs8 * 1.0e12 * (p.vs8 * 1.0e12);
  const double st = 2.0 * sigma / (rhol + rhog);
  p.fx = -st * dxinv;
  p.fy = -st * dyinv;
  p.fz = -st * dzinv;
  double *G = work[0], *pp = work[1], *n12 = work[2], *nside = work[3];
  chain(s, tile_grid(g.ni + 3, g.nj + 3, g.nk + 3, 128), 128, k_csf_grad)(g, p, phi, G, skip);
  // planes per walk: the first costs 9 additions more; as many as leave a warp for each
  // of the 608 quarter SMs, 8 at most
  const long cols = (long)(g.ni + 2) * (g.nj + 2);
  int m = 1;
  while (m < 8 && cols * (g.nk + 2) >= 2L * m * 768 * 32) m *= 2;
  chain(s, tile_grid(g.ni + 2, g.nj + 2, (g.nk + 2 + m - 1) / m, 128), 128, k_csf_normals)(g, p, m, G, pp, n12, nside,
                                                                                           skip);
  chain(s, tile_grid(g.ni, g.nj, g.nk, 256), 256, k_csf_force)(g, p, phi, pp, n12, nside, fu, fv, fw, skip);
  count_launch(3);
}
}  // namespace

bool csf_supported(const Grid& g) { return g.ni % TX == 0 && g.nj % TY == 0; }

void csf_force(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double rhol, double rhog,
               double sigma, const double* phi, double* fu, double* fv, double* fw, int prec, double* const* work,
               const int* skip) {
  if (prec == 1)
    launch_csf<float>(s, g, dxinv, dyinv, dzinv, rhol, rhog, sigma, phi, fu, fv, fw, skip);
  else if (prec == 2)
    launch_csf<Pr>(s, g, dxinv, dyinv, dzinv, rhol, rhog, sigma, phi, fu, fv, fw, skip);
  else if (!work)
    set_status(FMF_ERR_ARG);
  else
    csf_fp64(s, g, dxinv, dyinv, dzinv, rhol, rhog, sigma, phi, fu, fv, fw, work, skip);
}

}  // namespace fused
}  // namespace fmf
