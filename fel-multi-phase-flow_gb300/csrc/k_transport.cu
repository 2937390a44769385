// k_transport.cu -- the parts of the fused step's transport whose roundings the reference
// fixes (compiled without multiply-add contraction, operations in its order): the
// conservative update (solphi_mthinc2.f), the volume fix (solphi_mthinc3.f:121-160), the
// sum over bubbles (summation.f), the mixture properties (cal_arith_mean.f) and the
// scalar halos.
//
// Away from the interface phi is exactly 0 or 1 and the FP64 operations give zeros or
// the value they were given: there a warp takes that result from the bits of what it
// read, without the arithmetic (the FP64 pipe takes 64 cycles per warp instruction).
#include "bits.cuh"
#include "fused.cuh"
#include "ops.cuh"
#include "recip.cuh"

namespace fmf {
namespace fused {

namespace {
// solphi_mthinc2.f:19-45: phin = clip(phi (1 + dt div u) + the flux differences) on the
// interior.  In a warp where phi and the fluxes are 0 that is 0 (k_classify's flux of a
// velocity that is not finite is not 0); where phi is 1 and every flux is that of phi = 1
// (vel (dt dxinv), as k_classify forms it) it is 1 but for the roundings, and for a velocity
// that is not finite the clip's 1: 6 FP64 operations to see it, not 17.  (The snap takes the
// roundings of such cells away outside the band; inside it a cell is a few units in the last
// place nearer to 1 here than the operations one by one leave it.)
// 139 -> 66 us for a drop at 256x128x128.
__global__ void __launch_bounds__(256) k_advance(Grid g, double dxi, double dyi, double dzi, double dt, double cx,
                                                 double cy, double cz,
                                                 const double* __restrict__ u,
                                                 const double* __restrict__ v, const double* __restrict__ w,
                                                 const double* __restrict__ fx, const double* __restrict__ fy,
                                                 const double* __restrict__ fz, const double* __restrict__ phi,
                                                 double* __restrict__ phin) {
  after_previous();
  const Tile T = warp_tile(g.ni);
  const int i = 1 + T.x, j = 1 + T.y;
  if (i > g.ni || j > g.nj) return;
  const long X = 1, Y = g.sy, Z = g.sz;
  const long c = g.at(i, j, 1 + (int)blockIdx.z);
  const double q = __ldg(phi + c);
  const double f0 = __ldg(fx + c - X), f1 = __ldg(fx + c), f2 = __ldg(fy + c - Y), f3 = __ldg(fy + c),
               f4 = __ldg(fz + c - Z), f5 = __ldg(fz + c);
  if (!__any_sync(__activemask(), (mag(q) | mag(f0) | mag(f1) | mag(f2) | mag(f3) | mag(f4) | mag(f5)) != 0)) {
    phin[c] = 0.0;
    return;
  }
  const double ue = __ldg(u + c), uw = __ldg(u + c - X), vn = __ldg(v + c), vs = __ldg(v + c - Y), wt = __ldg(w + c),
               wb = __ldg(w + c - Z);
  bool pure = raw(q) == kOneBits;
  if (__all_sync(__activemask(), pure)) {
    auto differs = [](double f, double p) { return (unsigned long long)(raw(f) ^ raw(p)); };
    pure = (differs(f0, uw * cx) | differs(f1, ue * cx) | differs(f2, vs * cy) | differs(f3, vn * cy) |
            differs(f4, wb * cz) | differs(f5, wt * cz)) == 0;
    if (__all_sync(__activemask(), pure)) {
      phin[c] = 1.0;
      return;
    }
  }
  const double div = (ue - uw) * dxi + (vn - vs) * dyi + (wt - wb) * dzi;
  phin[c] = clip01(q * (1.0 + dt * div) + f0 - f1 + f2 - f3 + f4 - f5);
}

// solphi_mthinc3.f:138-160: phin += offset phin^2 (1 - phin), clipped, over the interior
// (exactly 0 and 1 keep their values); the offset (sums[2] >= 0: the Newton-Raphson
// reciprocal, no division) formed once per block.  phin0, the sum over the one bubble
// (summation.f:222-264), takes the same values.
__global__ void __launch_bounds__(256) k_offset(Grid g, const double* __restrict__ sums, double* __restrict__ phin,
                                                double* __restrict__ phin0) {
  after_previous();
  __shared__ double off;
  const Tile T = warp_tile(g.ni);
  const int i = 1 + T.x, j = 1 + T.y;
  const int k = 1 + (int)blockIdx.z;
  const bool in = i <= g.ni && j <= g.nj;
  const long c = in ? g.at(i, j, k) : 0;
  double p = in ? phin[c] : 0.0;  // in flight while the offset is formed
  const long long pb = raw(p);
  const bool between = pb != 0 && pb != kOneBits;
  if (__syncthreads_or(between)) {
    if (threadIdx.x == 0) off = (sums[0] - sums[1]) * recip_nr(sums[2] + 1.0e-99);
    __syncthreads();
    if (between) p = clip01(p + off * (p * p) * (1.0 - p));
  }
  if (!in) return;
  if (between) phin[c] = p;
  phin0[c] = p;
}

// The four cal_arith_mean calls of main.f90:526-529 (cal_arith_mean.f:13-27) in one pass:
// rho, rhon from (rhol, rhog) and rmu, rmun from (rmul, rmug) over phi0 and phin0; two
// points per thread per pass so that four loads are in flight.  Where phi is 0 or 1 the
// means are the fluids' own values.
struct Mix {
  double rl, rg, ml, mg;
  __device__ __forceinline__ void operator()(double a, double* rho, double* mu) const {
    const long long b = raw(a);
    if (b == 0 || b == kOneBits) {
      *rho = b ? rg : rl;
      *mu = b ? mg : ml;
    } else {
      const double d = 1.0 - a;
      *rho = rl * d + rg * a;
      *mu = ml * d + mg * a;
    }
  }
};
__global__ void __launch_bounds__(256) k_means4(long n, const double* __restrict__ p0, const double* __restrict__ p1,
                                                Mix mix, double* __restrict__ rho, double* __restrict__ rhon,
                                                double* __restrict__ rmu, double* __restrict__ rmun) {
  after_previous();
  const long stride = (long)gridDim.x * blockDim.x;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += 2 * stride) {
    const long t2 = t + stride;
    const bool two = t2 < n;
    const double a = p0[t], b = p1[t];
    const double a2 = two ? p0[t2] : 0.0, b2 = two ? p1[t2] : 0.0;
    mix(a, rho + t, rmu + t);
    mix(b, rhon + t, rmun + t);
    if (two) {
      mix(a2, rho + t2, rmu + t2);
      mix(b2, rhon + t2, rmun + t2);
    }
  }
}

// The x and z halos of q (bnd_periodic.f:173-205) and, WALLS, the reflected wall rows
// (bnd_neumann.f:222-252) in one pass: composed, every halo point holds the value of one
// interior point (of one point of its row, without WALLS), which no thread writes.
template <bool WALLS>
__global__ void __launch_bounds__(256) k_halos(Grid g, long nx, long nz, double* __restrict__ q) {
  after_previous();
  const int NI = g.ni, NJ = g.nj, NK = g.nk;
  auto wrap = [](int i, int n) { return i < 1 ? i + n : (i > n ? i - n : i); };
  auto row = [&](int j) { return !WALLS ? j : (j < 1 ? 1 - j : (j > NJ ? 2 * NJ + 1 - j : j)); };
  auto slot = [](int t, int n) { return t < 3 ? t - 2 : n + t - 2; };  // 0..5 -> -2, -1, 0, n+1, n+2, n+3
  long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  int i, j, k;
  if (t < nx) {  // x halos of every (j, k)
    i = slot((int)(t % 6), NI);
    t /= 6;
    j = (int)(t % (NJ + 6)) - 2;
    k = (int)(t / (NJ + 6)) - 2;
  } else if ((t -= nx) < nz) {  // z halos of the interior columns
    i = 1 + (int)(t % NI);
    t /= NI;
    j = (int)(t % (NJ + 6)) - 2;
    k = slot((int)(t / (NJ + 6)), NK);
  } else if (WALLS && (t -= nz) < 6L * NI * NK) {  // wall rows of the interior columns
    i = 1 + (int)(t % NI);
    t /= NI;
    k = 1 + (int)(t % NK);
    j = slot((int)(t / NK), NJ);
  } else {
    return;
  }
  q[g.at(i, j, k)] = q[g.at(wrap(i, NI), row(j), wrap(k, NK))];
}
template <bool WALLS>
void halos(cudaStream_t s, const Grid& g, double* q) {
  const long nx = 6L * (g.nj + 6) * (g.nk + 6), nz = 6L * g.ni * (g.nj + 6);
  const long n = nx + nz + (WALLS ? 6L * g.ni * g.nk : 0);
  chain(s, (unsigned)((n + 255) / 256), 256, k_halos<WALLS>)(g, nx, nz, q);
  count_launch();
}
}  // namespace

void halo_periodic(cudaStream_t s, const Grid& g, double* q) { halos<false>(s, g, q); }
void halo_neumann_periodic(cudaStream_t s, const Grid& g, double* q) { halos<true>(s, g, q); }

void mthinc_advance(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double dt,
                    const double* u, const double* v, const double* w, const double* fx, const double* fy,
                    const double* fz, const double* phi, double* phin) {
  chain(s, tile_grid(g.ni, g.nj, g.nk, 256), 256, k_advance)(g, dxinv, dyinv, dzinv, dt, dt * dxinv, dt * dyinv,
                                                          dt * dzinv, u, v, w, fx, fy, fz, phi, phin);
  count_launch();
}

void mthinc_volume_fix(cudaStream_t s, const Grid& g, double dxinv, double dyinv, double dzinv, double bet,
                       const double* gx, const double* gy, const double* gz, const double* phi, double* phin,
                       double* phin0, double* sums) {
  const Grid G = g;
  mthinc_snap(s, g, dxinv, dyinv, dzinv, bet, gx, gy, gz, phin);
  reduce_interior<3>(
      s, g,
      [=] __device__(int i, int j, int k, double* r) {
        const long c = G.at(i, j, k);
        const double p = phin[c];
        const long long b = raw(p);
        r[0] = phi[c];
        r[1] = p;
        r[2] = b == 0 || b == kOneBits ? 0.0 : p * p * (1.0 - p);
      },
      sums);
  chain(s, tile_grid(g.ni, g.nj, g.nk, 256), 256, k_offset)(g, sums, phin, phin0);
  count_launch();
}

void mixture_means(cudaStream_t s, const Grid& g, const double* phi0, const double* phin0, double rhol, double rhog,
                   double rmul, double rmug, double* rho, double* rhon, double* rmu, double* rmun) {
  chain(s, 152 * 8, 256, k_means4)(g.n, phi0, phin0, Mix{rhol, rhog, rmul, rmug}, rho, rhon, rmu, rmun);
  count_launch();
}

}  // namespace fused
}  // namespace fmf
