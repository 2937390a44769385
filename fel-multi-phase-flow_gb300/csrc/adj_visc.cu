// adj_visc.cu -- adjoint of the implicit viscous solve and of its coefficients
// (solu_sor4.f, cal_arith_coef_vis.f / cal_harm_coef_vis.f, cal_srcu.f), in the
// A/B/edge-viscosity form of fused_visc.cu.
//
// The forward solve iterates un <- G(un) (one outer iteration: 12 colour-pair
// sweeps, each followed by the wall/halo refresh) to its fixed point un*.  Its
// adjoint is the transposed fixed-point iteration  l <- lout + G'(un*)^T l  on the
// same sweep structure run backwards (each sweep transposed: the adjoint at the
// swept points is scattered to their 14 neighbours and cleared), followed by one
// more backward sweep that collects the gradients with respect to A, B, the edge
// viscosities, mu and the slip coefficients.  The forward states before each sweep
// of one cycle at the fixed point are replayed from un* (12 snapshots).
#include <algorithm>
#include <type_traits>

#include "../../include/fmf_capi.h"
#include "adj.cuh"
#include "fused.cuh"
#include "runtime.cuh"

namespace fmf {
namespace adj {

namespace {
struct VPa {
  double dx2, dy2, dz2, dxy, dxz, dyz;
};
VPa make_vpa(double dxi, double dyi, double dzi) {
  VPa p;
  p.dx2 = dxi * dxi;
  p.dy2 = dyi * dyi;
  p.dz2 = dzi * dzi;
  p.dxy = dxi * dyi;
  p.dxz = dxi * dzi;
  p.dyz = dyi * dzi;
  return p;
}
struct Arr3 {
  double* a[3];
};
struct CArr4 {
  const double* a[4];  // mu, exy, exz, eyz
};
struct Arr4 {
  double* a[4];
};
struct CArr3 {
  const double* a[3];
};

// The factors of visn of component COMP in the form of the forward sweeps: with S its own
// axis and, per transverse axis T with edge viscosity e and component F along T,
//   own (mu(S) q(S) + mu q(-S)) + sum_T k_T (e(-T) b(-T) + e b(T)),
//   b(T) = q(T) + r_T (F(S) - F(0)),  b(-T) = q(-T) + r_T (F(-T) - F(S-T)).
struct SwK {
  double own, k1, k2, r1, r2;
};
SwK make_swk(double dxi, double dyi, double dzi, int comp) {
  const double d[3] = {dxi, dyi, dzi};
  const double s = d[comp], a = d[comp == 0 ? 1 : 0], b = d[comp == 2 ? 1 : 2];
  return SwK{2.0 * s * s, a * a, b * b, s / a, s / b};
}
struct GradIn {
  const double *q0, *q1, *q2;  // the forward state before this sweep: own, T1's, T2's
  double *lA, *lB, *lmu, *le1, *le2;
};

// Transposed sweep of one colour pair: l at the swept points (OWN: with the adjoints of
// their x and z images, cleared; the wall rows of their columns hold none yet: within the
// component only the points of the wall row themselves scatter into those, after this, and
// before it the full transposed refresh cleared them) is scattered to their 14 neighbours
// (times A) and cleared.  blockIdx.z takes the planes of the first colour, then of the
// second.  Of the pair's points one at most reads a given point of another component
// (their four offsets have four parities in the two axes and one in the third, and the
// second colour has all three flipped), a given edge or a given mu: those adjoints are
// read, added to and stored; only the swept component's own neighbours are read by two and
// take atomics.
// GRAD: the gradients at the fixed point too: lB += l, lA += l visn(q), and those of mu and
// the edge viscosities.
// Bound by the latency of its one round of loads at these sizes and by the atomics: with
// all 14 as atomics, each point a thread for both colours and the full transposed refresh
// (8 us) before every pair, a pair took 13.7 + 8 us at 128x64x64; now 9.4, with the images
// 11; gradients in a kernel of their own 23 + 13.7, together 19.
template <int COMP, bool OWN, bool GRAD>
__global__ void __launch_bounds__(64, GRAD ? 10 : 16) k_pair_T(Grid g, SwK K, int pi, int pj, int pk, CArr4 cf,
                                                const double* __restrict__ A, Arr3 la, GradIn G) {
  after_previous();
  const bool h = (int)blockIdx.z >= g.nk / 2;
  const int i = (h ? 3 - pi : pi) + 2 * (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int j = (h ? 3 - pj : pj) + 2 * (int)(blockIdx.y * blockDim.y + threadIdx.y);
  const int k = (h ? 3 - pk : pk) + 2 * (int)(h ? blockIdx.z - g.nk / 2 : blockIdx.z);
  if (i > g.ni || j > (COMP == 1 ? g.nj - 1 : g.nj)) return;
  const long c = g.at(i, j, k), X = 1, Y = g.sy, Z = g.sz;
  const long S = COMP == 0 ? X : (COMP == 1 ? Y : Z), T1 = COMP == 0 ? Y : X, T2 = COMP == 2 ? Y : Z;
  double* l = la.a[COMP];
  double* f1 = la.a[COMP == 0 ? 1 : 0] + c;
  double* f2 = la.a[COMP == 2 ? 1 : 2] + c;
  const double* e1 = cf.a[COMP == 2 ? 2 : 1] + c;
  const double* e2 = cf.a[COMP == 0 ? 2 : 3] + c;
  double m = l[c];
  const double Ac = __ldg(A + c), m0 = __ldg(cf.a[0] + c), m1 = __ldg(cf.a[0] + c + S), e1n = __ldg(e1 - T1),
               e1p = __ldg(e1), e2n = __ldg(e2 - T2), e2p = __ldg(e2);
  const double a0 = f1[0], a1 = f1[S], a2 = f1[-T1], a3 = f1[S - T1];
  const double b0 = f2[0], b1 = f2[S], b2 = f2[-T2], b3 = f2[S - T2];
  if (OWN) {
    const bool hx = i <= 3 || i >= g.ni - 2, hz = k <= 3 || k >= g.nk - 2;
    const int ix = i <= 3 ? i + g.ni : i - g.ni, kx = k <= 3 ? k + g.nk : k - g.nk;
    if (hx || hz) {
      double *px = l + g.at(ix, j, k), *pz = l + g.at(i, j, kx), *pxz = l + g.at(ix, j, kx);
      const double vx = hx ? *px : 0.0, vz = hz ? *pz : 0.0, vxz = hx && hz ? *pxz : 0.0;
      m += (vx + vz) + vxz;
      if (hx) *px = 0.0;
      if (hz) *pz = 0.0;
      if (hx && hz) *pxz = 0.0;
      l[c] = 0.0;  // also where the images cancel it
    }
  }
  if (m == 0.0) return;
  l[c] = 0.0;
  const double ma = m * Ac, x1 = ma * K.k1, x2 = ma * K.k2;
  if (GRAD) {
    const double *q = G.q0 + c, *p1 = G.q1 + c, *p2 = G.q2 + c;
    const double qn = K.own * q[-S], qp = K.own * q[S];
    const double d1n = q[-T1] + K.r1 * (p1[-T1] - p1[S - T1]), d1p = q[T1] + K.r1 * (p1[S] - p1[0]);
    const double d2n = q[-T2] + K.r2 * (p2[-T2] - p2[S - T2]), d2p = q[T2] + K.r2 * (p2[S] - p2[0]);
    G.lB[c] += m;
    G.lA[c] += m * (m0 * qn + m1 * qp + K.k1 * (e1n * d1n + e1p * d1p) + K.k2 * (e2n * d2n + e2p * d2p));
    G.lmu[c] += ma * qn;
    G.lmu[c + S] += ma * qp;
    G.le1[c - T1] += x1 * d1n;
    G.le1[c] += x1 * d1p;
    G.le2[c - T2] += x2 * d2n;
    G.le2[c] += x2 * d2p;
  }
  const double xo = ma * K.own, n1 = x1 * e1n, w1 = x1 * e1p, n2 = x2 * e2n, w2 = x2 * e2p;
  aadd(l + c - S, xo * m0);
  aadd(l + c + S, xo * m1);
  aadd(l + c - T1, n1);
  aadd(l + c + T1, w1);
  aadd(l + c - T2, n2);
  aadd(l + c + T2, w2);
  f1[0] = a0 - K.r1 * w1;
  f1[S] = a1 + K.r1 * w1;
  f1[-T1] = a2 + K.r1 * n1;
  f1[S - T1] = a3 - K.r1 * n1;
  f2[0] = b0 - K.r2 * w2;
  f2[S] = b1 + K.r2 * w2;
  f2[-T2] = b2 + K.r2 * n2;
  f2[S - T2] = b3 - K.r2 * n2;
}
const int kPi[4] = {1, 1, 1, 2}, kPj[4] = {1, 1, 2, 1}, kPk[4] = {1, 2, 1, 1};
__global__ void k_copy3(long n, CArr3 a, double* __restrict__ b) {
  after_previous();
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    b[t] = a.a[0][t];
    b[t + n] = a.a[1][t];
    b[t + 2 * n] = a.a[2][t];
  }
}
// l holds G^T l_old, fb the feedback term l_old - lout: part[block] = sum of
// (l - fb)^2 = |l_new - l_old|^2, part[kParts + block] = sum of l^2, fb = l, l += lout
constexpr int kParts = 512;
__global__ void __launch_bounds__(256) k_add_diff3(long n, Arr3 l, CArr3 o, double* part, double* fb) {
  after_previous();
  __shared__ double sh[2][256];
  double acc = 0.0, acf = 0.0;
  const long step = kParts * 256L;
  for (int c = 0; c < 3; ++c) {
    double *lc = l.a[c], *fc = fb + c * n;
    const double* oc = o.a[c];
    for (long t0 = blockIdx.x * 256L + threadIdx.x; t0 < n; t0 += 4 * step) {
      double f[4], p[4], q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const long t = t0 + u * step;
        const bool on = t < n;
        f[u] = on ? lc[t] : 0.0;
        p[u] = on ? fc[t] : 0.0;
        q[u] = on ? oc[t] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const long t = t0 + u * step;
        if (t >= n) break;
        fc[t] = f[u];
        lc[t] = f[u] + q[u];
        const double d = f[u] - p[u];
        acf += f[u] * f[u];
        acc += d * d;
      }
    }
  }
  sh[0][threadIdx.x] = acc;
  sh[1][threadIdx.x] = acf;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st) {
      sh[0][threadIdx.x] += sh[0][threadIdx.x + st];
      sh[1][threadIdx.x] += sh[1][threadIdx.x + st];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[blockIdx.x] = sh[0][0];
    part[kParts + blockIdx.x] = sh[1][0];
  }
}
// The start: fbo = 0 (no fb), fb (the warm start) or 2 fb - fb2 (fb2 the feedback term one
// solve earlier: linear extrapolation in time; may be fbo itself), l = lout + fbo
__global__ void k_start3(long n, Arr3 l, CArr3 o, const double* fb, const double* fb2, double* fbo) {
  after_previous();
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
    for (int c = 0; c < 3; ++c) {
      double f = 0.0;
      if (fb) {
        f = fb[t + c * n];
        if (fb2) f += f - fb2[t + c * n];
      }
      fbo[t + c * n] = f;
      l.a[c][t] = o.a[c][t] + f;
    }
}
// out[0] = sum of part[0..n), out[1] = sum of part[kParts..kParts+n)
__global__ void k_sum_small(const double* part, int n, double* out) {
  after_previous();
  __shared__ double sh[2][256];
  double acc = 0.0, acf = 0.0;
  for (int t = threadIdx.x; t < n; t += 256) {
    acc += part[t];
    acf += part[kParts + t];
  }
  sh[0][threadIdx.x] = acc;
  sh[1][threadIdx.x] = acf;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st) {
      sh[0][threadIdx.x] += sh[0][threadIdx.x + st];
      sh[1][threadIdx.x] += sh[1][threadIdx.x + st];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = sh[0][0];
    out[1] = sh[1][0];
  }
}
}  // namespace

// Momentum factors of k_src_ab: per component T = 1/(r/dt + ap/2), A = T/2,
// B = rs T with r the 4-point density mean, ap the 6-term viscous diagonal and rs
// = r*(u/dt - 1.5 adv + 0.5 advo + 0.5 fst + 0.5 fstn + grav) - prs + 0.5 vis.
void src_ab_T(cudaStream_t s, const Grid& g, double dxi, double dyi, double dzi, double dt, double grvb,
              double grvp, const SrcArgs& a, const double* const* lAB, const SrcAdj& l) {
  const Grid G = g;
  const VPa p = make_vpa(dxi, dyi, dzi);
  const double dtinv = 1.0 / dt;
  const SrcArgs A = a;
  const SrcAdj L = l;
  const double *lA0 = lAB[0], *lB0 = lAB[1], *lA1 = lAB[2], *lB1 = lAB[3], *lA2 = lAB[4], *lB2 = lAB[5];
  range3(s, 1, g.ni, 1, g.nj, 1, g.nk, [=] __device__(int i, int j, int k) {
    const long X = 1, Y = G.sy, Z = G.sz;
    const long c = G.at(i, j, k);
    const double* mu = A.mu;
    const double *exy = A.E[0], *exz = A.E[1], *eyz = A.E[2];
    // q: component, o: its unit offset, lAq/lBq: adjoints; ap terms (array, index, factor)
    auto comp = [&](int q, long o, double lAq, double lBq, const double* vel, double grav, const double* ea,
                    long ia0, long ia1, double fa, const double* eb, long ib0, long ib1, double fb, double fm) {
      if (lAq == 0.0 && lBq == 0.0) return;
      const double r = (A.rho[c] + A.rho[c + o] + A.rhon[c] + A.rhon[c + o]) * 0.25;
      const double ap = fa * ea[ia0] + fb * eb[ib0] + fm * mu[c] * 2.0 + fm * mu[c + o] * 2.0 + fa * ea[ia1] +
                        fb * eb[ib1];
      const double Dd = r * dtinv + ap * 0.5, T = 1.0 / Dd;
      const double ex = vel[c] * dtinv - A.adv[q][c] * 1.5 + A.advo[q][c] * 0.5 + A.fst[q][c] * 0.5 +
                        A.fstn[q][c] * 0.5 + grav;
      const double rs = r * ex - A.prs[q][c] + A.vis[q][c] * 0.5;
      const double lT = 0.5 * lAq + rs * lBq, lrs = T * lBq;
      const double lD = -T * T * lT;
      const double lr = dtinv * lD + lrs * ex, lap = 0.5 * lD;
      aadd(L.u[q] + c, lrs * r * dtinv);
      L.adv[q][c] += -1.5 * r * lrs;
      L.advo[q][c] += 0.5 * r * lrs;
      L.fst[q][c] += 0.5 * r * lrs;
      L.fstn[q][c] += 0.5 * r * lrs;
      L.prs[q][c] += -lrs;
      L.vis[q][c] += 0.5 * lrs;
      aadd(L.rho + c, 0.25 * lr);
      aadd(L.rho + c + o, 0.25 * lr);
      aadd(L.rhon + c, 0.25 * lr);
      aadd(L.rhon + c + o, 0.25 * lr);
      aadd(L.ea[q] + ia0, fa * lap);
      aadd(L.ea[q] + ia1, fa * lap);
      aadd(L.eb[q] + ib0, fb * lap);
      aadd(L.eb[q] + ib1, fb * lap);
      aadd(L.mu + c, 2.0 * fm * lap);
      aadd(L.mu + c + o, 2.0 * fm * lap);
    };
    // u: ap = dz2 exz(-Z) + dy2 exy(-Y) + 2dx2 mu + 2dx2 mu(+X) + dy2 exy + dz2 exz
    comp(0, X, lA0[c], lB0[c], A.u, grvb, exz, c - Z, c, p.dz2, exy, c - Y, c, p.dy2, p.dx2);
    // v: dz2 eyz(-Z) + 2dy2 mu + dx2 exy(-X) + dx2 exy + 2dy2 mu(+Y) + dz2 eyz
    if (j <= G.nj - 1) comp(1, Y, lA1[c], lB1[c], A.v, grvp, eyz, c - Z, c, p.dz2, exy, c - X, c, p.dx2, p.dy2);
    // w: 2dz2 mu + dy2 eyz(-Y) + dx2 exz(-X) + dx2 exz + dy2 eyz + 2dz2 mu(+Z)
    comp(2, Z, lA2[c], lB2[c], A.w, 0.0, eyz, c - Y, c, p.dy2, exz, c - X, c, p.dx2, p.dz2);
  });
}

// k_edges: E(c) = 4-cell mean of mu over i,j,k in 0..n (arithmetic or harmonic)
void edges_T(cudaStream_t s, const Grid& g, int harmonic, const double* mu, const double* const* lE, double* lmu) {
  const Grid G = g;
  const double *l0 = lE[0], *l1 = lE[1], *l2 = lE[2];
  range3(s, 0, g.ni, 0, g.nj, 0, g.nk, [=] __device__(int i, int j, int k) {
    const long X = 1, Y = G.sy, Z = G.sz;
    const long c = G.at(i, j, k);
    auto one = [&](double L, long a, long b, long d, long e) {
      if (L == 0.0) return;
      if (!harmonic) {
        aadd(lmu + a, 0.25 * L);
        aadd(lmu + b, 0.25 * L);
        aadd(lmu + d, 0.25 * L);
        aadd(lmu + e, 0.25 * L);
      } else {
        const double sm = 1.0 / mu[a] + 1.0 / mu[b] + 1.0 / mu[d] + 1.0 / mu[e];
        const double f = 4.0 / (sm * sm) * L;  // d(4/sm)/d(mu_p) = 4/sm^2 / mu_p^2
        aadd(lmu + a, f / (mu[a] * mu[a]));
        aadd(lmu + b, f / (mu[b] * mu[b]));
        aadd(lmu + d, f / (mu[d] * mu[d]));
        aadd(lmu + e, f / (mu[e] * mu[e]));
      }
    };
    one(l0[c], c, c + X, c + Y, c + X + Y);
    one(l1[c], c, c + X, c + Z, c + X + Z);
    one(l2[c], c, c + Y, c + Z, c + Y + Z);
  });
}

// After a component's first pair the forward cycle changes that component alone, so the
// later pairs' states share the other two arrays (where the grid allows the one-pass
// refresh): 24 array copies, not 36.
namespace {
CArr3 replay_state(const Grid& g, const double* snaps, int comp, int pr) {
  const bool share = pr > 1 && fused::one_pass_refresh(g);
  CArr3 q;
  for (int c = 0; c < 3; ++c) q.a[c] = snaps + (3L * (4 * comp + (share && c != comp ? 1 : pr)) + c) * g.n;
  return q;
}
}  // namespace
void sor_replay(cudaStream_t s, const Grid& g, double dxi, double dyi, double dzi, int harmonic, const double* mu,
                double* const* E, double* const* AB, double uwall, const double* wallc, const double* const* ustar,
                double* snaps, double* part) {
  const long n = g.n;
  double* q[3] = {snaps + 36 * n, snaps + 37 * n, snaps + 38 * n};  // running state
  const CArr3 run{{q[0], q[1], q[2]}};
  chain(s, 608, 256, k_copy3)(n, CArr3{{ustar[0], ustar[1], ustar[2]}}, q[0]);
  count_launch();
  fused::sor_iteration(s, g, dxi, dyi, dzi, harmonic, mu, E, AB, uwall, wallc, q[0], q[1], q[2], part, nullptr,
                       fused::FlatFluid(),
                       [&](int comp, int pr) {
                         const CArr3 st = replay_state(g, snaps, comp, pr);
                         double* own = snaps + (3L * (4 * comp + pr) + comp) * n;
                         if (st.a[(comp + 1) % 3] == snaps + (3L * (4 * comp + pr) + (comp + 1) % 3) * n) {
                           chain(s, 608, 256, k_copy3)(n, run, snaps + 3L * (4 * comp + pr) * n);
                           count_launch();
                         } else {
                           FMF_CUDA(cudaMemcpyAsync(own, q[comp], sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
                         }
                       });
}

cudaGraphExec_t cached_graph(cudaStream_t s, GraphCache* cache, const std::vector<const void*>& key,
                             const std::function<void()>& body, long long* per_launch) {
  auto itc = cache->find(key);
  if (itc != cache->end()) {
    *per_launch = itc->second.second;
    return itc->second.first;
  }
  *per_launch = 0;
  cudaGraphExec_t exec = nullptr;
  cudaGraph_t graph = nullptr;
  const long long l0 = launches();
  if (!FMF_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed))) return nullptr;
  body();
  // the captured launches did not run: they are counted when the graph is replayed
  const long long captured = launches() - l0;
  count_launch((int)-captured);
  if (FMF_CUDA(cudaStreamEndCapture(s, &graph)) && FMF_CUDA(cudaGraphInstantiate(&exec, graph, 0))) {
    *per_launch = captured;
    (*cache)[key] = {exec, captured};
  } else {
    exec = nullptr;
  }
  if (graph) cudaGraphDestroy(graph);
  return exec;
}

int sor_T(cudaStream_t s, const Grid& g, double dxi, double dyi, double dzi, const double* mu, double* const* E,
          double* const* AB, double uwall, const double* wallc, const double* const* ustar, const double* snaps,
          const double* const* lout, double* const* lam, double* const* lAB, double* lmu, double* const* lE,
          double* lwc, double tol, int maxit, double* work, double* host_norm, GraphCache* cache, double* fb,
          double* fb_norm, const double* fb_prev, double* fb_out) {
  const long n = g.n;
  const CArr4 cf{{mu, E[0], E[1], E[2]}};
  double* part = work;             // 2 kParts
  double* nrm = work + 2 * kParts; // 2 doubles
  const Arr3 L3{{lam[0], lam[1], lam[2]}};
  const CArr3 O3{{lout[0], lout[1], lout[2]}};
  // l = lout, or lout plus the previous solve's feedback term
  const bool warm = *fb_norm > 0.0;
  chain(s, 608, 256, k_start3)(n, L3, O3, warm ? fb : nullptr, fb_prev, fb_out);
  count_launch();
  // The 12 sweeps backwards, the refresh after each transposed before it.  The forward
  // cycle after a component's second to fourth pair changes that component's ghosts
  // alone, which the swept points gather (OWN); the full refresh is after the first.
  // lout holds nothing in the wall rows (a transposed refresh has gone over it).
  const bool one_pass = fused::one_pass_refresh(g);
  const int bx = std::min(32, g.ni / 2), by = 64 / bx;
  const dim3 blk(bx, by), grd((g.ni / 2 + bx - 1) / bx, (g.nj / 2 + by - 1) / by, g.nk);
  auto backward_cycle = [&](auto grad) {
    constexpr bool GR = decltype(grad)::value;
    for (int comp = 2; comp >= 0; --comp) {
      const SwK K = make_swk(dxi, dyi, dzi, comp);
      for (int pr = 3; pr >= 0; --pr) {
        GradIn G{};
        if (GR) {
          const CArr3 q = replay_state(g, snaps, comp, pr);
          const int t1 = comp == 0 ? 1 : 0, t2 = comp == 2 ? 1 : 2;
          G = GradIn{q.a[comp],         q.a[t1], q.a[t2],                lAB[2 * comp],
                     lAB[2 * comp + 1], lmu,     lE[comp == 2 ? 1 : 0], lE[comp == 0 ? 1 : 2]};
        }
        const bool own = one_pass && pr > 0;
        // the slip-coefficient adjoint only in the gradient pass
        if (!own) wall_halo_T(s, g, 1 << comp, uwall, wallc, ustar[0], ustar[2], lam[0], lam[1], lam[2], GR ? lwc : nullptr);
        auto run = [&](auto fn) {
          chain(s, grd, blk, fn)(g, K, kPi[pr], kPj[pr], kPk[pr], cf, AB[2 * comp], L3, G);
          count_launch();
        };
        if (comp == 0) own ? run(k_pair_T<0, true, GR>) : run(k_pair_T<0, false, GR>);
        else if (comp == 1) own ? run(k_pair_T<1, true, GR>) : run(k_pair_T<1, false, GR>);
        else own ? run(k_pair_T<2, true, GR>) : run(k_pair_T<2, false, GR>);
      }
    }
  };
  // one iteration l <- lout + G^T l, |l_new - l_old|^2 and |G^T l|^2 into nrm and
  // the feedback term G^T l into fb: 17 kernels, replayed as a CUDA graph (one per
  // set of buffers)
  auto iteration = [&]() {
    backward_cycle(std::false_type());
    chain(s, kParts, 256, k_add_diff3)(n, L3, O3, part, fb_out);
    chain(s, 1, 256, k_sum_small)(part, kParts, nrm);
    count_launch(2);
  };
  long long per_launch = 0;
  cudaGraphExec_t exec =
      cache ? cached_graph(s, cache,
                           {lam[0], lam[1], lam[2], lout[0], lout[1], lout[2], mu, E[0], E[1], E[2], AB[0], AB[2],
                            AB[4], wallc, ustar[0], ustar[2], work, fb_out},
                           iteration, &per_launch)
            : nullptr;
  // The stop rule's scale: the change of the first iteration from l = lout (the
  // size of the feedback term G^T lout); from a warm start, the previous solve's
  // feedback norm, the same quantity one step later.
  double n0 = warm ? *fb_norm : -1.0;
  int it = 0;
  for (it = 0; it < maxit; ++it) {
    if (exec) {
      FMF_CUDA(cudaGraphLaunch(exec, s));
      count_launch((int)per_launch);
    } else {
      iteration();
    }
    FMF_CUDA(cudaMemcpyAsync(host_norm, nrm, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    FMF_CUDA(cudaStreamSynchronize(s));
    const double d = std::sqrt(host_norm[0]);
    if (!std::isfinite(d) || !std::isfinite(host_norm[1])) {
      set_status(FMF_ERR_NONFINITE);
      break;
    }
    *fb_norm = std::sqrt(host_norm[1]);
    if (n0 < 0.0) n0 = d;
    if (!(d > tol * (n0 + 1e-300))) break;
  }
  // gradient pass at the converged adjoint
  backward_cycle(std::true_type());
  return it + 1;
}

}  // namespace adj
}  // namespace fmf
