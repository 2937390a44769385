// fmf::adj::sor_T on host arrays, for tests/test_gpu_adjoint_images.py: the transposed
// viscous solve of one adjoint, no graphs, its gradients copied back.
#include <vector>

#include "adj.cuh"

// in: mu, E (3), AB (6), lout (3), ustar (3) and snaps (39) of n doubles each, then wallc;
// out: lAB (6), lmu, lE (3) of n doubles each.  Returns the CUDA status.
extern "C" int sor_T_check(int ni, int nj, int nk, const double* in, double* out) {
  const fmf::Grid g(ni, nj, nk);
  const long n = g.n, nwc = 4L * (nk + 6) * (ni + 6), nin = 55 * n + nwc, nwork = 10 * n + 6 * n + 3 * n + nwc + 2048;
  double *d = nullptr, *w = nullptr, *host_norm = nullptr;
  if (cudaMalloc(&d, sizeof(double) * nin) != cudaSuccess || cudaMalloc(&w, sizeof(double) * nwork) != cudaSuccess ||
      cudaMallocHost(&host_norm, 2 * sizeof(double)) != cudaSuccess)
    return -1;
  cudaMemcpy(d, in, sizeof(double) * nin, cudaMemcpyHostToDevice);
  cudaMemset(w, 0, sizeof(double) * nwork);
  double *mu = d, *E[3], *AB[6], *lout[3], *ustar[3], *snaps = d + 16 * n, *wallc = d + 55 * n;
  for (int q = 0; q < 3; ++q) {
    E[q] = d + (1 + q) * n;
    lout[q] = d + (10 + q) * n;
    ustar[q] = d + (13 + q) * n;
  }
  for (int q = 0; q < 6; ++q) AB[q] = d + (4 + q) * n;
  double *lAB[6], *lmu = w + 6 * n, *lE[3], *lam[3], *fb = w + 13 * n, *fb2 = w + 16 * n, *lwc = w + 19 * n;
  for (int q = 0; q < 6; ++q) lAB[q] = w + q * n;
  for (int q = 0; q < 3; ++q) {
    lE[q] = w + (7 + q) * n;
    lam[q] = w + (10 + q) * n;
  }
  double norm = 0.0;
  cudaStream_t s;
  cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  cudaDeviceSynchronize();
  fmf::adj::sor_T(s, g, (double)ni, (double)nj, (double)nk, mu, E, AB, 0.5, wallc, ustar, snaps, lout, lam, lAB, lmu, lE,
                  lwc, 1e-6, 4, lwc + nwc, host_norm, nullptr, fb, &norm, nullptr, fb2);
  const cudaError_t e = cudaStreamSynchronize(s);
  cudaMemcpy(out, w, sizeof(double) * 10 * n, cudaMemcpyDeviceToHost);
  cudaStreamDestroy(s);
  cudaFree(d);
  cudaFree(w);
  cudaFreeHost(host_norm);
  return (int)e;
}
