// Launches of fft_setup.cuh and the khat / potential of a disk on the tensor-core products.
#include <vector>

#include "fft_setup.cuh"
#include "kernels.h"

namespace dg {
namespace setup {

static bool make_plan(int n, Plan *pl) {
  pl->n = n;
  pl->n4 = pl->n2 = pl->n3 = pl->n5 = 0;
  int m = n;
  while (m % 4 == 0) { pl->n4++; m /= 4; }
  while (m % 2 == 0) { pl->n2++; m /= 2; }
  while (m % 3 == 0) { pl->n3++; m /= 3; }
  while (m % 5 == 0) { pl->n5++; m /= 5; }
  return m == 1 && n >= 1;
}

struct FftShape {
  int E, nb, threads;
  size_t smem;
};

template <typename V>
static FftShape fft_shape(int n, int count) {
  // Prefer 256 threads and 8 elements per thread; shrink nb to fill >= 2 waves of SMs.
  FftShape s;
  s.E = 8;
  s.threads = 256;
  if (n > s.E * s.threads) {
    s.threads = (n + s.E - 1) / s.E;
    s.threads = ((s.threads + 31) / 32) * 32;
    if (s.threads > 1024) s.threads = 1024;  // n <= 8192
  }
  s.nb = (s.E * s.threads) / n;
  if (s.nb < 1) s.nb = 1;
  int want = 2 * sm_count();
  while (s.nb > 1 && (count + s.nb - 1) / s.nb < want) s.nb /= 2;
  s.smem = (size_t)s.nb * n * sizeof(V);
  return s;
}

// (for each handle: the limit belongs to the device)
static cudaError_t prepare_kernels() {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const void *fns[] = {(const void *)k_phi_fwd<double, 8>, (const void *)k_u_conv<double, 8>,
                       (const void *)k_phi_inv<double, 8>};
  for (const void *f : fns) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

static cudaError_t phi_fwd(const double *src, int nrows, const double *rowscale, const Gravity &g, cudaStream_t st) {
  FftShape s = fft_shape<double2>(g.Nphi, (nrows + 1) / 2);
  const int blocks = (nrows + 2 * s.nb - 1) / (2 * s.nb);
  k_phi_fwd<double, 8><<<blocks, s.threads, s.smem, st>>>(src, nrows, g.Nphi, rowscale, g.W, 2 * g.Nu, g.phi, g.roots,
                                                          s.nb);
  return cudaGetLastError();
}

static cudaError_t u_conv(const Gravity &g, int nin, int nout, const double2 *khat, double2 *kout, cudaStream_t st) {
  const int Nc = g.Nphi / 2 + 1;
  FftShape s = fft_shape<double2>(g.u.n, Nc);
  k_u_conv<double, 8><<<(Nc + s.nb - 1) / s.nb, s.threads, s.smem, st>>>(g.W, 2 * g.Nu, Nc, nin, nout, g.u,
                                                                         g.roots + g.Nphi, khat, kout, s.nb);
  return cudaGetLastError();
}

cudaError_t build(int Nu, int Nphi, Gravity *g) {
  g->Nu = Nu;
  g->Nphi = Nphi;
  if (!make_plan(Nphi, &g->phi) || !make_plan(2 * Nu, &g->u)) return cudaErrorInvalidValue;
  std::vector<double2> r((size_t)Nphi + 2 * Nu);
  auto fill = [&](double2 *t, int n) {
    for (int k = 0; k < n; ++k) {
      const long double a = 2.0L * 3.141592653589793238462643383279502884L * (long double)k / (long double)n;
      t[k] = make_double2((double)cosl(a), (double)-sinl(a));
    }
  };
  fill(r.data(), Nphi);
  fill(r.data() + Nphi, 2 * Nu);
  const size_t spec = (size_t)(Nphi / 2 + 1) * 2 * Nu;
  cudaError_t e = cudaMalloc((void **)&g->W, spec * sizeof(double2));
  if (e == cudaSuccess) e = cudaMalloc((void **)&g->khat, spec * sizeof(double2));
  if (e == cudaSuccess) e = cudaMalloc((void **)&g->roots, r.size() * sizeof(double2));
  if (e == cudaSuccess) e = cudaMemcpy(g->roots, r.data(), r.size() * sizeof(double2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = prepare_kernels();
  return e;
}

void release(Gravity *g) {
  for (double2 *p : {g->W, g->khat, g->roots})
    if (p) cudaFree(p);
  *g = Gravity{};
}

cudaError_t khat(const double *samples, Gravity *g, cudaStream_t st) {
  const int M = 2 * g->Nu;
  const cudaError_t e = phi_fwd(samples, M, nullptr, *g, st);
  return e == cudaSuccess ? u_conv(*g, M, M, nullptr, g->khat, st) : e;
}

cudaError_t potential(const double *Sig, const double *rowscale, double pref, const double *sqrtR, double *out,
                      const Gravity &g, cudaStream_t st) {
  cudaError_t e = phi_fwd(Sig, g.Nu, rowscale, g, st);
  if (e == cudaSuccess) e = u_conv(g, g.Nu, g.Nu, g.khat, nullptr, st);
  if (e != cudaSuccess) return e;
  FftShape s = fft_shape<double2>(g.Nphi, (g.Nu + 1) / 2);
  const int blocks = (g.Nu + 2 * s.nb - 1) / (2 * s.nb);
  k_phi_inv<double, 8><<<blocks, s.threads, s.smem, st>>>(g.W, 2 * g.Nu, g.Nu, g.Nphi, g.phi, g.roots, pref, sqrtR, out,
                                                          s.nb);
  return cudaGetLastError();
}

}  // namespace setup
}  // namespace dg
