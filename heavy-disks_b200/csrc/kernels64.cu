// Small kernels of the plain method (FP64), some of them of mixed disks' set-up too, with their
// launchers: end of a step, CFL reduction, forces, mode sums, Kalnajs kernel samples, khat.  (A
// file's kernels are loaded together, so the large ones are in files of their own.)
#include <atomic>
#include <cmath>

#include "kernels.h"
#include "hydro64.cuh"
#include "fft_smem.cuh"
#include "step_ctl.cuh"

namespace dg {

// Mode-sum contribution of one cell: Sigma cos(m phi) dA and -Sigma sin(m phi) dA
// (diskmain.cpp:76-80).
__device__ __forceinline__ void add_modes(double *msum, int nmodes, double s, int j, double dphi, double dA) {
  double phi = (j + 0.5) * dphi;
  for (int m = 0; m < nmodes; ++m) {
    double sn, cs;
    sincos(m * phi, &sn, &cs);
    msum[2 * m] += s * cs * dA;
    msum[2 * m + 1] -= s * sn * dA;
  }
}

// ---------------------------------------------------------------------------------
// The end of a hydro launch that no gravity kernel takes care of.
__global__ void k_step_finalize(Ctl *ctl) {
  pdl_trigger();  // the next kernel's prologue may start; it waits for this one's completion
  pdl_wait();     // every CTA of the hydro launch has folded its sums
  if (threadIdx.x == 0) finalize_pending(ctl);
}
cudaError_t launch_step_finalize(Ctl *ctl, cudaStream_t st) {
  return launch_pdl(k_step_finalize, dim3(1), dim3(32), 0, st, ctl);
}

// CFL reduction over a state (DiskHydro::timestep, hydro.hpp:48-61); the last CTA stores
// dt = cfl / max (clipped to tlim unless fixed_dt).  Optionally accumulates mode sums.  Po, if
// given, takes the pressure, which the rate needs anyway.
__global__ void __launch_bounds__(256) k_cfl64(const double *__restrict__ Sig, const double *__restrict__ vR,
                                               const double *__restrict__ vp, double *__restrict__ Po, Ctl *ctl,
                                               Geom64 g, int nmodes, int record) {
  __shared__ double red[8];
  StepInfo si;
  si.t = ctl->t; si.dt = 0.0; si.tlim = ctl->tlim;
  si.active = false; si.advance_t = false;
  si.record = record != 0;
  si.nmodes = record && nmodes < 3 ? 3 : nmodes;
  nmodes = si.nmodes;
  double msum[2 * kMaxModes];
#pragma unroll
  for (int q = 0; q < 2 * kMaxModes; ++q) msum[q] = 0.0;
  double lmax = 0.0;
  const size_t n = (size_t)g.Nu * g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / g.Nphi), j = (int)(k % g.Nphi);
    double r;
    if (Po) {
      const double s = Sig[k], P = pres64(g, s);
      Po[k] = P;
      r = s < 1e-12 ? cfl_rate64(g, i, s, vR[k], vp[k]) : rate64(vR[k], vp[k], cs64(g, s, P), g.invdR[i], g.invdl[i]);
    } else {
      r = cfl_rate64(g, i, Sig[k], vR[k], vp[k]);
    }
    if (!(r == r)) lmax = r;
    else if (lmax == lmax) lmax = fmax(lmax, r);
    if (nmodes) {
      double dA = g.R[i] * (g.Rf[i + 1] - g.Rf[i]) * g.dphi;
      add_modes(msum, nmodes, Sig[k], j, g.dphi, dA);
    }
  }
  finish_launch<256>(ctl, si, lmax, msum, red);
}

// Sums Sigma e^{-i m phi} dA for m < nmodes (diskmain.cpp:72-84) into out[2m], out[2m+1].
__global__ void __launch_bounds__(256) k_modes64(const double *__restrict__ Sig, Geom64 g, int nmodes,
                                                 double *__restrict__ out) {
  __shared__ double red[8];
  double msum[2 * kMaxModes];
#pragma unroll
  for (int q = 0; q < 2 * kMaxModes; ++q) msum[q] = 0.0;
  const size_t n = (size_t)g.Nu * g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / g.Nphi), j = (int)(k % g.Nphi);
    double dA = g.R[i] * (g.Rf[i + 1] - g.Rf[i]) * g.dphi;
    add_modes(msum, nmodes, Sig[k], j, g.dphi, dA);
  }
  for (int q = 0; q < 2 * nmodes; ++q) {
    double v = warp_sum(msum[q]);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < 8; ++w) s += red[w];
      atomicAdd(&out[q], s);
    }
    __syncthreads();
  }
}

// KalnajsSolver::forces (kalnajs.hpp:65-80) as a standalone pass.
__global__ void k_forces64(const double *__restrict__ Phi, double *__restrict__ gR, double *__restrict__ gp,
                           Geom64 g) {
  const size_t n = (size_t)g.Nu * g.Nphi;
  const int Nu = g.Nu, Nphi = g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / Nphi), j = (int)(k % Nphi);
    int jm = (j - 1 + Nphi) % Nphi, jp = (j + 1) % Nphi;
    double dPhidphi = (Phi[(size_t)i * Nphi + jp] - Phi[(size_t)i * Nphi + jm]) / (2.0 * g.dphi);
    double dPhidu;
    if (i == 0) dPhidu = (Phi[(size_t)(i + 1) * Nphi + j] - Phi[k]) / g.du;
    else if (i == Nu - 1) dPhidu = (Phi[k] - Phi[(size_t)(i - 1) * Nphi + j]) / g.du;
    else dPhidu = (Phi[(size_t)(i + 1) * Nphi + j] - Phi[(size_t)(i - 1) * Nphi + j]) / (2.0 * g.du);
    gR[k] = -dPhidu / g.R[i];
    gp[k] = -dPhidphi / g.R[i];
  }
}

// Samples of the softened log-spiral kernel at wrapped offsets (kalnajs.hpp:106-112).
__global__ void k_kernel_samples64(double *__restrict__ out, int M, int Nphi, double du, double dphi, double eps) {
  const size_t n = (size_t)M * Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int p = (int)(k / Nphi), q = (int)(k % Nphi);
    int ioff = (p <= M / 2) ? p : p - M;
    double Du = ioff * du;
    double Dphi = q * dphi;
    out[k] = 1.0 / sqrt(2.0 * cosh(Du) - 2.0 * cos(Dphi) + eps);
  }
}

// global sums mass = sum Sigma dA, angmom = sum Sigma vphi R dA (FP64)
__global__ void k_conserved64(const double *__restrict__ Sig, const double *__restrict__ vp, Geom64 g,
                              double *__restrict__ out) {
  __shared__ double red[2][8];
  double m = 0.0, L = 0.0;
  const size_t n = (size_t)g.Nu * g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / g.Nphi);
    double dA = g.R[i] * (g.Rf[i + 1] - g.Rf[i]) * g.dphi;
    m += Sig[k] * dA;
    L += Sig[k] * vp[k] * g.R[i] * dA;
  }
  m = warp_sum(m);
  L = warp_sum(L);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = m; red[1][threadIdx.x >> 5] = L; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { a += red[0][w]; b += red[1][w]; }
    atomicAdd(&out[0], a);
    atomicAdd(&out[1], b);
  }
}

// ---------------------------------------------------------------------------------
// host launchers
int sm_count() {
  static std::atomic<int> known[64];  // by device; 0: not asked yet
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  if (dev >= 0 && dev < 64) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

cudaError_t launch_cfl64(const double *Sig, const double *vR, const double *vp, double *Po, Ctl *ctl, const Geom64 &g,
                         int nmodes, int record, cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  int cap = sm_count() * 4;
  if (blocks > cap) blocks = cap;
  k_cfl64<<<blocks, 256, 0, st>>>(Sig, vR, vp, Po, ctl, g, nmodes, record);
  return cudaGetLastError();
}

cudaError_t launch_modes64(const double *Sig, const Geom64 &g, int nmodes, double *out, cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 4) blocks = sm_count() * 4;
  cudaMemsetAsync(out, 0, 2 * nmodes * sizeof(double), st);
  k_modes64<<<blocks, 256, 0, st>>>(Sig, g, nmodes, out);
  return cudaGetLastError();
}

cudaError_t launch_forces64(const double *Phi, double *gR, double *gp, const Geom64 &g, cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  k_forces64<<<blocks, 256, 0, st>>>(Phi, gR, gp, g);
  return cudaGetLastError();
}

cudaError_t launch_conserved64(const double *Sig, const double *vp, const Geom64 &g, double *out2,
                               cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 4) blocks = sm_count() * 4;
  cudaMemsetAsync(out2, 0, 2 * sizeof(double), st);
  k_conserved64<<<blocks, 256, 0, st>>>(Sig, vp, g, out2);
  return cudaGetLastError();
}

cudaError_t launch_kernel_samples64(double *out, int M, int Nphi, double du, double dphi, double eps,
                                    cudaStream_t st) {
  size_t n = (size_t)M * Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  k_kernel_samples64<<<blocks, 256, 0, st>>>(out, M, Nphi, du, dphi, eps);
  return cudaGetLastError();
}

// the real khat table of the FP64 convolution (set-up)
cudaError_t launch_u_khat(const double2 *W, int ldw, int Nc, const FftTables<double2> &ft, double *kr,
                          cudaStream_t st) {
  const FftPlan &pl = ft.u;
  const cudaError_t e =
      cudaFuncSetAttribute(k_u_khat<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
  if (e != cudaSuccess) return e;
  k_u_khat<double2><<<2 * Nc, pl.threads, (size_t)fft_pad_len<double2>(pl.n) * sizeof(double2), st>>>(
      W, ldw, pl, ft.twU, ft.half, kr);
  return cudaGetLastError();
}

}  // namespace dg
