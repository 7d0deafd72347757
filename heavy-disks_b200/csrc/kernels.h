// Host-side declarations of the diskgpu kernel launchers.
#pragma once

#include <cuda_runtime.h>

#include <utility>
#include <vector>

#include "dg_common.cuh"
#include "hydro64.cuh"
#include "fft_plan.cuh"

namespace dg {

// plain-method (FP64) path
// Pin: the pressure of Sig, or NULL (Gamma = 2, or not known yet); Po takes the new state's
cudaError_t launch_hydro64(const double *Sig, const double *vR, const double *vp, const double *Phi,
                           const double *gR, const double *gp, int force_mode, const double *Pin, double *So,
                           double *vRo, double *vpo, double *Po, Ctl *ctl, const Geom64 &g, cudaStream_t st);
cudaError_t launch_step_finalize(Ctl *ctl, cudaStream_t st);
// Po: takes the pressure of Sig, or NULL
cudaError_t launch_cfl64(const double *Sig, const double *vR, const double *vp, double *Po, Ctl *ctl, const Geom64 &g,
                         int nmodes, int record, cudaStream_t st);
cudaError_t launch_modes64(const double *Sig, const Geom64 &g, int nmodes, double *out, cudaStream_t st);
cudaError_t launch_forces64(const double *Phi, double *gR, double *gp, const Geom64 &g, cudaStream_t st);
cudaError_t launch_conserved64(const double *Sig, const double *vp, const Geom64 &g, double *out2, cudaStream_t st);
cudaError_t launch_kernel_samples64(double *out, int M, int Nphi, double du, double dphi, double eps,
                                    cudaStream_t st);

// Launch with programmatic stream serialization: the kernel may begin (its prologue up to
// pdl_wait) while the previous kernel on the stream drains.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
  if (e != cudaSuccess) cudaGetLastError();  // reported here, and not by the next launch as well
  return e;
}

int sm_count();  // SMs of the current device

// Set-up gravity of disks on the tensor-core products (fft_setup.cuh).
namespace setup {
// n = 4^n4 * 2^n2 * 3^n3 * 5^n5; stages run in that order.
struct Plan {
  int n;
  int n4, n2, n3, n5;
};
struct Gravity {
  int Nu = 0, Nphi = 0;
  Plan phi{}, u{};
  double2 *W = nullptr, *khat = nullptr, *roots = nullptr;  // spectra and khat [m][2 Nu]; roots of both lengths
};
cudaError_t build(int Nu, int Nphi, Gravity *g);
void release(Gravity *g);
cudaError_t khat(const double *samples, Gravity *g, cudaStream_t st);
cudaError_t potential(const double *Sig, const double *rowscale, double pref, const double *sqrtR, double *out,
                      const Gravity &g, cudaStream_t st);
}  // namespace setup

// Compile-time lengths (fft_fixed.cuh): whether n is one, its five radices (1 = absent),
// kernel attributes, and the passes (nrows even).
template <typename V> bool fixed_length(int n);
template <typename V> void fixed_radices(int n, int *R);
template <typename V> cudaError_t fixed_attrs(int n);
template <typename V>
cudaError_t fixed_phi_fwd(int n, const FftDisk<V> &d, int b, int nrows, int ldw,
                          const V *tw, cudaStream_t st);
template <typename V>
cudaError_t fixed_u_conv(int n, const FftDisk<V> &d, int Nc, int ldw,
                         const V *tw, const V *half, cudaStream_t st);
template <typename V>
cudaError_t fixed_phi_inv(int n, const FftDisk<V> &d, int nrows, int ldw,
                          const V *tw, cudaStream_t st);
#define DG_FIXED_DECL(V)                                                                                             \
  template <> bool fixed_length<V>(int n);                                                                           \
  template <> void fixed_radices<V>(int n, int *R);                                                                  \
  template <> cudaError_t fixed_attrs<V>(int n);                                                                     \
  template <> cudaError_t fixed_phi_fwd<V>(int, const FftDisk<V> &, int, int, int,          \
                                           const V *, cudaStream_t);                                                 \
  template <> cudaError_t fixed_u_conv<V>(int, const FftDisk<V> &, int, int, const V *,     \
                                          const V *, cudaStream_t);                                                  \
  template <> cudaError_t fixed_phi_inv<V>(int, const FftDisk<V> &, int, int, const V *,    \
                                           cudaStream_t);
DG_FIXED_DECL(float2)
DG_FIXED_DECL(double2)
#undef DG_FIXED_DECL

// FFT gravity passes (fft_smem.cuh), V = double2 or float2; b picks the ping-pong input.
template <typename V> bool make_fft_plan(int n, FftPlan *pl);
template <> bool make_fft_plan<double2>(int n, FftPlan *pl);
template <> bool make_fft_plan<float2>(int n, FftPlan *pl);
template <typename V> cudaError_t build_fft_tables(int Nu, int Nphi, FftTables<V> *ft);
template <typename V>
cudaError_t launch_phi_fwd(const FftDisk<V> &d, int b, int nrows, int ldw,
                           const FftTables<V> &ft, cudaStream_t st);
template <typename V>
cudaError_t launch_u_conv(const FftDisk<V> &d, int Nc, int ldw,
                          const FftTables<V> &ft, cudaStream_t st);
template <typename V>
cudaError_t launch_phi_inv(const FftDisk<V> &d, int nrows, int ldw,
                           const FftTables<V> &ft, cudaStream_t st);
cudaError_t launch_u_khat(const double2 *W, int ldw, int Nc, const FftTables<double2> &ft, double *kr,
                          cudaStream_t st);

}  // namespace dg
