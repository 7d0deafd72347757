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
cudaError_t launch_hydro64(const double *Sig, const double *vR, const double *vp, const double *Phi,
                           const double *gR, const double *gp, int force_mode, const double *Pin, double *So,
                           double *vRo, double *vpo, double *Po, Ctl *ctl, const Geom64 &g, cudaStream_t st);
cudaError_t launch_pressure64(const double *Sig, double *P, const Geom64 &g, cudaStream_t st);
cudaError_t launch_cfl64(const double *Sig, const double *vR, const double *vp, Ctl *ctl, const Geom64 &g,
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
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

bool make_fft_plan(int n, FftPlan *pl);
void fft_tables(const FftPlan &pl, std::vector<double2> *tw, std::vector<unsigned short> *pos);
cudaError_t prepare_fft_kernels();
cudaError_t launch_phi_fwd(const double *src, int nrows, const double *rowscale, double2 *W, int ldw,
                           const FftPlan &pl, const double2 *tws, const unsigned short *pos, cudaStream_t st);
cudaError_t launch_u_conv(double2 *W, int ldw, int Nc, const FftPlan &pl, const double2 *tws, const double2 *half,
                          const double *kr, cudaStream_t st);
cudaError_t launch_u_khat(const double2 *W, int ldw, int Nc, const FftPlan &pl, const double2 *tws, const double2 *half,
                          double *kr, cudaStream_t st);
cudaError_t launch_phi_inv(const double2 *W, int ldw, int nrows, const FftPlan &pl, const double2 *tws,
                           const unsigned short *pos, double pref, const double *sqrtR, double *out, cudaStream_t st);

}  // namespace dg
