// Launch of the packed hydro step (hydro32p.cuh), SX: the forms that write the products' operand
// (mixed.cu) or those that do not (hydro32p_fft.cu: a file's kernels are loaded together, and a
// disk needs one kind).
#pragma once

#include <type_traits>

#include "kernels.h"  // ahead of hydro32p.cuh, which takes its force modes from here
#include "hydro32p.cuh"

namespace dg {

struct Hydro32pArgs {
  const CUtensorMap *S, *U, *W, *P;
  const float *sig, *u, *w, *Phi;
  const double *gR, *gp;
  float *so, *uo, *wo;
  SplitBf16 Sx;
  Ctl *ctl;
  const Rows32 *rows;
  int *rowpend, early_state;
};

template <bool SX> cudaError_t launch_hydro32p_as(const Hydro32pArgs &a, int fm, cudaStream_t st) {
  const Rows32 &g = *a.rows;
  const dim3 grid((g.Nphi + kTileJp - 1) / kTileJp, (g.Nu + kTileI - 1) / kTileI);
  auto go = [&](auto kern) {
    return launch_pdl(kern, grid, dim3(kThreads32t), kSmem32p, st, *a.S, *a.U, *a.W, *a.P, a.sig, a.u, a.w, a.Phi, a.gR,
                      a.gp, a.so, a.uo, a.wo, a.Sx, a.ctl, g, a.rowpend, a.early_state);
  };
  auto pick = [&](auto f) {
    constexpr int FM = decltype(f)::value;
    return g.gamma2 ? go(k_hydro32p<true, FM, SX>) : go(k_hydro32p<false, FM, SX>);
  };
  if (fm == kForcePhi) return pick(std::integral_constant<int, kForcePhi>{});
  if (fm == kForceArrays) return pick(std::integral_constant<int, kForceArrays>{});
  return pick(std::integral_constant<int, kForceNone>{});
}

template <bool SX> cudaError_t prepare_hydro32p_as() {
  cudaError_t e = cudaSuccess;
  for (const void *f : {(const void *)k_hydro32p<true, kForcePhi, SX>, (const void *)k_hydro32p<false, kForcePhi, SX>,
                        (const void *)k_hydro32p<true, kForceArrays, SX>,
                        (const void *)k_hydro32p<false, kForceArrays, SX>,
                        (const void *)k_hydro32p<true, kForceNone, SX>, (const void *)k_hydro32p<false, kForceNone, SX>}) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem32p);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  }
  return e;
}

template <bool SX> cudaError_t launch_hydro32p(const Hydro32pArgs &a, int fm, cudaStream_t st) {
  return launch_hydro32p_as<SX>(a, fm, st);
}
template <bool SX> cudaError_t prepare_hydro32p() { return prepare_hydro32p_as<SX>(); }
template <> cudaError_t launch_hydro32p<false>(const Hydro32pArgs &a, int fm, cudaStream_t st);
template <> cudaError_t prepare_hydro32p<false>();

}  // namespace dg
