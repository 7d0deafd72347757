// Host side of fft_fixed.cuh for one element type: the lengths it is built for and its
// launches (included once per type).
#pragma once

#include "fft_fixed.cuh"
#include "kernels.h"

namespace dg {

// CTAs for `count` pieces of work: all of them, or as few per SM as are resident together,
// evenly loaded.
static inline int fixed_grid(int count, int nt, size_t smem, int regs) {
  int per = 65536 / (regs * nt);
  const int by_smem = (int)((size_t)228 * 1024 / (smem + 1024));
  if (by_smem < per) per = by_smem;
  if (per < 1) per = 1;
  const int slots = sm_count() * per;
  if (count <= slots) return count;
  const int rounds = (count + slots - 1) / slots;
  return (count + rounds - 1) / rounds;
}

template <typename V, int N> struct FixedLen {
  using P = FixedPlan<V, N>;
  // Threads per CTA, and the CTAs per SM the registers are cut for.  128 registers (two CTAs of
  // 256) beat 80 and 64 on every length but the longest (FP64 1024^2 step: 62 us against 73 and
  // 80; mixed 512 x 1024: 27.9 against 30.8 and 33.7), whose phi passes take 64 (4096^2: 519
  // against 539 us).  Pass 2 of the longest holds its tables and both parities in one 512-thread
  // CTA (522 us against 531 with 256 threads).
  static constexpr bool kLong = sizeof(V) == 8 && N >= 4096;
  static constexpr int LB = 256, MINB = kLong ? 4 : 2, kRegs = 65536 / (LB * MINB);
  static constexpr int LBU = kLong ? 512 : 256, MINBU = kLong ? 1 : 2, kRegsU = 65536 / (LBU * MINBU);
  static constexpr int Q = N / P::LAST;
  // rows per group: up to 8 pairs (runs of W), to fill a warp or while every SM gets a CTA, and
  // where the rows divide
  static int log2_batch(int pairs) {
    int lg = 0;
    while (lg < 3 && (Q << (lg + 1)) <= LB && pairs % (2 << lg) == 0 &&
           ((Q << lg) < 32 || (pairs) >> (lg + 1) >= sm_count()))
      ++lg;
    return lg;
  }
  static int threads(int lg) {
    int T = Q;
    while ((T << (lg + 1)) <= LB && T < N / 8) T *= 2;
    return T;
  }
  static cudaError_t attrs() {
    cudaError_t e = cudaSuccess;
    for (const void *f : {(const void *)k_phi_fwd_n<V, N, LB, MINB>, (const void *)k_u_conv_n<V, N, LBU, MINBU>,
                          (const void *)k_phi_inv_n<V, N, LB, MINB>}) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    }
    return e;
  }
  static cudaError_t phi_fwd(const FftDisk<V> &d, int b, int nrows, int ldw,
                             const V *tw, cudaStream_t st) {
    const int pairs = nrows / 2, lg = log2_batch(pairs), nb = 1 << lg, T = threads(lg);
    const size_t sm = ((size_t)P::tab + (size_t)nb * P::np) * sizeof(V);
    return launch_pdl(k_phi_fwd_n<V, N, LB, MINB>, dim3(fixed_grid(pairs / nb, T * nb, sm, kRegs)),
                      dim3(T, nb), sm, st, d, b, pairs / nb, ldw, tw, lg);
  }
  static cudaError_t u_conv(const FftDisk<V> &d, int Nc, int ldw, const V *tw,
                            const V *half, cudaStream_t st) {
    int T = Q;
    while (T * 4 <= LBU && T < N / 8) T *= 2;
    if (T * 2 > LBU) T = LBU / 2;
    const size_t sm = ((size_t)P::tab + N + (size_t)2 * P::np) * sizeof(V);
    return launch_pdl(k_u_conv_n<V, N, LBU, MINBU>, dim3(fixed_grid(Nc, T * 2, sm, kRegsU)), dim3(T, 2), sm, st,
                      d, Nc, ldw, tw, half);
  }
  static cudaError_t phi_inv(const FftDisk<V> &d, int nrows, int ldw,
                             const V *tw, cudaStream_t st) {
    const int pairs = nrows / 2, lg = log2_batch(pairs), nb = 1 << lg, T = threads(lg);
    const size_t sm = ((size_t)P::tab + (size_t)nb * P::np) * sizeof(V);
    return launch_pdl(k_phi_inv_n<V, N, LB, MINB>, dim3(fixed_grid(pairs / nb, T * nb, sm, kRegs)),
                      dim3(T, nb), sm, st, d, pairs / nb, ldw, tw, lg);
  }
};

}  // namespace dg
