// Stage list of one FFT length of the plain (FP64) gravity path, and the layout of its khat
// table; the kernels are in fft_smem.cuh.
#pragma once

#include "dg_common.cuh"

namespace dg {

constexpr int kFftMaxStages = 14;   // 2^13 = 8192 by radix 2 alone
constexpr int kFftMaxThreads = 512;

// One length's stage list, kept by the host with its device tables.
struct FftPlan {
  int n = 0, ns = 0;
  int R[kFftMaxStages];                 // radix of DIF stage s (the inverse runs them backwards)
  int m[kFftMaxStages];                 // L / R: the stage's points of one butterfly are m apart
  unsigned magic[kFftMaxStages];        // ceil(2^32 / m): b / m = umulhi(b, magic) for b, m < 2^16
  int tw[kFftMaxStages];                // offset of the stage's twiddles w_L^{j q}, [q - 1][j]
  int threads = 0;                      // threads per transform
  int ntw = 0;                          // entries of the twiddle table
};

// khat(p, m) from that table: posu[q] is where an N-point transform leaves frequency q.
__device__ __forceinline__ double khat_at(const double *__restrict__ kr, const unsigned short *__restrict__ posu,
                                          int N, int m, int p) {
  return kr[((size_t)2 * m + (p & 1)) * N + posu[p >> 1]];
}

}  // namespace dg
