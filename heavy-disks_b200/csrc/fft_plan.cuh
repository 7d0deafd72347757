// Stage list of one FFT length, and what the gravity passes read and write of one disk; the
// kernels are in fft_smem.cuh and fft_fixed.cuh.
#pragma once

#include "dg_common.cuh"

namespace dg {

constexpr int kFftMaxStages = 14;   // 2^13 = 8192 by radix 2 alone
constexpr int kFftMaxThreads = 512;
constexpr size_t kMaxSmem = 227 * 1024;  // dynamic shared memory of a CTA (sm_100a)

// One length's stage list, kept by the host with its device tables.
struct FftPlan {
  int n = 0, ns = 0;
  int R[kFftMaxStages];                 // radix of DIF stage s (the inverse runs them backwards)
  int m[kFftMaxStages];                 // L / R: the stage's points of one butterfly are m apart
  unsigned magic[kFftMaxStages];        // ceil(2^32 / m): b / m = umulhi(b, magic) for b, m < 2^16
  int tw[kFftMaxStages];                // offset of the stage's twiddles w_L^{j q}, [q - 1][j]
  int threads = 0;                      // threads per transform
  int ntw = 0;                          // entries of the twiddle table
  bool fixed = false;                   // a length of fft_fixed.cuh, with its radices
};

// One disk's side of the three gravity passes, V = double2 (plain path) or float2 (mixed).
template <typename V> struct FftDisk {
  using T = decltype(V::x);
  const T *src[2];     // the two ping-pong inputs of pass 1
  const T *inscale;    // per row, or NULL
  V *W;                // half spectra [m][ldw]
  const T *kr;         // khat in transform order
  const T *outscale;   // per row
  T *out;              // the potential
  Ctl *ctl;            // whose due hydro end pass 2 finalises, or NULL
};

// Tables of one transform length for both directions of a grid.
template <typename V> struct FftTables {
  FftPlan phi, u;
  V *buf = nullptr;  // owns: stage twiddles of phi and u, e^{-2 pi i j / 2 Nu}, positions
  const V *twPhi = nullptr, *twU = nullptr, *half = nullptr;
  const unsigned short *posPhi = nullptr, *posU = nullptr;
};

}  // namespace dg
