// Shared-memory mixed-radix FFT of the plain (FP64) gravity path, and the three passes of
// the Kalnajs convolution built from it.
//
// The convolution restates diskfft/src/kalnajs.hpp:48-63 (potential) and :105-116
// (kernel table): a 2-D real-to-complex transform of the M x Nphi zero-padded field
// (M = 2 Nu), a multiply by khat, and the inverse.  It is split into:
//   pass 1  (phi_fwd)  rows i -> half spectrum in phi, two real rows packed per complex
//                      transform, written transposed as W[m][i] (mode-major);
//   pass 2  (u_conv)   per mode m: length-M transform along u (rows >= Nu are the
//                      implicit zero padding), multiply by khat[m][p], inverse, keep Nu;
//   pass 3  (phi_inv)  rows i <- Hermitian half spectrum (c2r), scaled by
//                      -G du dphi / (M Nphi) / sqrt(R_i).
//
// Transforms run in place in shared memory.  Forward: decimation in frequency, natural
// order in, digit-reversed order out; inverse: the same stages backwards (decimation in
// time), digit-reversed in, natural out.  A butterfly reads and writes only its own R
// points, so a stage needs one barrier, and threads loop over butterflies with one
// butterfly's points in registers.  The first stage reads its points from global memory
// and the last inverse stage writes there, so a transform of S stages makes S - 1 to S
// trips through shared memory.
//
// The zero padding of pass 2 is not transformed: the M = 2 N spectrum of N points is the
// N-point transform of x (even p) and of x[j] e^{-2 pi i j / M} (odd p), and the first N
// points of the inverse are E[j] + e^{+2 pi i j / M} O[j].  Both parities run side by side
// as transforms of length N = Nu.  The multiply by khat (real: the kernel is even in u and
// phi) sits between the last forward and the first inverse stage, in registers, with khat
// stored in digit-reversed order, so the spectrum is never written or reordered.
//
// What bounds it: latency.  Short transforms are a chain of barriers and L2 round trips, so
// their constant tables (twiddles, positions, khat) are copied to shared memory before the
// dependence wait, while the previous kernel still runs; long ones leave the tables to L1
// and the shared memory to more CTAs per SM.  The FP64 pipe's share is the butterflies,
// about 5 N log2 N operations per transform.  Against out-of-place radix-4 stages with two
// barriers each and a padded transform in u, 256 FP64 steps: 48.5 -> 37.3 ms at 1024^2,
// 9.0 -> 7.3 ms at 256^2.
#pragma once

#include "fft_plan.cuh"

namespace dg {

// Shared-memory position of element i: pads that spread strides of 8, 64 and 512 double2
// over the banks (a quarter-warp's eight 16-byte accesses hit distinct bank groups).
__host__ __device__ __forceinline__ int fft_pad(int i) { return i + (i >> 3) + (i >> 6) + (i >> 9); }
__host__ __device__ __forceinline__ int fft_pad_len(int n) { return fft_pad(n - 1) + 1; }

__host__ __device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ double2 cmulw(double2 a, double2 w) {
  return make_double2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
// a conj(w)
__host__ __device__ __forceinline__ double2 cmulc(double2 a, double2 w) {
  return make_double2(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y);
}
// multiply by -i (SIGN < 0) or +i (SIGN > 0)
template <int SIGN>
__host__ __device__ __forceinline__ double2 cmul_i(double2 a) {
  return SIGN < 0 ? make_double2(a.y, -a.x) : make_double2(-a.y, a.x);
}
// multiply by exp(SIGN 2 pi i k / n) given its cosine and sine
template <int SIGN>
__host__ __device__ __forceinline__ double2 crot(double2 a, double c, double s) {
  return SIGN < 0 ? make_double2(a.x * c + a.y * s, a.y * c - a.x * s)
                  : make_double2(a.x * c - a.y * s, a.y * c + a.x * s);
}

// R-point DFT in registers, natural order in and out; SIGN -1 forward, +1 inverse.
template <int R, int SIGN> struct Dft;
template <int SIGN> struct Dft<2, SIGN> {
  static __host__ __device__ __forceinline__ void run(double2 *v) {
    const double2 a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  }
};
template <int SIGN>
__host__ __device__ __forceinline__ void dft4(double2 &v0, double2 &v1, double2 &v2, double2 &v3) {
  const double2 a0 = cadd(v0, v2), a1 = csub(v0, v2), a2 = cadd(v1, v3), a3 = cmul_i<SIGN>(csub(v1, v3));
  v0 = cadd(a0, a2);
  v1 = cadd(a1, a3);
  v2 = csub(a0, a2);
  v3 = csub(a1, a3);
}
template <int SIGN> struct Dft<4, SIGN> {
  static __host__ __device__ __forceinline__ void run(double2 *v) { dft4<SIGN>(v[0], v[1], v[2], v[3]); }
};
template <int SIGN> struct Dft<3, SIGN> {
  static __host__ __device__ __forceinline__ void run(double2 *v) {
    const double h = 0.86602540378443864676;  // sqrt(3) / 2
    const double2 t1 = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const double2 t2 = make_double2(v[0].x - 0.5 * t1.x, v[0].y - 0.5 * t1.y);
    const double2 q = cmul_i<SIGN>(d), t3 = make_double2(q.x * h, q.y * h);
    v[0] = cadd(v[0], t1);
    v[1] = cadd(t2, t3);
    v[2] = csub(t2, t3);
  }
};
template <int SIGN> struct Dft<5, SIGN> {
  static __host__ __device__ __forceinline__ void run(double2 *v) {
    const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;  // cos 2pi/5, cos 4pi/5
    const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;   // sin 2pi/5, sin 4pi/5
    const double2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
    const double2 a1 = make_double2(v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y);
    const double2 a2 = make_double2(v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y);
    const double2 b1 = cmul_i<SIGN>(make_double2(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y));
    const double2 b2 = cmul_i<SIGN>(make_double2(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y));
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(a1, b1);
    v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2);
    v[3] = csub(a2, b2);
  }
};
template <int SIGN> struct Dft<8, SIGN> {
  static __host__ __device__ __forceinline__ void run(double2 *v) {
    const double h = 0.70710678118654752440;  // sqrt(1/2)
    dft4<SIGN>(v[0], v[2], v[4], v[6]);
    dft4<SIGN>(v[1], v[3], v[5], v[7]);
    const double2 o0 = v[1], o1 = crot<SIGN>(v[3], h, h), o2 = cmul_i<SIGN>(v[5]), o3 = crot<SIGN>(v[7], -h, h);
    const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  }
};
__host__ __device__ __forceinline__ int fft_div(int b, int m, unsigned magic) {
#ifdef __CUDA_ARCH__
  return m == 1 ? b : (int)__umulhi((unsigned)b, magic);
#else
  return m == 1 ? b : (int)(((unsigned long long)(unsigned)b * magic) >> 32);
#endif
}
// Stage s of one transform, threads tx = 0 .. T-1.  FWD: DFT, then twiddle (decimation in
// frequency); otherwise conjugate twiddle, then inverse DFT (decimation in time).  ld(i)
// and st(i, v) read and write element i; the same R elements are read and written.
template <int R, bool FWD, class LD, class ST>
__host__ __device__ __forceinline__ void fft_stage(const FftPlan &pl, int s, const double2 *__restrict__ tws, int tx,
                                                   int T, LD ld, ST st) {
  const int m = pl.m[s], L = m * R, nbf = pl.n / R;
  const double2 *tw = tws + pl.tw[s];
  for (int b = tx; b < nbf; b += T) {
    const int blk = fft_div(b, m, pl.magic[s]), j = b - blk * m, base = blk * L + j;
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(base + r * m);
    if (FWD) {
      Dft<R, -1>::run(v);
      if (m > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = cmulw(v[q], tw[(q - 1) * m + j]);
      }
    } else {
      if (m > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = cmulc(v[q], tw[(q - 1) * m + j]);
      }
      Dft<R, +1>::run(v);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) st(base + r * m, v[r]);
  }
}
template <bool FWD, class LD, class ST>
__host__ __device__ __forceinline__ void fft_stage_any(const FftPlan &pl, int s, const double2 *__restrict__ tws,
                                                       int tx, int T, LD ld, ST st) {
  switch (pl.R[s]) {  // uniform over the grid
    case 8: fft_stage<8, FWD>(pl, s, tws, tx, T, ld, st); break;
    case 5: fft_stage<5, FWD>(pl, s, tws, tx, T, ld, st); break;
    case 4: fft_stage<4, FWD>(pl, s, tws, tx, T, ld, st); break;
    case 3: fft_stage<3, FWD>(pl, s, tws, tx, T, ld, st); break;
    default: fft_stage<2, FWD>(pl, s, tws, tx, T, ld, st); break;
  }
}

// The middle of a convolution: the last forward stage (L = R, no twiddles), the multiply by
// the spectrum kr (position order, as the forward stages leave it), the first inverse stage.
template <int R, class LD, class ST>
__host__ __device__ __forceinline__ void fft_mid(const FftPlan &pl, const double *__restrict__ kr, int tx, int T,
                                                 LD ld, ST st) {
  for (int b = tx; b < pl.n / R; b += T) {
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(b * R + r);
    Dft<R, -1>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double k = kr[b * R + r];
      v[r].x *= k;
      v[r].y *= k;
    }
    Dft<R, +1>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) st(b * R + r, v[r]);
  }
}
template <class LD, class ST>
__host__ __device__ __forceinline__ void fft_mid_any(const FftPlan &pl, const double *__restrict__ kr, int tx, int T,
                                                     LD ld, ST st) {
  switch (pl.R[pl.ns - 1]) {
    case 8: fft_mid<8>(pl, kr, tx, T, ld, st); break;
    case 5: fft_mid<5>(pl, kr, tx, T, ld, st); break;
    case 4: fft_mid<4>(pl, kr, tx, T, ld, st); break;
    case 3: fft_mid<3>(pl, kr, tx, T, ld, st); break;
    default: fft_mid<2>(pl, kr, tx, T, ld, st); break;
  }
}

// A table of cnt entries: copied to shared memory at `to` (SMT; the caller's next barrier
// publishes it), or left where it is.
template <bool SMT, typename V>
__device__ __forceinline__ const V *fft_table(V *to, const V *__restrict__ from, int cnt, int flat, int nt) {
  if (!SMT) return from;
#pragma unroll 4
  for (int i = flat; i < cnt; i += nt) to[i] = __ldg(from + i);
  return to;
}
// shared memory of the tables: twiddles, then half (pass 2) or positions (passes 1 and 3),
// then khat (pass 2); in double2
__host__ __device__ __forceinline__ int fft_tab_phi(int n, int ntw) { return ntw + (n + 7) / 8; }
__host__ __device__ __forceinline__ int fft_tab_u(int n, int ntw) { return ntw + n + n; }

// Two neighbouring rows of one frequency of W as one 32-byte sector (W's row stride is even).
__device__ __forceinline__ void store_pair(double2 *w, double2 a, double2 b) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(w), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y) : "memory");
}
__device__ __forceinline__ void load_pair(const double2 *w, double2 &a, double2 &b) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(w) : "memory");
}

// ---------------------------------------------------------------------------------
// pass 1: rows -> transposed half spectrum.  The CTA's pairs of rows (threadIdx.y: pair;
// row0 = 2 blockDim.y blockIdx.x) of src (nrows x Nphi) are multiplied by rowscale[i]
// (kalnajs.hpp:51: R^{3/2} Sigma; NULL = 1), packed two rows per complex transform,
// transformed forward along phi and unpacked into W[m * ldw + i], m < Nc (ldw even).
// pos[m]: where the transform leaves frequency m.
template <bool SMT>
__global__ void __launch_bounds__(kFftMaxThreads, 2) k_phi_fwd(const double *__restrict__ src, int nrows,
                                                              const double *__restrict__ rowscale,
                                                              double2 *__restrict__ W, int ldw, const FftPlan pl,
                                                              const double2 *__restrict__ gtw,
                                                              const unsigned short *__restrict__ gpos, int log2nb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = pl.n, np = fft_pad_len(n), tx = threadIdx.x, T = blockDim.x, nb = 1 << log2nb;
  const int flat = threadIdx.y * T + tx, nt = nb * T;
  double2 *sm = reinterpret_cast<double2 *>(smem_raw), *all = sm + (SMT ? fft_tab_phi(n, pl.ntw) : 0);
  double2 *buf = all + threadIdx.y * np;
  const double2 *tws = fft_table<SMT>(sm, gtw, pl.ntw, flat, nt);
  const unsigned short *pos = fft_table<SMT>(reinterpret_cast<unsigned short *>(sm + pl.ntw), gpos, n, flat, nt);
  const int row0 = blockIdx.x * 2 * nb;
  const int r0 = row0 + 2 * threadIdx.y, r1 = r0 + 1;
  const double a0 = r0 < nrows ? (rowscale ? rowscale[r0] : 1.0) : 0.0;
  const double a1 = r1 < nrows ? (rowscale ? rowscale[r1] : 1.0) : 0.0;
  const double *s0 = src + (size_t)(r0 < nrows ? r0 : 0) * n, *s1 = src + (size_t)(r1 < nrows ? r1 : 0) * n;
  auto ldg = [&](int i) { return make_double2(r0 < nrows ? a0 * s0[i] : 0.0, r1 < nrows ? a1 * s1[i] : 0.0); };
  auto lds = [&](int i) { return buf[fft_pad(i)]; };
  auto sts = [&](int i, double2 v) { buf[fft_pad(i)] = v; };
  pdl_wait();
  pdl_trigger();
  if (SMT) __syncthreads();
  fft_stage_any<true>(pl, 0, tws, tx, T, ldg, sts);
  __syncthreads();
  for (int s = 1; s < pl.ns; ++s) {
    fft_stage_any<true>(pl, s, tws, tx, T, lds, sts);
    __syncthreads();
  }
  const int Nc = n / 2 + 1;
#pragma unroll 2
  for (int idx = flat; idx < nb * Nc; idx += nt) {
    const int m = idx >> log2nb, t = idx & (nb - 1);
    const double2 *Z = all + t * np;
    const double2 a = Z[fft_pad(pos[m])], c = Z[fft_pad(pos[m == 0 ? 0 : n - m])];
    const int q0 = row0 + 2 * t;
    double2 *w = W + (size_t)m * ldw + q0;
    // (an odd last row's partner is the row stride's padding)
    if (q0 < nrows)
      store_pair(w, make_double2(0.5 * (a.x + c.x), 0.5 * (a.y - c.y)),
                 make_double2(0.5 * (a.y + c.y), 0.5 * (c.x - a.x)));
  }
}

// pass 2: per mode m: the length-2N transform of W[m][0..N) (zero beyond), times khat
// (kalnajs.hpp:53-56), inverse, W[m][0..N).  One mode per CTA; threadIdx.y: parity of p.
// kr[(2 m + parity) N + position]; half[j] = e^{-2 pi i j / 2N}, j < N.
template <bool SMT>
__global__ void __launch_bounds__(kFftMaxThreads, 2) k_u_conv(double2 *__restrict__ W, int ldw, const FftPlan pl,
                                                             const double2 *__restrict__ gtw,
                                                             const double2 *__restrict__ ghalf,
                                                             const double *__restrict__ kr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = pl.n, np = fft_pad_len(n), tx = threadIdx.x, T = blockDim.x, odd = threadIdx.y;
  const int flat = odd * T + tx, nt = 2 * T;
  double2 *sm = reinterpret_cast<double2 *>(smem_raw), *all = sm + (SMT ? fft_tab_u(n, pl.ntw) : 0);
  double2 *buf = all + odd * np;
  const double2 *tws = fft_table<SMT>(sm, gtw, pl.ntw, flat, nt);
  const double2 *half = fft_table<SMT>(sm + pl.ntw, ghalf, n, flat, nt);
  const double *k = fft_table<SMT>(reinterpret_cast<double *>(sm + pl.ntw + n), kr + (size_t)2 * blockIdx.x * n, 2 * n,
                                   flat, nt) + odd * n;
  double2 *x = W + (size_t)blockIdx.x * ldw;
  auto ldg = [&](int i) { return odd ? cmulw(x[i], half[i]) : x[i]; };
  auto lds = [&](int i) { return buf[fft_pad(i)]; };
  auto sts = [&](int i, double2 v) { buf[fft_pad(i)] = v; };
  const int last = pl.ns - 1;
  pdl_wait();
  pdl_trigger();
  if (SMT) __syncthreads();
  if (last == 0) {
    fft_mid_any(pl, k, tx, T, ldg, sts);
  } else {
    fft_stage_any<true>(pl, 0, tws, tx, T, ldg, sts);
    __syncthreads();
    for (int s = 1; s < last; ++s) {
      fft_stage_any<true>(pl, s, tws, tx, T, lds, sts);
      __syncthreads();
    }
    fft_mid_any(pl, k, tx, T, lds, sts);
    for (int s = last - 1; s >= 0; --s) {
      __syncthreads();
      fft_stage_any<false>(pl, s, tws, tx, T, lds, sts);
    }
  }
  __syncthreads();
  // E[j] + conj(half[j]) O[j]: the threads of both transforms share the sums
#pragma unroll 4
  for (int j = flat; j < n; j += nt) x[j] = cadd(all[fft_pad(j)], cmulc(all[np + fft_pad(j)], half[j]));
}

// The spectrum table of pass 2: W holds the phi half spectra of the kernel samples at all
// 2N wrapped offsets, [m][p].  One CTA per (mode, parity): even frequencies transform
// x[j] + x[j + N], odd ones (x[j] - x[j + N]) e^{-2 pi i j / 2N}.  Only real parts are kept:
// the kernel is even in both offsets.
__global__ void __launch_bounds__(kFftMaxThreads) k_u_khat(const double2 *__restrict__ W, int ldw, const FftPlan pl,
                                                          const double2 *__restrict__ tws,
                                                          const double2 *__restrict__ half, double *__restrict__ kr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *buf = reinterpret_cast<double2 *>(smem_raw);
  const int n = pl.n, tx = threadIdx.x, T = blockDim.x, mode = blockIdx.x >> 1, odd = blockIdx.x & 1;
  const double2 *x = W + (size_t)mode * ldw;
  auto ldg = [&](int i) { return odd ? cmulw(csub(x[i], x[i + n]), half[i]) : cadd(x[i], x[i + n]); };
  auto lds = [&](int i) { return buf[fft_pad(i)]; };
  auto sts = [&](int i, double2 v) { buf[fft_pad(i)] = v; };
  fft_stage_any<true>(pl, 0, tws, tx, T, ldg, sts);
  __syncthreads();
  for (int s = 1; s < pl.ns; ++s) {
    fft_stage_any<true>(pl, s, tws, tx, T, lds, sts);
    __syncthreads();
  }
  double *k = kr + (size_t)blockIdx.x * n;
  for (int i = tx; i < n; i += T) k[i] = buf[fft_pad(i)].x;
}

// pass 3: transposed half spectrum -> rows.  Two Hermitian rows are packed into one
// complex inverse transform (FFTW c2r semantics: the imaginary parts of the m=0 and
// Nyquist bins are ignored), then out[i][j] = (pref / sqrtR[i]) x (kalnajs.hpp:58-62).
template <bool SMT>
__global__ void __launch_bounds__(kFftMaxThreads, 2) k_phi_inv(const double2 *__restrict__ W, int ldw, int nrows,
                                                              const FftPlan pl, const double2 *__restrict__ gtw,
                                                              const unsigned short *__restrict__ gpos, double pref,
                                                              const double *__restrict__ sqrtR,
                                                              double *__restrict__ out, int log2nb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = pl.n, np = fft_pad_len(n), tx = threadIdx.x, T = blockDim.x, nb = 1 << log2nb;
  const int flat = threadIdx.y * T + tx, nt = nb * T;
  double2 *sm = reinterpret_cast<double2 *>(smem_raw), *all = sm + (SMT ? fft_tab_phi(n, pl.ntw) : 0);
  double2 *buf = all + threadIdx.y * np;
  const double2 *tws = fft_table<SMT>(sm, gtw, pl.ntw, flat, nt);
  const unsigned short *pos = fft_table<SMT>(reinterpret_cast<unsigned short *>(sm + pl.ntw), gpos, n, flat, nt);
  const int row0 = blockIdx.x * 2 * nb;
  const int r0 = row0 + 2 * threadIdx.y, r1 = r0 + 1;
  const double p0 = r0 < nrows ? pref / sqrtR[r0] : 0.0, p1 = r1 < nrows ? pref / sqrtR[r1] : 0.0;
  pdl_wait();
  pdl_trigger();
  if (SMT) __syncthreads();
  const int Nc = n / 2 + 1;
#pragma unroll 2
  for (int idx = flat; idx < nb * Nc; idx += nt) {
    const int m = idx >> log2nb, t = idx & (nb - 1);
    const int q0 = row0 + 2 * t;
    const double2 *w = W + (size_t)m * ldw + q0;
    double2 A = make_double2(0.0, 0.0), B = A;
    if (q0 < nrows) load_pair(w, A, B);
    if (m == 0 || 2 * m == n) A.y = B.y = 0.0;
    double2 *Z = all + t * np;
    Z[fft_pad(pos[m])] = make_double2(A.x - B.y, A.y + B.x);
    if (m > 0 && n - m >= Nc) Z[fft_pad(pos[n - m])] = make_double2(A.x + B.y, B.x - A.y);
  }
  __syncthreads();
  auto lds = [&](int i) { return buf[fft_pad(i)]; };
  auto sts = [&](int i, double2 v) { buf[fft_pad(i)] = v; };
  const int o0 = r0 * n;  // at most 4096 x 8192 elements
  auto stg = [&](int i, double2 v) {
    if (r0 < nrows) out[o0 + i] = p0 * v.x;
    if (r1 < nrows) out[o0 + n + i] = p1 * v.y;
  };
  for (int s = pl.ns - 1; s > 0; --s) {
    fft_stage_any<false>(pl, s, tws, tx, T, lds, sts);
    __syncthreads();
  }
  fft_stage_any<false>(pl, 0, tws, tx, T, lds, stg);
}

}  // namespace dg
