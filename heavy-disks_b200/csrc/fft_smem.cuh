// Shared-memory mixed-radix FFT in FP64 (the plain path) and FP32 (the mixed path), and the
// three passes of the Kalnajs convolution built from it.
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
// barriers each and a padded transform in u, FP64, us a pass (forward / u / inverse, with their
// launches): 1000^2 21.2 / 43.4 / 20.8 -> 15.0 / 27.5 / 14.6, 640^2 15.1 / 27.1 / 14.7 ->
// 13.0 / 16.7 / 12.6, 300^2 11.0 / 18.8 / 10.6 -> 9.6 / 12.6 / 10.5.
#pragma once

#include "fft_plan.cuh"
#include "step_ctl.cuh"

namespace dg {

// Complex type of a transform: double2 or float2.
template <typename V> struct RealOf;
template <> struct RealOf<double2> { using type = double; };
template <> struct RealOf<float2> { using type = float; };
template <typename V> using real_t = typename RealOf<V>::type;
template <typename V>
__host__ __device__ __forceinline__ V cx(real_t<V> x, real_t<V> y) {
  V v;
  v.x = x;
  v.y = y;
  return v;
}

// Shared-memory position of element i, such that the accesses of one wavefront (eight
// 16-byte or sixteen 8-byte elements: consecutive, or strided by 4, 8, 16, 64) hit distinct
// banks.  FP64: pads after every 8, 64 and 512 elements.  FP32: the low four bits XORed with
// a mix of the higher ones.
template <typename V>
__host__ __device__ __forceinline__ int fft_pad(int i) {
  if (sizeof(V) == 16) return i + (i >> 3) + (i >> 6) + (i >> 9);
  const int h = i >> 4;
  return i ^ ((h ^ (h << 1) ^ (h << 2)) & 15);
}
template <typename V>
__host__ __device__ __forceinline__ int fft_pad_len(int n) {
  return sizeof(V) == 16 ? fft_pad<V>(n - 1) + 1 : (n + 15) & ~15;
}

template <typename V>
__host__ __device__ __forceinline__ V cadd(V a, V b) { return cx<V>(a.x + b.x, a.y + b.y); }
template <typename V>
__host__ __device__ __forceinline__ V csub(V a, V b) { return cx<V>(a.x - b.x, a.y - b.y); }
template <typename V>
__host__ __device__ __forceinline__ V cmulw(V a, V w) { return cx<V>(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x); }
// a conj(w)
template <typename V>
__host__ __device__ __forceinline__ V cmulc(V a, V w) { return cx<V>(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y); }
// multiply by -i (SIGN < 0) or +i (SIGN > 0)
template <int SIGN, typename V>
__host__ __device__ __forceinline__ V cmul_i(V a) { return SIGN < 0 ? cx<V>(a.y, -a.x) : cx<V>(-a.y, a.x); }
// multiply by exp(SIGN 2 pi i k / n) given its cosine and sine
template <int SIGN, typename V>
__host__ __device__ __forceinline__ V crot(V a, real_t<V> c, real_t<V> s) {
  return SIGN < 0 ? cx<V>(a.x * c + a.y * s, a.y * c - a.x * s) : cx<V>(a.x * c - a.y * s, a.y * c + a.x * s);
}

// R-point DFT in registers, natural order in and out; SIGN -1 forward, +1 inverse.
template <typename V, int R, int SIGN> struct Dft;
template <typename V, int SIGN> struct Dft<V, 2, SIGN> {
  static __host__ __device__ __forceinline__ void run(V *v) {
    const V a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  }
};
template <int SIGN, typename V>
__host__ __device__ __forceinline__ void dft4(V &v0, V &v1, V &v2, V &v3) {
  const V a0 = cadd(v0, v2), a1 = csub(v0, v2), a2 = cadd(v1, v3), a3 = cmul_i<SIGN>(csub(v1, v3));
  v0 = cadd(a0, a2);
  v1 = cadd(a1, a3);
  v2 = csub(a0, a2);
  v3 = csub(a1, a3);
}
template <typename V, int SIGN> struct Dft<V, 4, SIGN> {
  static __host__ __device__ __forceinline__ void run(V *v) { dft4<SIGN>(v[0], v[1], v[2], v[3]); }
};
template <typename V, int SIGN> struct Dft<V, 3, SIGN> {
  static __host__ __device__ __forceinline__ void run(V *v) {
    using T = real_t<V>;
    const T h = (T)0.86602540378443864676, hf = (T)0.5;  // sqrt(3) / 2
    const V t1 = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const V t2 = cx<V>(v[0].x - hf * t1.x, v[0].y - hf * t1.y);
    const V q = cmul_i<SIGN>(d), t3 = cx<V>(q.x * h, q.y * h);
    v[0] = cadd(v[0], t1);
    v[1] = cadd(t2, t3);
    v[2] = csub(t2, t3);
  }
};
template <typename V, int SIGN> struct Dft<V, 5, SIGN> {
  static __host__ __device__ __forceinline__ void run(V *v) {
    using T = real_t<V>;
    const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;  // cos 2pi/5, cos 4pi/5
    const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;   // sin 2pi/5, sin 4pi/5
    const V t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
    const V a1 = cx<V>(v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y);
    const V a2 = cx<V>(v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y);
    const V b1 = cmul_i<SIGN>(cx<V>(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y));
    const V b2 = cmul_i<SIGN>(cx<V>(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y));
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(a1, b1);
    v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2);
    v[3] = csub(a2, b2);
  }
};
template <typename V, int SIGN> struct Dft<V, 8, SIGN> {
  static __host__ __device__ __forceinline__ void run(V *v) {
    const real_t<V> h = (real_t<V>)0.70710678118654752440;  // sqrt(1/2)
    dft4<SIGN>(v[0], v[2], v[4], v[6]);
    dft4<SIGN>(v[1], v[3], v[5], v[7]);
    const V o0 = v[1], o1 = crot<SIGN>(v[3], h, h), o2 = cmul_i<SIGN>(v[5]), o3 = crot<SIGN>(v[7], -h, h);
    const V e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1); v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2); v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3); v[7] = csub(e3, o3);
  }
};
template <typename V, int SIGN> struct Dft<V, 16, SIGN> {
  static __host__ __device__ __forceinline__ void run(V *v) {
    using T = real_t<V>;
    const T c = (T)0.92387953251128675613, s = (T)0.38268343236508977173;  // cos, sin of pi / 8
    const T h = (T)0.70710678118654752440;
    // over n = r + 4 t: DFT over t for each r, twiddle w16^{r k}, DFT over r
    dft4<SIGN>(v[0], v[4], v[8], v[12]);
    dft4<SIGN>(v[1], v[5], v[9], v[13]);
    dft4<SIGN>(v[2], v[6], v[10], v[14]);
    dft4<SIGN>(v[3], v[7], v[11], v[15]);
    v[5] = crot<SIGN>(v[5], c, s);    v[9] = crot<SIGN>(v[9], h, h);     v[13] = crot<SIGN>(v[13], s, c);
    v[6] = crot<SIGN>(v[6], h, h);    v[10] = cmul_i<SIGN>(v[10]);       v[14] = crot<SIGN>(v[14], -h, h);
    v[7] = crot<SIGN>(v[7], s, c);    v[11] = crot<SIGN>(v[11], -h, h);  v[15] = crot<SIGN>(v[15], -c, -s);
    dft4<SIGN>(v[0], v[1], v[2], v[3]);
    dft4<SIGN>(v[4], v[5], v[6], v[7]);
    dft4<SIGN>(v[8], v[9], v[10], v[11]);
    dft4<SIGN>(v[12], v[13], v[14], v[15]);
    // v[4 k + q] is output k + 4 q: transpose
    V t;
    t = v[1]; v[1] = v[4]; v[4] = t;    t = v[2]; v[2] = v[8]; v[8] = t;     t = v[3]; v[3] = v[12]; v[12] = t;
    t = v[6]; v[6] = v[9]; v[9] = t;    t = v[7]; v[7] = v[13]; v[13] = t;   t = v[11]; v[11] = v[14]; v[14] = t;
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
template <typename V, int R, bool FWD, class LD, class ST>
__host__ __device__ __forceinline__ void fft_stage(const FftPlan &pl, int s, const V *__restrict__ tws, int tx, int T,
                                                   LD ld, ST st) {
  const int m = pl.m[s], L = m * R, nbf = pl.n / R;
  const V *tw = tws + pl.tw[s];
  for (int b = tx; b < nbf; b += T) {
    const int blk = fft_div(b, m, pl.magic[s]), j = b - blk * m, base = blk * L + j;
    V v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(base + r * m);
    if (FWD) {
      Dft<V, R, -1>::run(v);
      if (m > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = cmulw(v[q], tw[(q - 1) * m + j]);
      }
    } else {
      if (m > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) v[q] = cmulc(v[q], tw[(q - 1) * m + j]);
      }
      Dft<V, R, +1>::run(v);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) st(base + r * m, v[r]);
  }
}
// (only FP32 plans hold radix 16, and only at the lengths of fft_fixed.cuh)
template <typename V, bool FWD, class LD, class ST>
__host__ __device__ __forceinline__ void fft_stage_any(const FftPlan &pl, int s, const V *__restrict__ tws, int tx,
                                                       int T, LD ld, ST st) {
  switch (pl.R[s]) {  // uniform over the grid
    case 16:
      if (sizeof(V) == 8) fft_stage<V, sizeof(V) == 8 ? 16 : 2, FWD>(pl, s, tws, tx, T, ld, st);
      break;
    case 8: fft_stage<V, 8, FWD>(pl, s, tws, tx, T, ld, st); break;
    case 5: fft_stage<V, 5, FWD>(pl, s, tws, tx, T, ld, st); break;
    case 4: fft_stage<V, 4, FWD>(pl, s, tws, tx, T, ld, st); break;
    case 3: fft_stage<V, 3, FWD>(pl, s, tws, tx, T, ld, st); break;
    default: fft_stage<V, 2, FWD>(pl, s, tws, tx, T, ld, st); break;
  }
}

// The middle of a convolution: the last forward stage (L = R, no twiddles), the multiply by
// the spectrum kr (position order, as the forward stages leave it), the first inverse stage.
template <typename V, int R, class LD, class ST>
__host__ __device__ __forceinline__ void fft_mid(const FftPlan &pl, const real_t<V> *__restrict__ kr, int tx, int T,
                                                 LD ld, ST st) {
  for (int b = tx; b < pl.n / R; b += T) {
    V v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(b * R + r);
    Dft<V, R, -1>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const real_t<V> k = kr[b * R + r];
      v[r].x *= k;
      v[r].y *= k;
    }
    Dft<V, R, +1>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) st(b * R + r, v[r]);
  }
}
template <typename V, class LD, class ST>
__host__ __device__ __forceinline__ void fft_mid_any(const FftPlan &pl, const real_t<V> *__restrict__ kr, int tx,
                                                     int T, LD ld, ST st) {
  switch (pl.R[pl.ns - 1]) {
    case 16:
      if (sizeof(V) == 8) fft_mid<V, sizeof(V) == 8 ? 16 : 2>(pl, kr, tx, T, ld, st);
      break;
    case 8: fft_mid<V, 8>(pl, kr, tx, T, ld, st); break;
    case 5: fft_mid<V, 5>(pl, kr, tx, T, ld, st); break;
    case 4: fft_mid<V, 4>(pl, kr, tx, T, ld, st); break;
    case 3: fft_mid<V, 3>(pl, kr, tx, T, ld, st); break;
    default: fft_mid<V, 2>(pl, kr, tx, T, ld, st); break;
  }
}

// A table of cnt entries: copied to shared memory at `to` (SMT; the caller's next barrier
// publishes it), or left where it is.
template <bool SMT, typename E>
__device__ __forceinline__ const E *fft_table(E *to, const E *__restrict__ from, int cnt, int flat, int nt) {
  if (!SMT) return from;
#pragma unroll 4
  for (int i = flat; i < cnt; i += nt) to[i] = __ldg(from + i);
  return to;
}
// shared memory of the tables: twiddles, then positions (passes 1 and 3), or half and khat
// (pass 2); in complex elements, kept a multiple of 16 bytes
template <typename V>
__host__ __device__ __forceinline__ int fft_tab_phi(int n, int ntw) {
  return (ntw + (2 * n + (int)sizeof(V) - 1) / (int)sizeof(V) + 1) & ~1;
}
template <typename V>
__host__ __device__ __forceinline__ int fft_tab_u(int n, int ntw) { return (ntw + n + n + 1) & ~1; }

// Two neighbouring rows of one frequency of W (its row stride is even): one store.
__device__ __forceinline__ void store_pair(double2 *w, double2 a, double2 b) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(w), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y) : "memory");
}
__device__ __forceinline__ void store_pair(float2 *w, float2 a, float2 b) {
  *reinterpret_cast<float4 *>(w) = make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void load_pair(const double2 *w, double2 &a, double2 &b) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(w) : "memory");
}
__device__ __forceinline__ void load_pair(const float2 *w, float2 &a, float2 &b) {
  const float4 q = *reinterpret_cast<const float4 *>(w);
  a = make_float2(q.x, q.y);
  b = make_float2(q.z, q.w);
}

// ---------------------------------------------------------------------------------
// pass 1: rows -> transposed half spectrum.  The CTA's pairs of rows (threadIdx.y: pair;
// row0 = 2 blockDim.y blockIdx.x) of d.src (nrows x Nphi) are multiplied by d.inscale[i]
// (kalnajs.hpp:51: R^{3/2} Sigma; NULL = 1), packed two rows per complex transform,
// transformed forward along phi and unpacked into W[m * ldw + i], m < Nc (ldw even).
// pos[m]: where the transform leaves frequency m.
template <typename V, bool SMT>
__global__ void __launch_bounds__(kFftMaxThreads, 2) k_phi_fwd(const FftDisk<V> d, int b,
                                                              int nrows, int ldw, const FftPlan pl,
                                                              const V *__restrict__ gtw,
                                                              const unsigned short *__restrict__ gpos, int log2nb) {
  using T = real_t<V>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = pl.n, np = fft_pad_len<V>(n), tx = threadIdx.x, nx = blockDim.x, nb = 1 << log2nb;
  const int flat = threadIdx.y * nx + tx, nt = nb * nx;
  V *sm = reinterpret_cast<V *>(smem_raw), *all = sm + (SMT ? fft_tab_phi<V>(n, pl.ntw) : 0);
  V *buf = all + threadIdx.y * np;
  const V *tws = fft_table<SMT>(sm, gtw, pl.ntw, flat, nt);
  const unsigned short *pos = fft_table<SMT>(reinterpret_cast<unsigned short *>(sm + pl.ntw), gpos, n, flat, nt);
  const int row0 = blockIdx.x * 2 * nb;
  const int r0 = row0 + 2 * threadIdx.y, r1 = r0 + 1;
  const T a0 = r0 < nrows ? (d.inscale ? d.inscale[r0] : (T)1) : (T)0;
  const T a1 = r1 < nrows ? (d.inscale ? d.inscale[r1] : (T)1) : (T)0;
  const T *src = b ? d.src[1] : d.src[0];
  const T *s0 = src + (size_t)(r0 < nrows ? r0 : 0) * n, *s1 = src + (size_t)(r1 < nrows ? r1 : 0) * n;
  auto ldg = [&](int i) { return cx<V>(r0 < nrows ? a0 * s0[i] : (T)0, r1 < nrows ? a1 * s1[i] : (T)0); };
  auto lds = [&](int i) { return buf[fft_pad<V>(i)]; };
  auto sts = [&](int i, V v) { buf[fft_pad<V>(i)] = v; };
  pdl_wait();
  pdl_trigger();
  if (SMT) __syncthreads();
  fft_stage_any<V, true>(pl, 0, tws, tx, nx, ldg, sts);
  __syncthreads();
  for (int s = 1; s < pl.ns; ++s) {
    fft_stage_any<V, true>(pl, s, tws, tx, nx, lds, sts);
    __syncthreads();
  }
  const int Nc = n / 2 + 1;
  const T hf = (T)0.5;
#pragma unroll 2
  for (int idx = flat; idx < nb * Nc; idx += nt) {
    const int m = idx >> log2nb, t = idx & (nb - 1);
    const V *Z = all + t * np;
    const V a = Z[fft_pad<V>(pos[m])], c = Z[fft_pad<V>(pos[m == 0 ? 0 : n - m])];
    const int q0 = row0 + 2 * t;
    // (an odd last row's partner is the row stride's padding)
    if (q0 < nrows)
      store_pair(d.W + (size_t)m * ldw + q0, cx<V>(hf * (a.x + c.x), hf * (a.y - c.y)),
                 cx<V>(hf * (a.y + c.y), hf * (c.x - a.x)));
  }
}

// pass 2: per mode m: the length-2N transform of W[m][0..N) (zero beyond), times khat
// (kalnajs.hpp:53-56), inverse, W[m][0..N).  One mode per CTA; threadIdx.y: parity of p.
// d.kr[(2 m + parity) N + position]; half[j] = e^{-2 pi i j / 2N}, j < N.
template <typename V, bool SMT>
__global__ void __launch_bounds__(kFftMaxThreads, 2) k_u_conv(const FftDisk<V> d, int ldw,
                                                             const FftPlan pl, const V *__restrict__ gtw,
                                                             const V *__restrict__ ghalf) {
  using T = real_t<V>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = pl.n, np = fft_pad_len<V>(n), tx = threadIdx.x, nx = blockDim.x, odd = threadIdx.y;
  const int flat = odd * nx + tx, nt = 2 * nx;
  V *sm = reinterpret_cast<V *>(smem_raw), *all = sm + (SMT ? fft_tab_u<V>(n, pl.ntw) : 0);
  V *buf = all + odd * np;
  const V *tws = fft_table<SMT>(sm, gtw, pl.ntw, flat, nt);
  const V *half = fft_table<SMT>(sm + pl.ntw, ghalf, n, flat, nt);
  const T *k = fft_table<SMT>(reinterpret_cast<T *>(sm + pl.ntw + n), d.kr + (size_t)2 * blockIdx.x * n, 2 * n, flat,
                              nt) + odd * n;
  V *x = d.W + (size_t)blockIdx.x * ldw;
  auto ldg = [&](int i) { return odd ? cmulw(x[i], half[i]) : x[i]; };
  auto lds = [&](int i) { return buf[fft_pad<V>(i)]; };
  auto sts = [&](int i, V v) { buf[fft_pad<V>(i)] = v; };
  const int last = pl.ns - 1;
  pdl_wait();
  pdl_trigger();
  if (d.ctl && blockIdx.x == 0 && flat == nt - 1) finalize_pending(d.ctl);
  if (SMT) __syncthreads();
  if (last == 0) {
    fft_mid_any<V>(pl, k, tx, nx, ldg, sts);
  } else {
    fft_stage_any<V, true>(pl, 0, tws, tx, nx, ldg, sts);
    __syncthreads();
    for (int s = 1; s < last; ++s) {
      fft_stage_any<V, true>(pl, s, tws, tx, nx, lds, sts);
      __syncthreads();
    }
    fft_mid_any<V>(pl, k, tx, nx, lds, sts);
    for (int s = last - 1; s >= 0; --s) {
      __syncthreads();
      fft_stage_any<V, false>(pl, s, tws, tx, nx, lds, sts);
    }
  }
  __syncthreads();
  // E[j] + conj(half[j]) O[j]: the threads of both transforms share the sums
#pragma unroll 4
  for (int j = flat; j < n; j += nt) x[j] = cadd(all[fft_pad<V>(j)], cmulc(all[np + fft_pad<V>(j)], half[j]));
}

// The spectrum table of pass 2: W holds the phi half spectra of the kernel samples at all
// 2N wrapped offsets, [m][p].  One CTA per (mode, parity): even frequencies transform
// x[j] + x[j + N], odd ones (x[j] - x[j + N]) e^{-2 pi i j / 2N}.  Only real parts are kept:
// the kernel is even in both offsets.
template <typename V>
__global__ void __launch_bounds__(kFftMaxThreads) k_u_khat(const V *__restrict__ W, int ldw, const FftPlan pl,
                                                          const V *__restrict__ tws, const V *__restrict__ half,
                                                          real_t<V> *__restrict__ kr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *buf = reinterpret_cast<V *>(smem_raw);
  const int n = pl.n, tx = threadIdx.x, nx = blockDim.x, mode = blockIdx.x >> 1, odd = blockIdx.x & 1;
  const V *x = W + (size_t)mode * ldw;
  auto ldg = [&](int i) { return odd ? cmulw(csub(x[i], x[i + n]), half[i]) : cadd(x[i], x[i + n]); };
  auto lds = [&](int i) { return buf[fft_pad<V>(i)]; };
  auto sts = [&](int i, V v) { buf[fft_pad<V>(i)] = v; };
  fft_stage_any<V, true>(pl, 0, tws, tx, nx, ldg, sts);
  __syncthreads();
  for (int s = 1; s < pl.ns; ++s) {
    fft_stage_any<V, true>(pl, s, tws, tx, nx, lds, sts);
    __syncthreads();
  }
  real_t<V> *k = kr + (size_t)blockIdx.x * n;
  for (int i = tx; i < n; i += nx) k[i] = buf[fft_pad<V>(i)].x;
}

// pass 3: transposed half spectrum -> rows.  Two Hermitian rows are packed into one
// complex inverse transform (FFTW c2r semantics: the imaginary parts of the m=0 and
// Nyquist bins are ignored), then out[i][j] = d.outscale[i] x (kalnajs.hpp:58-62).
template <typename V, bool SMT>
__global__ void __launch_bounds__(kFftMaxThreads, 2) k_phi_inv(const FftDisk<V> d, int nrows,
                                                              int ldw, const FftPlan pl, const V *__restrict__ gtw,
                                                              const unsigned short *__restrict__ gpos, int log2nb) {
  using T = real_t<V>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = pl.n, np = fft_pad_len<V>(n), tx = threadIdx.x, nx = blockDim.x, nb = 1 << log2nb;
  const int flat = threadIdx.y * nx + tx, nt = nb * nx;
  V *sm = reinterpret_cast<V *>(smem_raw), *all = sm + (SMT ? fft_tab_phi<V>(n, pl.ntw) : 0);
  V *buf = all + threadIdx.y * np;
  const V *tws = fft_table<SMT>(sm, gtw, pl.ntw, flat, nt);
  const unsigned short *pos = fft_table<SMT>(reinterpret_cast<unsigned short *>(sm + pl.ntw), gpos, n, flat, nt);
  const int row0 = blockIdx.x * 2 * nb;
  const int r0 = row0 + 2 * threadIdx.y, r1 = r0 + 1;
  const T p0 = r0 < nrows ? d.outscale[r0] : (T)0, p1 = r1 < nrows ? d.outscale[r1] : (T)0;
  pdl_wait();
  pdl_trigger();
  if (SMT) __syncthreads();
  const int Nc = n / 2 + 1;
#pragma unroll 2
  for (int idx = flat; idx < nb * Nc; idx += nt) {
    const int m = idx >> log2nb, t = idx & (nb - 1);
    const int q0 = row0 + 2 * t;
    V A = cx<V>((T)0, (T)0), B = A;
    if (q0 < nrows) load_pair(d.W + (size_t)m * ldw + q0, A, B);
    if (m == 0 || 2 * m == n) A.y = B.y = (T)0;
    V *Z = all + t * np;
    Z[fft_pad<V>(pos[m])] = cx<V>(A.x - B.y, A.y + B.x);
    if (m > 0 && n - m >= Nc) Z[fft_pad<V>(pos[n - m])] = cx<V>(A.x + B.y, B.x - A.y);
  }
  __syncthreads();
  auto lds = [&](int i) { return buf[fft_pad<V>(i)]; };
  auto sts = [&](int i, V v) { buf[fft_pad<V>(i)] = v; };
  T *out = d.out;
  const int o0 = r0 * n;  // at most 4096 x 8192 elements
  auto stg = [&](int i, V v) {
    if (r0 < nrows) out[o0 + i] = p0 * v.x;
    if (r1 < nrows) out[o0 + n + i] = p1 * v.y;
  };
  for (int s = pl.ns - 1; s > 0; --s) {
    fft_stage_any<V, false>(pl, s, tws, tx, nx, lds, sts);
    __syncthreads();
  }
  fft_stage_any<V, false>(pl, 0, tws, tx, nx, lds, stg);
}

}  // namespace dg
