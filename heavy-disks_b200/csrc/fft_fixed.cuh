// The three passes of the Kalnajs convolution (fft_smem.cuh) for lengths known at compile
// time, those of the grids in use: FP64 64, 128, 256, 384, 512, 768, 1024 and 2048
// (fft_fixed_f64.cu), FP32 256 .. 4096 as 2^k, and 3 2^k and 5 2^k with k >= 7 (fft_fixed_f32.cu).
// A length is 200 to 270 KB of object code, so every other one takes the runtime form.  Same
// transforms, same tables layout per plan; what the compiler knows here is every stride.
//
// The runtime-length form is bound by instruction issue, two thirds of them index arithmetic
// (pass 2 at 1024 points, FP32: some 300 instructions per element, issue slots 64 % busy).
// Here element i sits at i + i / LAST with LAST the radix of the last stage, and every earlier
// stage's stride m is a multiple of LAST: then position(base + r m) = position(base) +
// r (m + m / LAST), an immediate offset, and each wavefront (LAST consecutive elements, or
// LAST blocks of the last stage) covers distinct banks.  Runtime lengths -> these, whole step:
// mixed 256^2 21.7 -> 16.7 us, 512^2 27.7 -> 20.9, 2048^2 162 -> 129, 4096^2 617 -> 519;
// FP64 1024^2 70 -> 62 us.
//
// Frequencies cross shared memory in natural order: the last forward stage of pass 1 writes
// them so and the first inverse stage of pass 3 reads them so (a barrier between reading and
// writing, each thread holding one butterfly), which makes the real-transform packing linear.
//
// CTAs walk their modes or row groups with a grid stride, so tables copied to shared memory
// serve several transforms where the grid is larger than the GPU.
#pragma once

#include "fft_smem.cuh"

namespace dg {

// Radices of length N: an odd factor 3 or 5, then powers of two, LAST at the end.
template <typename V, int N> struct FixedPlan {
  static constexpr int LAST = sizeof(V) == 8 ? 16 : 8;
  static constexpr int ODD = N % 3 == 0 ? 3 : (N % 5 == 0 ? 5 : 1);
  static constexpr int REST = N / ODD / LAST;  // a power of two
  static_assert(N == ODD * LAST * REST && (REST & (REST - 1)) == 0, "supported lengths");
  static constexpr int RMAX = sizeof(V) == 8 ? 16 : 8;
  // REST as radices A B C (1 = absent), balanced: a radix-2 stage costs a trip through shared
  // memory like any other (FP32 512 = 2 16 16 made the 512^2 step 25.9 us, 4 8 16 20.8)
  static constexpr int C =
      REST <= RMAX ? REST : (REST == 2 * RMAX ? RMAX / 2 : (REST == 64 && RMAX == 16 ? 8 : RMAX));
  static constexpr int RC = REST / C;
  static constexpr int B = RC <= RMAX ? RC : (RC == 2 * RMAX ? RMAX / 2 : RMAX);
  static constexpr int A = RC / B;
  static_assert(A <= RMAX, "supported lengths");
  static constexpr int R[5] = {ODD, A, B, C, LAST};
  static constexpr int first = ODD > 1 ? 0 : (A > 1 ? 1 : (B > 1 ? 2 : (C > 1 ? 3 : 4)));
  // stride and twiddle offset of slot s
  __host__ __device__ static constexpr int m(int s) {
    int L = N;
    for (int k = 0; k <= s; ++k) L /= R[k];
    return L;
  }
  __host__ __device__ static constexpr int tw(int s) {
    int o = 0;
    for (int k = 0; k < s; ++k) o += R[k] > 1 ? (R[k] - 1) * m(k) : 0;
    return o;
  }
  static constexpr int ntw = tw(4) + (LAST - 1);
  __host__ __device__ static constexpr int pad(int i) { return i + i / LAST; }
  static constexpr int np = N + N / LAST;
  // shared memory of the tables, in elements of V, rounded to 16 bytes
  static constexpr int tab = (ntw + 1) & ~1;
};

// Stage in slot S of one transform (fft_stage with every stride known): threads tx = 0 .. T-1.
template <typename V, int N, int S, bool FWD, class LD, class ST>
__device__ __forceinline__ void fixed_stage(const V *__restrict__ tws, int tx, int T, LD ld, ST st) {
  using P = FixedPlan<V, N>;
  constexpr int R = P::R[S], m = P::m(S), L = m * R;
  static_assert(m % P::LAST == 0, "strides keep the padding linear");
  const V *tw = tws + P::tw(S);
#pragma unroll 1
  for (int b = tx; b < N / R; b += T) {
    const int blk = b / m, j = b % m, base = blk * L + j;
    const V *twj = tw + j;
    V v[R];
    ld(v, base, m);
    if (FWD) {
      Dft<V, R, -1>::run(v);
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = cmulw(v[q], twj[(q - 1) * m]);
    } else {
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = cmulc(v[q], twj[(q - 1) * m]);
      Dft<V, R, +1>::run(v);
    }
    st(v, base, m);
  }
}

// Element access of a stage with stride m: shared memory ...
template <typename V, int N, int R> struct SmemIO {
  V *buf;
  __device__ __forceinline__ void operator()(V (&v)[R], int base, int m) const {
    const V *p = buf + FixedPlan<V, N>::pad(base);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[FixedPlan<V, N>::pad(r * m)];
  }
};
template <typename V, int N, int R> struct SmemSt {
  V *buf;
  __device__ __forceinline__ void operator()(V (&v)[R], int base, int m) const {
    V *p = buf + FixedPlan<V, N>::pad(base);
#pragma unroll
    for (int r = 0; r < R; ++r) p[FixedPlan<V, N>::pad(r * m)] = v[r];
  }
};

// The stages between the first and the last, in shared memory, each followed (forward) or
// preceded (inverse) by a barrier.
template <typename V, int N, int S, bool FWD>
__device__ __forceinline__ void fixed_smem_stage(const V *tws, V *buf, int tx, int T) {
  using P = FixedPlan<V, N>;
  if constexpr (P::R[S] > 1) {
    constexpr int R = P::R[S];
    fixed_stage<V, N, S, FWD>(tws, tx, T, SmemIO<V, N, R>{buf}, SmemSt<V, N, R>{buf});
    __syncthreads();
  }
}
template <typename V, int N>
__device__ __forceinline__ void fixed_forward_mid(const V *tws, V *buf, int tx, int T) {
  constexpr int f = FixedPlan<V, N>::first;
  if constexpr (f < 1) fixed_smem_stage<V, N, 1, true>(tws, buf, tx, T);
  if constexpr (f < 2) fixed_smem_stage<V, N, 2, true>(tws, buf, tx, T);
  if constexpr (f < 3) fixed_smem_stage<V, N, 3, true>(tws, buf, tx, T);
}
template <typename V, int N>
__device__ __forceinline__ void fixed_inverse_mid(const V *tws, V *buf, int tx, int T) {
  constexpr int f = FixedPlan<V, N>::first;
  if constexpr (f < 3) fixed_smem_stage<V, N, 3, false>(tws, buf, tx, T);
  if constexpr (f < 2) fixed_smem_stage<V, N, 2, false>(tws, buf, tx, T);
  if constexpr (f < 1) fixed_smem_stage<V, N, 1, false>(tws, buf, tx, T);
}

// Frequency of element 0 of block b of the last stage; its element q holds that + q N / LAST.
template <typename V, int N>
__device__ __forceinline__ int fixed_freq(int b) {
  using P = FixedPlan<V, N>;
  // b = ((d0 A + d1) B + d2) C + d3 -> d0 + ODD (d1 + A (d2 + B d3))
  const int d3 = b % P::C, b2 = b / P::C, d2 = b2 % P::B, b1 = b2 / P::B, d1 = b1 % P::A, d0 = b1 / P::A;
  return d0 + P::ODD * (d1 + P::A * (d2 + P::B * d3));
}

// ---------------------------------------------------------------------------------
// pass 1.  threadIdx.y: pair of rows within the group; nrows a multiple of 2 blockDim.y.
template <typename V, int N, int LB, int MINB>
__global__ void __launch_bounds__(LB, MINB) k_phi_fwd_n(const FftDisk<V> d,
                                                                    int b, int ngroups, int ldw,
                                                                    const V *__restrict__ gtw, int log2nb) {
  using T = real_t<V>;
  using P = FixedPlan<V, N>;
  constexpr int R0 = P::R[P::first], LAST = P::LAST, Q = N / LAST, Nc = N / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tx = threadIdx.x, nx = blockDim.x, nb = 1 << log2nb, flat = threadIdx.y * nx + tx, nt = nb * nx;
  V *tws = reinterpret_cast<V *>(smem_raw), *all = tws + P::tab, *buf = all + threadIdx.y * P::np;
  for (int i = flat; i < P::ntw; i += nt) tws[i] = __ldg(gtw + i);
  const T *src = b ? d.src[1] : d.src[0];
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
    const int row0 = g * 2 * nb, r0 = row0 + 2 * threadIdx.y;
    {
      const T a0 = d.inscale ? d.inscale[r0] : (T)1, a1 = d.inscale ? d.inscale[r0 + 1] : (T)1;
      const T *s0 = src + (size_t)r0 * N;
      auto ld = [&](V(&v)[R0], int base, int m) {
        const T *p = s0 + base;
#pragma unroll
        for (int r = 0; r < R0; ++r) v[r] = cx<V>(a0 * p[r * m], a1 * p[N + r * m]);
      };
      fixed_stage<V, N, P::first, true>(tws, tx, nx, ld, SmemSt<V, N, R0>{buf});
    }
    __syncthreads();
    fixed_forward_mid<V, N>(tws, buf, tx, nx);
    {
      V v[LAST];
      const bool on = tx < Q;
      if (on) {
        const V *p = buf + tx * (LAST + 1);
#pragma unroll
        for (int r = 0; r < LAST; ++r) v[r] = p[r];
        Dft<V, LAST, -1>::run(v);
      }
      __syncthreads();
      if (on) {
        const int k = fixed_freq<V, N>(tx);
        V *p = buf + P::pad(k);
        // k < Q: the pads of k and q Q add (Q is a multiple of LAST, or the sum stays below)
#pragma unroll
        for (int q = 0; q < LAST; ++q) {
          if (Q % LAST == 0) p[P::pad(q * Q)] = v[q];
          else buf[P::pad(k + q * Q)] = v[q];
        }
      }
      __syncthreads();
    }
    const T hf = (T)0.5;
#pragma unroll 2
    for (int idx = flat; idx < nb * Nc; idx += nt) {
      const int m = idx >> log2nb, t = idx & (nb - 1), mc = m == 0 ? 0 : N - m;
      const V *Z = all + t * P::np;
      const V a = Z[P::pad(m)], c = Z[P::pad(mc)];
      store_pair(d.W + (size_t)m * ldw + row0 + 2 * t, cx<V>(hf * (a.x + c.x), hf * (a.y - c.y)),
                 cx<V>(hf * (a.y + c.y), hf * (c.x - a.x)));
    }
    if (g + (int)gridDim.x < ngroups) __syncthreads();
  }
}

// pass 2.  threadIdx.y: parity of p.
template <typename V, int N, int LB, int MINB>
__global__ void __launch_bounds__(LB, MINB) k_u_conv_n(const FftDisk<V> d,
                                                                   int Nc, int ldw, const V *__restrict__ gtw,
                                                                   const V *__restrict__ ghalf) {
  using T = real_t<V>;
  using P = FixedPlan<V, N>;
  constexpr int R0 = P::R[P::first], LAST = P::LAST;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tx = threadIdx.x, nx = blockDim.x, odd = threadIdx.y, flat = odd * nx + tx, nt = 2 * nx;
  V *sm = reinterpret_cast<V *>(smem_raw), *all = sm + P::tab + N, *buf = all + odd * P::np;
  const V *tws = fft_table<true>(sm, gtw, P::ntw, flat, nt), *half = fft_table<true>(sm + P::tab, ghalf, N, flat, nt);
  pdl_wait();
  pdl_trigger();
  if (d.ctl && blockIdx.x == 0 && flat == nt - 1) finalize_pending(d.ctl);
  __syncthreads();
  for (int mode = blockIdx.x; mode < Nc; mode += gridDim.x) {
    V *x = d.W + (size_t)mode * ldw;
    const T *k = d.kr + ((size_t)2 * mode + odd) * N;
    auto ld = [&](V(&v)[R0], int base, int m) {
#pragma unroll
      for (int r = 0; r < R0; ++r) v[r] = x[base + r * m];
      if (odd) {
#pragma unroll
        for (int r = 0; r < R0; ++r) v[r] = cmulw(v[r], half[base + r * m]);
      }
    };
    fixed_stage<V, N, P::first, true>(tws, tx, nx, ld, SmemSt<V, N, R0>{buf});
    __syncthreads();
    fixed_forward_mid<V, N>(tws, buf, tx, nx);
#pragma unroll 1
    for (int b = tx; b < N / LAST; b += nx) {
      V v[LAST], *p = buf + b * (LAST + 1);
      // the spectrum's LAST values of this block, 16 bytes at a time
      T kk[LAST];
      const uint4 *k4 = reinterpret_cast<const uint4 *>(k + b * LAST);
#pragma unroll
      for (int r = 0; r < LAST * (int)sizeof(T) / 16; ++r) {
        const uint4 q = __ldg(k4 + r);
        memcpy(&kk[r * 16 / sizeof(T)], &q, 16);
      }
#pragma unroll
      for (int r = 0; r < LAST; ++r) v[r] = p[r];
      Dft<V, LAST, -1>::run(v);
#pragma unroll
      for (int r = 0; r < LAST; ++r) {
        v[r].x *= kk[r];
        v[r].y *= kk[r];
      }
      Dft<V, LAST, +1>::run(v);
#pragma unroll
      for (int r = 0; r < LAST; ++r) p[r] = v[r];
    }
    __syncthreads();
    fixed_inverse_mid<V, N>(tws, buf, tx, nx);
    fixed_stage<V, N, P::first, false>(tws, tx, nx, SmemIO<V, N, R0>{buf}, SmemSt<V, N, R0>{buf});
    __syncthreads();
#pragma unroll 4
    for (int j = flat; j < N; j += nt) x[j] = cadd(all[P::pad(j)], cmulc(all[P::np + P::pad(j)], half[j]));
    if (mode + (int)gridDim.x < Nc) __syncthreads();
  }
}

// pass 3.
template <typename V, int N, int LB, int MINB>
__global__ void __launch_bounds__(LB, MINB) k_phi_inv_n(const FftDisk<V> d,
                                                                    int ngroups, int ldw, const V *__restrict__ gtw,
                                                                    int log2nb) {
  using T = real_t<V>;
  using P = FixedPlan<V, N>;
  constexpr int R0 = P::R[P::first], LAST = P::LAST, Q = N / LAST, Nc = N / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tx = threadIdx.x, nx = blockDim.x, nb = 1 << log2nb, flat = threadIdx.y * nx + tx, nt = nb * nx;
  V *tws = reinterpret_cast<V *>(smem_raw), *all = tws + P::tab, *buf = all + threadIdx.y * P::np;
  for (int i = flat; i < P::ntw; i += nt) tws[i] = __ldg(gtw + i);
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
    const int row0 = g * 2 * nb, r0 = row0 + 2 * threadIdx.y;
#pragma unroll 2
    for (int idx = flat; idx < nb * Nc; idx += nt) {
      const int m = idx >> log2nb, t = idx & (nb - 1);
      V A, B;
      load_pair(d.W + (size_t)m * ldw + row0 + 2 * t, A, B);
      V *Z = all + t * P::np;
      if (m == 0 || m == N / 2) {
        Z[P::pad(m)] = cx<V>(A.x, B.x);
      } else {
        Z[P::pad(m)] = cx<V>(A.x - B.y, A.y + B.x);
        Z[P::pad(N - m)] = cx<V>(A.x + B.y, B.x - A.y);
      }
    }
    __syncthreads();
    {
      V v[LAST];
      const bool on = tx < Q;
      if (on) {
        const int k = fixed_freq<V, N>(tx);
        const V *p = buf + P::pad(k);
#pragma unroll
        for (int q = 0; q < LAST; ++q) {
          if (Q % LAST == 0) v[q] = p[P::pad(q * Q)];
          else v[q] = buf[P::pad(k + q * Q)];
        }
        Dft<V, LAST, +1>::run(v);
      }
      __syncthreads();
      if (on) {
        V *p = buf + tx * (LAST + 1);
#pragma unroll
        for (int r = 0; r < LAST; ++r) p[r] = v[r];
      }
      __syncthreads();
    }
    fixed_inverse_mid<V, N>(tws, buf, tx, nx);
    {
      const T p0 = d.outscale[r0], p1 = d.outscale[r0 + 1];
      T *out = d.out + (size_t)r0 * N;
      auto st = [&](V(&v)[R0], int base, int m) {
        T *o = out + base;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          o[r * m] = p0 * v[r].x;
          o[N + r * m] = p1 * v[r].y;
        }
      };
      fixed_stage<V, N, P::first, false>(tws, tx, nx, SmemIO<V, N, R0>{buf}, st);
    }
    if (g + (int)gridDim.x < ngroups) __syncthreads();
  }
}

}  // namespace dg
