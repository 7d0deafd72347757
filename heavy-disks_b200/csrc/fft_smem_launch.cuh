// Host side of fft_smem.cuh for one element type: plans, tables and launches (included once per
// type: a file's kernels are loaded as one image, so a disk loads those of its own type alone).
// First disk of a process, dg_create: FP64 128^2 11.1 ms with all kernels of the plain path in
// one file, 7.5 so; mixed 256^2 39 and 29.4.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "fft_smem.cuh"
#include "kernels.h"

namespace dg {

// Stage radices: those of fft_fixed.cuh for its lengths; else the factors 5 and 3 first, then
// the power of two in radices 8 and 4.
template <typename V> static bool make_plan(int n, FftPlan *pl) {
  *pl = FftPlan{};
  if (n < 1) return false;
  pl->n = n;
  auto add = [&](int R) { pl->R[pl->ns++] = R; };
  pl->fixed = fixed_length<V>(n);
  if (pl->fixed) {
    int R[5];
    fixed_radices<V>(n, R);
    for (int r : R)
      if (r > 1) add(r);
  } else {
    int e = 0, rest = n;
    while (rest % 2 == 0) { ++e; rest /= 2; }
    while (rest % 5 == 0) { add(5); rest /= 5; }
    while (rest % 3 == 0) { add(3); rest /= 3; }
    if (rest != 1) return false;
    while (e > 0) {
      const int k = (e <= 3) ? e : (e == 4 ? 2 : 3);
      add(1 << k);
      e -= k;
    }
  }
  if (pl->ns == 0) return false;  // n = 1
  int L = n;
  for (int s = 0; s < pl->ns; ++s) {
    const int R = pl->R[s], m = L / R;
    pl->m[s] = m;
    pl->magic[s] = m > 1 ? (unsigned)(((1ull << 32) + m - 1) / m) : 0u;
    pl->tw[s] = pl->ntw;
    pl->ntw += (R - 1) * m;
    L = m;
  }
  // threads per transform: one butterfly each in a radix-8 stage of a long transform; a
  // short one, whose few CTAs leave the SMs idle anyway, takes more for its loads and stores
  // (FP64 step at 64^2 / 128^2: 19.5 / 21.2 us with n / 4 threads, 18.6 / 20.5 with n / 2;
  // at 512^2 34.9 us with n / 4, 32.7 with n / 8)
  int T = n >= 512 ? (n + 7) / 8 : (n + 1) / 2;
  if (T > kFftMaxThreads / 2) T = kFftMaxThreads / 2;
  pl->threads = T < 1 ? 1 : T;
  return true;
}
// Host tables of a plan: the stage twiddles and the position of every frequency.
template <typename V>
void fft_tables(const FftPlan &pl, std::vector<V> *tw, std::vector<unsigned short> *pos) {
  using T = real_t<V>;
  tw->assign(pl.ntw, V{});
  for (int s = 0; s < pl.ns; ++s) {
    const int R = pl.R[s], m = pl.m[s], L = R * m;
    for (int q = 1; q < R; ++q)
      for (int j = 0; j < m; ++j) {
        const long double a = -2.0L * 3.141592653589793238462643383279502884L * (long double)(j * q) / (long double)L;
        (*tw)[pl.tw[s] + (q - 1) * m + j] = cx<V>((T)cosl(a), (T)sinl(a));
      }
  }
  pos->assign(pl.n, 0);
  for (int k = 0; k < pl.n; ++k) {  // k = q0 + R0 (q1 + R1 (...)) sits at q0 m0 + q1 m1 + ...
    int r = k, at = 0;
    for (int s = 0; s < pl.ns; ++s) {
      at += (r % pl.R[s]) * pl.m[s];
      r /= pl.R[s];
    }
    (*pos)[k] = (unsigned short)at;
  }
}

// Lengths whose tables go to shared memory (the SMT forms).
static bool fft_smt(int n) { return n <= 512; }

// Plans and device tables of an Nu x Nphi grid, in one buffer.
template <typename V>
cudaError_t build_fft_tables(int Nu, int Nphi, FftTables<V> *ft) {
  using T = real_t<V>;
  if (!make_fft_plan<V>(Nphi, &ft->phi) || !make_fft_plan<V>(Nu, &ft->u)) return cudaErrorInvalidValue;
  // Raise the dynamic shared-memory limit of the kernels that this grid launches, for each
  // handle: the limit belongs to the device, and a process may have handles on several.  (Of no
  // others: the first call that names a kernel loads it.)
  for (const FftPlan *pl : {&ft->phi, &ft->u}) {
    const cudaError_t e = pl->fixed ? fixed_attrs<V>(pl->n) : cudaSuccess;
    if (e != cudaSuccess) return e;
  }
  std::vector<const void *> fns;
  if (!ft->phi.fixed || Nu % 2) {
    const bool smt = fft_smt(Nphi);
    fns.push_back(smt ? (const void *)k_phi_fwd<V, true> : (const void *)k_phi_fwd<V, false>);
    fns.push_back(smt ? (const void *)k_phi_inv<V, true> : (const void *)k_phi_inv<V, false>);
  }
  if (!ft->u.fixed)
    fns.push_back(fft_smt(Nu) ? (const void *)k_u_conv<V, true> : (const void *)k_u_conv<V, false>);
  for (const void *f : fns) {
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
    if (e != cudaSuccess) return e;
  }
  std::vector<V> t1, t2;
  std::vector<unsigned short> p1, p2;
  fft_tables<V>(ft->phi, &t1, &p1);
  fft_tables<V>(ft->u, &t2, &p2);
  const size_t n1 = t1.size(), n2 = t2.size(), per = sizeof(V) / sizeof(unsigned short);
  std::vector<V> t(n1 + n2 + Nu + ((size_t)Nphi + Nu + per - 1) / per);
  std::copy(t1.begin(), t1.end(), t.begin());
  std::copy(t2.begin(), t2.end(), t.begin() + n1);
  for (int j = 0; j < Nu; ++j) {
    const long double a = -3.141592653589793238462643383279502884L * (long double)j / (long double)Nu;
    t[n1 + n2 + j] = cx<V>((T)cosl(a), (T)sinl(a));
  }
  unsigned short *ps = reinterpret_cast<unsigned short *>(t.data() + n1 + n2 + Nu);
  std::copy(p1.begin(), p1.end(), ps);
  std::copy(p2.begin(), p2.end(), ps + Nphi);
  cudaError_t e = cudaMalloc((void **)&ft->buf, t.size() * sizeof(V));
  if (e == cudaSuccess) e = cudaMemcpy(ft->buf, t.data(), t.size() * sizeof(V), cudaMemcpyHostToDevice);
  ft->twPhi = ft->buf;
  ft->twU = ft->buf + n1;
  ft->half = ft->twU + n2;
  ft->posPhi = reinterpret_cast<const unsigned short *>(ft->half + Nu);
  ft->posU = ft->posPhi + Nphi;
  return e;
}

// Transforms per CTA: up to 4 (their rows share the 128-byte runs of W), while every SM
// still gets a CTA and they fit its shared memory with their tables (two FP64 transforms do up
// to some 6300 points; one of 8192 takes 150 KB).
template <typename V> static int fft_log2_batch(const FftPlan &pl, int count) {
  const size_t one = fft_pad_len<V>(pl.n), tab = fft_smt(pl.n) ? fft_tab_phi<V>(pl.n, pl.ntw) : 0;
  int lg = 0;
  while (lg < 2 && (pl.threads << (lg + 1)) <= kFftMaxThreads && (count >> (lg + 1)) >= sm_count() &&
         ((one << (lg + 1)) + tab) * sizeof(V) <= kMaxSmem)
    ++lg;
  return lg;
}

template <typename V>
cudaError_t launch_phi_fwd(const FftDisk<V> &d, int b, int nrows, int ldw,
                           const FftTables<V> &ft, cudaStream_t st) {
  const FftPlan &pl = ft.phi;
  if (pl.fixed && nrows % 2 == 0) return fixed_phi_fwd<V>(pl.n, d, b, nrows, ldw, ft.twPhi, st);
  const int pairs = (nrows + 1) / 2, lg = fft_log2_batch<V>(pl, pairs), nb = 1 << lg;
  const bool smt = fft_smt(pl.n);
  const size_t sm = ((size_t)nb * fft_pad_len<V>(pl.n) + (smt ? fft_tab_phi<V>(pl.n, pl.ntw) : 0)) * sizeof(V);
  return launch_pdl(smt ? k_phi_fwd<V, true> : k_phi_fwd<V, false>, dim3((pairs + nb - 1) / nb),
                    dim3(pl.threads, nb), sm, st, d, b, nrows, ldw, pl, ft.twPhi, ft.posPhi, lg);
}

template <typename V>
cudaError_t launch_u_conv(const FftDisk<V> &d, int Nc, int ldw,
                          const FftTables<V> &ft, cudaStream_t st) {
  const FftPlan &pl = ft.u;
  if (pl.fixed) return fixed_u_conv<V>(pl.n, d, Nc, ldw, ft.twU, ft.half, st);
  const bool smt = fft_smt(pl.n);
  const size_t sm = ((size_t)2 * fft_pad_len<V>(pl.n) + (smt ? fft_tab_u<V>(pl.n, pl.ntw) : 0)) * sizeof(V);
  return launch_pdl(smt ? k_u_conv<V, true> : k_u_conv<V, false>, dim3(Nc), dim3(pl.threads, 2), sm, st, d,
                    ldw, pl, ft.twU, ft.half);
}

template <typename V>
cudaError_t launch_phi_inv(const FftDisk<V> &d, int nrows, int ldw,
                           const FftTables<V> &ft, cudaStream_t st) {
  const FftPlan &pl = ft.phi;
  if (pl.fixed && nrows % 2 == 0) return fixed_phi_inv<V>(pl.n, d, nrows, ldw, ft.twPhi, st);
  const int pairs = (nrows + 1) / 2, lg = fft_log2_batch<V>(pl, pairs), nb = 1 << lg;
  const bool smt = fft_smt(pl.n);
  const size_t sm = ((size_t)nb * fft_pad_len<V>(pl.n) + (smt ? fft_tab_phi<V>(pl.n, pl.ntw) : 0)) * sizeof(V);
  return launch_pdl(smt ? k_phi_inv<V, true> : k_phi_inv<V, false>, dim3((pairs + nb - 1) / nb),
                    dim3(pl.threads, nb), sm, st, d, nrows, ldw, pl, ft.twPhi, ft.posPhi, lg);
}

}  // namespace dg
