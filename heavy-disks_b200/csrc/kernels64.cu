// Plain-method (FP64) kernels: fused hydro step, CFL reduction, forces, mode sums,
// Kalnajs kernel samples, and launchers for the shared-memory FFT passes.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "kernels.h"
#include "hydro64.cuh"
#include "fft_smem.cuh"
#include "step_ctl.cuh"

namespace dg {

// Mode-sum contribution of one cell: Sigma cos(m phi) dA and -Sigma sin(m phi) dA
// (diskmain.cpp:76-80).
__device__ __forceinline__ void add_modes(double *msum, int nmodes, double s, int j, double dphi, double dA) {
  double phi = (j + 0.5) * dphi;
  for (int m = 0; m < nmodes; ++m) {
    double sn, cs;
    sincos(m * phi, &sn, &cs);
    msum[2 * m] += s * cs * dA;
    msum[2 * m + 1] -= s * sn * dA;
  }
}

// ---------------------------------------------------------------------------------
__device__ __forceinline__ double up1(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double dn1(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// One time step (hydro64.cuh).  blockIdx.x: group of blockDim.x / 32 strips; blockIdx.y: band
// of `band` rows.  PIN: the pressure comes from a field (Gamma != 2, all but the first step of an
// uploaded state).
template <bool G2, int FM, bool PIN>
__global__ void __launch_bounds__(32 * kMaxWarps64, 3) k_hydro64(
    const double *__restrict__ Sig, const double *__restrict__ vR, const double *__restrict__ vp,
    const double *__restrict__ Phi, const double *__restrict__ gRin, const double *__restrict__ gpin,
    const double *__restrict__ Pin, double *__restrict__ So, double *__restrict__ vRo, double *__restrict__ vpo,
    double *__restrict__ Po, Ctl *ctl, const Geom64 g, int band) {
  __shared__ __align__(16) double tab[(kMaxBand64 + 6) * kRow64W];
  __shared__ double red[kMaxWarps64];
  const int Nu = g.Nu, Nphi = g.Nphi, tid = threadIdx.x, lane = tid & 31, nt = blockDim.x;
  const int iA = blockIdx.y * band, iB = min(iA + band, Nu);
  const int strip = blockIdx.x * (nt >> 5) + (tid >> 5), j0 = strip * kOutCols64;
  int j = (j0 - kHalo64 + lane) % Nphi;
  if (j < 0) j += Nphi;
  const bool live = j0 < Nphi;
  const bool outp = live && lane >= kHalo64 && lane < kHalo64 + kOutCols64 && j0 - kHalo64 + lane < Nphi;

  pdl_wait();  // dt, the state and the potential come from earlier kernels on the stream
  pdl_trigger();
  const StepInfo si = read_step_info(ctl, true);
  const double dt = si.dt;
  double msum[2 * kMaxModes];  // set only when the launch accumulates modes
  double lmax = 0.0;
  bool bad = false;

  if (!si.active) {
    // pass-through so a launch after the loop has ended leaves the state unchanged
    if (outp)
      for (int i = iA; i < iB; ++i) {
        const size_t k = (size_t)i * Nphi + j;
        So[k] = Sig[k]; vRo[k] = vR[k]; vpo[k] = vp[k];
        if (!G2) Po[k] = PIN ? Pin[k] : pres64(g, Sig[k]);
        lmax = fmax(lmax, cfl_rate64(g, i, So[k], vRo[k], vpo[k]));
      }
    finish_launch_deferred<0>(ctl, si, lmax, msum, red);
    return;
  }

  // row constants of rows iA-3 .. iB+2 (edge rows repeat), products with dt included
  for (int c = tid; c < (iB - iA + 6) * kRow64W; c += nt) {
    const int q = c % kRow64W, i = iA - 3 + c / kRow64W;
    // faces f = 0 .. Nu; row constants of the rows outside the grid are the edge rows'
    const bool face = q == hAf || q == hCl || q == hCr;
    const int row = max(0, min(i, face ? Nu : Nu - 1));
    const double v = g.rowtab[(size_t)row * kRow64W + q];
    tab[c] = (q == hCvol || q == hCphi || q == hCl || q == hCr) ? dt * v : v;
  }
  __syncthreads();

  if (live) {
    auto at = [&](int r) { return max(0, min(r, Nu - 1)) * Nphi + j; };  // at most 4096 x 8192
    int r = iA - 3;
    // the next row, in flight
    int x = at(r);
    double nS = Sig[x], nU = vR[x], nW = vp[x], nP = PIN ? Pin[x] : 0.0, nPh = FM == kForcePhi ? Phi[x] : 0.0;
    // row r-1 as loaded; pressure and potential of rows r-1 and r-2
    double S1 = 0, U1 = 0, W1 = 0, P1 = 0, P2 = 0, Ph1 = 0, Ph2 = 0;
    // rows r-2 and r-3 after the source; differences (row r-2) - (row r-3); slopes of row r-3
    double S2 = 0, u2 = 0, w2 = 0, S3 = 0, u3 = 0, w3 = 0, dS = 0, du = 0, dw = 0, kS = 0, kU = 0, kW = 0;
    // fluxes through the face between rows r-4 and r-3
    double F0 = 0, FR0 = 0, FP0 = 0, tsum = 0;
    const double *tc = tab;  // constants of row r
#pragma unroll 2  // the windows' shifts become renames
    for (int k = 0; r <= iB + 2; ++k, ++r, tc += kRow64W) {
      const double S = nS, U = nU, W = nW, Ph = nPh, P = G2 ? g.Kpoly * (S * S) : (PIN ? nP : pres64(g, S));
      x = at(r + 1);
      nS = Sig[x]; nU = vR[x]; nW = vp[x];
      if (PIN) nP = Pin[x];
      if (FM == kForcePhi) nPh = Phi[x];
      double s1 = 0, u1 = 0, w1 = 0;  // row r-1 after the source
      if (k >= 2) {
        // ---- source of row r-1 (hydro.hpp:73-96; kalnajs.hpp:71-78 for the forces) ----
        const double *t = tc - kRow64W;
        const double dPR = P - P2, dPp = dn1(P1) - up1(P1);
        double aR = t[hGstar], gp = 0.0;
        if (FM == kForcePhi) {
          aR = fma(Ph - Ph2, t[hPhiu], aR);
          gp = dn1(Ph1) - up1(Ph1);  // times -1 / (2 R dphi) below
        } else if (FM == kForceArrays) {
          aR += gRin[at(r - 1)];
        }
        double rs, tR = dPR * t[hInvdRc];
        if (rcp_ok64(S1)) rs = rcp64(S1);
        else rs = 1.0 / S1;
        aR = fma(-tR, rs, aR);
        const double wR = W1 * t[hInvR];
        aR = fma(W1, wR, aR);
        double ap = fma(t[hPhip], fma(dPp, rs, gp), -(U1 * wR));
        if (FM == kForceArrays) ap += gpin[at(r - 1)];
        s1 = S1;
        u1 = fma(dt, aR, U1);
        w1 = fma(dt, ap, W1);
      }
      const double eS = s1 - S2, eU = u1 - u2, eW = w1 - w2;  // (row r-1) - (row r-2)
      double lS = 0, lU = 0, lW = 0;                          // slopes of row r-2
      double F = 0, FR = 0, FP = 0;                           // face between rows r-3 and r-2
      if (k >= 4) {
        if (r - 2 > 0 && r - 2 < Nu - 1) {  // no slope in the first and last row (hydro.hpp:117-119)
          lS = vanleer64(eS, dS);
          lU = vanleer64(eU, du);
          lW = vanleer64(eW, dw);
        }
        // ---- radial flux (hydro.hpp:107-130) through face f = r-2 ----
        if (k >= 5 && r - 2 >= 1 && r - 2 <= Nu - 1) {
          const double *t = tc - 2 * kRow64W;
          const double vf = 0.5 * (u3 + u2);
          const bool up = pos64(vf);
          // q_u + k_u (+-1/2 - vf dt / (2 dR_u))
          const double h = fma(-vf, up ? t[hCl] : t[hCr], up ? 0.5 : -0.5);
          const double sf = fma(h, up ? kS : lS, up ? S3 : S2);
          const double uf = fma(h, up ? kU : lU, up ? u3 : u2);
          const double wf = fma(h, up ? kW : lW, up ? w3 : w2);
          F = vf * sf * t[hAf];
          FR = F * uf;
          FP = F * wf;
        }
        if (k >= 6) {
          // ---- row i = r-3: radial gather (hydro.hpp:131-139) ----
          const double *t = tc - 3 * kRow64W;
          const double cv = t[hCvol];
          const double ns = fma(cv, F0 - F, S3);
          const double mR = fma(S3, u3, cv * (FR0 - FR)), mP = fma(S3, w3, cv * (FP0 - FP));
          double d = dmax_ref(ns, 1e-10);
          double y = rcp_approx64(d);
          const double a = quot64(mR, d, y), b = quot64(mP, d, y);
          // ---- azimuthal sweep (hydro.hpp:150-178): this lane's left face and cell ----
          const double sm = up1(ns), am = up1(a), bm = up1(b);
          const double qS = vanleer64(dn1(ns) - ns, ns - sm), qA = vanleer64(dn1(a) - a, a - am),
                       qB = vanleer64(dn1(b) - b, b - bm);
          const double qSm = up1(qS), qAm = up1(qA), qBm = up1(qB);
          const double vf = 0.5 * (bm + b);
          const bool up = pos64(vf);
          const double h = fma(-vf, t[hCphi], up ? 0.5 : -0.5);
          const double sf = fma(h, up ? qSm : qS, up ? sm : ns);
          const double af = fma(h, up ? qAm : qA, up ? am : a);
          const double bf = fma(h, up ? qBm : qB, up ? bm : b);
          const double G = vf * sf * t[hAphi], GR = G * af, GP = G * bf;
          const double n2 = fma(cv, G - dn1(G), ns);
          const double mR2 = fma(ns, a, cv * (GR - dn1(GR))), mP2 = fma(ns, b, cv * (GP - dn1(GP)));
          d = dmax_ref(n2, 1e-10);  // the quotients' floor and the state's (hydro.hpp:69)
          y = rcp_approx64(d);
          const double uo = quot64(mR2, d, y), wo = quot64(mP2, d, y);
          if (outp) {
            const int q = (r - 3) * Nphi + j;
            So[q] = d;
            vRo[q] = uo;
            vpo[q] = wo;
            double Pn = 0.0;
            if (!G2) Po[q] = Pn = pres64(g, d);
            // CFL rate of the new state; d is above the 1e-12 of the reference's cs
            const double rate = rate64(uo, wo, cs64(g, d, Pn), t[hInvdR], t[hInvdl]);
            bad |= !(rate == rate) || !(uo == uo) || !(wo == wo);
            lmax = fmax(lmax, rate);
            if (si.nmodes) tsum = fma(d, t[hDA], tsum);
          }
        }
      }
      F0 = F; FR0 = FR; FP0 = FP;
      S3 = S2; u3 = u2; w3 = w2; kS = lS; kU = lU; kW = lW;
      S2 = s1; u2 = u1; w2 = w1; dS = eS; du = eU; dw = eW;
      S1 = S; U1 = U; W1 = W;
      P2 = P1; P1 = P; Ph2 = Ph1; Ph1 = Ph;
    }
    // mode sums of the column (diskmain.cpp:76-80): Sigma dA summed over the band's rows
    if (si.nmodes) {
      const double phi = (j + 0.5) * g.dphi;
      for (int m = 0; m < si.nmodes; ++m) {
        double sn, cs;
        sincos(m * phi, &sn, &cs);
        msum[2 * m] = tsum * cs;
        msum[2 * m + 1] = -tsum * sn;
      }
    }
  } else {
    for (int q = 0; q < 2 * si.nmodes; ++q) msum[q] = 0.0;
  }
  if (bad) lmax = __longlong_as_double(0x7ff8000000000000ll);
  finish_launch_deferred<0>(ctl, si, lmax, msum, red);
}

// The end of a hydro launch that no gravity kernel takes care of.
__global__ void k_step_finalize(Ctl *ctl) {
  pdl_trigger();  // the next kernel's prologue may start; it waits for this one's completion
  pdl_wait();     // every CTA of the hydro launch has folded its sums
  if (threadIdx.x == 0) finalize_pending(ctl);
}
cudaError_t launch_step_finalize(Ctl *ctl, cudaStream_t st) {
  return launch_pdl(k_step_finalize, dim3(1), dim3(32), 0, st, ctl);
}

// CFL reduction over a state (DiskHydro::timestep, hydro.hpp:48-61); the last CTA stores
// dt = cfl / max (clipped to tlim unless fixed_dt).  Optionally accumulates mode sums.  Po, if
// given, takes the pressure, which the rate needs anyway.
__global__ void __launch_bounds__(256) k_cfl64(const double *__restrict__ Sig, const double *__restrict__ vR,
                                               const double *__restrict__ vp, double *__restrict__ Po, Ctl *ctl,
                                               Geom64 g, int nmodes, int record) {
  __shared__ double red[8];
  StepInfo si;
  si.t = ctl->t; si.dt = 0.0; si.tlim = ctl->tlim;
  si.active = false; si.advance_t = false;
  si.record = record != 0;
  si.nmodes = record && nmodes < 3 ? 3 : nmodes;
  nmodes = si.nmodes;
  double msum[2 * kMaxModes];
#pragma unroll
  for (int q = 0; q < 2 * kMaxModes; ++q) msum[q] = 0.0;
  double lmax = 0.0;
  const size_t n = (size_t)g.Nu * g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / g.Nphi), j = (int)(k % g.Nphi);
    double r;
    if (Po) {
      const double s = Sig[k], P = pres64(g, s);
      Po[k] = P;
      r = s < 1e-12 ? cfl_rate64(g, i, s, vR[k], vp[k]) : rate64(vR[k], vp[k], cs64(g, s, P), g.invdR[i], g.invdl[i]);
    } else {
      r = cfl_rate64(g, i, Sig[k], vR[k], vp[k]);
    }
    if (!(r == r)) lmax = r;
    else if (lmax == lmax) lmax = fmax(lmax, r);
    if (nmodes) {
      double dA = g.R[i] * (g.Rf[i + 1] - g.Rf[i]) * g.dphi;
      add_modes(msum, nmodes, Sig[k], j, g.dphi, dA);
    }
  }
  finish_launch<256>(ctl, si, lmax, msum, red);
}

// Sums Sigma e^{-i m phi} dA for m < nmodes (diskmain.cpp:72-84) into out[2m], out[2m+1].
__global__ void __launch_bounds__(256) k_modes64(const double *__restrict__ Sig, Geom64 g, int nmodes,
                                                 double *__restrict__ out) {
  __shared__ double red[8];
  double msum[2 * kMaxModes];
#pragma unroll
  for (int q = 0; q < 2 * kMaxModes; ++q) msum[q] = 0.0;
  const size_t n = (size_t)g.Nu * g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / g.Nphi), j = (int)(k % g.Nphi);
    double dA = g.R[i] * (g.Rf[i + 1] - g.Rf[i]) * g.dphi;
    add_modes(msum, nmodes, Sig[k], j, g.dphi, dA);
  }
  for (int q = 0; q < 2 * nmodes; ++q) {
    double v = warp_sum(msum[q]);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < 8; ++w) s += red[w];
      atomicAdd(&out[q], s);
    }
    __syncthreads();
  }
}

// KalnajsSolver::forces (kalnajs.hpp:65-80) as a standalone pass.
__global__ void k_forces64(const double *__restrict__ Phi, double *__restrict__ gR, double *__restrict__ gp,
                           Geom64 g) {
  const size_t n = (size_t)g.Nu * g.Nphi;
  const int Nu = g.Nu, Nphi = g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / Nphi), j = (int)(k % Nphi);
    int jm = (j - 1 + Nphi) % Nphi, jp = (j + 1) % Nphi;
    double dPhidphi = (Phi[(size_t)i * Nphi + jp] - Phi[(size_t)i * Nphi + jm]) / (2.0 * g.dphi);
    double dPhidu;
    if (i == 0) dPhidu = (Phi[(size_t)(i + 1) * Nphi + j] - Phi[k]) / g.du;
    else if (i == Nu - 1) dPhidu = (Phi[k] - Phi[(size_t)(i - 1) * Nphi + j]) / g.du;
    else dPhidu = (Phi[(size_t)(i + 1) * Nphi + j] - Phi[(size_t)(i - 1) * Nphi + j]) / (2.0 * g.du);
    gR[k] = -dPhidu / g.R[i];
    gp[k] = -dPhidphi / g.R[i];
  }
}

// Samples of the softened log-spiral kernel at wrapped offsets (kalnajs.hpp:106-112).
__global__ void k_kernel_samples64(double *__restrict__ out, int M, int Nphi, double du, double dphi, double eps) {
  const size_t n = (size_t)M * Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int p = (int)(k / Nphi), q = (int)(k % Nphi);
    int ioff = (p <= M / 2) ? p : p - M;
    double Du = ioff * du;
    double Dphi = q * dphi;
    out[k] = 1.0 / sqrt(2.0 * cosh(Du) - 2.0 * cos(Dphi) + eps);
  }
}

// global sums mass = sum Sigma dA, angmom = sum Sigma vphi R dA (FP64)
__global__ void k_conserved64(const double *__restrict__ Sig, const double *__restrict__ vp, Geom64 g,
                              double *__restrict__ out) {
  __shared__ double red[2][8];
  double m = 0.0, L = 0.0;
  const size_t n = (size_t)g.Nu * g.Nphi;
  for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(k / g.Nphi);
    double dA = g.R[i] * (g.Rf[i + 1] - g.Rf[i]) * g.dphi;
    m += Sig[k] * dA;
    L += Sig[k] * vp[k] * g.R[i] * dA;
  }
  m = warp_sum(m);
  L = warp_sum(L);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = m; red[1][threadIdx.x >> 5] = L; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { a += red[0][w]; b += red[1][w]; }
    atomicAdd(&out[0], a);
    atomicAdd(&out[1], b);
  }
}

// ---------------------------------------------------------------------------------
// host launchers
int sm_count() {
  static std::atomic<int> known[64];  // by device; 0: not asked yet
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  if (dev >= 0 && dev < 64) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

cudaError_t launch_hydro64(const double *Sig, const double *vR, const double *vp, const double *Phi,
                           const double *gR, const double *gp, int force_mode, const double *Pin, double *So,
                           double *vRo, double *vpo, double *Po, Ctl *ctl, const Geom64 &g, cudaStream_t st) {
  // strips per CTA: the count that leaves the fewest idle warps; rows per band: the GPU's
  // warps (16 per SM) shared among the strips.  A grid too small to fill the GPU takes
  // one-row bands: seven row visits for one, but the shortest chain (128^2 step: 19.99 us,
  // 21.15 with at least two rows, 23.21 with four).
  const int strips = (g.Nphi + kOutCols64 - 1) / kOutCols64;
  int wc = strips <= kMaxWarps64 ? strips : 4;
  if (strips > kMaxWarps64)
    for (int c : {5, 3})
      if ((strips + c - 1) / c * c < (strips + wc - 1) / wc * wc) wc = c;
  const int cols = (strips + wc - 1) / wc, slots = sm_count() * (16 / wc);  // 16 warps per SM
  int bands = slots / cols;
  if (bands < 1) bands = 1;
  int band = (g.Nu + bands - 1) / bands;
  if (band < 1) band = 1;
  if (band > kMaxBand64) band = kMaxBand64;
  auto go = [&](auto kern) {
    return launch_pdl(kern, dim3(cols, (g.Nu + band - 1) / band), dim3(32 * wc), 0, st, Sig, vR, vp, Phi, gR, gp, Pin,
                      So, vRo, vpo, Po, ctl, g, band);
  };
  auto pick = [&](auto fm) {
    constexpr int FM = decltype(fm)::value;
    if (g.gamma2) return go(k_hydro64<true, FM, false>);
    return Pin ? go(k_hydro64<false, FM, true>) : go(k_hydro64<false, FM, false>);
  };
  if (force_mode == kForcePhi) return pick(std::integral_constant<int, kForcePhi>{});
  if (force_mode == kForceArrays) return pick(std::integral_constant<int, kForceArrays>{});
  return pick(std::integral_constant<int, kForceNone>{});
}

cudaError_t launch_cfl64(const double *Sig, const double *vR, const double *vp, double *Po, Ctl *ctl, const Geom64 &g,
                         int nmodes, int record, cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  int cap = sm_count() * 4;
  if (blocks > cap) blocks = cap;
  k_cfl64<<<blocks, 256, 0, st>>>(Sig, vR, vp, Po, ctl, g, nmodes, record);
  return cudaGetLastError();
}

cudaError_t launch_modes64(const double *Sig, const Geom64 &g, int nmodes, double *out, cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 4) blocks = sm_count() * 4;
  cudaMemsetAsync(out, 0, 2 * nmodes * sizeof(double), st);
  k_modes64<<<blocks, 256, 0, st>>>(Sig, g, nmodes, out);
  return cudaGetLastError();
}

cudaError_t launch_forces64(const double *Phi, double *gR, double *gp, const Geom64 &g, cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  k_forces64<<<blocks, 256, 0, st>>>(Phi, gR, gp, g);
  return cudaGetLastError();
}

cudaError_t launch_conserved64(const double *Sig, const double *vp, const Geom64 &g, double *out2,
                               cudaStream_t st) {
  size_t n = (size_t)g.Nu * g.Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 4) blocks = sm_count() * 4;
  cudaMemsetAsync(out2, 0, 2 * sizeof(double), st);
  k_conserved64<<<blocks, 256, 0, st>>>(Sig, vp, g, out2);
  return cudaGetLastError();
}

cudaError_t launch_kernel_samples64(double *out, int M, int Nphi, double du, double dphi, double eps,
                                    cudaStream_t st) {
  size_t n = (size_t)M * Nphi;
  int blocks = (int)((n + 255) / 256);
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  k_kernel_samples64<<<blocks, 256, 0, st>>>(out, M, Nphi, du, dphi, eps);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------
// FFT plans and pass launchers.

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
template <> bool make_fft_plan<double2>(int n, FftPlan *pl) { return make_plan<double2>(n, pl); }
template <> bool make_fft_plan<float2>(int n, FftPlan *pl) { return make_plan<float2>(n, pl); }

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

// Plans and device tables of an Nu x Nphi grid, in one buffer.
template <typename V>
cudaError_t build_fft_tables(int Nu, int Nphi, FftTables<V> *ft) {
  using T = real_t<V>;
  if (!make_fft_plan<V>(Nphi, &ft->phi) || !make_fft_plan<V>(Nu, &ft->u)) return cudaErrorInvalidValue;
  for (const FftPlan *pl : {&ft->phi, &ft->u}) {
    const cudaError_t e = pl->fixed ? fixed_attrs<V>(pl->n) : cudaSuccess;
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

// Lengths whose tables go to shared memory (the SMT forms).
static bool fft_smt(int n) { return n <= 512; }

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

// Raise the dynamic shared-memory limit of every FFT pass, for each handle: the limit belongs to
// the device, and a process may have handles on several.
cudaError_t prepare_fft_kernels() {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const void *fns[] = {(const void *)k_phi_fwd<double2, true>, (const void *)k_phi_fwd<double2, false>,
                       (const void *)k_u_conv<double2, true>,  (const void *)k_u_conv<double2, false>,
                       (const void *)k_phi_inv<double2, true>, (const void *)k_phi_inv<double2, false>,
                       (const void *)k_phi_fwd<float2, true>,  (const void *)k_phi_fwd<float2, false>,
                       (const void *)k_u_conv<float2, true>,   (const void *)k_u_conv<float2, false>,
                       (const void *)k_phi_inv<float2, true>,  (const void *)k_phi_inv<float2, false>,
                       (const void *)k_u_khat<double2>};
  for (const void *f : fns) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
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

cudaError_t launch_u_khat(const double2 *W, int ldw, int Nc, const FftTables<double2> &ft, double *kr,
                          cudaStream_t st) {
  const FftPlan &pl = ft.u;
  k_u_khat<double2><<<2 * Nc, pl.threads, (size_t)fft_pad_len<double2>(pl.n) * sizeof(double2), st>>>(
      W, ldw, pl, ft.twU, ft.half, kr);
  return cudaGetLastError();
}

#define DG_FFT_INSTANCES(V)                                                                                        \
  template cudaError_t build_fft_tables<V>(int, int, FftTables<V> *);                                              \
  template cudaError_t launch_phi_fwd<V>(const FftDisk<V> &, int, int, int,               \
                                         const FftTables<V> &, cudaStream_t);                                     \
  template cudaError_t launch_u_conv<V>(const FftDisk<V> &, int, int, const FftTables<V> &, \
                                        cudaStream_t);                                                            \
  template cudaError_t launch_phi_inv<V>(const FftDisk<V> &, int, int,                    \
                                         const FftTables<V> &, cudaStream_t);
DG_FFT_INSTANCES(double2)
DG_FFT_INSTANCES(float2)
#undef DG_FFT_INSTANCES

}  // namespace dg
