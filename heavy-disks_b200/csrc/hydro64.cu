// The FP64 hydro step's kernel (hydro64.cuh) and its launch.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "hydro64.cuh"
#include "kernels.h"
#include "step_ctl.cuh"

namespace dg {

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

}  // namespace dg
