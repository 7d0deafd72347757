// Plain-method (FP64) hydro: one fused kernel per time step.
//
// It restates DiskHydro::step (diskfft/src/hydro.hpp:63-70) =
//   source (:73-96) -> transportR (:99-140) -> transportPhi (:143-179) -> floor (:69)
// with the self-gravity forces of KalnajsSolver::forces (kalnajs.hpp:65-80) computed
// from the potential in the same pass, and the CFL reduction of DiskHydro::timestep
// (:48-61) for the NEXT step fused into the epilogue.  Results agree to round-off, not bit for
// bit: the expressions are regrouped (fused multiply-adds, row constants and dt multiplied
// ahead, quotients through shared reciprocals).  Each is grouped so that no rounding is added
// where it counts: a momentum after a sweep is fma(Sigma, v, dt/Vol dF), which rounds the small
// term of the sum and not the large one, and quotients are good to half a unit in the last
// place.  Error of one step against 80-bit arithmetic, rms over a field: velocities
// 1.20 - 1.29e-16, sigma 6.6 - 6.8e-17, the same to 0.5 % as with IEEE divisions in the
// reference's order (64^2 .. 256^2, Gamma 1.55 .. 2); rounding Sigma v by itself costs 6 % more.
//
// A warp marches down a strip of 32 columns (26 outputs and 3 halo columns on each side),
// one column per lane, with the rows a stage needs in registers: at row r it loads row r,
// applies the source to row r-1, limits the radial slopes of row r-2, forms the radial flux
// between rows r-3 and r-2, and finishes row r-3 (radial gather, azimuthal sweep, floor,
// outputs, CFL rate).  Azimuthal neighbours come from the neighbouring lanes.  Nothing but
// the row constants goes through shared memory and no stage waits at a barrier.
//
// What bounds it: the FP64 pipe (two warp instructions per SM and cycle), so the march does
// each operation once per zone: a cell's slopes are limited once and picked by the upwind
// side, a row's constants (products with dt included) come from a table, and quotients share
// reciprocals.  A strip of a band of B rows costs B + 6 row visits, so B is as large as the
// grid allows with every SM full (launch_hydro64).  At 1024^2 (Gamma = 2) a launch takes 40 us
// cold against 85 us of the tiled form this replaced (every stage through shared memory, all
// quotients by division), with 2.3 instructions issued per active cycle and the FP64 pipe a
// third busy; 256 steps 37.3 -> 24.6 ms, at 256^2 7.3 -> 6.3 ms.
//
// For Gamma != 2 the pressure is a field of its own: a step computes it once per zone from
// the density it stores (the CFL rate needs it there anyway) and the next step loads it,
// instead of a pow per row visit and another per output (768 x 1024, Gamma = 1.75: 95.8 ->
// 80.1 us a step; 240 x 180: 26.8 -> 21.7).  An uploaded state has none: the CFL pass before a
// run of steps stores it beside the rate, and a lone step straight after an upload takes the
// form with a pow per row visit (a kernel of its own in the upload cost 5 to 8 us there).
//
// phi is periodic (wrapped loads).  Rows outside [0, Nu) load the edge row, which is what
// the reference's clamped pressure and one-sided potential differences read there; slopes
// of the first and last row and the fluxes through the radial edges are zero.
#pragma once

#include "dg_common.cuh"

namespace dg {

// Row table of the hydro kernel, [Nu + 1][kRow64W]: row constants of row i, constants of the
// face f = i between rows i - 1 and i (row Nu holds only that face).  Entries marked dt are
// multiplied by the step's dt when a CTA stages its rows.
enum Row64 : int {
  hGstar = 0,   // -GM* / R^2
  hInvR = 1,    // 1 / R
  hInvdRc = 2,  // 1 / (R[ip] - R[im]) (clamped neighbours)
  hPhiu = 3,    // -1 / (R du (ip - im)): radial potential differences to force
  hPhip = 4,    // -1 / (2 R dphi): azimuthal differences to acceleration
  hCvol = 5,    // dt / Vol
  hAphi = 6,    // Rf[i+1] - Rf[i]: azimuthal face length
  hCphi = 7,    // dt / (2 R dphi)
  hInvdR = 8,   // 1 / (Rf[i+1] - Rf[i])
  hInvdl = 9,   // 1 / (R dphi)
  hAf = 10,     // Rf[f] dphi: radial face length
  hCl = 11,     // dt / (2 (Rf[f] - Rf[f-1]))
  hCr = 12,     // dt / (2 (Rf[f+1] - Rf[f]))
  hDA = 13,     // R (Rf[i+1] - Rf[i]) dphi
  kRow64W = 16
};

struct Geom64 {
  const double *R, *Rf, *Vol;
  const double *invdR, *invdl;  // per row: 1 / (Rf[i+1] - Rf[i]), 1 / (R dphi) (CFL)
  const double *rowtab;         // [Nu + 1][kRow64W]
  int Nu, Nphi;
  double dphi, du, Kpoly, gamma, gmstar;
  int gamma2;  // gamma == 2: P = K s^2, cs^2 = 2 K s without pow
};

// Which self-gravity the kernel applies (hydro.hpp:86-88).
enum ForceMode : int { kForceNone = 0, kForcePhi = 1, kForceArrays = 2 };

constexpr int kOutCols64 = 26, kHalo64 = 3;  // columns of a strip: 3 + 26 + 3
constexpr int kMaxWarps64 = 5;               // strips per CTA
constexpr int kMaxBand64 = 32;               // rows of a band

// Quotients by Newton's method on the hardware's approximate reciprocal (PTX rcp.approx,
// relative error at most 2^-20): a step squares the error, and Markstein's residual
// correction (IBM J. Res. Dev. 34, 1990) leaves n / b the error of its last rounding, half a unit
// in the last place.  b must be a normal number whose reciprocal is one; 0, infinities and NaN
// give NaN.
__device__ __forceinline__ double rcp_approx64(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return fma(y, fma(-b, y, 1.0), y);  // about 2^-40
}
__device__ __forceinline__ double quot64(double n, double b, double y) {  // y = rcp_approx64(b)
  const double q = n * y;
  return fma(fma(-b, q, n), y, q);
}
__device__ __forceinline__ double rcp64(double b) {
  const double y = rcp_approx64(b);
  return fma(y, fma(-b, y, 1.0), y);
}
// whether 1 / b is a normal number (b neither tiny, huge, infinite nor NaN)
__device__ __forceinline__ bool rcp_ok64(double b) {
  return ((unsigned)__double2hiint(b) & 0x7fffffffu) - 0x00300000u < 0x7fa00000u;
}
__device__ __forceinline__ bool pos64(double x) { return __double2hiint(x) > 0; }  // x > 0 beyond 2^-1042

// hydro.hpp:16-18.  a b > 0 (beyond underflow) puts |a + b| above 10^-162: the quotient is
// in range
__device__ __forceinline__ double vanleer64(double a, double b) {
  const double p = a * b, s = a + b;
  const double q = quot64(p + p, s, rcp_approx64(s));
  return pos64(p) ? q : 0.0;
}
__device__ __forceinline__ double dmax_ref(double a, double b) { return (a < b) ? b : a; }  // std::max

__device__ __forceinline__ double pres64(const Geom64 &g, double s) {  // hydro.hpp:46
  return g.gamma2 ? g.Kpoly * (s * s) : g.Kpoly * pow(s, g.gamma);
}
// sound speed (hydro.hpp:45) of s > 0 whose pressure is P: cs^2 = Gamma P / Sigma, so a zone
// costs one pow.  Product and quotient round together, which leaves as many roundings as
// Gamma K Sigma^(Gamma - 1) has
__device__ __forceinline__ double cs64(const Geom64 &g, double s, double P) {
  if (g.gamma2) return sqrt(g.gamma * g.Kpoly * s);
  const double y = rcp_approx64(s), n = g.gamma * P, e = fma(g.gamma, P, -n);  // Gamma P = n + e
  const double q = n * y;
  return sqrt(fma(fma(-s, q, n) + e, y, q));
}
// (|vR| + cs)/dR + (|vp| + cs)/(R dphi)  (hydro.hpp:54-57)
__device__ __forceinline__ double rate64(double vr, double vp, double cs, double invdR, double invdl) {
  return fma(fabs(vr) + cs, invdR, (fabs(vp) + cs) * invdl);
}
__device__ __forceinline__ double cfl_rate64(const Geom64 &g, int i, double s, double vr, double vp) {
  s = dmax_ref(s, 1e-12);
  return rate64(vr, vp, cs64(g, s, g.gamma2 ? 0.0 : pres64(g, s)), g.invdR[i], g.invdl[i]);
}

}  // namespace dg
