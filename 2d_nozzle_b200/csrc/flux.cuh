// flux.cuh -- the interface fluxes of physics.cuh with fewer and shorter divisions
// and square roots, for the tile and the generic kernels.
//
// A division or square root is an iterative sequence of a dozen and more
// instructions and over 100 cycles of latency (a 1 / x chain measured 135 cycles a
// step, sqrt 103, against 13 for a multiply-add), and they are most of a flux.  The Roe
// weights need only r = sqrt(rho_R / rho_L), and reciprocals and roots are the short ones
// below.  Each takes its own: one reciprocal of a product for two denominators (both
// traces' 1 / rho, the star state's) has as many multiply-adds, three roundings where one
// is enough, and overflows where neither denominator does.
// Together with shorter address arithmetic in the loads, a residual of 480 000 linear
// triangles went 199 -> 173 us, of 240 000 cubic quadrilaterals 235 -> 195 us (tile
// kernel before its asynchronous copies).  The values differ from the templates' in the last
// bits, so the one-thread kernels keep those.
//
// Arguments of the roots are positive: rho and p are floored at FLOOR (a NaN stays one).
#pragma once
#include "physics.cuh"

namespace nzb {

// 1 / a, sqrt(a) and 1 / sqrt(a) for normal, finite a (a > 0 for the roots) from the hardware's
// approximations x, y (rcp / rsqrt.approx.ftz.f64, about 20 bits).  The reciprocal takes one third-order
// Householder step: with e = 1 - a x,  x (1 + e + e^2), whose remainder e^3 = 2^-60 is below the rounding.
// The root is s = a y and two Heron steps s + (a - s^2) y / 2, which square the relative error and then
// multiply it by y's: 2^-59; both residuals come exact from a multiply-add, so one rounding is left, as
// in the division and root they replace, without their range checks and branch.  The root's reciprocal is
// a Householder step on 1 - s y.
// Over 4 x 10^6 arguments per decade, 1e-30 to 1e30, reciprocal and root are the division's and sqrt's
// but for one unit in the last place at 4 of 10^4 (nzb_reciprocals and nzb_roots expose them to the tests).
// With the first such forms a stage of 480 000 cubic triangles went 380 -> 332 us, of 240 000 cubic
// quadrilaterals 291 -> 260, the 72-member sweep's step 547 -> 493; these, with a rounding fewer a root and
// two fewer a pair of denominators, take 1 % more of the sweep (51 steps 25.1 -> 25.4 ms).
// Arguments of zero, a denormal or an infinity give a NaN; the floors and guards of the callers keep them
// above 1e-10, and a NaN stays one.
__device__ __forceinline__ double lean_rcp(double a) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  const double e = fma(-a, x, 1.0);
  return fma(x, fma(e, e, e), x);
}
__device__ __forceinline__ double rsqrt_approx(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  return y;
}
__device__ __forceinline__ double root_from(double a, double y) {
  const double h = 0.5 * y;
  double s = a * y;
  s = fma(fma(-s, s, a), h, s);
  return fma(fma(-s, s, a), h, s);
}
__device__ __forceinline__ double lean_sqrt(double a) { return root_from(a, rsqrt_approx(a)); }
// sqrt(a), and its reciprocal in rcp
__device__ __forceinline__ double lean_sqrt(double a, double& rcp) {
  const double y = rsqrt_approx(a), s = root_from(a, y);
  const double e = fma(-s, y, 1.0);
  rcp = fma(y, fma(e, e, e), y);
  return s;
}
// A sound speed from its square s = lean_sqrt(a): an infinite one (infinite energy) stays infinite, so the
// local step it bounds is zero.
__device__ __forceinline__ double sound_speed(double a, double s) {
  return (__double2hiint(a) & 0x7ff00000) == 0x7ff00000 ? a : s;
}
__device__ __forceinline__ double sound_speed(double a) { return sound_speed(a, lean_sqrt(a)); }

// primitives(U, g) of physics.cuh with lean_rcp.
__device__ __forceinline__ Prim lean_primitives(const double* U, double g) {
  Prim s;
  s.rho = floor_at(U[0], FLOOR);
  s.inv = lean_rcp(s.rho);
  s.vx = U[1] * s.inv;
  s.vy = U[2] * s.inv;
  s.p = floor_at((g - 1.0) * (U[3] - 0.5 * s.rho * (s.vx * s.vx + s.vy * s.vy)), FLOOR);
  s.H = (U[3] + s.p) * s.inv;
  return s;
}

__device__ __forceinline__ double lean_roe_flux(const double* UL, const double* UR, double nx, double ny, double g,
                                           double efix, double* F) {
  const Prim L = lean_primitives(UL, g), R = lean_primitives(UR, g);
  double FL[4], FR[4];
  normal_flux(L, nx, ny, FL);
  normal_flux(R, nx, ny, FR);
  const double r = lean_sqrt(R.rho * L.inv);
  const double iden = lean_rcp(1.0 + r);
  const double vx = (L.vx + r * R.vx) * iden;
  const double vy = (L.vy + r * R.vy) * iden;
  const double H = (L.H + r * R.H) * iden;
  const double q2 = vx * vx + vy * vy;
  const double c2 = floor_at((g - 1.0) * (H - 0.5 * q2), FLOOR);
  double ic;
  const double c = sound_speed(c2, lean_sqrt(c2, ic));
  const double vn = vx * nx + vy * ny;
  double l1 = fabs(vn + c), l2 = fabs(vn - c), l3 = fabs(vn);
  const double smax = l1 < l2 ? l2 : l1;
  const double eps = efix * c;
  if (l1 < eps || l2 < eps || l3 < eps) {
    const double h = 0.5 * lean_rcp(eps), e2 = eps * eps;
    if (l1 < eps) l1 = (l1 * l1 + e2) * h;
    if (l2 < eps) l2 = (l2 * l2 + e2) * h;
    if (l3 < eps) l3 = (l3 * l3 + e2) * h;
  }
  const double d0 = UR[0] - UL[0], d1 = UR[1] - UL[1], d2 = UR[2] - UL[2], d3 = UR[3] - UL[3];
  const double G1 = (g - 1.0) * (0.5 * q2 * d0 - vx * d1 - vy * d2 + d3);
  const double G2 = -vn * d0 + d1 * nx + d2 * ny;
  const double s1 = 0.5 * (l1 + l2), s2 = 0.5 * (l1 - l2);
  const double C1 = (G1 * (ic * ic)) * (s1 - l3) + (G2 * ic) * s2;
  const double C2 = (G1 * ic) * s2 + (s1 - l3) * G2;
  F[0] = 0.5 * (FL[0] + FR[0]) - 0.5 * (l3 * d0 + C1);
  F[1] = 0.5 * (FL[1] + FR[1]) - 0.5 * (l3 * d1 + C1 * vx + C2 * nx);
  F[2] = 0.5 * (FL[2] + FR[2]) - 0.5 * (l3 * d2 + C1 * vy + C2 * ny);
  F[3] = 0.5 * (FL[3] + FR[3]) - 0.5 * (l3 * d3 + C1 * H + C2 * vn);
  return smax;
}

__device__ __forceinline__ double lean_hllc_flux(const double* UL, const double* UR, double nx, double ny, double g,
                                            double low_mach, double* F) {
  const Prim L = lean_primitives(UL, g), R = lean_primitives(UR, g);
  const double vnL = L.vx * nx + L.vy * ny;
  const double vnR = R.vx * nx + R.vy * ny;
  const double aL = sound_speed(floor_at(g * L.p * L.inv, FLOOR)), aR = sound_speed(floor_at(g * R.p * R.inv, FLOOR));
  const double r = lean_sqrt(R.rho * L.inv);
  const double iden = lean_rcp(1.0 + r);
  const double vx = (L.vx + r * R.vx) * iden;
  const double vy = (L.vy + r * R.vy) * iden;
  const double H = (L.H + r * R.H) * iden;
  const double vt = vx * nx + vy * ny;
  const double at = lean_sqrt(floor_at((g - 1.0) * (H - 0.5 * (vx * vx + vy * vy)), FLOOR));
  double SL = fmin(vnL - aL, vt - at);
  double SR = fmax(vnR + aR, vt + at);
  if (low_mach > 0.0) {
    const double mach = fmax(fabs(vnL) / aL, fabs(vnR) / aR);
    const double phi = fmin(1.0, mach / low_mach);
    const double bL = fmin(vnL, vt), bR = fmax(vnR, vt);
    SL = bL - phi * (bL - SL);
    SR = bR + phi * (SR - bR);
  }
  const double smax = fmax(fabs(SL), fabs(SR));
  const double mL = L.rho * (SL - vnL), mR = R.rho * (SR - vnR);
  const double dm = fabs(mR - mL) > FLOOR ? mR - mL : FLOOR;
  const double SM = (vnR * mR - vnL * mL + L.p - R.p) * lean_rcp(dm);
  // the side the face lies on: left of SL or of the contact, the left one; its star
  // state applies between SL and SR
  const bool left = SL >= 0.0 || (!(SR <= 0.0) && SM >= 0.0);
  const bool star = !(SL >= 0.0) && !(SR <= 0.0);
  const double rho = left ? L.rho : R.rho, ux = left ? L.vx : R.vx, uy = left ? L.vy : R.vy, p = left ? L.p : R.p;
  const double E = left ? UL[3] : UR[3], vn = left ? vnL : vnR, S = left ? SL : SR, m = left ? mL : mR;
  const double mf = rho * vn;
  F[0] = mf;
  F[1] = mf * ux + p * nx;
  F[2] = mf * uy + p * ny;
  F[3] = vn * (E + p);
  if (star) {
    const double rs = m * lean_rcp(guard(S - SM));  // rho (S - vn) / (S - SM)
    const double dv = SM - vn;
    const double Es = E * (left ? L.inv : R.inv) + dv * (SM + p * lean_rcp(guard(m)));
    F[0] += S * (rs - (left ? UL[0] : UR[0]));
    F[1] += S * (rs * (ux + dv * nx) - (left ? UL[1] : UR[1]));
    F[2] += S * (rs * (uy + dv * ny) - (left ? UL[2] : UR[2]));
    F[3] += S * (rs * Es - E);
  }
  return smax;
}

__device__ __forceinline__ double lean_ausm_up_flux(const double* UL, const double* UR, double nx, double ny, double g,
                                               double* F) {
  constexpr double BETA = 0.125, ALPHA = 0.1875, KP = 0.4, KU = 0.2;
  const Prim L = lean_primitives(UL, g), R = lean_primitives(UR, g);
  const double vnL = L.vx * nx + L.vy * ny;
  const double vnR = R.vx * nx + R.vy * ny;
  const double aL = sound_speed(g * L.p * L.inv), aR = sound_speed(g * R.p * R.inv);
  const double ah = 0.5 * (aL + aR), rh = 0.5 * (L.rho + R.rho);
  const double iah = lean_rcp(ah), mL = vnL * iah, mR = vnR * iah;
  const double mb2 = 0.5 * (mL * mL + mR * mR);
  const double pL2 = 0.25 * ((mL + 1.0) * (mL + 1.0)), mL2 = -0.25 * ((mL - 1.0) * (mL - 1.0));
  const double pR2 = 0.25 * ((mR + 1.0) * (mR + 1.0)), mR2 = -0.25 * ((mR - 1.0) * (mR - 1.0));
  const double m4p = fabs(mL) >= 1.0 ? 0.5 * (mL + fabs(mL)) : pL2 * (1.0 - 16.0 * BETA * mL2);
  const double m4m = fabs(mR) >= 1.0 ? 0.5 * (mR - fabs(mR)) : mR2 * (1.0 + 16.0 * BETA * pR2);
  const double dif = 1.0 - mb2;
  const double uh = ah * (m4p + m4m) + KP * (dif < 0.0 ? 0.0 : dif) * (L.p - R.p) * lean_rcp(rh * ah);
  const double p5p = fabs(mL) >= 1.0 ? (mL > 0.0 ? 1.0 : 0.0) : pL2 * ((2.0 - mL) - 16.0 * ALPHA * mL * mL2);
  const double p5m = fabs(mR) >= 1.0 ? (mR > 0.0 ? 0.0 : 1.0) : mR2 * ((-2.0 - mR) + 16.0 * ALPHA * mR * pR2);
  const double ph = p5p * L.p + p5m * R.p + KU * p5p * p5m * rh * ah * (vnL - vnR);
  // upwind: 1/2 u (PsiL + PsiR) - 1/2 |u| (PsiR - PsiL) = max(u, 0) PsiL + min(u, 0) PsiR
  const double up = 0.5 * (uh + fabs(uh)), um = 0.5 * (uh - fabs(uh));
  F[0] = up * L.rho + um * R.rho;
  F[1] = up * UL[1] + um * UR[1] + ph * nx;
  F[2] = up * UL[2] + um * UR[2] + ph * ny;
  F[3] = up * (UL[3] + L.p) + um * (UR[3] + R.p);
  return fmax(fabs(vnL) + aL, fabs(vnR) + aR);
}

__device__ __forceinline__ double lean_interface_flux(const double* UL, const double* UR, double nx, double ny,
                                                      const nzb_physics& ph, double* F) {
  if (ph.flux == NZB_HLLC) return lean_hllc_flux(UL, UR, nx, ny, ph.gamma, ph.hllc_low_mach, F);
  if (ph.flux == NZB_AUSMUP) return lean_ausm_up_flux(UL, UR, nx, ny, ph.gamma, F);
  return lean_roe_flux(UL, UR, nx, ny, ph.gamma, ph.entropy_fix, F);
}

}  // namespace nzb
