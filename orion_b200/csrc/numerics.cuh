// Point- and face-level numerics of ORION's per-step path, as device functions.
//
// Every function reproduces the reference's arithmetic operation by operation
// (same operands, same association, no contraction: the FP64 translation unit is
// compiled with --fmad=false), so the plain FP64 path is bit-identical to the
// reference wherever the reference uses only + - * / sqrt.  Templated on the
// compute type T so the mixed-precision path runs the same formulas in FP32.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace orion {

template <typename T> __device__ __forceinline__ T tabs(T x) { return x < T(0) ? -x : x; }
template <> __device__ __forceinline__ double tabs<double>(double x) { return fabs(x); }
template <> __device__ __forceinline__ float tabs<float>(float x) { return fabsf(x); }
template <typename T> __device__ __forceinline__ T tsqrt(T x);
template <> __device__ __forceinline__ double tsqrt<double>(double x) { return sqrt(x); }
template <> __device__ __forceinline__ float tsqrt<float>(float x) { return sqrtf(x); }
template <typename T> __device__ __forceinline__ T tmax(T a, T b) { return (a < b) ? b : a; }  // std::max

// a / b, correctly rounded, from r = RN(1/b), b > 0: two Newton corrections of
// the quotient with an exact remainder (Markstein, IBM J. Res. Dev. 34, 1990:
// with r correctly rounded and q within one ulp, RN(q + r (a - b q)) = RN(a / b)).
// The first correction brings q = RN(a r) within one ulp, the second is the
// theorem's step.  The remainder is formed as b q - a and subtracted, so that a
// zero keeps its sign.  Exact while the remainder and 1/b are normal numbers
// (|a| from 2^-959, b from 2^-1021 to 2^1021) and the quotient is one or zero;
// below that the last bit may differ, and a b whose reciprocal overflows gives
// an infinity.  Where the corrections meet an infinity (an infinite or zero
// denominator, an infinite quotient) they end in a NaN, and the product a r is
// what the division gives; the test is on the high word, off the FP64 pipe.
__device__ __forceinline__ double quotient(double a, double b, double r) {
  const double q0 = a * r;
  const double q1 = __fma_rn(-__fma_rn(b, q0, -a), r, q0);
  const double q2 = __fma_rn(-__fma_rn(b, q1, -a), r, q1);
  return (__double2hiint(q2) & 0x7ff00000) == 0x7ff00000 ? q0 : q2;
}
// 0, and so quotient 0, for a denominator outside 1e-290 .. 1e290 (a sound speed
// no flow has).
__device__ __forceinline__ double quotient_rcp(double b) {
  return (b > 1.0e-290 && b < 1.0e290) ? __drcp_rn(b) : 0.0;
}

// ---------------------------------------------------------------------------
// Roe flux with Harten entropy fix: flux_Roe + calc_physical_flux
// (src/solver/InviscidFluxComputer.cpp:14-131).  q = (rho,u,v,w,p).
// ---------------------------------------------------------------------------
// Quotients by one denominator: FP64 rounded as the division (quotient), FP32
// the product with the reciprocal.
template <typename T> struct Over {
  T b, r;
};
__device__ __forceinline__ Over<double> over(double b) { return Over<double>{b, __drcp_rn(b)}; }
__device__ __forceinline__ Over<float> over(float b) { return Over<float>{b, __fdividef(1.f, b)}; }
__device__ __forceinline__ double div(double a, const Over<double>& o) { return quotient(a, o.b, o.r); }
__device__ __forceinline__ float div(float a, const Over<float>& o) { return a * o.r; }

template <typename T>
__device__ __forceinline__ void physical_flux(const T q[5], const Over<T>& rg1, const Over<T>& rrho, T nx, T ny, T nz,
                                              T nt, T f[5]) {
  const T rho = q[0], u = q[1], v = q[2], w = q[3], p = q[4];
  const T V = u * nx + v * ny + w * nz + nt;
  const T E = div(p, rg1) + T(0.5) * rho * (u * u + v * v + w * w);
  const T H = div(E + p, rrho);
  f[0] = rho * V;
  f[1] = rho * u * V + p * nx;
  f[2] = rho * v * V + p * ny;
  f[3] = rho * w * V + p * nz;
  f[4] = rho * H * V + p * nt;
}

template <typename T>
__device__ __forceinline__ void roe_flux(const T ql[5], const T qr[5], T nx, T ny, T nz, T nt, T efix, T gamma,
                                         T f[5]) {
  T fl[5], fr[5];
  const T gamma1 = gamma - T(1);
  const T gamma2 = gamma / gamma1;
  const Over<T> rg1 = over(gamma1), rl = over(ql[0]), rr = over(qr[0]);
  physical_flux(ql, rg1, rl, nx, ny, nz, nt, fl);
  physical_flux(qr, rg1, rr, nx, ny, nz, nt, fr);
  const T drho = qr[0] - ql[0], du = qr[1] - ql[1], dv = qr[2] - ql[2], dw = qr[3] - ql[3], dp = qr[4] - ql[4];
  const T hl = div(gamma2 * ql[4], rl) + T(0.5) * (ql[1] * ql[1] + ql[2] * ql[2] + ql[3] * ql[3]);
  const T hr = div(gamma2 * qr[4], rr) + T(0.5) * (qr[1] * qr[1] + qr[2] * qr[2] + qr[3] * qr[3]);
  const T sqrt_rL = tsqrt(ql[0]);
  const T sqrt_rR = tsqrt(qr[0]);
  const T inv_den = over(sqrt_rL + sqrt_rR).r;
  const T rho_roe = sqrt_rL * sqrt_rR;
  const T u_roe = (sqrt_rL * ql[1] + sqrt_rR * qr[1]) * inv_den;
  const T v_roe = (sqrt_rL * ql[2] + sqrt_rR * qr[2]) * inv_den;
  const T w_roe = (sqrt_rL * ql[3] + sqrt_rR * qr[3]) * inv_den;
  const T h_roe = (sqrt_rL * hl + sqrt_rR * hr) * inv_den;
  const T v2 = u_roe * u_roe + v_roe * v_roe + w_roe * w_roe;
  T c2 = (h_roe - T(0.5) * v2) * gamma1;
  if (c2 <= T(0)) c2 = T(1.0e-6);
  const T c = tsqrt(c2);
  const T U_contra = u_roe * nx + v_roe * ny + w_roe * nz + nt;
  T grad_mag = tsqrt(nx * nx + ny * ny + nz * nz);
  grad_mag = tmax(grad_mag, T(1.0e-30));
  const T inv_mag = over(grad_mag).r;
  const T nx_n = nx * inv_mag, ny_n = ny * inv_mag, nz_n = nz * inv_mag;
  const T c_mag = c * grad_mag;
  T l1 = tabs(U_contra - c_mag);
  T l4 = tabs(U_contra);
  T l5 = tabs(U_contra + c_mag);
  const T delta = efix * c_mag;
  const T delta2 = delta * delta;
  if (l1 < delta) l1 = tsqrt(l1 * l1 + delta2);
  if (l4 < delta) l4 = tsqrt(l4 * l4 + delta2);
  if (l5 < delta) l5 = tsqrt(l5 * l5 + delta2);
  const T rodcta = rho_roe * (du * nx_n + dv * ny_n + dw * nz_n);
  const T dp_c2 = div(dp, over(c2));
  const T rodctac = div(rodcta, over(c));
  const T a1 = l4 * (drho - dp_c2);
  const T a2 = l5 * (dp_c2 + rodctac) * T(0.5);
  const T a3 = l1 * (dp_c2 - rodctac) * T(0.5);
  const T a4 = a1 + a2 + a3;
  const T a5 = c * (a2 - a3);
  const T a6 = l4 * (rho_roe * du - nx_n * rodcta);
  const T a7 = l4 * (rho_roe * dv - ny_n * rodcta);
  const T a8 = l4 * (rho_roe * dw - nz_n * rodcta);
  const T df0 = a4;
  const T df1 = u_roe * a4 + nx_n * a5 + a6;
  const T df2 = v_roe * a4 + ny_n * a5 + a7;
  const T df3 = w_roe * a4 + nz_n * a5 + a8;
  const T df4 = h_roe * a4 + U_contra * inv_mag * a5 + u_roe * a6 + v_roe * a7 + w_roe * a8 - div(c2 * a1, rg1);
  f[0] = T(0.5) * (fl[0] + fr[0] - df0);
  f[1] = T(0.5) * (fl[1] + fr[1] - df1);
  f[2] = T(0.5) * (fl[2] + fr[2] - df2);
  f[3] = T(0.5) * (fl[3] + fr[3] - df3);
  f[4] = T(0.5) * (fl[4] + fr[4] - df4);
}

// a / 6, a / 12, a / 24 and a / 1920, FP64 rounded as the divisions.
__device__ __forceinline__ double div6(double a) { return quotient(a, 6.0, 1.0 / 6.0); }
__device__ __forceinline__ float div6(float a) { return a * (1.f / 6.f); }
__device__ __forceinline__ double div12(double a) { return quotient(a, 12.0, 1.0 / 12.0); }
__device__ __forceinline__ float div12(float a) { return a * (1.f / 12.f); }
__device__ __forceinline__ double div24(double a) { return quotient(a, 24.0, 1.0 / 24.0); }
__device__ __forceinline__ float div24(float a) { return a * (1.f / 24.f); }
__device__ __forceinline__ double div1920(double a) { return quotient(a, 1920.0, 1.0 / 1920.0); }
__device__ __forceinline__ float div1920(float a) { return a * (1.f / 1920.f); }

// 6th-order / boundary flux differences (FLUX_DXYZ,
// src/solver/InviscidFluxComputer.cpp:197-233 and src/solver/FluxComputer.cpp:257-296,
// identical formulas) at point t in [0,ni); f(k) is face k's flux (faces 0..ni).
template <typename T, typename F>
__device__ __forceinline__ T flux_diff_at(F f, int t, int ni) {
  if (t >= 2 && t < ni - 2) {
    const T term1 = T(2250) * (f(t + 1) - f(t));
    const T term2 = T(-125) * (f(t + 2) - f(t - 1));
    const T term3 = T(9) * (f(t + 3) - f(t - 2));
    return div1920(term1 + term2 + term3);
  }
  if (t == 0) return div24(T(-23) * f(0) + T(21) * f(1) + T(3) * f(2) - f(3));
  if (t == 1) return div24(f(0) - T(27) * f(1) + T(27) * f(2) - f(3));
  if (t == ni - 1) return -div24(T(-23) * f(ni) + T(21) * f(ni - 1) + T(3) * f(ni - 2) - f(ni - 3));
  // t == ni - 2
  return -div24(f(ni) - T(27) * f(ni - 1) + T(27) * f(ni - 2) - f(ni - 3));
}

// ---------------------------------------------------------------------------
// Spectral radii of the implicit sweeps (src/solver/StateUpdater.cpp:175-215).
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T spectral_radius(T rho, T u, T v, T w, T p, T gamma, T kx, T ky, T kz) {
  if (rho < T(1e-30)) rho = T(1e-30);
  if (p < T(1e-30)) p = T(1e-30);
  const T c2 = gamma * p / rho;
  const T c = tsqrt(c2);
  const T U = u * kx + v * ky + w * kz + T(0);
  const T grad_mag = tsqrt(kx * kx + ky * ky + kz * kz);
  return tabs(U) + c * grad_mag;
}

template <typename T>
__device__ __forceinline__ T visc_spectral_radius(T rho, T mu, T vol, T reynolds, T kx, T ky, T kz) {
  if (rho < T(1e-30)) rho = T(1e-30);
  const T grad2 = kx * kx + ky * ky + kz * kz;
  const T rm_vol = rho * vol;
  const T coef = T(2) * mu / (tabs(reynolds) * rm_vol + T(1.0e-30));
  return coef * grad2;
}

}  // namespace orion
