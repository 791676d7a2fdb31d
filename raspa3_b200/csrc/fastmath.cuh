// Reciprocal, reciprocal square root and erfc for the pair kernels, FP32 and FP64 (own code: hardware approximations
// refined by one Newton or Householder step, and erfc as exp(-x^2) times a fitted rational-in-t polynomial).
#pragma once

namespace rgd
{
// FP32 reciprocal: the hardware approximation refined by one Newton step (x (2 - a x)), ~0.5 ulp
__device__ __forceinline__ float rcpRn(float a)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  const float e = fmaf(-a, r, 1.0f);
  return fmaf(r, e, r);
}
// FP32 reciprocal square root, refined by one Newton step (r (3 - a r^2) / 2)
__device__ __forceinline__ float rsqrtRn(float a)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  const float h = 0.5f * a * r;
  return r * fmaf(-h, r, 1.5f);
}
// exp(x) as 2^(x log2 e) from the hardware base-2 exponential (ex2.approx, a few ulp): the Gaussian factor of the FP32
// Ewald grid terms, whose FP32 rounding of the large cancelling pair terms already dominates the grid error
__device__ __forceinline__ float expApprox(float x)
{
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950408889634f));
  return r;
}
// the hardware reciprocal and reciprocal square root unrefined (a few ulp): the FP32 grid kernels, whose error is
// dominated by the FP32 rounding of the large cancelling pair terms
__device__ __forceinline__ float rcpApprox(float a)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float rsqrtApprox(float a)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
// erfc(x) = exp(-x^2) R(x) for 0 <= x <= 4, with R(x) = exp(x^2) erfc(x) fitted (weighted least squares in Chebyshev
// form, relative error 4e-8 in FP64, ~2 ulp in FP32) as a degree-9 polynomial in t = 1 / (1 + x/2); the caller passes
// exp(-x^2), which the derivative factors need anyway. REFINED = false takes t from the unrefined reciprocal.
template <bool REFINED = true>
__device__ __forceinline__ float erfcFromExp(float x, float expmx2)
{
  const float t = REFINED ? rcpRn(fmaf(0.5f, x, 1.0f)) : rcpApprox(fmaf(0.5f, x, 1.0f));
  float r = -0.02496027760207653f;
  r = fmaf(r, t, 0.09420006722211838f);
  r = fmaf(r, t, -0.024484887719154358f);
  r = fmaf(r, t, -0.36430737376213074f);
  r = fmaf(r, t, 0.534475564956665f);
  r = fmaf(r, t, -0.11705945432186127f);
  r = fmaf(r, t, 0.3620023727416992f);
  r = fmaf(r, t, 0.25453805923461914f);
  r = fmaf(r, t, 0.2858136296272278f);
  r = fmaf(r, t, -0.00021772264153696597f);
  return expmx2 * r;
}
// FP64 reciprocal and reciprocal square root of a normal positive number: the hardware's approximation (about 2^-20)
// refined by one third-order Householder step, r (1 + e + e^2) with e = 1 - a r and y (1 + h/2 + 3 h^2 / 8) with
// h = 1 - a y^2 (remainders e^3 and 5/16 h^3, below 2^-59): about 1 ulp, four and five FP64 instructions, no branch.
__device__ __forceinline__ double rcpHouseholder(double a)
{
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
  const double e = fma(-a, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double rsqrtHouseholder(double a)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double h = fma(-a, y * y, 1.0);
  return fma(y * h, fma(h, 0.375, 0.5), y);
}
// FP64 erfc(x) = exp(-x^2) erfcx(x) with the caller's exp(-x^2): erfcx on 0 <= x <= 6 as a degree-18 polynomial in
// 1/(x + 4), a Chebyshev interpolant against a 50-digit reference (relative error 4e-17, evaluated in FP64 8e-16).
// 24 FP64 instructions against the several branches of erfc(). Beyond x = 6 (erfc < 3e-17): the library function with
// CHECK; without it the caller has made sure that such a value is not used.
constexpr double kErfcxMax = 6.0;
template <bool CHECK>
__device__ __forceinline__ double erfcFromExp64(double x, double expmx2)
{
  const double z = fma(rcpHouseholder(x + 4.0), -13.333333333333334, 2.3333333333333335);
  double r = -4.868322297166477e-13;
  r = fma(r, z, -2.0813034355240175e-11);
  r = fma(r, z, 1.46441923632205e-11);
  r = fma(r, z, 6.313930979988944e-10);
  r = fma(r, z, -8.634552068758454e-10);
  r = fma(r, z, -1.648679324397335e-08);
  r = fma(r, z, 5.58422882224548e-08);
  r = fma(r, z, 3.49334672916577e-07);
  r = fma(r, z, -2.99897571043269e-06);
  r = fma(r, z, 2.049727284062024e-06);
  r = fma(r, z, 9.612949174094587e-05);
  r = fma(r, z, -0.0008244984060164637);
  r = fma(r, z, 0.004160948981895034);
  r = fma(r, z, -0.015418189713472417);
  r = fma(r, z, 0.04501085509437996);
  r = fma(r, z, -0.10664603114075659);
  r = fma(r, z, 0.2074011779915091);
  r = fma(r, z, -0.33072538002522917);
  r = fma(r, z, 0.28972211632346423);
  double ec = expmx2 * r;
  if constexpr (CHECK)
    if (__double2hiint(x) >= 0x40180000) ec = erfc(x);  // the high word of 6.0
  return ec;
}
// The radial factors of C q erfc(alpha r) / r: B_k = (-1/r d/dr)^k of erfc(alpha r) / r for k = 0..N-1 by the recursion
// B_{k+1} = ((2k + 1) B_k + (2 alpha^2)^{k+1} exp(-alpha^2 r^2) / (alpha sqrt(pi))) / r^2 (W. Smith, CCP5 Newsletter 46
// (1998)); every term is positive, so nothing cancels. c1 = 2 alpha / sqrt(pi), two_a2 = 2 alpha^2.
template <int N, bool CHECK = true>
__device__ __forceinline__ void ewaldLadder(double rr, double alpha, double c1, double two_a2, double B[N])
{
  const double invr = rsqrtHouseholder(rr);
  const double ex = exp(-0.5 * two_a2 * rr);
  B[0] = erfcFromExp64<CHECK>(alpha * (rr * invr), ex) * invr;
  const double inv = invr * invr;
  double e = c1 * ex;
#pragma unroll
  for (int k = 1; k < N; ++k)
  {
    B[k] = fma(static_cast<double>(2 * k - 1), B[k - 1], e) * inv;
    e *= two_a2;
  }
}

// erf(x)/x as a polynomial in u = x^2 for 0 <= x <= 2 (FP64): a Chebyshev least-squares fit of erf(sqrt(u))/sqrt(u) on
// u in [0, 4] against a 40-digit reference, in monomial form, relative error 2e-15. erf(x)/x is entire, so the
// complement erfc(x)/x = 1/x - erf(x)/x needs no exponential and no branch (relative error 4e-13 for x <= 2).
constexpr double kErfOverXMax = 2.0;
__device__ __forceinline__ double erfOverX(double u)
{
  double r = 1.805761181299233e-16;
  r = fma(r, u, -1.0300117447682573e-14);
  r = fma(r, u, 2.927836726213971e-13);
  r = fma(r, u, -5.731081299066304e-12);
  r = fma(r, u, 8.96014012256378e-11);
  r = fma(r, u, -1.2127292658512346e-09);
  r = fma(r, u, 1.4763819202890526e-08);
  r = fma(r, u, -1.635716222383698e-07);
  r = fma(r, u, 1.6460811429838825e-06);
  r = fma(r, u, -1.4925505494318574e-05);
  r = fma(r, u, 0.00012055321281183126);
  r = fma(r, u, -0.000854832635719831);
  r = fma(r, u, 0.005223977599866574);
  r = fma(r, u, -0.026866170638949895);
  r = fma(r, u, 0.11283791670871149);
  r = fma(r, u, -0.37612638903178647);
  return fma(r, u, 1.1283791670955123);
}
}  // namespace rgd
