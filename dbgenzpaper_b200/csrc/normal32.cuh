// normal32.cuh -- FP32 normal tail mass and inverse of the mixed-precision
// step, written for this library (no dependencies: device code only).
//
//   tail_mass_f32(x) = erfc(x) / 2 = Phi(-sqrt(2) x),   0 <= x <= 9,
//
// in the form erfc(x) = t exp(P(t) - x^2), t = 1 / (1 + x/2), with P a
// degree-9 polynomial: the form of the Chebyshev-fitted complementary error
// function of Press, Teukolsky, Vetterling and Flannery (Numerical Recipes,
// "erfcc").  The coefficients here are our own: a least-squares fit of
// P(t) = ln(erfcx(x)) - ln(t) on 400,001 points of [0, 9] in double
// precision (maximum error of the fit 2.2e-7 in P), times log2(e), so that
// t 2^(P'(t) - x (x log2 e)) takes no multiply after the polynomial; the last
// three, given as floats, are within two units of that, chosen for the least
// mean error of the float evaluation.
// Evaluated in FP32 with one reciprocal, ten FMAs and one exp2 and no branches; the relative error
// against erfc is below 3e-6 for x <= 4.5 and below 1.5e-5 up to x = 9 (the
// FP32 rounding of the exponent P - x^2 dominates there, where the mass is
// below 1e-10).
#pragma once

namespace dbgz {

// 2^z by the SFU (ex2.approx.ftz: relative error about 2^-22; results below
// 2^-126 flush to zero, -inf gives 0).
__device__ __forceinline__ float exp2_sfu(float z) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z));
  return e;
}

// The SFU's reciprocal, base-2 logarithm and reciprocal square root in the
// forms that flush subnormals: their arguments here are normal (or 0 where
// the result is not used), and the plain forms (__fdividef, __logf, rsqrtf)
// spend two to five instructions each on scaling subnormal arguments.
__device__ __forceinline__ float rcp_sfu(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float log2_sfu(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_sfu(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

constexpr double kL2 = 1.4426950408889634;  // log2(e)
constexpr float kLog2e = (float)kL2;
__device__ __forceinline__ float tail_mass_f32(float x) {
  const float t = rcp_sfu(fmaf(0.5f, x, 1.0f));
  const float xl = x * kLog2e;
  float p = (float)(1.6112529716e-01 * kL2);
  p = fmaf(p, t, (float)(-7.6098558876e-01 * kL2));
  p = fmaf(p, t, (float)(1.3262850294e+00 * kL2));
  p = fmaf(p, t, (float)(-8.9638341094e-01 * kL2));
  p = fmaf(p, t, (float)(6.4102997549e-02 * kL2));
  p = fmaf(p, t, (float)(-6.4260147179e-02 * kL2));
  p = fmaf(p, t, (float)(5.3133554076e-02 * kL2));
  p = fmaf(p, t, 5.533192754e-01f);
  p = fmaf(p, t, 1.441120148e+00f);
  p = fmaf(p, t, -1.825669408e+00f);
  return 0.5f * t * exp2_sfu(fmaf(-xl, x, p));
}

constexpr double kR2 = 1.4142135623730951;

// -Phi^-1(p) for 0 < p <= 1/2 (the smaller tail: the step forms u or 1 - u,
// whichever is below 1/2), FP32, without branches.  The form is M. Giles'
// ("Approximating the erfinv function", GPU Computing Gems Jade, 2011):
// with x = 1 - 2p and w = -ln(4 p (1 - p)) = -ln(1 - x^2),
//   erfinv(x) = x P(w - 2.5)          for w < 5   (p > 1.69e-3),
//   erfinv(x) = T(sqrt(w) - 4)        for w >= 5  (p down to 2.2e-16, w <= 34.7),
// and Phi^-1(p) = -sqrt(2) erfinv(x).  P (degree 8) and T (degree 9) are our
// own weighted least-squares fits of the relative error in double precision
// (maximum 9.4e-8 and 5.8e-8), the coefficients times sqrt(2); w enters as
// -log2(4 p (1 - p)) with ln 2 in the two arguments' FMAs (one coefficient,
// given as a float, is two units off for the least mean error of the float
// evaluation).  Both are evaluated and the region selected, so the code has
// no branch.  Relative error in FP32 below 4e-7 for p >= 2.2e-16.
__device__ __forceinline__ float phi_inv_mag_f32(float p) {
  const float lg = log2_sfu(4.0f * p * (1.0f - p));
  const float x = fmaf(-2.0f, p, 1.0f);
  const float tc = fmaf(lg, -0.69314718056f, -2.5f);
  float pc = (float)(2.854775242e-08 * kR2);
  pc = fmaf(pc, tc, (float)(3.437494356e-07 * kR2));
  pc = fmaf(pc, tc, (float)(-3.528993161e-06 * kR2));
  pc = fmaf(pc, tc, (float)(-4.396994196e-06 * kR2));
  pc = fmaf(pc, tc, (float)(2.186026004e-04 * kR2));
  pc = fmaf(pc, tc, (float)(-1.253706953e-03 * kR2));
  pc = fmaf(pc, tc, (float)(-4.177708101e-03 * kR2));
  pc = fmaf(pc, tc, 3.488027155e-01f);
  pc = fmaf(pc, tc, (float)(1.501409422e+00 * kR2));
  const float ts = fmaf(-lg * rsqrt_sfu(-lg), 0.83255461116f, -4.0f);  // sqrt(w) - 4
  float pt = (float)(8.193106379e-07 * kR2);
  pt = fmaf(pt, ts, (float)(-1.490730122e-06 * kR2));
  pt = fmaf(pt, ts, (float)(-6.624017282e-06 * kR2));
  pt = fmaf(pt, ts, (float)(2.765589313e-05 * kR2));
  pt = fmaf(pt, ts, (float)(-8.117484620e-05 * kR2));
  pt = fmaf(pt, ts, (float)(2.877970689e-04 * kR2));
  pt = fmaf(pt, ts, (float)(-8.563289957e-04 * kR2));
  pt = fmaf(pt, ts, (float)(1.256645993e-03 * kR2));
  pt = fmaf(pt, ts, (float)(1.009495442e+00 * kR2));
  pt = fmaf(pt, ts, (float)(3.839783388e+00 * kR2));
  return lg > -7.2134752044f ? pc * x : pt;  // w < 5
}
// Phi^-1(p), 0 < p <= 1/2
__device__ __forceinline__ float phi_inv_lower_f32(float p) { return -phi_inv_mag_f32(p); }

}  // namespace dbgz
