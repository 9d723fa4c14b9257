// normal64.cuh -- FP64 erf and inverse erf of the integration loops, written
// for this library.
//
// Both expand around the nearest a = i/32 of a 193-entry table in shared
// memory (erfc, its derivative g and 1/g there, correctly rounded;
// normtab_fit.py), with delta = x - a, |delta| <= 1/64:
//   erfc(a + delta) = erfc(a) - g(a) delta Q(a delta, delta^2),
//   Q = sum_n (-1)^n H_n(a) delta^n / (n + 1)!,
// the Taylor series of the integral of exp(-2 a t - t^2) over [0, delta]; the
// Hermite polynomials H_n are homogeneous in z = a delta and w = delta^2, so
// Q is one polynomial in (z, w) for every table entry.  n <= 7 leaves less
// than 1e-18 absolute in erfc, and n <= 9 (its larger terms; kTail) less than
// 5e-16 in an x up to 5.8 taken from erfc.
//
// Why a table: the FP64 pipe bounds the loops, and a warp-wide operation on
// it takes 2 cycles.  CUDA's erf and erfinv measured 147 and 179 cycles a
// warp (4 warps a scheduler); 26 and 42 operations here make 52 and 84, and
// there is no branch for the lanes to diverge on.
#pragma once
#include <cuda_runtime.h>

#include "normal32.cuh"

namespace dbgz {

constexpr int kNormTab = 193;
static __device__ const double kNormTabSrc[kNormTab][3] = {
#include "normtab.h"
};

// The table in shared memory; norm_tab_load by `nt` threads, then a barrier.
struct NormTab {
  double2 eg[kNormTab];  // erfc(a), g(a)
  double rg[kNormTab];   // 1 / g(a)
};
__device__ __forceinline__ void norm_tab_load(NormTab &t, int tid, int nt) {
  for (int i = tid; i < kNormTab; i += nt) {
    t.eg[i] = make_double2(kNormTabSrc[i][0], kNormTabSrc[i][1]);
    t.rg[i] = kNormTabSrc[i][2];
  }
}

// delta Q of x = a + delta, 0 <= x <= 6: i = 32 a, zd = i delta = 32 z
struct NormNode {
  int i;
  double delta, z32, w;
  __device__ __forceinline__ explicit NormNode(double x) {
    const double m = 6755399441055744.0;  // 1.5 2^52: adding it rounds to an integer
    const double t = fma(x, 32.0, m);
    i = __double2loint(t);
    const double r = t - m;
    delta = fma(r, -0.03125, x);
    z32 = r * delta;
    w = delta * delta;
  }
  template <bool kTail>
  __device__ __forceinline__ double q() const {
    constexpr double s = 1.0 / 32.0, s2 = s * s, s3 = s2 * s, s4 = s2 * s2, s5 = s4 * s, s6 = s3 * s3, s7 = s6 * s;
    constexpr double s8 = s4 * s4, s9 = s8 * s;
    const double a0 = fma(fma(fma(w, -1.0 / 42.0, 0.1), w, -1.0 / 3.0), w, 1.0);
    const double a1 = fma(fma(fma(w, s / 24.0, -s / 6.0), w, s / 2.0), w, -s);
    const double a2 = fma(fma(w, s2 / 7.0, -0.4 * s2), w, s2 * 2.0 / 3.0);
    const double a3 = fma(fma(w, -s3 / 12.0, s3 * 2.0 / 9.0), w, -s3 / 3.0);
    const double a4 = fma(kTail ? fma(w, s4 / 27.0, -s4 * 2.0 / 21.0) : -s4 * 2.0 / 21.0, w, s4 * 2.0 / 15.0);
    const double a5 = fma(w, s5 / 30.0, -s5 * 2.0 / 45.0);
    // even and odd parts in z^2, two chains
    const double zz = z32 * z32;
    double a6 = s6 * 4.0 / 315.0, a7 = -s7 / 315.0;
    if (kTail) {
      a6 = fma(zz, s8 * 2.0 / 2835.0, fma(w, -s6 * 4.0 / 405.0, a6));
      a7 = fma(zz, -s9 * 2.0 / 14175.0, a7);
    }
    const double ev = fma(fma(fma(zz, a6, a4), zz, a2), zz, a0);
    const double od = fma(fma(fma(zz, a7, a5), zz, a3), zz, a1);
    return fma(od, z32, ev);
  }
};

// erf(x) for any x that is not NaN (|x| > 6 rounds to 1)
__device__ __forceinline__ double erf_tab(const NormTab &t, double x) {
  const double ax = fabs(x);
  const NormNode n(ax < 6.0 ? ax : 6.0);
  const double2 eg = t.eg[n.i];
  const double ec = fma(-(eg.y * n.delta), n.q<false>(), eg.x);
  return copysign(1.0 - ec, x);
}

// sqrt(2) erfinv(v) = Phi^-1((1 + v) / 2), 2^-52 <= 1 - |v|: the FP32 quantile
// (relative error 4e-7) and one third-order correction, with the residual
// taken in erfc(|x|) - (1 - |v|), which is exact to the last bits of v in
// the tails:  D = R / g(x0),  x = x0 + D + x0 D^2  (the next term is below
// 3e-16 at x0 = 5).  1 / g(x0) = exp(2 a delta + delta^2) / g(a).
__device__ __forceinline__ double sqrt2_erfinv_tab(const NormTab &t, double v) {
  const double q = 1.0 - fabs(v);
  const double x0 = (double)fminf(-0.70710678f * phi_inv_lower_f32(0.5f * (float)q), 6.0f);
  const NormNode n(x0);
  const double2 eg = t.eg[n.i];
  const double res = fma(-(eg.y * n.delta), n.q<true>(), eg.x - q);
  const double u = fma(n.z32, 1.0 / 16.0, n.w);  // 2 a delta + delta^2, below 0.19
  double e = fma(u, 1.0 / 5040.0, 1.0 / 720.0);
  e = fma(e, u, 1.0 / 120.0);
  e = fma(e, u, 1.0 / 24.0);
  e = fma(e, u, 1.0 / 6.0);
  e = fma(e, u, 0.5);
  e = fma(e, u, 1.0);
  e = fma(e, u, 1.0);
  const double D = res * (t.rg[n.i] * e);
  const double x = fma(fma(x0, D, 1.0), D, x0);
  return copysign(1.4142135623730951 * x, v);
}

}  // namespace dbgz
