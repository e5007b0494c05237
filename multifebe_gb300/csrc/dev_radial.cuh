// Radial functions of the time-harmonic fundamental solutions as piecewise
// polynomials. psi, chi, TT1..TT3 (bem_harela3d.f90:654-688) and S1..S5
// (:219-283, 2573-2662) depend on the distance r alone: each is a singular
// part (a 1/r, 1/r^2, 1/r^3 term, for S1..S5 a 1/r term too) plus an entire
// function of r. Once per call, k_radial samples the entire parts of every
// frequency on intervals of length h = kRadKh / max(|k1|, |k2|) that cover the
// mesh and turns them into polynomials of degree kRadD in the interval's
// coordinate; a quadrature point then costs a table row and a Horner sum
// instead of two decomposed exponentials (2 x ~15 series terms or exp and
// sincos) and their 50 complex combinations.
//
// Truncation: with |k| h / 2 = 1/16 the Chebyshev coefficients fall like
// (1/32)^m / m!, so degree 7 leaves at most 3e-17 of the function (checked in
// 40 digits for nu = 0 .. 0.49, xi = 0 .. 0.1; degree 8 on intervals twice as
// long leaves 5e-17, at 10 more operations per point and function). The
// samples themselves are formed in binary64 with the E_n series up to
// |z| = 4, so they lose less to cancellation near |z| = 1 than a direct
// evaluation with the reference's switch to exp at |z| = 1.
//
// The functions are stored with the constants of u* (cte_u), t* / d* (cte_t =
// cte_d) and s* (cte_s) multiplied in, so the flush of a pair does not scale.
#pragma once
#include "dev_complex.cuh"
#include "dev_df64.cuh"

namespace mfb {

constexpr double kRadKh = 0.125;
constexpr int kRadD = 7;             // polynomial degree
constexpr int kRadC = kRadD + 1;
constexpr int kRadDF = 4;            // double-float path: terms up to this degree in df64, the rest in FP32
constexpr int kRadRowF = kRadDF + 3; // float4 per function and interval of the double-float table
// intervals per frequency at most: rows of 640 B (1280 with S1..S5, and 560 more
// for the double-float ones), 40 to 120 MB per frequency. Beyond it (|k| times the
// mesh's extent above 8192, 1300 wavelengths across) the kernels evaluate E_n
// directly.
constexpr int kRadMaxN = 65536;

// singular coefficients (scaled) and the interval of one frequency
struct RadF {
  double inv2h;  // 2 / h
  cd s[5];       // psi(1), chi(1) [1/r], T1(1), T2(1), T3(1) [1/r^2]
  cd s3[5], s1[5];  // S1..S5: the 1/r^3 and 1/r terms (HBIE only)
};
struct RadFF {
  ff inv2h;
  cf s[5];
};
// double-float rows: per function kRadDF + 1 coefficients {re.hi, im.hi, re.lo,
// im.lo}, then the FP32 ones in pairs {re, im, re, im}
// table of all frequencies: rows [f][interval][function][kRadC] complex; nfun
// 5 (psi, chi, TT1..TT3) or 10 (with S1..S5); n = 0: no table
struct RadTab {
  const double2* c = nullptr;
  const float4* cf4 = nullptr;  // double-float rows [f][interval][5][kRadRowF], or null
  const RadF* f = nullptr;
  const RadFF* ff_ = nullptr;
  int n = 0, nfun = 5;
};

#ifdef __CUDACC__
// the interval of r and the coordinate x in [-1, 1] inside it
__device__ __forceinline__ const double2* rad_row(const RadTab& t, int f, const RadF& q, double r, double& x) {
  const double s = r * q.inv2h;
  const int i = min(max((int)(0.5 * s), 0), t.n - 1);
  x = s - (double)(2 * i + 1);
  return t.c + ((size_t)f * t.n + i) * t.nfun * kRadC;
}
// Horner sum of one function's row
__device__ __forceinline__ cd rad_eval(const double2* c, double x) {
  double2 v = __ldg(c + kRadD);
  double re = v.x, im = v.y;
#pragma unroll
  for (int m = kRadD - 1; m >= 0; --m) {
    v = __ldg(c + m);
    re = fma(re, x, v.x);
    im = fma(im, x, v.y);
  }
  return mk(re, im);
}
#endif

}  // namespace mfb
