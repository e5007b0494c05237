// Builder of the radial tables (dev_radial.cuh): one warp per (interval,
// frequency). Lanes 0..15 form E_2..E_6 of k1 and lanes 16..31 those of k2 at
// 16 Chebyshev nodes of the interval, lanes 0..15 combine them into the entire
// parts of the functions, then all lanes form the Chebyshev coefficients
// (discrete orthogonality) and the monomial ones. About 20 k binary64 lane
// operations per row: 20 us for the 29 intervals x 20 frequencies of the 8x8
// cube's sweep, against tens of milliseconds of pair kernels.
#pragma once

namespace mfb {

// E_2..E_6 of z for the tables: the series up to |z| = 4 (terms to z^34), then
// e^z minus its leading terms
__device__ __forceinline__ void rad_zexp(cd z, cd E[7]) {
  const double az2 = z.re * z.re + z.im * z.im;
  const cd z2 = z * z, z3 = z2 * z, z4 = z3 * z, z5 = z4 * z;
  if (az2 <= 16.0) {
    cd t = mk(1.0);
    for (int k = 34; k >= 7; --k) t = 1.0 + t * z * (1.0 / (double)k);
    E[6] = ((z5 * z) * (1.0 / 720.0)) * t;
    E[5] = E[6] + z5 * (1.0 / 120.0);
    E[4] = E[5] + z4 * (1.0 / 24.0);
    E[3] = E[4] + z3 * (1.0 / 6.0);
    E[2] = E[3] + z2 * 0.5;
  } else {
    E[2] = (cexp_(z) - 1.0) - z;
    E[3] = E[2] - 0.5 * z2;
    E[4] = E[3] - (1.0 / 6.0) * z3;
    E[5] = E[4] - (1.0 / 24.0) * z4;
    E[6] = E[5] - (1.0 / 120.0) * z5;
  }
}

// Chebyshev polynomials T_j as monomials, rows j, columns m
__constant__ double c_cheb[8][8] = {{1, 0, 0, 0, 0, 0, 0, 0},     {0, 1, 0, 0, 0, 0, 0, 0},
                                    {-1, 0, 2, 0, 0, 0, 0, 0},    {0, -3, 0, 4, 0, 0, 0, 0},
                                    {1, 0, -8, 0, 8, 0, 0, 0},    {0, 5, 0, -20, 0, 16, 0, 0},
                                    {-1, 0, 18, 0, -48, 0, 32, 0}, {0, -7, 0, 56, 0, -112, 0, 64}};

template <int NFUN>
__global__ void __launch_bounds__(32) k_radial(const HarParD* par, const HarParH* parh, const double* hlen, int n,
                                               double2* tab, float4* tabf, RadF* rf, RadFF* rff) {
  static_assert(kRadC == 8, "conversion matrix");
  __shared__ cd E[2][16][7];        // [n]: E_n scaled by r^-(n-1), n = 2..6, per wavenumber and node
  __shared__ double F[16][2 * NFUN];  // function samples
  __shared__ double C[kRadC][2 * NFUN];
  __shared__ double M[kRadC][2 * NFUN];
  __shared__ double cs[33];           // cos(pi j / 32)
  const int lane = threadIdx.x, iv = blockIdx.x, f = blockIdx.y;
  const HarParD& q = par[f];
  const double h = hlen[f];
  cs[lane] = cospi(lane / 32.0);
  if (lane == 0) cs[32] = -1.0;
  __syncwarp();
  {
    const int k = lane & 15;
    const double r = h * (iv + 0.5 * (1.0 + cs[2 * k + 1]));
    const cd kk = lane < 16 ? q.k1 : q.k2;
    cd e[7];
    rad_zexp(mk(kk.im * r, -kk.re * r), e);
    const double d1 = 1.0 / r;
    double s = d1;
#pragma unroll
    for (int j = 2; j < 7; ++j, s *= d1) E[lane >> 4][k][j] = e[j] * s;
  }
  __syncwarp();
  if (lane < 16) {
    const cd* a = E[0][lane];  // a[n] = E_n(-i k1 r) r^-(n-1)
    const cd* b = E[1][lane];
    cd X[NFUN];
    X[0] = q.psi[1] + b[2] + q.psi[2] * a[3] + q.psi[3] * b[3] + q.psi[4] * a[4] + q.psi[5] * b[4];
    X[1] = q.chi[1] * a[2] + b[2] + q.chi[2] * a[3] + q.chi[3] * b[3] + q.chi[4] * a[4] + q.chi[5] * b[4];
    X[2] = q.T1[1] + q.T1[2] * a[2] + q.T1[3] * b[2] + q.T1[4] * a[3] + q.T1[5] * b[3] + q.T1[6] * a[4] +
           q.T1[7] * b[4] + q.T1[8] * a[5] + q.T1[9] * b[5];
    X[3] = q.T2[1] + q.T2[2] * b[2] + q.T2[3] * a[3] + q.T2[4] * b[3] + q.T2[5] * a[4] + q.T2[6] * b[4] +
           q.T2[7] * a[5] + q.T2[8] * b[5];
    X[4] = q.T3[1] + q.T3[2] * a[2] + q.T3[3] * a[3] + q.T3[4] * b[3] + q.T3[5] * a[4] + q.T3[6] * b[4] +
           q.T3[7] * a[5] + q.T3[8] * b[5];
    X[0] = q.cte_u * X[0];
    X[1] = q.cte_u * X[1];
#pragma unroll
    for (int t = 2; t < 5; ++t) X[t] = q.cte_t * X[t];
    if constexpr (NFUN == 10) {
      const HarParH& s = parh[f];
      X[5] = s.S1[2] * b[2] + s.S1[3] * a[3] + s.S1[4] * b[3] + s.S1[5] * a[4] + s.S1[6] * b[4] + s.S1[7] * a[5] +
             s.S1[8] * b[5] + s.S1[9] * a[6] + s.S1[10] * b[6];
      X[6] = s.S2[2] * a[2] + s.S2[3] * a[3] + s.S2[4] * b[3] + s.S2[5] * a[4] + s.S2[6] * b[4] + s.S2[7] * a[5] +
             s.S2[8] * b[5] + s.S2[9] * a[6] + s.S2[10] * b[6];
      X[7] = s.S3[2] * a[2] + s.S3[3] * b[2] + s.S3[4] * a[3] + s.S3[5] * b[3] + s.S3[6] * a[4] + s.S3[7] * b[4] +
             s.S3[8] * a[5] + s.S3[9] * b[5] + s.S3[10] * a[6] + s.S3[11] * b[6];
      X[8] = s.S4[2] + s.S4[3] * b[3] + s.S4[4] * a[4] + s.S4[5] * b[4] + s.S4[6] * a[5] + s.S4[7] * b[5] +
             s.S4[8] * a[6] + s.S4[9] * b[6];
      X[9] = s.S5[2] + s.S5[3] * a[2] + s.S5[4] * a[3] + s.S5[5] * a[4] + s.S5[6] * b[4] + s.S5[7] * a[5] +
             s.S5[8] * b[5] + s.S5[9] * a[6] + s.S5[10] * b[6];
#pragma unroll
      for (int t = 5; t < 10; ++t) X[t] = s.cte_s * X[t];
    }
#pragma unroll
    for (int t = 0; t < NFUN; ++t) {
      F[lane][2 * t] = X[t].re;
      F[lane][2 * t + 1] = X[t].im;
    }
  }
  __syncwarp();
  for (int o = lane; o < kRadC * 2 * NFUN; o += 32) {
    const int j = o / (2 * NFUN), c = o - j * (2 * NFUN);
    double s = 0.0;
#pragma unroll 4
    for (int k = 0; k < 16; ++k) {
      const int m = (j * (2 * k + 1)) & 63;
      s = fma(F[k][c], cs[m <= 32 ? m : 64 - m], s);
    }
    C[j][c] = s * (j == 0 ? 0.0625 : 0.125);
  }
  __syncwarp();
  double2* T = tab + ((size_t)f * n + iv) * NFUN * kRadC;
  for (int o = lane; o < kRadC * 2 * NFUN; o += 32) {
    const int m = o / (2 * NFUN), c = o - m * (2 * NFUN);
    double s = 0.0;
#pragma unroll
    for (int j = kRadC - 1; j >= 0; --j) s = fma(c_cheb[j][m], C[j][c], s);
    M[m][c] = s;
    reinterpret_cast<double*>(T)[2 * ((size_t)(c >> 1) * kRadC + m) + (c & 1)] = s;
  }
  __syncwarp();
  if (tabf) {
    float4* Tf = tabf + ((size_t)f * n + iv) * 5 * kRadRowF;
    for (int o = lane; o < 5 * kRadRowF; o += 32) {
      const int t = o / kRadRowF, m = o - t * kRadRowF;
      if (m <= kRadDF) {
        const ff re = ff_from(M[m][2 * t]), im = ff_from(M[m][2 * t + 1]);
        Tf[o] = make_float4(re.hi, im.hi, re.lo, im.lo);
      } else {
        const int a = 2 * m - kRadDF - 1;  // first of the two FP32 terms of this float4
        const float2 u = make_float2((float)M[a][2 * t], (float)M[a][2 * t + 1]);
        const float2 v = a + 1 <= kRadD ? make_float2((float)M[a + 1][2 * t], (float)M[a + 1][2 * t + 1])
                                        : make_float2(0.0f, 0.0f);
        Tf[o] = make_float4(u.x, u.y, v.x, v.y);
      }
    }
  }
  if (iv == 0 && lane == 0) {
    RadF o;
    o.inv2h = 2.0 / h;
    o.s[0] = q.cte_u * q.psi[0];
    o.s[1] = q.cte_u * q.chi[0];
    o.s[2] = q.cte_t * q.T1[0];
    o.s[3] = q.cte_t * q.T2[0];
    o.s[4] = q.cte_t * q.T3[0];
#pragma unroll
    for (int t = 0; t < 5; ++t) o.s3[t] = o.s1[t] = mk(0.0);
    if constexpr (NFUN == 10) {
      const HarParH& s = parh[f];
      o.s3[0] = s.cte_s * s.S1[0]; o.s1[0] = s.cte_s * s.S1[1];
      o.s3[1] = s.cte_s * s.S2[0]; o.s1[1] = s.cte_s * s.S2[1];
      o.s3[2] = s.cte_s * s.S3[0]; o.s1[2] = s.cte_s * s.S3[1];
      o.s3[3] = s.cte_s * s.S4[0]; o.s1[3] = s.cte_s * s.S4[1];
      o.s3[4] = s.cte_s * s.S5[0]; o.s1[4] = s.cte_s * s.S5[1];
    }
    rf[f] = o;
    if (rff) {
      RadFF w;
      w.inv2h = ff_from(o.inv2h);
      for (int t = 0; t < 5; ++t) w.s[t] = cf_from(o.s[t].re, o.s[t].im);
      rff[f] = w;
    }
  }
}

}  // namespace mfb
