// Dense LU with partial pivoting (LAPACK getrf semantics: row interchanges
// recorded in ipiv, unit lower L and upper U overwrite A) and the triangular
// solves of getrs, for a batch of column-major matrices with a common size.
// Replaces the LAPACK calls of src/solve_lse_r.f90:137,189 and
// src/solve_lse_c.f90:124,176.
//
// Right-looking blocked algorithm, panel width NB:
//   panel   column-by-column partial pivoting inside the panel (k_panel_*),
//   laswp   the panel's interchanges applied to the other columns,
//   trsm    U12 = L11^{-1} A12,
//   update  A22 -= L21 U12 (a GEMM; issued by the host layer).
#pragma once
#include <cuda_runtime.h>
#include "dev_complex.cuh"
#include <cooperative_groups.h>

namespace mfb {

// scalar traits ---------------------------------------------------------------
template <typename S> struct Sc;
template <> struct Sc<double> {
  typedef double R;
  __device__ static double zero() { return 0.0; }
  __device__ static double one() { return 1.0; }
  __device__ static double abs1(double a) { return fabs(a); }
  __device__ static double mul(double a, double b) { return a * b; }
  __device__ static double sub(double a, double b) { return a - b; }
  __device__ static double add(double a, double b) { return a + b; }
  __device__ static double div(double a, double b) { return a / b; }
  __device__ static double rcp(double a) { return 1.0 / a; }
  __device__ static bool iszero(double a) { return a == 0.0; }
  __device__ static double conj(double a) { return a; }
  __device__ static double from(double v) { return v; }
  __device__ static double re(double a) { return a; }
};
template <> struct Sc<float> {
  typedef float R;
  __device__ static float zero() { return 0.0f; }
  __device__ static float one() { return 1.0f; }
  __device__ static float abs1(float a) { return fabsf(a); }
  __device__ static float mul(float a, float b) { return a * b; }
  __device__ static float sub(float a, float b) { return a - b; }
  __device__ static float add(float a, float b) { return a + b; }
  __device__ static float div(float a, float b) { return a / b; }
  __device__ static float rcp(float a) { return 1.0f / a; }
  __device__ static bool iszero(float a) { return a == 0.0f; }
  __device__ static float conj(float a) { return a; }
  __device__ static float from(double v) { return (float)v; }
  __device__ static float re(float a) { return a; }
};
template <> struct Sc<double2> {
  typedef double R;
  __device__ static double2 zero() { return make_double2(0.0, 0.0); }
  __device__ static double2 one() { return make_double2(1.0, 0.0); }
  // |re| + |im|, the pivot measure of LAPACK's izamax (dcabs1)
  __device__ static double abs1(double2 a) { return fabs(a.x) + fabs(a.y); }
  __device__ static double2 mul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
  __device__ static double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
  __device__ static double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
  __device__ static double2 div(double2 a, double2 b) {
    cd q = mk(a.x, a.y) / mk(b.x, b.y);
    return make_double2(q.re, q.im);
  }
  __device__ static double2 rcp(double2 a) { return div(one(), a); }
  __device__ static bool iszero(double2 a) { return a.x == 0.0 && a.y == 0.0; }
  __device__ static double2 conj(double2 a) { return make_double2(a.x, -a.y); }
  __device__ static double2 from(double v) { return make_double2(v, 0.0); }
  __device__ static double re(double2 a) { return a.x; }
};
template <> struct Sc<float2> {
  typedef float R;
  __device__ static float2 zero() { return make_float2(0.f, 0.f); }
  __device__ static float2 one() { return make_float2(1.f, 0.f); }
  __device__ static float abs1(float2 a) { return fabsf(a.x) + fabsf(a.y); }
  __device__ static float2 mul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
  __device__ static float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
  __device__ static float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
  __device__ static float2 div(float2 a, float2 b) {
    if (fabsf(b.x) >= fabsf(b.y)) {
      float r = b.y / b.x, den = b.x + b.y * r;
      return make_float2((a.x + a.y * r) / den, (a.y - a.x * r) / den);
    }
    float r = b.x / b.y, den = b.y + b.x * r;
    return make_float2((a.x * r + a.y) / den, (a.y * r - a.x) / den);
  }
  __device__ static float2 rcp(float2 a) { return div(one(), a); }
  __device__ static bool iszero(float2 a) { return a.x == 0.f && a.y == 0.f; }
  __device__ static float2 conj(float2 a) { return make_float2(a.x, -a.y); }
  __device__ static float2 from(double v) { return make_float2((float)v, 0.f); }
  __device__ static float re(float2 a) { return a.x; }
};

// biased exponent of the larger component's modulus; 0 for zero and subnormal
// values, and for non-finite ones, which stay so under any scale
__device__ __forceinline__ int tq_exp(float2 v) {
  const int x = (__float_as_uint(v.x) >> 23) & 255, y = (__float_as_uint(v.y) >> 23) & 255;
  return max(x == 255 ? 0 : x, y == 255 ? 0 : y);
}

// a value of another lane
template <typename S> __device__ __forceinline__ S shfl_s(S v, int src);
template <> __device__ __forceinline__ float2 shfl_s(float2 v, int src) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
template <> __device__ __forceinline__ double2 shfl_s(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
template <> __device__ __forceinline__ float shfl_s(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <> __device__ __forceinline__ double shfl_s(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// 1 / d by two Newton steps from the binary32 reciprocal (2^-23 -> 2^-46 -> the
// rounding of the last step: half a unit in the last place, as a division) where
// d and 1 / d are well inside binary32's range: on the chain of every column,
// where a dependent binary64 operation takes 63 cycles and more
__device__ __forceinline__ double piv_rcp(double d) {
  const float f = fabsf((float)d);
  if (!(f > 1e-36f && f < 1e36f)) return 1.0 / d;
  double y = (double)__frcp_rn((float)d);
  y = fma(y, fma(-d, y, 1.0), y);
  return fma(y, fma(-d, y, 1.0), y);
}
// conj(d) / |d|^2 where |d|^2 stays within that range, else Smith's form. |d|^2 as
// q + lo, lo the rounding errors of the squares and of their sum (formed while the
// first step runs), and the second step's correction c applied to the products,
// so that each part is rounded once: 0.44 x 2^-53 of |1 / d| rms, 1.0 at most, over
// 2e7 values (Smith's form 0.61 and 1.6; without lo and c 0.79 and 3.0)
__device__ __forceinline__ double2 piv_rcp(double2 d) {
  const bool xm = fabs(d.x) >= fabs(d.y);
  const double a = xm ? d.x : d.y, b = xm ? d.y : d.x;  // |a| >= |b|: aa - q is exact
  const double aa = a * a, q = fma(b, b, aa);
  const float f = (float)q;
  if (!(f > 1e-36f && f < 1e36f)) return Sc<double2>::rcp(d);
  const double lo = fma(b, b, aa - q) + fma(a, a, -aa);
  double y = (double)__frcp_rn(f);
  y = fma(y, fma(-q, y, 1.0), y);
  const double c = y * fma(-lo, y, fma(-q, y, 1.0));
  return make_double2(fma(d.x, y, d.x * c), -fma(d.y, y, d.y * c));
}
__device__ __forceinline__ float piv_rcp(float d) { return 1.0f / d; }
__device__ __forceinline__ float2 piv_rcp(float2 d) { return Sc<float2>::rcp(d); }

// ---------------------------------------------------------------------------
// Panel factorisation, one CTA per matrix (used where the panel's arithmetic
// is cheap relative to synchronisation: FP32 and small FP64 problems).
// A: batch of matrices at A + b*strideA; panel = columns [k, k+nb).
// ipiv (1-based global row indices) at ipiv + b*n; info (first zero pivot).
// ---------------------------------------------------------------------------
template <typename S, int NT>
__global__ void __launch_bounds__(NT) k_panel_cta(S* A, long long strideA, int lda, int n, int k, int nb, int* ipiv,
                                                  int* info) {
  typedef typename Sc<S>::R R;
  const int bidx = blockIdx.x;
  S* M = A + strideA * bidx;
  int* piv = ipiv + (size_t)n * bidx;
  __shared__ R sv[NT / 32];
  __shared__ int si[NT / 32];
  __shared__ int sp;
  __shared__ S prow[128];
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  const int kend = min(k + nb, n);
  for (int j = k; j < kend; ++j) {
    // argmax |A(i,j)|, i >= j (first index on ties, as i?amax)
    R best = -1;
    int bi = j;
    for (int i = j + threadIdx.x; i < n; i += NT) {
      R v = Sc<S>::abs1(M[(size_t)j * lda + i]);
      if (v > best) { best = v; bi = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      R ov = __shfl_xor_sync(0xffffffffu, best, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) { sv[wid] = best; si[wid] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      R b0 = sv[0];
      int i0 = si[0];
      for (int w = 1; w < NT / 32; ++w)
        if (sv[w] > b0 || (sv[w] == b0 && si[w] < i0)) { b0 = sv[w]; i0 = si[w]; }
      sp = i0;
      piv[j] = i0 + 1;
      if (Sc<S>::iszero(M[(size_t)j * lda + i0]) && info[bidx] == 0) info[bidx] = j + 1;
    }
    __syncthreads();
    const int p = sp;
    // swap rows j and p inside the panel and keep the pivot row in shared memory
    for (int c = k + threadIdx.x; c < kend; c += NT) {
      S a = M[(size_t)c * lda + j], bb = M[(size_t)c * lda + p];
      M[(size_t)c * lda + j] = bb;
      M[(size_t)c * lda + p] = a;
      prow[c - k] = bb;
    }
    __syncthreads();
    S dj = prow[j - k];
    if (!Sc<S>::iszero(dj)) {
      S r = Sc<S>::rcp(dj);
      for (int i = j + 1 + threadIdx.x; i < n; i += NT) {
        S l = Sc<S>::mul(M[(size_t)j * lda + i], r);
        M[(size_t)j * lda + i] = l;
        for (int c = j + 1; c < kend; ++c) M[(size_t)c * lda + i] = Sc<S>::sub(M[(size_t)c * lda + i], Sc<S>::mul(l, prow[c - k]));
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Multi-CTA panel step for one column j (FP64 problems, where a single SM's
// FP64 rate would serialise the panel). Two launches per column:
//   k_pcol_pivot:  one CTA per matrix, pivot search, ipiv, interchange in the panel
//   k_pcol_update: G CTAs per matrix, scale column j and rank-1 update of the
//                  panel columns j+1..k+nb-1 over row chunks
// ---------------------------------------------------------------------------
template <typename S, int NT>
__global__ void __launch_bounds__(NT) k_pcol_pivot(S* A, long long strideA, int lda, int n, int k, int nb, int j,
                                                   int* ipiv, int* info) {
  typedef typename Sc<S>::R R;
  const int bidx = blockIdx.x;
  S* M = A + strideA * bidx;
  __shared__ R sv[NT / 32];
  __shared__ int si[NT / 32];
  __shared__ int sp;
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  R best = -1;
  int bi = j;
  for (int i = j + threadIdx.x; i < n; i += NT) {
    R v = Sc<S>::abs1(M[(size_t)j * lda + i]);
    if (v > best) { best = v; bi = i; }
  }
  for (int o = 16; o > 0; o >>= 1) {
    R ov = __shfl_xor_sync(0xffffffffu, best, o);
    int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  if (lane == 0) { sv[wid] = best; si[wid] = bi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    R b0 = sv[0];
    int i0 = si[0];
    for (int w = 1; w < NT / 32; ++w)
      if (sv[w] > b0 || (sv[w] == b0 && si[w] < i0)) { b0 = sv[w]; i0 = si[w]; }
    sp = i0;
    ipiv[(size_t)n * bidx + j] = i0 + 1;
    if (Sc<S>::iszero(M[(size_t)j * lda + i0]) && info[bidx] == 0) info[bidx] = j + 1;
  }
  __syncthreads();
  const int p = sp;
  if (p != j) {
    const int kend = min(k + nb, n);
    for (int c = k + threadIdx.x; c < kend; c += NT) {
      S a = M[(size_t)c * lda + j];
      M[(size_t)c * lda + j] = M[(size_t)c * lda + p];
      M[(size_t)c * lda + p] = a;
    }
  }
}
template <typename S, int NT>
__global__ void __launch_bounds__(NT) k_pcol_update(S* A, long long strideA, int lda, int n, int k, int nb, int j) {
  const int bidx = blockIdx.y;
  S* M = A + strideA * bidx;
  const int kend = min(k + nb, n);
  __shared__ S prow[128];
  for (int c = j + threadIdx.x; c < kend; c += NT) prow[c - j] = M[(size_t)c * lda + j];
  __syncthreads();
  S dj = prow[0];
  if (Sc<S>::iszero(dj)) return;
  S r = Sc<S>::rcp(dj);
  for (int i = j + 1 + blockIdx.x * NT + threadIdx.x; i < n; i += gridDim.x * NT) {
    S l = Sc<S>::mul(M[(size_t)j * lda + i], r);
    M[(size_t)j * lda + i] = l;
    for (int c = j + 1; c < kend; ++c) M[(size_t)c * lda + i] = Sc<S>::sub(M[(size_t)c * lda + i], Sc<S>::mul(l, prow[c - j]));
  }
}

// ---------------------------------------------------------------------------
// Cooperative panel factorisation: the panel columns [k, k+kb) of each matrix
// are split by rows over G CTAs (row chunk of `chunk` rows each) and held in
// shared memory for the whole panel; per column one barrier among the matrix's
// G CTAs exchanges the chunk-local pivot candidates. Launched with
// cudaLaunchCooperativeKernel, so all CTAs are co-resident; every barrier wait
// is bounded (about a second), after which the kernel sets *err and returns.
//
// Per column j (global row/column jj = k + j):
//   every CTA   argmax |A(i,jj)| (LAPACK's |re|+|im| for complex) over its rows
//               i >= jj, publishes (value, row, the row's kb panel values); the
//               owner of row jj publishes that row too (slot jj % 2)
//   barrier
//   every CTA   picks the winner (largest value, smallest row on ties), swaps
//               the two rows inside its chunk where it owns them, then scales
//               column jj below the diagonal and updates columns jj+1.. of its rows
// Counters ctr[matrix] count barrier arrivals over the whole factorisation
// (zeroed once per getrf), so the target of column jj is (jj + 1) * G.
// ---------------------------------------------------------------------------
constexpr long long kCoopSpin = 1LL << 24;

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <typename S, int NT>
__global__ void __launch_bounds__(NT) k_panel_coop(S* A, long long strideA, int lda, int n, int k, int kb, int G,
                                                   int chunk, int b0, int* ipiv, int* info, unsigned* ctr, S* xrow,
                                                   typename Sc<S>::R* xval, int* xidx, int* err, long long spin) {
  typedef typename Sc<S>::R R;
  extern __shared__ __align__(16) unsigned char smraw[];
  S* pan = reinterpret_cast<S*>(smraw);  // [kb][chunk]
  S* prow = pan + (size_t)kb * chunk;     // [kb] pivot row
  __shared__ R sv[NT / 32];
  __shared__ int si[NT / 32], sg[NT / 32];
  __shared__ int s_ok, s_p, s_g;
  const int mat = b0 + blockIdx.x / G, g = blockIdx.x % G;
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  S* M = A + strideA * mat;
  int* piv = ipiv + (size_t)n * mat;
  const int r0 = k + g * chunk, r1 = min(n, r0 + chunk), nr = max(0, r1 - r0);
  // exchange slots of this matrix: [2][G][kb] rows, [2][G] values / indices, then
  // [2][kb] for the current diagonal row (stored at candidate index G)
  S* XR = xrow + (size_t)(mat) * 2 * (G + 1) * kb;
  R* XV = xval + (size_t)(mat) * 2 * G;
  int* XI = xidx + (size_t)(mat) * 2 * G;
  for (int t = threadIdx.x; t < kb * nr; t += NT) {
    const int c = t / nr, i = t - c * nr;
    pan[(size_t)c * chunk + i] = M[(size_t)(k + c) * lda + r0 + i];
  }
  __syncthreads();
  for (int j = 0; j < kb; ++j) {
    const int jj = k + j, slot = jj & 1;
    // chunk-local candidate
    R best = -1;
    int bi = -1;
    for (int i = max(jj, r0) - r0 + threadIdx.x; i < nr; i += NT) {
      const R v = Sc<S>::abs1(pan[(size_t)j * chunk + i]);
      if (v > best) { best = v; bi = r0 + i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const R ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi >= 0 && (bi < 0 || oi < bi))) { best = ov; bi = oi; }
    }
    if (lane == 0) { sv[wid] = best; si[wid] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      R b_ = sv[0];
      int i_ = si[0];
      for (int w = 1; w < NT / 32; ++w)
        if (sv[w] > b_ || (sv[w] == b_ && si[w] >= 0 && (i_ < 0 || si[w] < i_))) { b_ = sv[w]; i_ = si[w]; }
      XV[slot * G + g] = b_;
      XI[slot * G + g] = i_;
      s_p = i_;
    }
    __syncthreads();
    const int myc = s_p;
    if (myc >= 0 && (int)threadIdx.x < kb)
      XR[((size_t)slot * (G + 1) + g) * kb + threadIdx.x] = pan[(size_t)threadIdx.x * chunk + (myc - r0)];
    if (jj >= r0 && jj < r1 && (int)threadIdx.x < kb)
      XR[((size_t)slot * (G + 1) + G) * kb + threadIdx.x] = pan[(size_t)threadIdx.x * chunk + (jj - r0)];
    // barrier among the G CTAs of this matrix
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(ctr + mat, 1u);
      const unsigned target = (unsigned)(jj + 1) * (unsigned)G;
      long long it = 0;
      int ok = 1;
      const long long lim = spin > 0 ? spin : kCoopSpin;
      while (ld_acquire_u32(ctr + mat) < target) {
        if (++it > lim) { ok = 0; atomicExch(err, 1); break; }
        __nanosleep(32);
      }
      __threadfence();
      s_ok = ok;
    }
    __syncthreads();
    if (!s_ok) return;
    // winner over the G candidates (parallel loads, block argmax)
    {
      R b_ = -1;
      int i_ = -1, g_ = 0;
      for (int q = threadIdx.x; q < G; q += NT) {
        const R v = __ldcg(XV + slot * G + q);
        const int ix = __ldcg(XI + slot * G + q);
        if (ix >= 0 && (v > b_ || (v == b_ && ix < i_))) { b_ = v; i_ = ix; g_ = q; }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const R ov = __shfl_xor_sync(0xffffffffu, b_, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i_, o);
        const int og = __shfl_xor_sync(0xffffffffu, g_, o);
        if (oi >= 0 && (ov > b_ || (ov == b_ && (i_ < 0 || oi < i_)))) { b_ = ov; i_ = oi; g_ = og; }
      }
      if (lane == 0) { sv[wid] = b_; si[wid] = i_; sg[wid] = g_; }
      __syncthreads();
      if (threadIdx.x == 0) {
        R bb = sv[0];
        int ii = si[0], gg = sg[0];
        for (int w = 1; w < NT / 32; ++w)
          if (si[w] >= 0 && (sv[w] > bb || (sv[w] == bb && (ii < 0 || si[w] < ii)))) { bb = sv[w]; ii = si[w]; gg = sg[w]; }
        s_p = ii;
        s_g = gg;
      }
      __syncthreads();
    }
    const int p = s_p;
    if ((int)threadIdx.x < kb)
      prow[threadIdx.x] = __ldcg(XR + ((size_t)slot * (G + 1) + s_g) * kb + threadIdx.x);
    __syncthreads();
    if (g == 0 && threadIdx.x == 0) {
      piv[jj] = p + 1;
      if (Sc<S>::iszero(prow[j]) && info[mat] == 0) info[mat] = jj + 1;
    }
    if (p != jj) {
      // row p <- old row jj, row jj <- pivot row, where this CTA owns them
      if (p >= r0 && p < r1 && (int)threadIdx.x < kb)
        pan[(size_t)threadIdx.x * chunk + (p - r0)] = __ldcg(XR + ((size_t)slot * (G + 1) + G) * kb + threadIdx.x);
      if (jj >= r0 && jj < r1 && (int)threadIdx.x < kb) pan[(size_t)threadIdx.x * chunk + (jj - r0)] = prow[threadIdx.x];
    }
    __syncthreads();
    const S dj = prow[j];
    if (!Sc<S>::iszero(dj)) {
      const S rcp = piv_rcp(dj);
      for (int i = max(jj + 1, r0) - r0 + threadIdx.x; i < nr; i += NT) {
        const S l = Sc<S>::mul(pan[(size_t)j * chunk + i], rcp);
        pan[(size_t)j * chunk + i] = l;
        for (int c = j + 1; c < kb; ++c)
          pan[(size_t)c * chunk + i] = Sc<S>::sub(pan[(size_t)c * chunk + i], Sc<S>::mul(l, prow[c]));
      }
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < kb * nr; t += NT) {
    const int c = t / nr, i = t - c * nr;
    M[(size_t)(k + c) * lda + r0 + i] = pan[(size_t)c * chunk + i];
  }
}

// ---------------------------------------------------------------------------
// Cluster panel: the same pivoting as k_panel_coop with the G CTAs of a matrix
// forming one thread-block cluster (cluster rank = row chunk). Per column each
// CTA pushes its candidate (|a| as an ordered integer key, row, the row's kb
// values, the reciprocal of its pivot) into every CTA's shared memory, one
// hardware cluster barrier follows, and each warp picks the winner from local
// memory: no remote read and no block barrier lies between the cluster barrier
// and the update. The candidate of the next column is taken while its values
// are updated. Slots are double-buffered by column parity: a slot of column
// j + 2 is written after the barrier of column j + 1, which every CTA enters
// after its last read of column j's.
//
// GB300's binary64 pipe takes 16 cycles per warp instruction whatever the
// number of active lanes, so binary64 operations outside the rank-1 update
// decide the time of a small panel: the reciprocal of the pivot is formed by
// one warp per CTA, while the others push the rows, instead of by every thread
// (30 to 100 operations each); the pivot search compares integers (redux);
// complex updates use four FMAs. A column of an 870-row real panel takes 4800
// cycles (barriers and exchange 1600, reciprocal and pushes 1500, update 1400),
// 7600 before; 217 panels of four complex 3462-row systems 32.1 -> 12 ms with
// 16 CTAs per matrix.
// A NaN counts as zero in the search; the row jj itself is then taken.
// ---------------------------------------------------------------------------
// |a| ordered as an unsigned integer, 0 for NaN
__device__ __forceinline__ unsigned long long piv_key(double v) {
  const unsigned long long k = (unsigned long long)__double_as_longlong(v);
  return k > 0x7ff0000000000000ull ? 0ull : k;
}
__device__ __forceinline__ unsigned long long piv_key(float v) {
  const unsigned k = __float_as_uint(v);
  return k > 0x7f800000u ? 0ull : (unsigned long long)k;
}
// the warp's largest key and, among its holders, the smallest row (key + 1 and
// row as unsigned; no candidate: key1 = 0, row = ~0u)
__device__ __forceinline__ void piv_reduce(unsigned long long& key1, unsigned& row) {
  const unsigned hi = (unsigned)(key1 >> 32), lo = (unsigned)key1;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  row = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? row : 0xffffffffu);
  key1 = ((unsigned long long)mh << 32) | ml;
}
// a - l p
__device__ __forceinline__ double lu_fnma(double l, double p, double a) { return fma(-l, p, a); }
__device__ __forceinline__ float lu_fnma(float l, float p, float a) { return fmaf(-l, p, a); }
__device__ __forceinline__ double2 lu_fnma(double2 l, double2 p, double2 a) {
  return make_double2(fma(-l.x, p.x, fma(l.y, p.y, a.x)), fma(-l.x, p.y, fma(-l.y, p.x, a.y)));
}
__device__ __forceinline__ float2 lu_fnma(float2 l, float2 p, float2 a) {
  return make_float2(fmaf(-l.x, p.x, fmaf(l.y, p.y, a.x)), fmaf(-l.x, p.y, fmaf(-l.y, p.x, a.y)));
}
// bytes of dynamic shared memory of k_panel_cluster
template <typename S>
inline size_t panel_cluster_smem(int G, int kb, int chunk) {
  return sizeof(S) * (((size_t)kb * chunk + 3) / 4 * 4 + 2 * (size_t)G * (kb + 1) + 2 * (size_t)kb) + 2 * (size_t)G * 16 + 32;
}
template <typename S, int NT>
__global__ void __launch_bounds__(NT) k_panel_cluster(S* A, long long strideA, int lda, int n, int k, int kb,
                                                      int chunk, int* ipiv, int* info) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int G = (int)cl.num_blocks(), g = (int)cl.block_rank();
  extern __shared__ __align__(16) unsigned char smraw[];
  S* pan = reinterpret_cast<S*>(smraw);          // [kb][chunk]
  S* cand = pan + ((size_t)kb * chunk + 3) / 4 * 4;  // [2][G][kb + 1]: candidate row, reciprocal of its pivot
  S* rowj = cand + 2 * (size_t)G * (kb + 1);     // [2][kb]: row jj before the interchange
  unsigned long long* ckey = reinterpret_cast<unsigned long long*>(rowj + 2 * (size_t)kb);  // [2][G] key + 1
  unsigned* crow = reinterpret_cast<unsigned*>(ckey + 2 * (size_t)G);                      // [2][G]
  __shared__ unsigned long long wkey[NT / 32];
  __shared__ unsigned wrow[NT / 32];
  const int mat = blockIdx.x / G;
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  S* M = A + strideA * mat;
  int* piv = ipiv + (size_t)n * mat;
  const int r0 = k + g * chunk, r1 = min(n, r0 + chunk), nr = max(0, r1 - r0);
  for (int t = threadIdx.x; t < kb * nr; t += NT) {
    const int c = t / nr, i = t - c * nr;
    pan[(size_t)c * chunk + i] = M[(size_t)(k + c) * lda + r0 + i];
  }
  __syncthreads();
  unsigned long long bk = 0;  // this thread's candidate: key + 1, row
  unsigned br = 0xffffffffu;
  for (int i = threadIdx.x; i < nr; i += NT) {
    const unsigned long long q = piv_key(Sc<S>::abs1(pan[i])) + 1;
    if (q > bk) { bk = q; br = (unsigned)(r0 + i); }
  }
  cl.sync();  // every CTA of the cluster runs before the first push
  for (int j = 0; j < kb; ++j) {
    const int jj = k + j, slot = j & 1;
    piv_reduce(bk, br);
    if (lane == 0) { wkey[wid] = bk; wrow[wid] = br; }
    __syncthreads();
    {
      // every warp finds the CTA's candidate; warp 0 pushes its key and the
      // reciprocal of its pivot, the others its row (and row jj)
      unsigned long long q = lane < NT / 32 ? wkey[lane] : 0ull;
      unsigned r = lane < NT / 32 ? wrow[lane] : 0xffffffffu;
      piv_reduce(q, r);
      const bool have = q != 0ull, own = jj >= r0 && jj < r1;
      const int ix = have ? (int)r - r0 : 0;
      if (wid == 0) {
        if (have) {
          const S d = pan[(size_t)j * chunk + ix];
          const S rc = q == 1ull && Sc<S>::iszero(d) ? d : piv_rcp(d);
          if (lane < G) cl.map_shared_rank(cand, lane)[((size_t)slot * G + g) * (kb + 1) + kb] = rc;
        }
        if (lane < G) {
          cl.map_shared_rank(ckey, lane)[slot * G + g] = q;
          cl.map_shared_rank(crow, lane)[slot * G + g] = r;
        }
      } else if (lane < kb) {
        const S v = pan[(size_t)lane * chunk + ix], vj = own ? pan[(size_t)lane * chunk + (jj - r0)] : v;
        for (int rk = wid - 1; rk < G; rk += NT / 32 - 1) {
          if (have) cl.map_shared_rank(cand, rk)[((size_t)slot * G + g) * (kb + 1) + lane] = v;
          if (own) cl.map_shared_rank(rowj, rk)[slot * kb + lane] = vj;
        }
      }
    }
    cl.sync();
    unsigned long long q = lane < G ? ckey[slot * G + lane] : 0ull;
    const unsigned long long q0 = q;
    unsigned r = lane < G ? crow[slot * G + lane] : 0xffffffffu;
    const unsigned rr = r;
    piv_reduce(q, r);
    const int win = __ffs(__ballot_sync(0xffffffffu, lane < G && q0 == q && rr == r)) - 1;
    const int p = (int)r;
    const S* pr = cand + ((size_t)slot * G + win) * (kb + 1);
    const S* oj = rowj + slot * kb;
    const bool zero = q == 1ull && Sc<S>::iszero(pr[j]);  // key 0: zero or NaN
    if (g == 0 && threadIdx.x == 0) {
      piv[jj] = p + 1;
      if (zero && info[mat] == 0) info[mat] = jj + 1;
    }
    if (jj >= r0 && jj < r1 && p != jj && (int)threadIdx.x < kb)
      pan[(size_t)threadIdx.x * chunk + (jj - r0)] = pr[threadIdx.x];
    const S rcp = pr[kb];
    bk = 0;
    br = 0xffffffffu;
    for (int i = max(jj + 1, r0) - r0 + threadIdx.x; i < nr; i += NT) {
      S* x = pan + i;
      if (r0 + i == p) {  // takes row jj's place in the interchange
        for (int c = 0; c < kb; ++c) x[(size_t)c * chunk] = oj[c];
      }
      if (!zero) {
        const S l = Sc<S>::mul(x[(size_t)j * chunk], rcp);
        x[(size_t)j * chunk] = l;
#pragma unroll 5
        for (int c = j + 1; c < kb; ++c) x[(size_t)c * chunk] = lu_fnma(l, pr[c], x[(size_t)c * chunk]);
      }
      if (j + 1 < kb) {
        const unsigned long long qn = piv_key(Sc<S>::abs1(x[(size_t)(j + 1) * chunk])) + 1;
        if (qn > bk) { bk = qn; br = (unsigned)(r0 + i); }
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kb * nr; t += NT) {
    const int c = t / nr, i = t - c * nr;
    M[(size_t)(k + c) * lda + r0 + i] = pan[(size_t)c * chunk + i];
  }
}

// ---------------------------------------------------------------------------
// Interchanges of a 16-column panel applied to every column outside it and, for
// the columns [k + kb, ce), U12 = inv(L11) A12 in the same pass (one launch in
// place of k_laswp and k_trsm_cols). A warp composes the up to 16 interchanges
// into "position R_q takes the entry of C_q" for at most 32 positions (lanes 0..
// 15: the panel's rows, the others: rows below it), so a thread's loads of its
// column are independent instead of a chain of 16 exchanges through memory;
// the substitution runs on registers. One column per thread, 32 per CTA.
// ---------------------------------------------------------------------------
template <typename S>
__global__ void __launch_bounds__(32) k_swap_trsm16(S* A, long long strideA, int lda, int n, int k, int kb, int ce,
                                                    const int* ipiv) {
  __shared__ S L[16 * 16];
  __shared__ int R_[32], C_[32];
  const int bidx = blockIdx.y, t = threadIdx.x;
  S* M = A + strideA * bidx;
  const int* piv = ipiv + (size_t)n * bidx;
  int R = t < kb ? k + t : -1, C = R, nx = kb;
  const int myp = t < kb ? piv[k + t] - 1 : 0;
  for (int j = 0; j < kb; ++j) {
    const int p = __shfl_sync(0xffffffffu, myp, j);
    unsigned at = __ballot_sync(0xffffffffu, R == p);
    if (!at) {
      if (t == nx) R = C = p;
      at = 1u << nx;
      ++nx;
    }
    const int q = __ffs(at) - 1;
    const int cj = __shfl_sync(0xffffffffu, C, j), cq = __shfl_sync(0xffffffffu, C, q);
    if (t == j) C = cq;
    if (t == q && q != j) C = cj;
  }
  R_[t] = R;
  C_[t] = C;
  for (int e = t; e < 256; e += 32) {
    const int i = e & 15, jj = e >> 4;
    L[e] = (i < kb && jj < kb && i > jj) ? M[(size_t)(k + jj) * lda + k + i] : Sc<S>::zero();
  }
  __syncwarp();
  const int c = blockIdx.x * 32 + t;
  if (c >= n - kb) return;
  const int col = c < k ? c : c + kb;
  S* Ac = M + (size_t)col * lda;
  S x[16], y[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q] = q < kb ? Ac[C_[q]] : Sc<S>::zero();
#pragma unroll
  for (int q = 0; q < 16; ++q)
    if (kb + q < nx) y[q] = Ac[C_[kb + q]];
  const bool solve = col >= k + kb && col < ce;
  if (solve) {
#pragma unroll
    for (int jj = 0; jj < 16; ++jj)
#pragma unroll
      for (int i = jj + 1; i < 16; ++i) x[i] = lu_fnma(L[jj * 16 + i], x[jj], x[i]);
  }
#pragma unroll
  for (int q = 0; q < 16; ++q)
    if (q < kb && (solve || C_[q] != R_[q])) Ac[k + q] = x[q];
#pragma unroll
  for (int q = 0; q < 16; ++q)
    if (kb + q < nx && C_[kb + q] != R_[kb + q]) Ac[R_[kb + q]] = y[q];
}

// ---------------------------------------------------------------------------
// U12 = inv(L11) A12 of a whole outer block (w <= 128 rows from K, columns
// [c0, c1)) in one launch: a CTA holds NC columns in shared memory and walks the
// block in steps of 16 rows: a step's rows are solved (16 lanes per column,
// shuffles), then the threads subtract their multiples from the rows below;
// binary32: each thread CT columns of one row in four (a warp's lanes on
// consecutive rows, so L's column is read without conflict and X's entries are
// broadcasts), 4 + CT shared-memory loads for 4 CT multiply-adds. In place of a TRSM and a GEMM
// launch per 16 or 32 rows, each with a fixed cost (copies, a tile of the SMs
// idle, for the tensor-core paths an operand split). kexp: as in k_trsm_cols.
// ---------------------------------------------------------------------------
template <typename S, int NC>
__global__ void __launch_bounds__(256) k_trsm_block(S* A, long long strideA, int lda, int K, int w, int c0, int c1,
                                                    int* kexp, int kst) {
  constexpr int CT = NC >= 8 ? NC / 8 : 1, CG = NC / CT;  // columns per thread, column groups
  constexpr int RT = 4;                                   // rows per thread (32 apart)
  constexpr bool F64 = sizeof(typename Sc<S>::R) == 8;
  extern __shared__ __align__(16) unsigned char tbraw[];
  S* X = reinterpret_cast<S*>(tbraw);       // [NC][129]
  S* L = X + NC * 129;                      // [16][128 + 1]: the step's columns of L11
  S* M = A + strideA * blockIdx.y;
  const int cb = c0 + blockIdx.x * NC, nc = min(NC, c1 - cb), t = threadIdx.x;
  for (int e = t; e < NC * w; e += 256) {
    const int i = e % w, c = e / w;
    X[c * 129 + i] = c < nc ? M[(size_t)(cb + c) * lda + K + i] : Sc<S>::zero();
  }
  for (int s = 0; s < w; s += 16) {
    const int sb = min(16, w - s), rows = w - s;
    __syncthreads();  // X of the step before, and its reads of L, are done
    for (int e = t; e < 16 * rows; e += 256) {
      const int i = e % rows, c = e / rows;
      L[c * 129 + i] = c < sb ? M[(size_t)(K + s + c) * lda + K + s + i] : Sc<S>::zero();
    }
    __syncthreads();
    // 16 lanes per column, lane = row: one multiply-add per lane and step
    for (int u = t; u < 16 * NC; u += 256) {
      const int i = u & 15, c = u >> 4;
      const bool on = i < sb;
      S x = on ? X[c * 129 + s + i] : Sc<S>::zero();
#pragma unroll
      for (int jj = 0; jj < 15; ++jj) {
        const S l = on ? L[jj * 129 + i] : Sc<S>::zero();
        const S xj = shfl_s(x, (u & 16) | jj);
        if (i > jj) x = lu_fnma(l, xj, x);
      }
      if (on) X[c * 129 + s + i] = x;
    }
    __syncthreads();
    // rows below (none unless sb = 16)
    const int below = rows - sb;
    if constexpr (F64) {
      // binary64: bound by its pipe, so one output per thread and all threads
      for (int e = t; e < below * nc; e += 256) {
        const int i = e % below, c = e / below;
        S v = X[c * 129 + s + sb + i];
#pragma unroll
        for (int jj = 0; jj < 16; ++jj) v = lu_fnma(L[jj * 129 + sb + i], X[c * 129 + s + jj], v);
        X[c * 129 + s + sb + i] = v;
      }
      continue;
    }
    // 32 RT rows at a time
    const int lane = t & 31, wid = t >> 5;
    // warps over (column group, group of 32 RT rows)
    for (int u = wid; u < CG * ((below + 32 * RT - 1) / (32 * RT)); u += 8) {
      const int cg = u % CG, rb = (u / CG) * 32 * RT + lane;
      S v[RT][CT];
#pragma unroll
      for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int c = 0; c < CT; ++c)
          if (rb + 32 * r < below) v[r][c] = X[(cg * CT + c) * 129 + s + sb + rb + 32 * r];
#pragma unroll 4
      for (int jj = 0; jj < 16; ++jj) {
        S xj[CT];
#pragma unroll
        for (int c = 0; c < CT; ++c) xj[c] = X[(cg * CT + c) * 129 + s + jj];
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          if (rb + 32 * r < below) {
            const S l = L[jj * 129 + sb + rb + 32 * r];
#pragma unroll
            for (int c = 0; c < CT; ++c) v[r][c] = lu_fnma(l, xj[c], v[r][c]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int c = 0; c < CT; ++c)
          if (rb + 32 * r < below) X[(cg * CT + c) * 129 + s + sb + rb + 32 * r] = v[r][c];
    }
  }
  __syncthreads();
  for (int e = t; e < nc * w; e += 256) {
    const int i = e % w, c = e / w;
    M[(size_t)(cb + c) * lda + K + i] = X[c * 129 + i];
  }
  if constexpr (std::is_same<S, float2>::value) {
    if (kexp && t < w) {
      int e = 0;
      for (int c = 0; c < nc; ++c) e = max(e, tq_exp(X[c * 129 + t]));
      atomicMax(kexp + (size_t)kst * blockIdx.y + K + t, e);
    }
  }
}

// Apply the panel interchanges (rows k..k+nb-1 with ipiv) to the columns
// outside the panel: one thread per column.
template <typename S>
__global__ void k_laswp(S* A, long long strideA, int lda, int n, int k, int nb, const int* ipiv) {
  const int bidx = blockIdx.y;
  S* M = A + strideA * bidx;
  const int* piv = ipiv + (size_t)n * bidx;
  const int kend = min(k + nb, n);
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  int nout = n - (kend - k);
  if (c >= nout) return;
  int col = c < k ? c : c + (kend - k);
  S* Ac = M + (size_t)col * lda;
  for (int j = k; j < kend; ++j) {
    int p = piv[j] - 1;
    if (p != j) {
      S t = Ac[j];
      Ac[j] = Ac[p];
      Ac[p] = t;
    }
  }
}

// U12 = L11^{-1} A12 (L11 unit lower, nb x nb at (k,k)); one thread per column.
template <typename S>
__global__ void k_trsm_llu(S* A, long long strideA, int lda, int n, int k, int nb) {
  const int bidx = blockIdx.y;
  S* M = A + strideA * bidx;
  const int kend = min(k + nb, n), w = kend - k;
  extern __shared__ unsigned char smraw[];
  S* L = reinterpret_cast<S*>(smraw);  // w x w
  for (int t = threadIdx.x; t < w * w; t += blockDim.x) {
    int i = t % w, jj = t / w;
    L[t] = M[(size_t)(k + jj) * lda + k + i];
  }
  __syncthreads();
  int col = kend + blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= n) return;
  S* Ac = M + (size_t)col * lda + k;
  S x[128];
  for (int i = 0; i < w; ++i) x[i] = Ac[i];
  for (int jj = 0; jj < w; ++jj)
    for (int i = jj + 1; i < w; ++i) x[i] = Sc<S>::sub(x[i], Sc<S>::mul(L[jj * w + i], x[jj]));
  for (int i = 0; i < w; ++i) Ac[i] = x[i];
}

// U12 = L11^{-1} A12 for the columns [c0, c1) (L11 unit lower, w x w at (k,k),
// w <= 32). A CTA of trsm_cols<S>() threads stages a 32-row tile of as many
// columns (coalesced along each column), thread t solves column t in shared
// memory, and the tile is written back. kexp (complex64, else null): [batch][kst]
// by absolute row, raised to the largest exponent in each solved row; the
// operand split of the updates balances its scales with it (mfbem_tc.cuh), and
// a row of U gets its parts by several solves, so the maxima gather over one
// factorisation.
template <typename S> __host__ __device__ constexpr int trsm_cols() { return sizeof(S) > 8 ? 32 : 64; }
template <typename S>
__global__ void __launch_bounds__(trsm_cols<S>()) k_trsm_cols(S* A, long long strideA, int lda, int k, int w, int c0,
                                                              int c1, int* kexp, int kst) {
  constexpr int NC = trsm_cols<S>();
  const int bidx = blockIdx.y;
  S* M = A + strideA * bidx;
  __shared__ S L[32 * 32];
  __shared__ S T[NC * 33];  // [column][row], padded
  const int cb = c0 + blockIdx.x * NC;
  const int ncol = min(NC, c1 - cb);
  for (int t = threadIdx.x; t < w * w; t += NC) {
    const int i = t % w, jj = t / w;
    L[t] = M[(size_t)(k + jj) * lda + k + i];
  }
  // the 32 rows of one column are contiguous
  for (int t = threadIdx.x; t < 32 * ncol; t += NC) {
    const int i = t & 31, c = t >> 5;
    if (i < w) T[c * 33 + i] = M[(size_t)(cb + c) * lda + k + i];
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (c < ncol) {
    S* x = T + c * 33;
    if (w == 32) {
      // full panel width: the column in registers, the substitution unrolled
      // (L read from shared memory as a broadcast, no read-modify-write of x)
      S xr[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) xr[i] = x[i];
#pragma unroll
      for (int jj = 0; jj < 32; ++jj)
#pragma unroll
        for (int i = jj + 1; i < 32; ++i) xr[i] = Sc<S>::sub(xr[i], Sc<S>::mul(L[jj * 32 + i], xr[jj]));
#pragma unroll
      for (int i = 0; i < 32; ++i) x[i] = xr[i];
    } else {
      for (int jj = 0; jj < w; ++jj) {
        const S xj = x[jj];
        for (int i = jj + 1; i < w; ++i) x[i] = Sc<S>::sub(x[i], Sc<S>::mul(L[jj * w + i], xj));
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 32 * ncol; t += NC) {
    const int i = t & 31, cc = t >> 5;
    if (i < w) M[(size_t)(cb + cc) * lda + k + i] = T[cc * 33 + i];
  }
  if constexpr (std::is_same<S, float2>::value) {
    if (kexp && (int)threadIdx.x < w) {
      int e = 0;
      for (int q = 0; q < ncol; ++q) e = max(e, tq_exp(T[q * 33 + threadIdx.x]));
      atomicMax(kexp + (size_t)kst * bidx + k + threadIdx.x, e);
    }
  }
}

// Diagonal block solve of getrs by one warp: the w x w block (w <= 64) staged
// in shared memory, lane l holding rows l and l + 32 of the block; the solved
// component is broadcast by a shuffle, no block-wide barrier per row.
// LOWER: unit lower forward substitution; else upper backward substitution.
// Stage the w x w diagonal block at (r0, r0) into D[col * 65 + row] with 128
// threads, eight loads in flight per thread before their stores (the block is
// usually cold in L2; one load per iteration would serialise on its latency).
template <typename S>
__device__ __forceinline__ void stage_diag64(const S* M, int lda, int r0, int w, S* D) {
  for (int t0 = threadIdx.x; t0 < w * 64; t0 += 128 * 8) {
    S v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = t0 + 128 * u, i = t & 63, j = t >> 6;
      if (t < w * 64 && i < w) v[u] = M[(size_t)(r0 + j) * lda + r0 + i];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = t0 + 128 * u, i = t & 63, j = t >> 6;
      if (t < w * 64 && i < w) D[j * 65 + i] = v[u];
    }
  }
}

template <typename S, bool LOWER>
__global__ void __launch_bounds__(128) k_trsv_diag64(const S* A, long long strideA, int lda, S* b, long long strideb,
                                                     int r0, int w) {
  const int bidx = blockIdx.x;
  const S* M = A + strideA * bidx;
  S* xg = b + strideb * bidx;
  extern __shared__ __align__(16) unsigned char smraw[];
  S* D = reinterpret_cast<S*>(smraw);  // [col][row], w x w, padded to 65 rows
  stage_diag64(M, lda, r0, w, D);
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int l = threadIdx.x;
  S x0 = l < w ? xg[r0 + l] : Sc<S>::zero();
  S x1 = l + 32 < w ? xg[r0 + l + 32] : Sc<S>::zero();
  if (LOWER) {
    for (int j = 0; j < w; ++j) {
      const S xj = shfl_s(j < 32 ? x0 : x1, j & 31);
      if (l > j && l < w) x0 = Sc<S>::sub(x0, Sc<S>::mul(D[j * 65 + l], xj));
      if (l + 32 > j && l + 32 < w) x1 = Sc<S>::sub(x1, Sc<S>::mul(D[j * 65 + l + 32], xj));
    }
  } else {
    for (int j = w - 1; j >= 0; --j) {
      if (j < 32) { if (l == j) x0 = Sc<S>::div(x0, D[j * 65 + j]); }
      else { if (l + 32 == j) x1 = Sc<S>::div(x1, D[j * 65 + j]); }
      const S xj = shfl_s(j < 32 ? x0 : x1, j & 31);
      if (l < j) x0 = Sc<S>::sub(x0, Sc<S>::mul(D[j * 65 + l], xj));
      if (l + 32 < j) x1 = Sc<S>::sub(x1, Sc<S>::mul(D[j * 65 + l + 32], xj));
    }
  }
  if (l < w) xg[r0 + l] = x0;
  if (l + 32 < w) xg[r0 + l + 32] = x1;
}

// ---------------------------------------------------------------------------
// Inner panel without row interchanges (the mixed path's first attempt; its
// factors are only a preconditioner for FP64 refinement, which falls back to
// partial pivoting when it stalls), one launch: every CTA factorises the
// kb x kb diagonal block in shared memory (the same operations in the same
// order, so every copy is bitwise the one written back), takes the
// reciprocals of U11's diagonal, then solves its 128 rows of
// L21 = A21 inv(U11), one thread per row. No cross-CTA pivot search per
// column and no launch between the diagonal block and its rows (a separate
// diagonal kernel cost one dependent launch per 32 columns). The factorised
// block goes back in place only after every CTA has read the original: each
// CTA takes a ticket from cnt[b], and the last one writes and resets the
// counter (zero on entry, zero on exit). The ticket is taken once the factors
// are in shared memory: they are computed from the loaded entries, so all of
// the CTA's loads have returned before the barrier that precedes it (a barrier
// alone does not wait for loads whose registers nothing has read), and fences
// on both sides of the counter order them before the last CTA's stores. The
// counter's round trip is hidden behind the CTA's own rows. A zero or
// non-finite pivot sets info and leaves the block and the rows as they are.
// Grid: (max(1, ceil((r1 - r0) / 128)), batch).
// ---------------------------------------------------------------------------
// The diagonal block sits in registers, warp g holding the columns g + 4 q of
// row = lane: a step takes one reciprocal, one exchange of the column of
// multipliers through shared memory with one barrier, and shuffles of the
// pivot row inside each warp (a copy in shared memory with two barriers and an
// index division per element took twice as long). The rows of L21 update to the
// right, so their multiply-adds are independent. Factorisation before and after,
// together with the deep outer blocks: 58.5 and 53.2 ms at 14883 unknowns; a
// static mixed solve of 870 unknowns 2.55 and 2.34 ms.
__device__ __forceinline__ float diag_rcp(float d) { return 1.0f / d; }
// (as the binary64 piv_rcp: |d|^2 with its rounding errors, each part rounded once)
__device__ __forceinline__ float2 diag_rcp(float2 d) {
  const bool xm = fabsf(d.x) >= fabsf(d.y);
  const float a = xm ? d.x : d.y, b = xm ? d.y : d.x;
  const float aa = a * a, q = fmaf(b, b, aa);
  if (!(q > 1e-30f && q < 1e30f)) return Sc<float2>::rcp(d);
  const float lo = fmaf(b, b, aa - q) + fmaf(a, a, -aa);
  const float y = 1.0f / q, c = y * fmaf(-lo, y, fmaf(-q, y, 1.0f));
  return make_float2(fmaf(d.x, y, d.x * c), -fmaf(d.y, y, d.y * c));
}
template <typename S>
__global__ void __launch_bounds__(128) k_panel_nopiv(S* A, long long sA, int lda, int k, int kb, int r0, int r1,
                                                     int* info, int* cnt) {
  __shared__ S D[32 * 33];
  __shared__ S ur[32];  // reciprocals of U11's diagonal: the row chains multiply, no division
  __shared__ S lc[2][32];  // multipliers of the step's column, by step parity
  __shared__ int s_bad, s_last;
  const int b = blockIdx.y, t = threadIdx.x, lane = t & 31, g = t >> 5;
  S* M = A + sA * b;
  // entries beyond kb: those of the identity
  S v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = g + 4 * q;
    v[q] = lane < kb && c < kb ? M[(size_t)(k + c) * lda + k + lane] : (lane == c ? Sc<S>::one() : Sc<S>::zero());
  }
  if (t == 0) s_bad = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (g == (j & 3)) {
      const S d = shfl_s(v[j >> 2], j);
      const float m = (float)Sc<S>::abs1(d);
      const bool bad = !(m > 0.0f) || !isfinite(m);
      const S rc = diag_rcp(d);
      const S l = Sc<S>::mul(v[j >> 2], rc);
      if (lane > j) v[j >> 2] = l;
      lc[j & 1][lane] = l;
      if (lane == 0) {
        ur[j] = rc;
        if (bad && s_bad == 0) s_bad = j + 1;
      }
    }
    __syncthreads();
    const S l = lc[j & 1][lane];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (4 * q + 3 > j) {
        const S u = shfl_s(v[q], j);
        if (lane > j && g + 4 * q > j) v[q] = lu_fnma(l, u, v[q]);
      }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) D[(g + 4 * q) * 33 + lane] = v[q];
  __syncthreads();
  int ticket = 0;
  if (t == 0) {
    __threadfence();
    ticket = atomicAdd(cnt + b, 1);
  }
  const int row = r0 + blockIdx.x * 128 + t;
  if (!s_bad && row < r1) {
    S x[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = j < kb ? M[(size_t)(k + j) * lda + row] : Sc<S>::zero();
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      x[j] = Sc<S>::mul(x[j], ur[j]);
#pragma unroll
      for (int c = j + 1; c < 32; ++c) x[c] = lu_fnma(x[j], D[c * 33 + j], x[c]);
    }
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < kb) M[(size_t)(k + j) * lda + row] = x[j];
  }
  if (t == 0) {
    s_last = ticket == (int)gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  // a zero or non-finite pivot at column s_bad - 1: nothing is written back
  if (s_last) {
    if (s_bad) {
      if (t == 0 && info[b] == 0) info[b] = k + s_bad;
    } else {
      for (int e = t; e < 1024; e += 128) {
        const int i = e & 31, c = e >> 5;
        if (i < kb && c < kb) M[(size_t)(k + c) * lda + k + i] = D[c * 33 + i];
      }
    }
    if (t == 0) cnt[b] = 0;
  }
}

// ---------------------------------------------------------------------------
// Triangular solve of getrs in one launch per triangle (no counterpart in the
// reference, which calls ?getrs): the rows are cut in blocks of 64; a CTA takes
// work items (system, block) in solve order from a global counter, adds the
// contributions of the blocks already solved as their ready flags appear
// (L or U read once, 64 contiguous entries per column), solves its 64 x 64
// diagonal block in one warp (shuffles) and publishes x and its flag. Items are
// claimed in dependency order, so every block an item waits for is held by a
// CTA that is already running: no co-residency is needed. Waits on flags are
// bounded; a wait that gives up sets *err and the CTA publishes its block
// anyway, so every other wait ends too.
// OP: unit lower L (forward), U (backward), or the conjugate-transposed factors
// U^H (forward) and L^H (backward) of getrs 'C' and the norm estimates, read
// with the roles of rows and columns exchanged (a thread's loads of a tile then
// touch one column each; they are prefetched before the wait).
// ready[b * nb + blk] must be 0 and *counter 0 on entry. Dynamic shared
// memory: trsv_sf_smem<S>() bytes.
// ---------------------------------------------------------------------------
enum TrOp { TR_L = 0, TR_U = 1, TR_UH = 2, TR_LH = 3 };
constexpr long long kTrsvSpin = 1LL << 22;
template <typename S>
constexpr size_t trsv_sf_smem() {
  return sizeof(S) * (64 * 65 + 4 * 64 + 64 + 64);
}
__device__ __forceinline__ int ld_acquire_s32(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Loads of the factors issued where they stand in the program: the
// prefetch of the next solved block's tile must leave before the wait on
// that block's flag (a plain load may be scheduled next to its first use,
// behind the wait). The factors are read-only during the solve.
__device__ __forceinline__ float ld_pinned(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_pinned(const double* p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 ld_pinned(const float2* p) {
  float2 v;
  asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_pinned(const double2* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
template <typename S, int OP>
__global__ void __launch_bounds__(256) k_trsv_sf(const S* A, long long sA, int lda, int n, S* x, long long sx,
                                                 int batch, int nb, unsigned* counter, int* ready, int* err,
                                                 long long spin) {
  // dynamic shared memory: D [64 x 65] (diagonal block, column-major), part [4][64],
  // xs [64] (the solved block being applied), rinv [64] (reciprocals of U's
  // diagonal, formed before the wait so that no division lies on the chain)
  extern __shared__ __align__(16) unsigned char sfraw[];
  constexpr bool FWD = OP == TR_L || OP == TR_UH;    // order of the blocks
  constexpr bool UNIT = OP == TR_L || OP == TR_LH;   // unit diagonal
  constexpr bool CT = OP == TR_UH || OP == TR_LH;    // conjugate-transposed factor
  S* D = reinterpret_cast<S*>(sfraw);
  S (*part)[64] = reinterpret_cast<S (*)[64]>(D + 64 * 65);
  S* xs = D + 64 * 65 + 4 * 64;
  S* rinv = xs + 64;
  __shared__ int s_item, s_end;
  const int t = threadIdx.x, row = t & 63, grp = t >> 6;
  const long long lim = spin > 0 ? spin : kTrsvSpin;
  for (;;) {
    if (t == 0) s_item = (int)atomicAdd(counter, 1u);
    __syncthreads();
    const int item = s_item;
    if (item >= nb * batch) break;
    const int b = item % batch, q = item / batch;
    const int blk = FWD ? q : nb - 1 - q;
    const int r0 = blk * 64, w = min(64, n - r0);
    const S* M = A + sA * b;
    S* xb = x + sx * b;
    // this thread's 16 entries (row, columns grp + 4i) of the next solved
    // block's tile: loaded before that block is published (the factors do not
    // depend on it), so applying a newly solved block costs one load of its
    // 64 values and 16 FMAs
    S mreg[16];
    auto load_tile = [&](int qq) {
      const int jb = FWD ? qq : nb - 1 - qq;
      const int c0 = jb * 64, wc = min(64, n - c0);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int c = grp + 4 * i;
        if (CT) mreg[i] = (row < w && c < wc) ? Sc<S>::conj(ld_pinned(M + (size_t)(r0 + row) * lda + c0 + c)) : Sc<S>::zero();
        else mreg[i] = (row < w && c < wc) ? ld_pinned(M + (size_t)(c0 + c) * lda + r0 + row) : Sc<S>::zero();
      }
    };
    if (q > 0) load_tile(0);
    // diagonal block into shared memory (used after the contributions),
    // transposed and conjugated for CT; without a unit diagonal its rows scaled
    // by the reciprocals of the diagonal, so that the substitution chain below
    // carries no multiplication by them
    if (!UNIT) {
      if (t < w) {
        const S d = M[(size_t)(r0 + t) * lda + r0 + t];
        rinv[t] = Sc<S>::rcp(CT ? Sc<S>::conj(d) : d);
      }
      __syncthreads();
    }
    for (int e = t; e < 64 * 64; e += 256) {
      const int i = e & 63, j = e >> 6;
      if (i < w && j < w) {
        // e & 63 runs along a column of the factor either way
        const S v = M[(size_t)(r0 + j) * lda + r0 + i];
        if (CT) D[i * 65 + j] = UNIT ? Sc<S>::conj(v) : Sc<S>::mul(Sc<S>::conj(v), rinv[j]);
        else D[j * 65 + i] = UNIT ? v : Sc<S>::mul(v, rinv[i]);
      }
    }
    // contributions of the solved blocks, in the order they were solved:
    // thread 0 waits for the next one, then takes every later one already
    // published too, so a CTA that is behind catches up with one barrier
    S acc = Sc<S>::zero();
    for (int done = 0; done < q;) {
      if (t == 0) {
        long long it = 0;
        const int jb0 = FWD ? done : nb - 1 - done;
        while (ld_acquire_s32(ready + (size_t)b * nb + jb0) == 0) {
          if (++it > lim) {
            atomicExch(err, 1);
            break;
          }
          if (it > 64) __nanosleep(64);
        }
        int e = done + 1;
        while (e < q && ld_acquire_s32(ready + (size_t)b * nb + (FWD ? e : nb - 1 - e)) != 0) ++e;
        s_end = e;
      }
      __syncthreads();
      const int end = s_end;
      for (int qq = done; qq < end; ++qq) {
        const int jb = FWD ? qq : nb - 1 - qq;
        const int c0 = jb * 64, wc = min(64, n - c0);
        if (t < 64) xs[t] = t < wc ? __ldcg(xb + c0 + t) : Sc<S>::zero();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc = lu_fnma(mreg[i], xs[grp + 4 * i], acc);
        __syncthreads();
        if (qq + 1 < q) load_tile(qq + 1);
      }
      done = end;
    }
    part[grp][row] = acc;
    __syncthreads();
    if (t < 32) {
      const int l = t;
      S x0 = Sc<S>::zero(), x1 = Sc<S>::zero();
      if (l < w) x0 = Sc<S>::add(xb[r0 + l], Sc<S>::add(Sc<S>::add(part[0][l], part[1][l]), Sc<S>::add(part[2][l], part[3][l])));
      if (l + 32 < w)
        x1 = Sc<S>::add(xb[r0 + l + 32], Sc<S>::add(Sc<S>::add(part[0][l + 32], part[1][l + 32]),
                                                    Sc<S>::add(part[2][l + 32], part[3][l + 32])));
      if (!UNIT) {
        // rows pre-scaled: x_l = y_l / d_l - sum_j (d_lj / d_l) x_j
        if (l < w) x0 = Sc<S>::mul(x0, rinv[l]);
        if (l + 32 < w) x1 = Sc<S>::mul(x1, rinv[l + 32]);
      }
      if (FWD) {
        for (int j = 0; j < w; ++j) {
          const S xj = shfl_s(j < 32 ? x0 : x1, j & 31);
          if (l > j && l < w) x0 = lu_fnma(D[j * 65 + l], xj, x0);
          if (l + 32 > j && l + 32 < w) x1 = lu_fnma(D[j * 65 + l + 32], xj, x1);
        }
      } else {
        for (int j = w - 1; j >= 0; --j) {
          const S xj = shfl_s(j < 32 ? x0 : x1, j & 31);
          if (l < j) x0 = lu_fnma(D[j * 65 + l], xj, x0);
          if (l + 32 < j) x1 = lu_fnma(D[j * 65 + l + 32], xj, x1);
        }
      }
      if (l < w) xb[r0 + l] = x0;
      if (l + 32 < w) xb[r0 + l + 32] = x1;
      __threadfence();
      __syncwarp();
      if (l == 0) atomicExch(ready + (size_t)b * nb + blk, 1);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// getrs (no transpose) for one right-hand side per matrix, blocked by TB rows:
//   k_rhs_swap:     apply all interchanges to b (sequential, one thread per matrix)
//   k_trsv_diag:    solve the TB x TB diagonal block (one CTA per matrix)
//   k_trsv_update:  b[rest] -= A[rest, blk] x[blk] (GEMV, many CTAs)
// ---------------------------------------------------------------------------
template <typename S>
__global__ void k_rhs_swap(S* b, long long strideb, int n, const int* ipiv, int nbatch) {
  int bidx = blockIdx.x * blockDim.x + threadIdx.x;
  if (bidx >= nbatch) return;
  S* x = b + strideb * bidx;
  const int* piv = ipiv + (size_t)n * bidx;
  for (int j = 0; j < n; ++j) {
    int p = piv[j] - 1;
    if (p != j) {
      S t = x[j];
      x[j] = x[p];
      x[p] = t;
    }
  }
}
// lower (unit) forward / upper backward solve of the diagonal block [r0, r0+w)
template <typename S, bool LOWER>
__global__ void k_trsv_diag(const S* A, long long strideA, int lda, S* b, long long strideb, int r0, int w) {
  const int bidx = blockIdx.x;
  const S* M = A + strideA * bidx;
  S* x = b + strideb * bidx;
  __shared__ S xs[256];
  if ((int)threadIdx.x < w) xs[threadIdx.x] = x[r0 + threadIdx.x];
  __syncthreads();
  if (LOWER) {
    for (int j = 0; j < w; ++j) {
      S xj = xs[j];
      int i = threadIdx.x;
      if (i > j && i < w) xs[i] = Sc<S>::sub(xs[i], Sc<S>::mul(M[(size_t)(r0 + j) * lda + r0 + i], xj));
      __syncthreads();
    }
  } else {
    for (int j = w - 1; j >= 0; --j) {
      if (threadIdx.x == 0) xs[j] = Sc<S>::div(xs[j], M[(size_t)(r0 + j) * lda + r0 + j]);
      __syncthreads();
      S xj = xs[j];
      int i = threadIdx.x;
      if (i < j) xs[i] = Sc<S>::sub(xs[i], Sc<S>::mul(M[(size_t)(r0 + j) * lda + r0 + i], xj));
      __syncthreads();
    }
  }
  if ((int)threadIdx.x < w) x[r0 + threadIdx.x] = xs[threadIdx.x];
}
// rows [i0, i1) -= A[rows, r0:r0+w] x[r0:r0+w]
template <typename S>
__global__ void k_trsv_update(const S* A, long long strideA, int lda, S* b, long long strideb, int r0, int w, int i0,
                              int i1) {
  const int bidx = blockIdx.y;
  const S* M = A + strideA * bidx;
  S* x = b + strideb * bidx;
  __shared__ S xs[256];
  if ((int)threadIdx.x < w) xs[threadIdx.x] = x[r0 + threadIdx.x];
  __syncthreads();
  int i = i0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= i1) return;
  S acc = Sc<S>::zero();
#pragma unroll 8
  for (int j = 0; j < w; ++j) acc = Sc<S>::add(acc, Sc<S>::mul(M[(size_t)(r0 + j) * lda + i], xs[j]));
  x[i] = Sc<S>::sub(x[i], acc);
}

}  // namespace mfb
