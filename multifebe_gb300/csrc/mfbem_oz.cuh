// FP64-accurate GEMM update C -= A B on the bf16 tensor cores (tcgen05,
// kind::f16), for the trailing updates of the plain FP64 LU (the drop-in
// zgetrf / dgetrf of solve_lse_c / solve_lse_r). GB300 runs binary64 FMA at
// 1/64 of its FP32 rate; the update is instead computed exactly in integer
// pieces on the tensor cores and recombined in binary64 (the Ozaki scheme:
// Ozaki, Ogita, Oishi, "Error-free transformations of matrix multiplication
// by using fast routines of matrix multiplication", Numer. Algorithms 2012;
// on tensor cores: Mukunoki, Ozaki, Ogita, Imamura, ICCS 2020).
// Included into mfbem_abi.cu.
//
// Splitting. Row r of A (real view, m' rows) gets a power-of-two scale 2^e_r
// with |a_rk| < 2^(e_r - 1); column j of B gets 2^f_j likewise. The integer
// X = a_rk 2^(55 - e_r) (|X| < 2^54, the row's largest entries exactly, the
// others rounded at 2^-55 of the row scale) is written with seven signed
// digits, X = sum_p d_p 2^(48 - 8p), |d_0| <= 64, |d_p| <= 128, and slice p is
// stored as the bf16 value d_p 2^(-8p) (exact). Then
//     a_rk b_kj = 2^(e_r + f_j - 14) sum_{p,q} slice_p(a) slice_q(b).
// Products with p + q >= 7 are dropped (below 2^-56 of the scales). For
// t = p + q <= 4 every product is an integer multiple of 2^(-8t) and the sum
// over a K of at most 256 stays within 2^24 units, so an FP32 accumulator per
// level t holds it exactly; levels 5..6 (13 products, 2^-40 and smaller) share
// a sixth accumulator, whose FP32 accumulation (rounded or truncated by the
// tensor core) stays near 2^-53 of the result. The epilogue rebuilds the
// exact integer sum of levels 0..4 in int64 (below 2^53 in units of 2^-32),
// converts it to binary64, adds the tail with one FMA that applies the scale
// 2^(e_r + f_j - 14) too, and subtracts the result from C by a reduction at the
// L2: two binary64 operations per output (at two lanes per cycle and SM) and no
// wait for C. The scaled tail is put together from the bits of the FP32 one; the
// FMA rounds sum + tail once, as the scale is a power of two.
//
// Complex: C~ (2m x n real) -= A~ (2m x 2k) B~ (2k x n) with A~ realified in
// 2 x 2 blocks [[re, -im], [im, re]] and B~, C~ the complex arrays viewed as
// real (as in the TF32 kernel of mfbem_tc.cuh).
//
// Kernels: k_oz_split (row tiles of A, column tiles of B) computes the scales and writes the slices
// pre-tiled in the canonical K-major no-swizzle UMMA layout (8-row x 16-byte
// core matrices), all seven slices of a (tile, K chunk) contiguous, so the
// GEMM streams one bulk copy of A slices and one of B slices per chunk into a
// two-stage pipeline; one thread issues 28 tcgen05.mma (M 128, N 80, K 16)
// per K step into six TMEM accumulators (480 columns); four warps run the
// binary64 epilogue. Every wait is bounded (error flag, drain, TMEM freed).
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

namespace mfb {

constexpr int OZ_BM = 128;                    // real rows of C~ per CTA
constexpr int OZ_BN = 80;                     // columns per CTA
constexpr int OZ_KC = 32;                     // real K per chunk (bf16 elements)
constexpr int OZ_S = 7;                       // slices per operand
constexpr int OZ_NACC = 6;                    // TMEM accumulators: levels 0..4 exact, 5..6 tail
constexpr int OZ_WPR = OZ_KC / 2;             // 32-bit words per tile row per chunk (16)
constexpr int OZ_TWA = OZ_BM * OZ_WPR;        // words of one A slice tile (2048 = 8 KB)
constexpr int OZ_TWB = OZ_BN * OZ_WPR;        // words of one B slice tile (1280 = 5 KB)
constexpr int OZ_STAGE_A = OZ_S * OZ_TWA * 4; // bytes of a stage's A slices (56 KB)
constexpr int OZ_STAGE_B = OZ_S * OZ_TWB * 4; // bytes of a stage's B slices (35 KB)
constexpr int OZ_STAGE = OZ_STAGE_A + OZ_STAGE_B;
constexpr int OZ_SMEM = 2 * OZ_STAGE + 64 + OZ_BN * 4;
constexpr int OZ_SBO = OZ_WPR / 4 * 128;      // bytes between 8-row groups (512)
constexpr int OZ_MAXK = 256;                  // real K of one update (exactness bound)

// word w of a tile (OZ_WPR words per row) <-> (row, word column): core matrix
// w / 32 (OZ_WPR / 4 of them along K per 8-row group), row (w % 32) / 4
// inside it, word w % 4 of the row's 16 bytes
__host__ __device__ __forceinline__ void oz_rw(int w, int& r, int& kw) {
  const int cm = w >> 5;
  r = (cm / (OZ_WPR / 4)) * 8 + ((w & 31) >> 2);
  kw = (cm % (OZ_WPR / 4)) * 4 + (w & 3);
}

// e such that max |v| < 2^(e - 1) for max |v| = mx (0 for mx = 0)
__device__ __forceinline__ int oz_scale_exp(double mx) { return mx > 0.0 ? ilogb(mx) + 2 : 0; }

// the seven signed digits of v 2^(55 - e) (|v| < 2^(e - 1))
__device__ __forceinline__ void oz_digits(double v, int e, int d[OZ_S]) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const int be = (int)((u >> 52) & 0x7FF);
  long long mt = (long long)(u & 0xFFFFFFFFFFFFFULL);
  int E = -1022;
  if (be) {
    mt |= 1LL << 52;
    E = be - 1023;
  }
  const int sh = E - e + 3;  // X = mt 2^sh, sh <= 1
  long long X;
  if (mt == 0) X = 0;
  else if (sh >= 0) X = mt << sh;
  else if (sh > -63) X = (mt + (1LL << (-sh - 1))) >> (-sh);
  else X = 0;
  if (u >> 63) X = -X;
  long long R = X;
#pragma unroll
  for (int p = 0; p < OZ_S - 1; ++p) {
    const int s = 48 - 8 * p;
    const long long dp = (R + (1LL << (s - 1))) >> s;
    d[p] = (int)dp;
    R -= dp << s;
  }
  d[OZ_S - 1] = (int)R;
}

// 2^s, a normal number
__device__ __forceinline__ double oz_pow2(int s) { return __hiloint2double((s + 1023) << 20, 0); }
// v 2^s where 2^s need not be a number (|s| beyond 2040: zero or infinity):
// two factors, so that the one rounding is that of a subnormal result
__device__ __forceinline__ double oz_scale2(double v, int s) {
  s = s < -2040 ? -2040 : (s > 2040 ? 2040 : s);
  const int h = s >> 1;
  return v * oz_pow2(h) * oz_pow2(s - h);
}

// bf16 pair (lo: d0 2^(-8p), hi: d1 2^(-8p)) as one word
__device__ __forceinline__ uint32_t oz_pack(int d0, int d1, int p) {
  const float sc = __int_as_float((127 - 8 * p) << 23);  // 2^(-8p)
  const __nv_bfloat16 a = __float2bfloat16_rn((float)d0 * sc), b = __float2bfloat16_rn((float)d1 * sc);
  return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}

template <bool CPLX> struct OzT;
template <> struct OzT<true> { typedef double2 S; };
template <> struct OzT<false> { typedef double S; };

__device__ __forceinline__ double oz_absmax(double2 v) { return fmax(fabs(v.x), fabs(v.y)); }
__device__ __forceinline__ double oz_absmax(double v) { return fabs(v); }

// A slices. Real view: m' = 2m (complex) or m rows, K = 2k or k. One CTA
// (256 threads) per (row tile, batch): row scales over the whole K, then the
// slices of every K chunk. Output: tiles [batch][mt][kc][slice][word],
// exponents erow[batch][nmt * OZ_BM].
template <bool CPLX>
__device__ __forceinline__ void oz_split_a_tile(const typename OzT<CPLX>::S* A, int lda, long long sA, int m, int k,
                                                int nmt, int nkc, uint32_t* tiles, int* erow, int mt, int b) {
  typedef typename OzT<CPLX>::S S;
  __shared__ double smax[4][OZ_BM];
  __shared__ int se[OZ_BM];
  const int t = threadIdx.x;
  const S* Ab = A + sA * b;
  // rows of the source matrix in this tile: 64 complex or 128 real
  constexpr int RS = CPLX ? OZ_BM / 2 : OZ_BM;
  const int i0 = mt * RS;
  {
    const int il = t % RS, part = t / RS, nparts = 256 / RS;
    const int i = i0 + il;
    double mx = 0.0;
    if (i < m)
      for (int l = part; l < k; l += nparts) mx = fmax(mx, oz_absmax(Ab[(size_t)l * lda + i]));
    smax[part][il] = mx;
  }
  __syncthreads();
  if (t < RS) {
    double mx = smax[0][t];
    for (int q = 1; q < 256 / RS; ++q) mx = fmax(mx, smax[q][t]);
    const int e = oz_scale_exp(mx);
    if (CPLX) {
      se[2 * t] = e;
      se[2 * t + 1] = e;
    } else {
      se[t] = e;
    }
  }
  __syncthreads();
  if (t < OZ_BM) erow[(size_t)b * nmt * OZ_BM + (size_t)mt * OZ_BM + t] = se[t];
  const int Kr = CPLX ? 2 * k : k;  // real K
  for (int kc = 0; kc < nkc; ++kc) {
    uint32_t* dst = tiles + (((size_t)b * nmt + mt) * nkc + kc) * (OZ_S * OZ_TWA);
    for (int w = t; w < OZ_TWA; w += 256) {
      int r, kw;
      oz_rw(w, r, kw);
      const int kk = kc * OZ_KC + 2 * kw;  // real K of the word's low half
      int d0[OZ_S], d1[OZ_S];
      if (CPLX) {
        const int i = i0 + (r >> 1), l = kk >> 1;
        double2 a = make_double2(0.0, 0.0);
        if (i < m && l < k) a = reinterpret_cast<const double2*>(Ab)[(size_t)l * lda + i];
        // row 2i: (re, -im); row 2i+1: (im, re)
        if (r & 1) {
          oz_digits(a.y, se[r], d0);
          oz_digits(a.x, se[r], d1);
        } else {
          oz_digits(a.x, se[r], d0);
          oz_digits(a.y, se[r], d1);
#pragma unroll
          for (int p = 0; p < OZ_S; ++p) d1[p] = -d1[p];
        }
      } else {
        const int i = i0 + r;
        double a0 = 0.0, a1 = 0.0;
        if (i < m && kk < Kr) a0 = reinterpret_cast<const double*>(Ab)[(size_t)kk * lda + i];
        if (i < m && kk + 1 < Kr) a1 = reinterpret_cast<const double*>(Ab)[(size_t)(kk + 1) * lda + i];
        oz_digits(a0, se[r], d0);
        oz_digits(a1, se[r], d1);
      }
#pragma unroll
      for (int p = 0; p < OZ_S; ++p) dst[(size_t)p * OZ_TWA + w] = oz_pack(d0[p], d1[p], p);
    }
  }
}

// B slices: tile rows are the columns j of B (OZ_BN per tile), K along the
// rows of B. One CTA (256 threads) per (column tile, batch). Output: tiles
// [batch][nt][kc][slice][word], exponents fcol[batch][nnt * OZ_BN].
template <bool CPLX>
__device__ __forceinline__ void oz_split_b_tile(const typename OzT<CPLX>::S* B, int ldb, long long sB, int k, int n,
                                                int nnt, int nkc, uint32_t* tiles, int* fcol, int nt, int b) {
  typedef typename OzT<CPLX>::S S;
  __shared__ int sf[OZ_BN];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const S* Bb = B + sB * b;
  const int j0 = nt * OZ_BN;
  // column scales: a warp per column, lanes along K
  for (int c = wid; c < OZ_BN; c += 8) {
    const int j = j0 + c;
    double mx = 0.0;
    if (j < n)
      for (int l = lane; l < k; l += 32) mx = fmax(mx, oz_absmax(Bb[(size_t)j * ldb + l]));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) sf[c] = oz_scale_exp(mx);
  }
  __syncthreads();
  if (t < OZ_BN) fcol[(size_t)b * nnt * OZ_BN + (size_t)nt * OZ_BN + t] = sf[t];
  const int Kr = CPLX ? 2 * k : k;
  for (int kc = 0; kc < nkc; ++kc) {
    uint32_t* dst = tiles + (((size_t)b * nnt + nt) * nkc + kc) * (OZ_S * OZ_TWB);
    for (int w = t; w < OZ_TWB; w += 256) {
      int c, kw;
      oz_rw(w, c, kw);
      const int j = j0 + c, kk = kc * OZ_KC + 2 * kw;
      int d0[OZ_S], d1[OZ_S];
      if (CPLX) {
        const int l = kk >> 1;
        double2 v = make_double2(0.0, 0.0);
        if (j < n && l < k) v = reinterpret_cast<const double2*>(Bb)[(size_t)j * ldb + l];
        oz_digits(v.x, sf[c], d0);
        oz_digits(v.y, sf[c], d1);
      } else {
        double v0 = 0.0, v1 = 0.0;
        if (j < n && kk < Kr) v0 = reinterpret_cast<const double*>(Bb)[(size_t)j * ldb + kk];
        if (j < n && kk + 1 < Kr) v1 = reinterpret_cast<const double*>(Bb)[(size_t)j * ldb + kk + 1];
        oz_digits(v0, sf[c], d0);
        oz_digits(v1, sf[c], d1);
      }
#pragma unroll
      for (int p = 0; p < OZ_S; ++p) dst[(size_t)p * OZ_TWB + w] = oz_pack(d0[p], d1[p], p);
    }
  }
}

// Both operands' slices in one launch: blocks [0, nmt) split row tiles of A,
// blocks [nmt, nmt + nnt) column tiles of B (blockIdx.y: the matrix).
template <bool CPLX>
__global__ void __launch_bounds__(256) k_oz_split(const typename OzT<CPLX>::S* A, int lda, long long sA, int m,
                                                  const typename OzT<CPLX>::S* B, int ldb, long long sB, int n, int k,
                                                  int nmt, int nnt, int nkc, uint32_t* at, int* erow, uint32_t* bt,
                                                  int* fcol) {
  if ((int)blockIdx.x < nmt) oz_split_a_tile<CPLX>(A, lda, sA, m, k, nmt, nkc, at, erow, blockIdx.x, blockIdx.y);
  else oz_split_b_tile<CPLX>(B, ldb, sB, k, n, nnt, nkc, bt, fcol, blockIdx.x - nmt, blockIdx.y);
}

__device__ __forceinline__ uint64_t oz_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(128 >> 4) << 16;
  d |= (uint64_t)(OZ_SBO >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}
// instruction descriptor, kind::f16: D f32, A and B bf16, both K-major, N, M
__host__ __device__ constexpr uint32_t oz_idesc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void oz_ld16(uint32_t ta, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(ta)
      : "memory");
}

// C~ (real view: m' rows, n columns, ld ldc, batch stride sC, in doubles) -=
// A~ B~ from the slice tiles; CTA (row tile, column tile, batch).
__global__ void __launch_bounds__(128, 1) k_oz_gemm(const uint32_t* At, const uint32_t* Bt, const int* erow,
                                                    const int* fcol, int nmt, int nnt, int nkc, double* C,
                                                    long long ldc, long long sC, int mr, int n, int* err,
                                                    long long spin) {
  extern __shared__ __align__(1024) unsigned char osm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(osm + 2 * OZ_STAGE);  // fb[2], mb[2]
  uint32_t* tslot = reinterpret_cast<uint32_t*>(osm + 2 * OZ_STAGE + 32);
  int* sfc = reinterpret_cast<int*>(osm + 2 * OZ_STAGE + 64);
  __shared__ int s_ok;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int mt = blockIdx.x, nt = blockIdx.y, bz = blockIdx.z;
  const uint32_t* ta0 = At + ((size_t)bz * nmt + mt) * nkc * (OZ_S * OZ_TWA);
  const uint32_t* tb0 = Bt + ((size_t)bz * nnt + nt) * nkc * (OZ_S * OZ_TWB);
  const uint32_t fb[2] = {smem_u32(bars), smem_u32(bars + 1)}, mb[2] = {smem_u32(bars + 2), smem_u32(bars + 3)};
  const uint32_t st0 = smem_u32(osm);
  if (t == 0) {
    for (int q = 0; q < 2; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(fb[q]) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb[q]) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_ok = 1;
  }
  if (t < OZ_BN) sfc[t] = fcol[(size_t)bz * nnt * OZ_BN + (size_t)nt * OZ_BN + t];
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  constexpr uint32_t idesc = oz_idesc(OZ_BM, OZ_BN);
  int issued = 0, loaded = 0, landed = 0;
  if (t == 0) {
    auto load = [&](int kc, int sidx) {
      const uint32_t d = st0 + sidx * OZ_STAGE;
      tc_expect(fb[sidx], (uint32_t)OZ_STAGE);
      tc_bulk(d, ta0 + (size_t)kc * (OZ_S * OZ_TWA), OZ_STAGE_A, fb[sidx]);
      tc_bulk(d + OZ_STAGE_A, tb0 + (size_t)kc * (OZ_S * OZ_TWB), OZ_STAGE_B, fb[sidx]);
      loaded = kc + 1;
    };
    bool ok = true;
    if (nkc > 0) load(0, 0);
    for (int kc = 0; kc < nkc && ok; ++kc) {
      const int s = kc & 1;
      if (kc + 1 < nkc) {
        // stage s^1 was read by the MMAs of chunk kc - 1
        if (kc >= 1 && !tc_wait(mb[s ^ 1], (uint32_t)(((kc - 1) >> 1) & 1), spin)) { ok = false; break; }
        load(kc + 1, s ^ 1);
      }
      if (!tc_wait(fb[s], (uint32_t)((kc >> 1) & 1), spin)) { ok = false; break; }
      landed = kc + 1;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sa = st0 + s * OZ_STAGE, sb = sa + OZ_STAGE_A;
#pragma unroll
      for (int ks = 0; ks < OZ_KC / 16; ++ks) {
#pragma unroll
        for (int p = 0; p < OZ_S; ++p) {
          const uint64_t da = oz_desc(sa + p * (OZ_TWA * 4) + ks * 256);
#pragma unroll
          for (int q = 0; q + p < OZ_S; ++q) {
            const int lev = p + q;
            const int acc = lev < OZ_NACC - 1 ? lev : OZ_NACC - 1;
            const bool first = kc == 0 && ks == 0 && p == 0 && (lev < OZ_NACC - 1 || q == OZ_NACC - 1);
            const uint64_t db = oz_desc(sb + q * (OZ_TWB * 4) + ks * 256);
            const uint32_t dt = tmem + (uint32_t)(acc * OZ_BN);
            asm volatile(
                "{\n .reg .pred pa;\n setp.ne.u32 pa, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, pa;\n}\n" ::"r"(
                    dt),
                "l"(da), "l"(db), "r"(idesc), "r"(first ? 0u : 1u)
                : "memory");
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mb[s])
                   : "memory");
      issued = kc + 1;
    }
    // the last commit covers every earlier MMA
    if (ok && issued > 0 && !tc_wait(mb[(issued - 1) & 1], (uint32_t)(((issued - 1) >> 1) & 1), spin)) ok = false;
    if (!ok) {
      atomicExch(err, 1);
      s_ok = 0;
      // drain (full limit): the MMAs issued so far, then the copies not yet waited for
      if (issued > 0) tc_wait(mb[(issued - 1) & 1], (uint32_t)(((issued - 1) >> 1) & 1));
      for (int c = landed; c < loaded; ++c) tc_wait(fb[c & 1], (uint32_t)((c >> 1) & 1));
    }
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (s_ok && nkc > 0) {
    const int r = 32 * warp + lane;
    const int row = mt * OZ_BM + r;
    const bool live = row < mr;
    const int er = live ? erow[(size_t)bz * nmt * OZ_BM + row] : 0;
    double* Cb = C + sC * bz;
    for (int c0 = 0; c0 < OZ_BN; c0 += 16) {
      uint32_t v[OZ_NACC][16];
      const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c0;
#pragma unroll
      for (int a = 0; a < OZ_NACC; ++a) oz_ld16(ta + (uint32_t)(a * OZ_BN), v[a]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (live) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          // exact integer sum of levels 0..4 in units of 2^-32 (|V| < 2^53)
          const long long i0 = (long long)__float2int_rn(__uint_as_float(v[0][q]));
          const long long i1 = (long long)__float2int_rn(__uint_as_float(v[1][q]) * 0x1p8f);
          const long long i2 = (long long)__float2int_rn(__uint_as_float(v[2][q]) * 0x1p16f);
          const long long i3 = (long long)__float2int_rn(__uint_as_float(v[3][q]) * 0x1p24f);
          const long long i4 = (long long)__float2int_rn(__uint_as_float(v[4][q]) * 0x1p32f);
          const long long V = (i0 << 32) + (i1 << 24) + (i2 << 16) + (i3 << 8) + i4;
          const int s = er + sfc[c0 + q] - 14;
          double r;
          if (s >= -960 && s <= 1000) {
            // the tail is a multiple of 2^-48 (its products are) or zero
            const uint32_t te = (v[5][q] >> 23) & 255;
            const int hi = (int)((v[5][q] & 0x80000000u) | ((te + (uint32_t)(s + 896)) << 20) | ((v[5][q] >> 3) & 0xFFFFFu));
            r = fma((double)V, oz_pow2(s - 32), te ? __hiloint2double(hi, (int)(v[5][q] << 29)) : 0.0);
          } else {  // operands near the ends of the exponent range
            r = oz_scale2(fma((double)V, 0x1p-32, (double)__uint_as_float(v[5][q])), s);
          }
          const int j = nt * OZ_BN + c0 + q;
          // a reduction at the L2: no wait for C; one addition per entry and update
          if (j < n) atomicAdd(Cb + (size_t)j * ldc + row, -r);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

}  // namespace mfb
