// Internal points: calculate_internal_points_mechanics_bem_{staela,harela}
// (src/calculate_internal_points_mechanics_static.f90:188-502,
// src/calculate_internal_points_mechanics_bem_harela.f90:22-505), the step
// after the solve. Displacement and stress tensor at points inside the region
// from the nodal solution, for ordinary BE boundaries without symmetry planes,
// body loads or incident field:
//   u_il        = sum_e sum_kn g(kn,il,ik) t_ik - h(kn,il,ik) u_ik      (sbie_auto)
//   sigma_il,kc = sum_e sum_kn l(kn,il,ik) t_ik - m(kn,il,ik) u_ik      (hbie_auto, n_i = e_kc)
// with the HBIE kernels d* (l) and s* (m) of bem_staela3d.f90:4376-4446 and
// bem_harela3d.f90:2573-2662, classified like sbie_auto with the 1/r^7
// quasi-singular estimate. A point at a boundary node (distance / csize of the
// node's first element < 1e-12) takes the node's displacement and zero
// stresses (calculate_internal_points_mechanics_bem_harela.f90:190-208).
//
// Layout of the work: the shape-function weights of every quadrature point are
// contracted with the element's nodal values first (t_w = sum_kn phi_kn J w t_kn,
// the same for u), so no 8x3x3 kernel block is formed; for the precalculated
// rules that is done once per call and dataset point (k_ip_weights), since it
// does not depend on the internal point. Kernel and nodal vectors are
// contracted before the tensors are formed: sigma is symmetric, and with
// a = dr.T, b = dr.U, w = n.U, d = dr/dn its six components take about 150
// multiply-adds a point instead of the 1350 of 3 x 9 components of d* and s*.
// One warp per (point, frequency, 32 elements) spreads the quadrature points of
// its elements over the lanes (elements with a 2 x 2 rule no longer leave 28
// lanes idle), one thread per quasi-singular (point, element) pair walks the
// subdivision tree; partial sums are added per point in element order
// (deterministic). FP64. 300 points in a harmonic 6 x 6 cube, the
// whole call: 27.5 ms with one warp per point and lanes on one element's points,
// 2.7 ms here (0.7 ms of it the classification).
#pragma once

namespace mfb {

// Contraction of one quadrature point with t_w (T) and u_w (U): the u-part
// (SBIE) and the sigma-part (HBIE with the three unit normals; six components,
// (0,0) (0,1) (0,2) (1,1) (1,2) (2,2)). rs = -1 for a reversed element. With
//   g = psi I - chi dr dr^T, h = TT1 d dr dr^T + TT2 (n dr^T + d I) + TT3 dr n^T
//   d*, s* of hbie_point_s / hbie_point_h with n_i = e_c
// and the constants of u*, t*, d*, s* in the coefficients.
template <typename T>
struct IpCoef {
  T psi, chi, TT1, TT2, TT3, S1, S2, S3, S4, S5;
};
template <typename T>
__device__ __forceinline__ void ip_sbie(const IpCoef<T>& c, const double dr[3], const double n[3], double d, const T ut[3],
                                        const T uu[3], double rs, T du[3]) {
  const T a = ut[0] * dr[0] + ut[1] * dr[1] + ut[2] * dr[2], b = uu[0] * dr[0] + uu[1] * dr[1] + uu[2] * dr[2];
  const T w = uu[0] * n[0] + uu[1] * n[1] + uu[2] * n[2];
  const T A = -(c.chi * a) - (c.TT1 * (b * d) + c.TT3 * w) * rs;
  const T h2 = c.TT2 * rs;
#pragma unroll
  for (int l = 0; l < 3; ++l) du[l] = du[l] + c.psi * ut[l] + A * dr[l] - h2 * (b * n[l] + uu[l] * d);
}
template <typename T>
__device__ __forceinline__ void ip_hbie(const IpCoef<T>& c, const double dr[3], const double n[3], double d, const T ut[3],
                                        const T uu[3], double rs, T sg[6]) {
  const T a = ut[0] * dr[0] + ut[1] * dr[1] + ut[2] * dr[2], b = uu[0] * dr[0] + uu[1] * dr[1] + uu[2] * dr[2];
  const T w = uu[0] * n[0] + uu[1] * n[1] + uu[2] * n[2];
  const T bd = b * d;
  const T A = -(c.TT1 * a) - (c.S2 * w - c.S3 * bd) * rs, D = -(c.TT3 * a) - (c.S2 * bd + c.S5 * w) * rs;
  const T s1 = c.S1 * (-rs), s4 = c.S4 * (-rs);
  T V[3], W[3];
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    V[l] = s1 * (uu[l] * d + b * n[l]) - c.TT2 * ut[l];
    W[l] = s4 * uu[l];
  }
  int q = 0;
#pragma unroll
  for (int l = 0; l < 3; ++l)
#pragma unroll
    for (int k = l; k < 3; ++k, ++q) {
      T v = A * (dr[l] * dr[k]) + V[l] * dr[k] + V[k] * dr[l] + W[l] * n[k] + W[k] * n[l];
      if (l == k) v = v + D;
      sg[q] = sg[q] + v;
    }
}
__device__ __forceinline__ double ip_geo(const double rv[3], const double n[3], double dr[3], double& d1r, double& drdn) {
  const double r = sqrt(rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2]);
  d1r = 1.0 / r;
#pragma unroll
  for (int c = 0; c < 3; ++c) dr[c] = rv[c] * d1r;
  drdn = dr[0] * n[0] + dr[1] * n[1] + dr[2] * n[2];
  return r;
}

struct IpStatic {
  typedef double T;
  StaelaP k;
  double nu, cted1, cted2, ctes1, ctes2, ctes3, mu = 0.0;
  __device__ void sbie(int, const double*, const double rv[3], const double n[3], const T ut[3], const T uu[3], double rs,
                       T du[3]) const {
    double dr[3], d1r, d;
    ip_geo(rv, n, dr, d1r, d);
    const double cu = k.cteu1 * d1r, ct = k.ctet1 * d1r * d1r;
    IpCoef<double> c;
    c.psi = cu * k.cteu2; c.chi = -cu; c.TT1 = 3.0 * ct; c.TT2 = k.ctet2 * ct; c.TT3 = -c.TT2;
    ip_sbie(c, dr, n, d, ut, uu, rs, du);
  }
  __device__ void hbie(int, const double*, const double rv[3], const double n[3], const T ut[3], const T uu[3], double rs,
                       T sg[6]) const {
    double dr[3], d1r, d;
    ip_geo(rv, n, dr, d1r, d);
    const double cd_ = cted1 * d1r * d1r, cs = ctes1 * d1r * d1r * d1r;
    IpCoef<double> c;
    c.TT1 = 3.0 * cd_; c.TT2 = cted2 * cd_; c.TT3 = -c.TT2;
    c.S1 = 3.0 * nu * cs; c.S2 = 3.0 * ctes2 * cs; c.S3 = 15.0 * cs; c.S4 = ctes2 * cs; c.S5 = -ctes3 * cs;
    ip_hbie(c, dr, n, d, ut, uu, rs, sg);
  }
};

// E_n evaluated directly (wavenumbers or distances beyond the radial table)
struct IpHarmonic {
  typedef cd T;
  const HarParD* p;
  const HarParH* ph;
  __device__ void sbie(int f, const double*, const double rv[3], const double n[3], const T ut[3], const T uu[3], double rs,
                       T du[3]) const {
    double dr[3], d1r, d, d1, d2;
    const HarParD& q = p[f];
    const double r = ip_geo(rv, n, dr, d1r, d);
    IpCoef<cd> c;
    harela_coeffs(q, r, c.psi, c.chi, c.TT1, c.TT2, c.TT3, d1, d2, true);
    c.psi = q.cte_u * c.psi; c.chi = q.cte_u * c.chi;
    c.TT1 = q.cte_t * c.TT1; c.TT2 = q.cte_t * c.TT2; c.TT3 = q.cte_t * c.TT3;
    ip_sbie(c, dr, n, d, ut, uu, rs, du);
  }
  __device__ void hbie(int f, const double*, const double rv[3], const double n[3], const T ut[3], const T uu[3], double rs,
                       T sg[6]) const {
    double dr[3], d1r, d;
    const double r = ip_geo(rv, n, dr, d1r, d);
    HbieCoefH k;
    hbie_coef_h(p[f], ph[f], r, true, k);
    const cd cl = ph[f].cte_d, cm = ph[f].cte_s;
    IpCoef<cd> c;
    c.TT1 = cl * k.TT1; c.TT2 = cl * k.TT2; c.TT3 = cl * k.TT3;
    c.S1 = cm * k.S1; c.S2 = cm * k.S2; c.S3 = cm * k.S3; c.S4 = cm * k.S4; c.S5 = cm * k.S5;
    ip_hbie(c, dr, n, d, ut, uu, rs, sg);
  }
};
// the same from the call's radial table
struct IpHarmonicRad {
  typedef cd T;
  RadTab t;
  __device__ void sbie(int f, const double*, const double rv[3], const double n[3], const T ut[3], const T uu[3], double rs,
                       T du[3]) const {
    double dr[3], d1r, d, x;
    const double r = ip_geo(rv, n, dr, d1r, d);
    const RadF& q = t.f[f];
    const double2* w = rad_row(t, f, q, r, x);
    const double d2 = d1r * d1r;
    IpCoef<cd> c;
    c.psi = rad_eval(w, x) + q.s[0] * d1r;
    c.chi = rad_eval(w + kRadC, x) + q.s[1] * d1r;
    c.TT1 = rad_eval(w + 2 * kRadC, x) + q.s[2] * d2;
    c.TT2 = rad_eval(w + 3 * kRadC, x) + q.s[3] * d2;
    c.TT3 = rad_eval(w + 4 * kRadC, x) + q.s[4] * d2;
    ip_sbie(c, dr, n, d, ut, uu, rs, du);
  }
  __device__ void hbie(int f, const double*, const double rv[3], const double n[3], const T ut[3], const T uu[3], double rs,
                       T sg[6]) const {
    double dr[3], d1r, d;
    const double r = ip_geo(rv, n, dr, d1r, d);
    HbieCoefH k;
    hbie_coef_rad(t, f, r, d1r, true, k);
    IpCoef<cd> c;
    c.TT1 = k.TT1; c.TT2 = k.TT2; c.TT3 = k.TT3;
    c.S1 = k.S1; c.S2 = k.S2; c.S3 = k.S3; c.S4 = k.S4; c.S5 = k.S5;
    ip_hbie(c, dr, n, d, ut, uu, rs, sg);
  }
};

// Half-space (static, x3 >= xp, traction-free surface): the complementary
// kernels added at internal points (calculate_internal_points_mechanics_static.f90:
// 288-310,401-418). rv is measured from the image of the point (the pairs are
// classified on it, as fbem_bem_staela3d_hsc_sbie_auto / _hsc_hbie_auto do);
// xi is the point. u*, t*: hsc_point (fbem_bem_staela3d_hsc_sbie). d*, s*
// (fbem_bem_staela3d_hsc_hbie, bem_staela3d.f90:10882-11102): built from the
// first and mixed second derivatives of the complementary u* in x and x_i,
// here by forward-mode differentiation of u* in Cartesian form (HJet: value,
// the gradients in x and x_i and the mixed Hessian block).
struct HJet {
  double v, gx[3], gi[3], H[3][3];
};
__device__ __forceinline__ HJet hj_const(double c) {
  HJet r;
  r.v = c;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.gx[j] = r.gi[j] = 0.0;
#pragma unroll
    for (int p = 0; p < 3; ++p) r.H[j][p] = 0.0;
  }
  return r;
}
__device__ __forceinline__ HJet hj_axpy(double a, const HJet& x, const HJet& y) {  // a x + y
  HJet r;
  r.v = a * x.v + y.v;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.gx[j] = a * x.gx[j] + y.gx[j];
    r.gi[j] = a * x.gi[j] + y.gi[j];
#pragma unroll
    for (int p = 0; p < 3; ++p) r.H[j][p] = a * x.H[j][p] + y.H[j][p];
  }
  return r;
}
__device__ __forceinline__ HJet hj_add(const HJet& x, const HJet& y) { return hj_axpy(1.0, x, y); }
__device__ __forceinline__ HJet hj_sub(const HJet& x, const HJet& y) { return hj_axpy(-1.0, y, x); }
__device__ __forceinline__ HJet hj_scale(double a, const HJet& x) { return hj_axpy(a, x, hj_const(0.0)); }
__device__ __forceinline__ HJet hj_mul(const HJet& a, const HJet& b) {
  HJet r;
  r.v = a.v * b.v;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.gx[j] = a.v * b.gx[j] + a.gx[j] * b.v;
    r.gi[j] = a.v * b.gi[j] + a.gi[j] * b.v;
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int p = 0; p < 3; ++p) r.H[j][p] = a.v * b.H[j][p] + a.H[j][p] * b.v + a.gx[j] * b.gi[p] + a.gi[p] * b.gx[j];
  return r;
}
__device__ __forceinline__ HJet hj_chain(const HJet& a, double g, double d1, double d2) {
  HJet r;
  r.v = g;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    r.gx[j] = d1 * a.gx[j];
    r.gi[j] = d1 * a.gi[j];
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int p = 0; p < 3; ++p) r.H[j][p] = d1 * a.H[j][p] + d2 * a.gx[j] * a.gi[p];
  return r;
}
__device__ __forceinline__ HJet hj_inv(const HJet& a) {
  const double q = 1.0 / a.v;
  return hj_chain(a, q, -q * q, 2.0 * q * q * q);
}
__device__ __forceinline__ HJet hj_sqrt(const HJet& a) {
  const double s = sqrt(a.v);
  return hj_chain(a, s, 0.5 / s, -0.25 / (s * a.v));
}
// complementary u*[l][k] without 1 / (16 pi mu (1 - nu)); x, xi seeded jets
__device__ void hsc_u_jets(double nu, const HJet x[3], const HJet xi[3], double xp, HJet u[3][3]) {
  const double c1 = 1.0 - nu, c2 = 1.0 - 2.0 * nu, c4 = 3.0 - 4.0 * nu, k12 = 4.0 * c1 * c2;
  const HJet rx = hj_sub(x[0], xi[0]), ry = hj_sub(x[1], xi[1]);
  const HJet z = hj_axpy(1.0, x[2], hj_const(-xp)), c = hj_axpy(1.0, xi[2], hj_const(-xp)), zc = hj_add(z, c);
  const HJet rp = hj_sqrt(hj_add(hj_add(hj_mul(rx, rx), hj_mul(ry, ry)), hj_mul(zc, zc)));
  const HJet irp = hj_inv(rp), irp2 = hj_mul(irp, irp), irp3 = hj_mul(irp2, irp), irp5 = hj_mul(irp3, irp2);
  const HJet iq = hj_inv(hj_add(rp, zc)), iq2 = hj_mul(iq, iq);
  const HJet cz = hj_mul(c, z), zmc = hj_sub(z, c);
  const HJet one = hj_const(1.0);
  const HJet irpiq = hj_mul(irp, iq);
  // shared radial factors of the tangential / normal loads
  const HJet tA = hj_sub(hj_scale(c4, hj_mul(zmc, irp3)), hj_scale(6.0, hj_mul(hj_mul(cz, zc), irp5)));
  const HJet Bt = hj_axpy(k12, irpiq, tA);   // load tangential, component 3
  const HJet Bn = hj_axpy(-k12, irpiq, hj_axpy(12.0, hj_mul(hj_mul(cz, zc), irp5), tA));  // normal load, components 1, 2
#pragma unroll 1
  for (int a = 0; a < 2; ++a) {
    const HJet ra = a ? ry : rx, ra2 = hj_mul(ra, ra);
    HJet v = hj_add(irp, hj_scale(c4, hj_mul(ra2, irp3)));
    v = hj_add(v, hj_mul(hj_scale(2.0, hj_mul(cz, irp3)), hj_axpy(-3.0, hj_mul(ra2, irp2), one)));
    v = hj_add(v, hj_mul(hj_scale(k12, iq), hj_sub(one, hj_mul(ra2, irpiq))));
    u[a][a] = v;
    u[a][2] = hj_mul(ra, Bt);
    u[2][a] = hj_mul(ra, Bn);
  }
  u[0][1] = hj_mul(hj_mul(rx, ry), hj_sub(hj_sub(hj_scale(c4, irp3), hj_scale(6.0, hj_mul(cz, irp5))),
                                          hj_scale(k12, hj_mul(irp, iq2))));
  u[1][0] = u[0][1];
  const HJet zc2 = hj_mul(zc, zc);
  u[2][2] = hj_add(hj_add(hj_scale(8.0 * c1 * c1 - c4, irp), hj_mul(hj_sub(hj_scale(c4, zc2), hj_scale(2.0, cz)), irp3)),
                   hj_scale(6.0, hj_mul(hj_mul(cz, zc2), irp5)));
}
struct IpHsc {
  typedef double T;
  double mu, nu, xp;
  __device__ void sbie(int, const double* xi, const double rv[3], const double n[3], const T ut[3], const T uu[3],
                       double rs, T du[3]) const {
    const double c = xi[2] - xp;
    double fu[9], ft[9];
    hsc_point(nu, rv[0], rv[1], c, rv[2] - c, rv[2] + 2.0 * xp, n, fu, ft);
    const double cu = 1.0 / (16.0 * kPi * mu * (1.0 - nu)), ct = 1.0 / (8.0 * kPi * (1.0 - nu));
#pragma unroll
    for (int il = 0; il < 3; ++il) {
      double g = 0.0, h = 0.0;
#pragma unroll
      for (int ik = 0; ik < 3; ++ik) {
        g += fu[3 * il + ik] * ut[ik];
        h += ft[3 * il + ik] * uu[ik];
      }
      du[il] += cu * g - rs * ct * h;
    }
  }
  __device__ void hbie(int, const double* xi, const double rv[3], const double n[3], const T ut[3], const T uu[3],
                       double rs, T sg[6]) const {
    // x = image + rv
    const double xq[3] = {xi[0] + rv[0], xi[1] + rv[1], 2.0 * xp - xi[2] + rv[2]};
    HJet xj[3], ij[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      xj[c] = hj_const(xq[c]);
      xj[c].gx[c] = 1.0;
      ij[c] = hj_const(xi[c]);
      ij[c].gi[c] = 1.0;
    }
    HJet u[3][3];
    hsc_u_jets(nu, xj, ij, xp, u);
    const double Ku = 1.0 / (16.0 * kPi * mu * (1.0 - nu)), lam = 2.0 * mu * nu / (1.0 - 2.0 * nu);
    // x_i derivative of t* = sigma*(x) n, sigma*_{l,kj} = lam d_kj div u_l + mu (u_lk,j + u_lj,k)
    double dt[3][3][3];
#pragma unroll 1
    for (int l = 0; l < 3; ++l)
#pragma unroll 1
      for (int k = 0; k < 3; ++k)
#pragma unroll 1
        for (int p = 0; p < 3; ++p) {
          const double div = u[l][0].H[0][p] + u[l][1].H[1][p] + u[l][2].H[2][p];
          double v = 0.0;
          for (int j = 0; j < 3; ++j) {
            double sj = mu * (u[l][k].H[j][p] + u[l][j].H[k][p]);
            if (j == k) sj += lam * div;
            v += sj * n[j];
          }
          dt[l][k][p] = Ku * v;
        }
    // d*_lkp, s*_lkp contracted with n_i = e_kc: sg(l, kc) += d ut - rs s uu,
    // symmetric in (l, kc)
#pragma unroll 1
    for (int l = 0; l < 3; ++l)
#pragma unroll 1
      for (int kc = l; kc < 3; ++kc) {
        double acc = 0.0;
        for (int k = 0; k < 3; ++k) {
          double dl = mu * Ku * (u[l][k].gi[kc] + u[kc][k].gi[l]);
          double sl = mu * (dt[l][k][kc] + dt[kc][k][l]);
          if (l == kc) {
            dl += lam * Ku * (u[0][k].gi[0] + u[1][k].gi[1] + u[2][k].gi[2]);
            sl += lam * (dt[0][k][0] + dt[1][k][1] + dt[2][k][2]);
          }
          acc += dl * ut[k] - rs * sl * uu[k];
        }
        sg[kc + (l == 1 ? 2 : (l == 2 ? 3 : 0))] += acc;
      }
  }
};

// inputs of the internal-point kernels
struct IpArgs {
  int nip, nf;
  const double* xip;     // [nip][3]
  const int* enode;      // [ne][8] 0-based node of each element node
  const double* nodex;   // [nn][3]
  const double* nodecl;  // [nn] csize of the node's first element
  int nn;
  const void* uval;      // [nf][nn][3] T
  const void* tval;      // [nf][nn][3] T
  uint8_t* cls_s;        // [nip][ne]
  uint8_t* cls_h;
  int* onnode;           // [nip] node index or -1
  int* npair;            // [nip] quasi-singular pairs per point, then exclusive offsets [nip+1]
  int* poff;
  int* pair_e;           // [npairs]
  int* pair_ip;
  int* err;              // first point (1-based) on an element away from its nodes, 0 if none
  void* slot;            // [nf][npairs][9] T: u (3), sigma (6)
  int npairs;
  int e0, nec;           // elements of this launch (e0 a multiple of 32)
  void* uw;              // [nf][nec ptot][6] T: u_w, t_w at the dataset points
  void* part;            // [nf][nip][nch][9] T: partial sums of gpc groups of 32 elements each
  int nch, gpc;
  void* out;             // [nf][nip][12] T: u(3), then sigma(:, kc) for kc = 0..2
  // image pass of a half-space region: pairs classified and integrated from
  // the image (x_i1, x_i2, 2 xp - x_i3) of each point; points at a node add 0
  int image;
  double hs_xp;
};
// the point the pair geometry is measured from: the point, or its image
__device__ __forceinline__ void ip_ref(const IpArgs& a, const double* xi, double xr[3]) {
  xr[0] = xi[0];
  xr[1] = xi[1];
  xr[2] = a.image ? 2.0 * a.hs_xp - xi[2] : xi[2];
}

// point at a node: the last node (in node order) within 1e-12 csize; one warp
// per point
__global__ void k_ip_onnode(IpArgs a) {
  const int ip = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (ip >= a.nip) return;
  const double* x = a.xip + 3 * (size_t)ip;
  int last = -1;
  for (int s = threadIdx.x & 31; s < a.nn; s += 32) {
    if (a.nodecl[s] <= 0.0) continue;  // node of no element
    const double r0 = x[0] - a.nodex[3 * s], r1 = x[1] - a.nodex[3 * s + 1], r2 = x[2] - a.nodex[3 * s + 2];
    if (sqrt(r0 * r0 + r1 * r1 + r2 * r2) / a.nodecl[s] < 1e-12) last = s;
  }
  last = __reduce_max_sync(0xffffffffu, last);
  if ((threadIdx.x & 31) == 0) a.onnode[ip] = last;
}

// sbie_auto / hbie_auto classification of every (point, element) pair
__global__ void k_ip_classify(DMesh m, IpArgs a, const QsCurves* __restrict__ qs) {
  const long long total = (long long)a.nip * m.ne;
  for (long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x; id < total;
       id += (long long)gridDim.x * blockDim.x) {
    const int ip = (int)(id / m.ne), e = (int)(id % m.ne);
    double xi[3];
    ip_ref(a, a.xip + 3 * (size_t)ip, xi);
    const double* b = m.ball + 4 * (size_t)e;
    const double r0 = b[0] - xi[0], r1 = b[1] - xi[1], r2 = b[2] - xi[2];
    double rmin = sqrt(r0 * r0 + r1 * r1 + r2 * r2) - b[3];
    double bx[2] = {0.0, 0.0}, d;
    bool sing = false;
    if (rmin > 4.0 * b[3]) {
      d = rmin / m.cl[e];
    } else {
      int method;
      nearest_q8(m.ex + 24 * (size_t)e, m.cl[e], xi, bx, &rmin, &d, &method);
      sing = d <= 1e-12;
    }
    uint8_t c[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (sing) {
        c[h] = CLS_SING;
        continue;
      }
      const int gn = qs_estimate(*qs, 2, h ? 7 : 5, d, bx, false);
      const int gln = max(m.gln_far[e], gn);
      c[h] = CLS_ADP;
      if (gln <= m.ps_gln_max && gn > 0)
        for (int i = 0; i < m.nps; ++i)
          if (m.ps_gln[i] >= gln) { c[h] = (uint8_t)i; break; }
    }
    a.cls_s[id] = c[0];
    a.cls_h[id] = c[1];
  }
}

// quasi-singular pairs per point (one warp per point); a singular pair of a
// point that is not at a node records the point in err
__global__ void k_ip_count(DMesh m, IpArgs a) {
  const int ip = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), l = threadIdx.x & 31;
  if (ip >= a.nip) return;
  int cnt = 0, sing = 0;
  if (a.onnode[ip] < 0)
    for (int e = l; e < m.ne; e += 32) {
      const size_t id = (size_t)ip * m.ne + e;
      const uint8_t s = a.cls_s[id], h = a.cls_h[id];
      if (s == CLS_SING || h == CLS_SING) sing = 1;
      else if (s == CLS_ADP || h == CLS_ADP) ++cnt;
    }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    sing |= __shfl_xor_sync(0xffffffffu, sing, o);
  }
  if (l == 0) {
    a.npair[ip] = sing ? 0 : cnt;
    if (sing) atomicMin(a.err, ip + 1);
  }
}
__global__ void k_ip_fill(DMesh m, IpArgs a) {
  const int ip = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), l = threadIdx.x & 31;
  if (ip >= a.nip || a.onnode[ip] >= 0) return;
  int o = a.poff[ip];
  const int o1 = a.poff[ip + 1];
  for (int e0 = 0; e0 < m.ne && o < o1; e0 += 32) {
    const int e = e0 + l;
    bool q = false;
    if (e < m.ne) {
      const size_t id = (size_t)ip * m.ne + e;
      const uint8_t s = a.cls_s[id], h = a.cls_h[id];
      q = s != CLS_SING && h != CLS_SING && (s == CLS_ADP || h == CLS_ADP);
    }
    const unsigned mq = __ballot_sync(0xffffffffu, q);
    if (q) {
      const int j = o + __popc(mq & ((1u << l) - 1u));
      a.pair_e[j] = e;
      a.pair_ip[j] = ip;
    }
    o += __popc(mq);
  }
}

// weighted sums of the element's nodal values at one quadrature point
template <typename T>
__device__ __forceinline__ void ip_weights(const T* un, const T* tn, const double w[8], T uu[3], T ut[3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    uu[c] = VT<T>::zero();
    ut[c] = VT<T>::zero();
  }
#pragma unroll
  for (int kn = 0; kn < 8; ++kn)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      uu[c] = uu[c] + un[3 * kn + c] * w[kn];
      ut[c] = ut[c] + tn[3 * kn + c] * w[kn];
    }
}

// One quasi-singular (point, element) pair and frequency per thread: the
// subdivision tree of sbie_ext_adp / hbie_ext_adp (bem_staela3d.f90:973-1096,
// 4790-4914) walked depth-first with an explicit stack, every leaf integrated
// with its Telles-mapped rule (sbie_ext_st / hbie_ext_st) as it is reached.
template <class POL>
__global__ void k_ip_adp(DMesh m, IpArgs a, POL pol, const QsCurves* __restrict__ qs) {
  typedef typename POL::T T;
  const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (id >= (long long)a.npairs * a.nf) return;
  const int pr = (int)(id % a.npairs), f = (int)(id / a.npairs);
  const int ip = a.pair_ip[pr], e = a.pair_e[pr];
  const double* xi = a.xip + 3 * (size_t)ip;
  double xr[3];
  ip_ref(a, xi, xr);
  const double* x = m.ex + 24 * (size_t)e;
  const T* uv = (const T*)a.uval + (size_t)f * a.nn * 3;
  const T* tv = (const T*)a.tval + (size_t)f * a.nn * 3;
  T un[24], tn[24];
  for (int kn = 0; kn < 8; ++kn) {
    const int s = a.enode[8 * e + kn];
    for (int c = 0; c < 3; ++c) {
      un[3 * kn + c] = uv[3 * s + c];
      tn[3 * kn + c] = tv[3 * s + c];
    }
  }
  const double rs = (m.rev[e] & 1) ? -1.0 : 1.0;
  T du[3], sg[6];
  for (int c = 0; c < 3; ++c) du[c] = VT<T>::zero();
  for (int c = 0; c < 6; ++c) sg[c] = VT<T>::zero();
  const size_t cid = (size_t)ip * m.ne + e;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    if ((h ? a.cls_h[cid] : a.cls_s[cid]) != CLS_ADP) continue;
    const int F = h ? 7 : 5;
    AdpNode st[52];
    int top = 0;
    st[0].xs[0] = -1; st[0].xs[1] = -1; st[0].xs[2] = 1; st[0].xs[3] = -1;
    st[0].xs[4] = 1;  st[0].xs[5] = 1;  st[0].xs[6] = -1; st[0].xs[7] = 1;
    st[0].ks = 1;
    top = 1;
    while (top > 0) {
      const AdpNode nd = st[--top];
      double bx[2], rmin, d;
      int method;
      if (nd.ks == 1) {
        nearest_q8(x, m.cl[e], xr, bx, &rmin, &d, &method);
      } else {
        double xsub[24];
        subdiv_q8(x, nd.xs, xsub);
        nearest_q8(xsub, clen_q8(xsub, 1e-12), xr, bx, &rmin, &d, &method);
      }
      int gn = qs_estimate(*qs, 2, F, d, bx, true);
      bool sub = false;
      if (nd.ks == m.ns_max) {
        if (gn == 0) gn = 30;
      } else if (gn == 0) {
        sub = true;
      }
      if (sub && top + 4 <= 52) {
        const double* s = nd.xs;
        const double c0 = 0.25 * (s[0] + s[2] + s[4] + s[6]), c1 = 0.25 * (s[1] + s[3] + s[5] + s[7]);
        const double q[4][8] = {
            {s[0], s[1], 0.5 * (s[0] + s[2]), 0.5 * (s[1] + s[3]), c0, c1, 0.5 * (s[0] + s[6]), 0.5 * (s[1] + s[7])},
            {0.5 * (s[0] + s[2]), 0.5 * (s[1] + s[3]), s[2], s[3], 0.5 * (s[2] + s[4]), 0.5 * (s[3] + s[5]), c0, c1},
            {c0, c1, 0.5 * (s[2] + s[4]), 0.5 * (s[3] + s[5]), s[4], s[5], 0.5 * (s[4] + s[6]), 0.5 * (s[5] + s[7])},
            {0.5 * (s[0] + s[6]), 0.5 * (s[1] + s[7]), c0, c1, 0.5 * (s[4] + s[6]), 0.5 * (s[5] + s[7]), s[6], s[7]}};
        for (int i = 3; i >= 0; --i) {
          for (int j = 0; j < 8; ++j) st[top].xs[j] = q[i][j];
          st[top].ks = nd.ks + 1;
          ++top;
        }
        continue;
      }
      // leaf: Telles-mapped rule of order max(gn, gln_far) on the sub-square
      const int g = max(gn, m.gln_far[e]);
      const double barr = telles_barr(d);
      const Telles t1 = telles11(bx[0], barr), t2 = telles11(bx[1], barr);
      for (int k1 = 1; k1 <= g; ++k1) {
        double xp1, jt1;
        telles_map(t1, gl11x(k1, g), xp1, jt1);
        for (int k2 = 1; k2 <= g; ++k2) {
          double xp2, jt2;
          telles_map(t2, gl11x(k2, g), xp2, jt2);
          double sp[4], sd1[4], sd2[4];
          phi_q4(xp1, xp2, sp);
          dphi_q4(xp1, xp2, sd1, sd2);
          double xa = 0, xb = 0, a11 = 0, a12 = 0, a21 = 0, a22 = 0;
          for (int qq = 0; qq < 4; ++qq) {
            xa += sp[qq] * nd.xs[2 * qq];
            xb += sp[qq] * nd.xs[2 * qq + 1];
            a11 += sd1[qq] * nd.xs[2 * qq];
            a12 += sd1[qq] * nd.xs[2 * qq + 1];
            a21 += sd2[qq] * nd.xs[2 * qq];
            a22 += sd2[qq] * nd.xs[2 * qq + 1];
          }
          const double js = a11 * a22 - a12 * a21;
          double xq[3], T1[3], T2[3], phi[8], N[3];
          geom_q8(x, xa, xb, xq, T1, T2, phi);
          cross3(T1, T2, N);
          const double jg = norm3(N);
          const double n[3] = {N[0] / jg, N[1] / jg, N[2] / jg};
          const double rv[3] = {xq[0] - xr[0], xq[1] - xr[1], xq[2] - xr[2]};
          const double jw = jg * js * jt1 * jt2 * gl11w(k1, g) * gl11w(k2, g);
          double w[8];
          for (int qq = 0; qq < 8; ++qq) w[qq] = phi[qq] * jw;
          T uu[3], ut[3];
          ip_weights<T>(un, tn, w, uu, ut);
          if (h) pol.hbie(f, xi, rv, n, ut, uu, rs, sg);
          else pol.sbie(f, xi, rv, n, ut, uu, rs, du);
        }
      }
    }
  }
  T* sl = (T*)a.slot + ((size_t)f * a.npairs + pr) * 9;
  for (int c = 0; c < 3; ++c) sl[c] = du[c];
  for (int c = 0; c < 6; ++c) sl[3 + c] = sg[c];
}

// u_w, t_w at every dataset point (all precalculated rules) of the launch's elements
template <typename T>
__global__ void k_ip_weights(DMesh m, IpArgs a) {
  const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x, np = (long long)a.nec * m.ptot;
  if (id >= np * a.nf) return;
  const int f = (int)(id / np);
  const long long pt = id - f * np + (long long)a.e0 * m.ptot;
  const int e = (int)(pt / m.ptot);
  const T* uv = (const T*)a.uval + (size_t)f * a.nn * 3;
  const T* tv = (const T*)a.tval + (size_t)f * a.nn * 3;
  T un[24], tn[24];
  double w[8];
#pragma unroll
  for (int kn = 0; kn < 8; ++kn) {
    const int s = a.enode[8 * e + kn];
    w[kn] = m.pphi[8 * pt + kn];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      un[3 * kn + c] = uv[3 * s + c];
      tn[3 * kn + c] = tv[3 * s + c];
    }
  }
  T* o = (T*)a.uw + 6 * id;
  ip_weights<T>(un, tn, w, o, o + 3);
}

// One warp per (gpc groups of 32 elements, point, frequency): the
// precalculated-rule pairs of the launch's elements, added to the sums of the
// launches before. gpc is 1 until the points alone fill the GPU.
// A lane looks up one element's rule; a scan of the point counts then deals the
// quadrature points of all 32 out to the lanes.
template <class POL, int WPB>
__global__ void __launch_bounds__(WPB * 32) k_ip_reg(DMesh m, IpArgs a, POL pol) {
  typedef typename POL::T T;
  const int lane = threadIdx.x & 31;
  const long long gw = blockIdx.x * (long long)WPB + (threadIdx.x >> 5);
  if (gw >= (long long)a.nip * a.nf * a.nch) return;
  const int ch = (int)(gw % a.nch), ip = (int)((gw / a.nch) % a.nip), f = (int)(gw / a.nch / a.nip);
  if (a.onnode[ip] >= 0) return;
  const double* xi = a.xip + 3 * (size_t)ip;
  double xr[3];
  ip_ref(a, xi, xr);
  const T* uw = (const T*)a.uw + (size_t)f * a.nec * m.ptot * 6;
  const size_t pt0 = (size_t)a.e0 * m.ptot;
  T du[3], sg[6];
  for (int c = 0; c < 3; ++c) du[c] = VT<T>::zero();
  for (int c = 0; c < 6; ++c) sg[c] = VT<T>::zero();
  unsigned revs = 0;
  int cls_s = CLS_SING, cls_h = CLS_SING, e = 0;
  const int g0 = ch * a.gpc, g1 = min(g0 + a.gpc, (a.nec + 31) / 32);
#pragma unroll 1
  for (int hg = 2 * g0; hg < 2 * g1; ++hg) {
    const int h = hg & 1;
    if (h == 0) {
      e = 16 * hg + lane;
      int rev = 0;
      cls_s = cls_h = CLS_SING;
      if (e < a.nec) {
        const size_t cid = (size_t)ip * m.ne + a.e0 + e;
        cls_s = a.cls_s[cid];
        cls_h = a.cls_h[cid];
        rev = m.rev[a.e0 + e] & 1;
        if (cls_s == CLS_SING || cls_h == CLS_SING) cls_s = cls_h = CLS_SING;
      }
      revs = __ballot_sync(0xffffffffu, rev);
    }
    const int c = h ? cls_h : cls_s, P = c >= CLS_ADP ? 0 : m.ps_gln[c] * m.ps_gln[c];
    int end = P;  // inclusive scan
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    const int total = __shfl_sync(0xffffffffu, end, 31);
    // dataset index, from the launch's first element, of scan position q of this
    // lane's element: first + q
    const int first = P > 0 ? e * m.ptot + m.ps_off[c] - (end - P) : 0;
#pragma unroll 1
    for (int base = 0; base < total; base += 32) {
      const int q = base + lane;
      int j = 0;  // lanes whose range ends at or before q
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(0xffffffffu, end, j + o - 1) <= q) j += o;
      j = min(j, 31);
      const int pt = __shfl_sync(0xffffffffu, first, j) + q;
      if (q < total) {
        const double rs = (revs >> j) & 1 ? -1.0 : 1.0;
        const double* px = m.px + 3 * (pt0 + pt);
        const double* pn = m.pn + 3 * (pt0 + pt);
        const double rv[3] = {px[0] - xr[0], px[1] - xr[1], px[2] - xr[2]};
        const double n[3] = {pn[0], pn[1], pn[2]};
        const T* v = uw + 6 * (size_t)pt;
        const T uu[3] = {v[0], v[1], v[2]}, ut[3] = {v[3], v[4], v[5]};
        if (h) pol.hbie(f, xi, rv, n, ut, uu, rs, sg);
        else pol.sbie(f, xi, rv, n, ut, uu, rs, du);
      }
    }
  }
  T* o = (T*)a.part + 9 * (size_t)(((size_t)f * a.nip + ip) * a.nch + ch);
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    T v = j < 3 ? du[j < 3 ? j : 0] : sg[j < 3 ? 0 : j - 3];
    for (int off = 16; off > 0; off >>= 1) v = v + shfl_x(v, off);
    if (lane == 0) o[j] = a.e0 > 0 ? o[j] + v : v;
  }
}

// Sums of a point: its element groups, then its quasi-singular slots, in
// order; one thread per (component, point, frequency)
template <typename T>
__global__ void k_ip_sum(IpArgs a) {
  const long long id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (id >= 9LL * a.nip * a.nf) return;
  const int j = (int)(id % 9), ip = (int)((id / 9) % a.nip), f = (int)(id / 9 / a.nip);
  const int on = a.onnode[ip];
  T v = VT<T>::zero();
  if (on >= 0) {
    if (j < 3 && !a.image) v = ((const T*)a.uval)[((size_t)f * a.nn + on) * 3 + j];
  } else {
    const T* p = (const T*)a.part + 9 * (size_t)(((size_t)f * a.nip + ip) * a.nch);
    for (int ch = 0; ch < a.nch; ++ch) v = v + p[9 * ch + j];
    const T* sl = (const T*)a.slot;
    for (int pr = a.poff[ip]; pr < a.poff[ip + 1]; ++pr) v = v + sl[((size_t)f * a.npairs + pr) * 9 + j];
  }
  T* o = (T*)a.out + ((size_t)f * a.nip + ip) * 12;
  if (j < 3) {
    o[j] = v;
  } else {
    const int l = sym_il(j - 3), k = sym_ik(j - 3);
    o[3 + 3 * k + l] = v;
    o[3 + 3 * l + k] = v;
  }
}

}  // namespace mfb
