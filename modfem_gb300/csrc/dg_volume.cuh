// Volume integrals of DG tensor-basis prisms of degree P (FP64), shared by
// the per-degree kernel and the persistent mixed kernel.
//
// Reference: apr_num_int_el of apd_dg_prism (aps_dg_prism_intf.c:1239-1728):
// K_uw = sum_q vol_q sum_ij a_ij d_i phi_w d_j phi_u, R_w = sum_q vol_q f phi_w.
// With the adjugate rows c_a of the Jacobian every point contributes
// D_q^T G_q D_q (D_q: 3 x ns reference derivatives, G_q = (w_q/|det|) C^T A C,
// 6 entries for symmetric A).
//
// The basis is monomial, phi_u = xi^a eta^b zeta^c, so a product of two
// derivatives is a monomial again and every entry needs only the moments
//   M_cd[i, j][k] = sum_q G_q,cd xi^i eta^j zeta^k :
//   K_uw = a a' M_00 + (a b' + b a') M_01 + b b' M_11
//        + (a c' + c a') M_02 + (b c' + c b') M_12 + c c' M_22
// at the exponents of the product (u: a b c, w: a' b' c').  The rules are
// tensor products (triangle points x Gauss line points), so the moments are
// summed over the line points first, then over the triangle points.  FMA an
// element, p = 1/2/3/4: 0.5k / 3.4k / 18k / 49k besides the point geometry,
// against 0.5k / 12k / 135k / 738k of the sum over points per entry
// (nq (9 ns + 3 ns (ns + 1) / 2)).  All terms of a sum keep their sign
// pattern (monomials of xi, eta >= 0 and powers of zeta), so the error stays
// that of an FP64 dot product of the same length.  Measured (GB300, isolated):
// p = 3, 54,000 prisms 13.1 ms (sum over points) -> 2.06 ms, the FP64 issue
// bound of its 710 warp instructions an element; p = 4, 21,296 prisms 2.19 ms.
//
// A CTA integrates NE elements; each stage runs over the flattened (element,
// item) index, so that full warps issue: GB300 issues an FP64 instruction of
// a warp once in 16 clocks per SM, whatever the number of its active lanes,
// and integer and shared-memory instructions are nearly free beside it.
// Every sum has a fixed order: results do not depend on NE or the CTA size.
#pragma once

#include "prism_std.cuh"

namespace gbfem {

__host__ __device__ constexpr int dg_tri(int d) { return (d + 1) * (d + 2) / 2; }  // monomials of degree <= d

// One upper entry (u, w) of the matrix: the moment offsets and the integer
// coefficients of the components 00, 01, 11, 02, 12, 22 (a zero coefficient
// goes with offset 0).
struct DgVolEntry {
  unsigned short off[6];
  unsigned char coef[6];
  unsigned char u, w;
};

template <int P>
struct DgVol {
  static constexpr int NS = P == 1 ? 6 : P == 2 ? 18 : P == 3 ? 40 : 75;
  static constexpr int NQ = P == 1 ? 6 : P == 2 ? 18 : P == 3 ? 48 : 80;
  static constexpr int NZ = P + 1, NT = NQ / NZ;  // line and triangle points
  static constexpr int NSYM = NS * (NS + 1) / 2;
  // powers of zeta and monomials of (xi, eta) per component: order 00 01 11
  // (derivatives in the triangle only), 02 12, 22, and the load vector's
  static constexpr int K0 = 2 * P + 1, K1 = 2 * P, K2 = 2 * P - 1, KV = P + 1;
  static constexpr int T0 = dg_tri(2 * P - 2), T1 = dg_tri(2 * P - 1), T2 = dg_tri(2 * P), TV = dg_tri(P);
  static constexpr int NCK = 3 * K0 + 2 * K1 + K2 + KV;  // line sums per triangle point
  static constexpr int ZS = NT | 1;                      // their row stride (odd: no bank conflicts)
  static constexpr int NM = 3 * T0 * K0 + 2 * T1 * K1 + T2 * K2;  // moments
  // doubles of scratch per element: vertex differences and tensor, then the
  // point factors (7 per point, dead once the line sums exist) or the
  // moments, then the line sums
  static constexpr int GM = NM > 7 * NQ ? NM : 7 * NQ;
  static constexpr int PER_EL = 30 + GM + NCK * ZS;
  // tables copied to shared memory: triangle monomials [T2][NT], powers of
  // the line points [NZ][K0], the doubles 0 .. 2 P^2
  static constexpr int TAB = T2 * NT + NZ * K0 + 2 * P * P + 1;
};
__host__ __device__ constexpr int dg_vol_per_el(int p) {
  return p == 1 ? DgVol<1>::PER_EL : p == 2 ? DgVol<2>::PER_EL : p == 3 ? DgVol<3>::PER_EL : DgVol<4>::PER_EL;
}
__host__ __device__ constexpr int dg_vol_tab(int p) {
  return p == 1 ? DgVol<1>::TAB : p == 2 ? DgVol<2>::TAB : p == 3 ? DgVol<3>::TAB : DgVol<4>::TAB;
}

// Elements per CTA (launch variants, chosen by the autotuners): enough to
// fill the warps of the point stage (6 / 18 / 48 / 80 points an element) and
// few enough for three or more CTAs of 256 threads per SM.
constexpr int DG_VOL_VARIANTS = 3;
constexpr int DG_VOL_THREADS = 256;
__host__ __device__ constexpr int dg_vol_elems(int p, int v) {
  return p == 1 ? (v == 0 ? 16 : v == 1 ? 8 : 32)
       : p == 2 ? (v == 0 ? 8 : v == 1 ? 4 : 12)
       : p == 3 ? (v == 0 ? 4 : v == 1 ? 2 : 1)
                : (v == 0 ? 2 : 1);
}
__host__ __device__ constexpr int dg_vol_smem(int p, int v) {  // doubles
  return dg_vol_tab(p) + dg_vol_elems(p, v) * dg_vol_per_el(p);
}

// The element matrices and load vectors of `count` <= NE elements.  Element
// el's vertices and tensor are read through src(el, i), i < 18: coordinate
// i % 3 of vertex i / 3, i < 27: tensor entry i - 18 (row-major, symmetric); its block (column-major
// NS x NS) and load vector go to blk(el), rhs(el).  smem: dg_vol_smem(P)
// doubles; the whole CTA of DG_VOL_THREADS threads calls.
template <int P, class Src, class Blk, class Rhs>
__device__ __forceinline__ void dg_prism_volume_tile(int count, double f, const double *__restrict__ tab,
                                                     const double *__restrict__ QP, const DgVolEntry *__restrict__ ent, double *smem,
                                                     Src src, Blk blk, Rhs rhs) {
  using D = DgVol<P>;
  constexpr int NS = D::NS, NQ = D::NQ, NT = D::NT, NZ = D::NZ, ZS = D::ZS, TH = DG_VOL_THREADS;
  const int tid = threadIdx.x;
  double *sX = smem, *sZ = sX + D::T2 * NT, *sI = sZ + NZ * D::K0, *el0 = sI + 2 * P * P + 1;
  for (int t = tid; t < D::TAB; t += TH) smem[t] = tab[t];
  // vertex differences e_a = X1 - X0, e_b = X4 - X3 (xi edges), f_a = X2 -
  // X0, f_b = X5 - X3 (eta edges), C_i = X_{i+3} - X_i (zeta edges); tensor
  for (int t = tid; t < count * 30; t += TH) {
    const int el = t / 30, r = t % 30;
    double v;
    if (r < 21) {
      const int g = r / 3, d = r % 3;
      const int hi = g == 0 ? 1 : g == 1 ? 4 : g == 2 ? 2 : g == 3 ? 5 : g - 1;
      const int lo = g == 0 || g == 2 ? 0 : g == 1 || g == 3 ? 3 : g - 4;
      v = src(el, 3 * hi + d) - src(el, 3 * lo + d);
    } else {
      v = src(el, 18 + r - 21);
    }
    el0[el * D::PER_EL + r] = v;
  }
  __syncthreads();
  // point factors G (00 01 11 02 12 22) and w |det|, [factor][point]
  for (int t = tid; t < count * NQ; t += TH) {
    const int el = t / NQ, q = t % NQ;
    double *B = el0 + el * D::PER_EL, *G = B + 30 + q;
    const double xi = QP[4 * q], eta = QP[4 * q + 1], zeta = QP[4 * q + 2], w = QP[4 * q + 3];
    const double lo = 0.5 - 0.5 * zeta, hi = 0.5 + 0.5 * zeta, l0 = 0.5 - 0.5 * xi - 0.5 * eta, l1 = 0.5 * xi,
                 l2 = 0.5 * eta;
    const v3 ea = {B[0], B[1], B[2]}, eb = {B[3], B[4], B[5]}, fa = {B[6], B[7], B[8]}, fb = {B[9], B[10], B[11]};
    const v3 c0 = {B[12], B[13], B[14]}, c1v = {B[15], B[16], B[17]}, c2v = {B[18], B[19], B[20]};
    const double *A = B + 21;
    // columns of the Jacobian of the linear prism (apr_elem_calc_3D geometry)
    const v3 j1 = v3_fma(lo, ea, v3_scale(hi, eb)), j2 = v3_fma(lo, fa, v3_scale(hi, fb)),
             j3 = v3_fma(l0, c0, v3_fma(l1, c1v, v3_scale(l2, c2v)));
    const v3 cb[3] = {v3_cross(j2, j3), v3_cross(j3, j1), v3_cross(j1, j2)};
    const double adet = fabs(v3_dot(j1, cb[0]));
    const double s = w / adet;
    // G_ab = s c_a^T A c_b: the tensor a_ij multiplies d_i(test) d_j(trial)
    v3 Ac[3];
#pragma unroll
    for (int b = 0; b < 3; b++)
      Ac[b] = {s * fma(A[0], cb[b].x, fma(A[1], cb[b].y, A[2] * cb[b].z)),
               s * fma(A[3], cb[b].x, fma(A[4], cb[b].y, A[5] * cb[b].z)),
               s * fma(A[6], cb[b].x, fma(A[7], cb[b].y, A[8] * cb[b].z))};
    G[0 * NQ] = v3_dot(cb[0], Ac[0]);
    G[1 * NQ] = v3_dot(cb[0], Ac[1]);
    G[2 * NQ] = v3_dot(cb[1], Ac[1]);
    G[3 * NQ] = v3_dot(cb[0], Ac[2]);
    G[4 * NQ] = v3_dot(cb[1], Ac[2]);
    G[5 * NQ] = v3_dot(cb[2], Ac[2]);
    G[6 * NQ] = w * adet;
  }
  __syncthreads();
  // sums over the line points: row ck of component c, power k
  for (int t = tid; t < count * D::NCK * NT; t += TH) {
    const int el = t / (D::NCK * NT), r = t % (D::NCK * NT), ck = r / NT, m = r % NT;
    int c, k;
    if (ck < 3 * D::K0) {
      c = ck / D::K0;
      k = ck % D::K0;
    } else if (ck < 3 * D::K0 + 2 * D::K1) {
      c = 3 + (ck - 3 * D::K0) / D::K1;
      k = (ck - 3 * D::K0) % D::K1;
    } else if (ck < 3 * D::K0 + 2 * D::K1 + D::K2) {
      c = 5;
      k = ck - 3 * D::K0 - 2 * D::K1;
    } else {
      c = 6;
      k = ck - 3 * D::K0 - 2 * D::K1 - D::K2;
    }
    double *B = el0 + el * D::PER_EL;
    const double *G = B + 30 + c * NQ + m;
    double a = 0.0;
#pragma unroll
    for (int n = 0; n < NZ; n++) a = fma(G[n * NT], sZ[n * D::K0 + k], a);
    B[30 + D::GM + ck * ZS + m] = a;
  }
  __syncthreads();
  // moments (component, monomial, power) and the load vector: sums over the
  // triangle points
  constexpr int NL = D::TV * D::KV;
  for (int t = tid; t < count * (D::NM + NL); t += TH) {
    const int el = t / (D::NM + NL), r = t % (D::NM + NL);
    int al, ck;  // monomial, line-sum row
    if (r < 3 * D::T0 * D::K0) {
      const int c = r / (D::T0 * D::K0), s = r % (D::T0 * D::K0);
      al = s / D::K0;
      ck = c * D::K0 + s % D::K0;
    } else if (r < 3 * D::T0 * D::K0 + 2 * D::T1 * D::K1) {
      const int r1 = r - 3 * D::T0 * D::K0, c = r1 / (D::T1 * D::K1), s = r1 % (D::T1 * D::K1);
      al = s / D::K1;
      ck = 3 * D::K0 + c * D::K1 + s % D::K1;
    } else if (r < D::NM) {
      const int s = r - 3 * D::T0 * D::K0 - 2 * D::T1 * D::K1;
      al = s / D::K2;
      ck = 3 * D::K0 + 2 * D::K1 + s % D::K2;
    } else {
      const int s = r - D::NM;
      al = s / D::KV;
      ck = 3 * D::K0 + 2 * D::K1 + D::K2 + s % D::KV;
    }
    double *B = el0 + el * D::PER_EL;
    const double *Z = B + 30 + D::GM + ck * ZS, *X = sX + al * NT;
    double a = 0.0;
#pragma unroll
    for (int m = 0; m < NT; m++) a = fma(Z[m], X[m], a);
    if (r < D::NM)
      B[30 + r] = a;
    else
      rhs(el)[ent[D::NSYM + r - D::NM].u] = f * a;  // the function of (monomial, power)
  }
  __syncthreads();
  // entries (u, w), u <= w: K_uw is column-major in the block, blk[w + NS u]
  for (int k = tid; k < D::NSYM; k += TH) {
    const DgVolEntry E = ent[k];
    double cf[6];
#pragma unroll
    for (int c = 0; c < 6; c++) cf[c] = sI[E.coef[c]];
    const int lo = E.w + NS * E.u, up = E.u + NS * E.w;
    for (int el = 0; el < count; el++) {
      const double *M = el0 + el * D::PER_EL + 30;
      double a = cf[0] * M[E.off[0]];
#pragma unroll
      for (int c = 1; c < 6; c++) a = fma(cf[c], M[E.off[c]], a);
      double *b = blk(el);
      b[lo] = a;
      if (lo != up) b[up] = a;
    }
  }
}

}  // namespace gbfem
