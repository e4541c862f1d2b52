// DG tetrahedron face integrals on the device, one CTA per owner element,
// FP64.  The reference's DG module is prism-only (apd_dg_prism); this is the
// interior-penalty form of its weak form (pds_conv_diff_weakform_dg.c:
// 232-1140) with the algebra of the prism face kernel (dg_face.cuh,
// dg_faces.cu) on affine tetrahedra:
//   rows i of e (side s_i), columns j of both sides (side s_j), per point q
//   of the face rule: a_q [ s_j phi_j (f g_i + s_i c phi_i) - s_i f phi_i g_j ],
// g = (A^T n) . grad phi = v . grad_xi phi with v = J^-1 A^T n constant per
// side (affine map), f = 1/2 inside and 1 on the Dirichlet boundary,
// c = pen min(p1, p2) / sqrt(area) (pen p1 / sqrt(area) on the boundary),
// n the unit normal out of the first neighbour, a_q = |ds| w_q.  The face
// rule is the triangle rule of the prism kernel for max(p1, p2) (order
// 2 max(p1, p2)); the point in each neighbour's reference coordinates comes
// through the face-vertex weights.  Basis: complete monomials xi^a eta^b
// zeta^c, a + b + c <= p, ordered by total degree, then a, then b
// descending.  Ownership as in the prism kernel: e's CTA writes e's rows of
// the off-diagonal blocks and adds its share of the diagonal block once.
//
// The derivatives of a monomial are monomials, v and n are constant on the face
// and the rule is exact for every product that occurs, so an entry needs only the
// face mass matrix S_ij = sum_q w_q phi_i phi_j of the two sides:
//   E_ij = |ds| [ s_j f sum_k v_i,k e_k(i) S_{i-k,j} + s_i s_j c S_ij
//                 - s_i f sum_k v_j,k e_k(j) S_{i,j-k} ],
// e_k(i) the exponent of direction k in phi_i and i - k the function with one
// less.  S depends on how the face sits in the two elements only (the owner's
// side, and which of the neighbour's vertices meets each of the owner's in
// ascending order: 4 x 24), and a lower degree's is the leading part: one table
// of 96 x 35 x 35 values for all degrees.  An entry is 7 FP64 operations
// instead of 4 nq (or 2 nq double-word products).  2,300 tetrahedra of each degree
// p = 1..4: 52, 84, 150, 346 us; 191, 247, 335, 721 us in double words over the points.

#include "dg_face.cuh"
#include "gbfem_internal.h"

namespace gbfem {

static __device__ const double tt_fq[GB_DG_PMAX][2][GB_DG_MAXNQF][3] = GB_DG_FQ_INIT;

// threads per CTA by the owner's degree: the diagonal share has NS^2 = 16,
// 100, 400, 1225 entries
__host__ __device__ constexpr int tt_threads(int p) { return p == 1 ? 32 : p == 2 ? 64 : p == 3 ? 128 : 256; }
constexpr int TT_NS = 35;   // functions for p = 4
constexpr int TT_NF = 4;    // faces of an owner

__host__ __device__ constexpr int tt_ns(int p) { return (p + 1) * (p + 2) * (p + 3) / 6; }

// function (a, b, c) in the order of the basis
__host__ __device__ constexpr int tt_index(int a, int b, int c) {
  return (a + b + c) * (a + b + c + 1) * (a + b + c + 2) / 6 + (b + c) * (b + c + 1) / 2 + c;
}
__device__ __forceinline__ void tt_exponents(int k, int (&e)[3]) {
  int d = 0, r = 0;
  while (tt_ns(d) <= k) d++;
  const int t = k - d * (d + 1) * (d + 2) / 6;
  while ((r + 1) * (r + 2) / 2 <= t) r++;
  e[0] = d - r;
  e[2] = t - r * (r + 1) / 2;
  e[1] = r - e[2];
}

// S of configuration blockIdx.x = 24 side + code: tab[cfg][j * 35 + i], i the
// owner's function, j the neighbour's, by the rule of degree 4
__global__ void dg_tet_face_table_kernel(double *__restrict__ tab) {
  __shared__ double mo[GB_DG_MAXNQF][TT_NS], mn[GB_DG_MAXNQF][TT_NS];
  constexpr int NQ = 16;
  const int side = blockIdx.x / 24, code = blockIdx.x % 24;
  int lo[3], ln[3];
  for (int i = 0, v = 0; v < 4; v++)
    if (v != side) lo[i++] = v;
  ln[0] = code / 6;
  ln[1] = code / 2 % 3;
  ln[1] += ln[1] >= ln[0];
  ln[2] = code % 2;
  const int x = min(ln[0], ln[1]), y = max(ln[0], ln[1]);
  ln[2] += ln[2] >= x;
  ln[2] += ln[2] >= y;
  for (int t = threadIdx.x; t < NQ * TT_NS * 2; t += blockDim.x) {
    const int sd = t % 2, k = t / 2 % TT_NS, q = t / 2 / TT_NS;
    const double *fq = tt_fq[GB_DG_PMAX - 1][0][q];
    const double w[3] = {1.0 - fq[0] - fq[1], fq[0], fq[1]};
    double X[3] = {0.0, 0.0, 0.0};
    for (int i = 0; i < 3; i++) {
      const int v = sd ? ln[i] : lo[i];
      if (v > 0) X[v - 1] += w[i];
    }
    int e[3];
    tt_exponents(k, e);
    double m = sd ? 1.0 : fq[2];
    for (int d = 0; d < 3; d++)
      for (int i = 0; i < e[d]; i++) m *= X[d];
    (sd ? mn : mo)[q][k] = m;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < TT_NS * TT_NS; t += blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < NQ; q++) s = fma(mo[q][t % TT_NS], mn[q][t / TT_NS], s);
    tab[(size_t)blockIdx.x * TT_NS * TT_NS + t] = s;
  }
}

template <int P, int T = tt_threads(P)>
__global__ void __launch_bounds__(T) dg_tet_faces_kernel(
    int count, const int *__restrict__ ent_el, const int *__restrict__ hf_ptr, const DgHalfFace *__restrict__ hf,
    const int *__restrict__ el_p, const int *__restrict__ el_nodes, const double *__restrict__ xyz,
    const double *__restrict__ k_el, const double *__restrict__ D_el, double pen, double gval,
    const double *__restrict__ tab, const long long *__restrict__ boff_diag, const int *__restrict__ roff,
    double *__restrict__ val, double *__restrict__ rhs) {
  constexpr int NS = tt_ns(P), NP = NS * (NS + 1) / 2, PER = (NP + T - 1) / T;
  __shared__ double sO[NS * NS], sN[TT_NS * NS];      // S owner-owner and owner-neighbour, [j][i]
  __shared__ double sV[TT_NF][2][3], sC[TT_NF][2];    // v of both sides; |ds|, |ds| c
  __shared__ double sCo[3][NS], sCn[3][TT_NS];        // |ds| f v_k e_k of the owner's and the neighbour's functions
  __shared__ signed char sDec[3][TT_NS], sExp[3][TT_NS];  // function with one less (itself if there is none), exponent
  const int bi = blockIdx.x, tid = threadIdx.x;
  if (bi >= count) return;
  const int e = ent_el[bi];
  for (int k = tid; k < TT_NS; k += T) {
    int x[3];
    tt_exponents(k, x);
    for (int d = 0; d < 3; d++) {
      sExp[d][k] = (signed char)x[d];
      sDec[d][k] = (signed char)(x[d] ? tt_index(x[0] - (d == 0), x[1] - (d == 1), x[2] - (d == 2)) : k);
    }
  }
  // diagonal share: thread's pairs (i <= j) of functions, both entries of each.  With
  // R_ij = sum_k v_k e_k(i) S_{i-k,j} entry (i, j) is so (R_ij - R_ji) + c S_ij: R_ij
  // and R_ji serve both
  double acc[PER], acd[PER];
  int pair[PER];
#pragma unroll
  for (int m = 0; m < PER; m++) {
    acc[m] = acd[m] = 0.0;
    const int k = min(tid + m * T, NP - 1);
    int j = (int)((sqrtf(8.0f * k + 1.0f) - 1.0f) * 0.5f);
    j += (j + 1) * (j + 2) / 2 <= k;
    j -= j * (j + 1) / 2 > k;
    pair[m] = (k - j * (j + 1) / 2) | j << 8;
  }
  double racc[(NS + T - 1) / T];
#pragma unroll
  for (int m = 0; m < (NS + T - 1) / T; m++) racc[m] = 0.0;
  const int h0 = hf_ptr[e], h1 = hf_ptr[e + 1];
  for (int h = h0; h < h1; h++) {
    const int slot = (h - h0) % TT_NF;
    __syncthreads();  // shared arrays of the previous face are free
    // the geometry of up to four faces at once, one thread a face and side
    if (slot == 0 && tid < 2 * TT_NF && h + tid / 2 < h1) {
      const int f = tid / 2, sd = tid & 1;
      const DgHalfFace F = hf[h + f];
      if (sd == 0 || F.el2 >= 0) {
        auto node = [&](int el, int v) -> v3 {
          const double *x = xyz + 3 * (size_t)el_nodes[4 * (size_t)el + v];
          return {x[0], x[1], x[2]};
        };
        // face vertices in face order from the first neighbour; the normal
        // points away from its vertex off the face (local index side1)
        const v3 va = node(F.el1, F.loc1[0]), vb = node(F.el1, F.loc1[1]), vc = node(F.el1, F.loc1[2]);
        const v3 ds = v3_cross(v3_sub(vb, va), v3_sub(vc, va));
        const double d = sqrt(v3_dot(ds, ds));
        v3 n = v3_scale(1.0 / d, ds);
        if (v3_dot(n, v3_sub(node(F.el1, F.side1), va)) > 0.0) n = v3_scale(-1.0, n);
        const int el = sd ? F.el2 : F.el1;
        double X[12], A[9];
        for (int v = 0; v < 4; v++) {
          const v3 x = node(el, v);
          X[3 * v] = x.x;
          X[3 * v + 1] = x.y;
          X[3 * v + 2] = x.z;
        }
        for (int r = 0; r < 9; r++) A[r] = D_el ? D_el[9 * (size_t)el + r] : (r % 4 == 0 ? (k_el ? k_el[el] : 1.0) : 0.0);
        const v3 v = tet_face_v(X, A, n);
        sV[f][sd][0] = v.x;
        sV[f][sd][1] = v.y;
        sV[f][sd][2] = v.z;
        if (sd == 0) {
          const int p1 = el_p[F.el1], p2 = F.el2 >= 0 ? el_p[F.el2] : p1;
          sC[f][0] = d;
          sC[f][1] = d * (pen * (p1 < p2 ? p1 : p2) / sqrt(0.5 * d));
        }
      }
    }
    const DgHalfFace F = hf[h];
    const bool interior = F.el2 >= 0;
    const int own = F.owner_is_2, ns_nb = interior ? tt_ns(el_p[own ? F.el1 : F.el2]) : 0;
    const unsigned char *lo = own ? F.loc2 : F.loc1, *ln = own ? F.loc1 : F.loc2;
    const double *to = tab + (size_t)tet_face_config(lo, lo) * TT_NS * TT_NS;
    for (int t = tid; t < NS * NS; t += T) sO[t] = to[t / NS * TT_NS + t % NS];
    if (interior) {
      const double *tn = tab + (size_t)tet_face_config(lo, ln) * TT_NS * TT_NS;
      for (int t = tid; t < NS * ns_nb; t += T) sN[t] = tn[t / NS * TT_NS + t % NS];
    }
    __syncthreads();
    const double so = own ? -1.0 : 1.0, df = sC[slot][0] * (interior ? 0.5 : 1.0), pc = sC[slot][1];
    for (int t = tid; t < 3 * (NS + ns_nb); t += T) {
      const int d = t % 3, k = t / 3;
      if (k < NS)
        sCo[d][k] = df * sV[slot][own][d] * sExp[d][k];
      else
        sCn[d][k - NS] = df * sV[slot][own ^ 1][d] * sExp[d][k - NS];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < PER; m++) {
      if (tid + m * T < NP) {
        const int i = pair[m] & 255, j = pair[m] >> 8;
        double r = 0.0, c = 0.0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
          r = fma(sCo[d][i], sO[sDec[d][i] + NS * j], r);
          c = fma(sCo[d][j], sO[sDec[d][j] + NS * i], c);
        }
        const double q = so * (r - c), g = pc * sO[i + NS * j];
        acc[m] += g + q;
        acd[m] += g - q;
      }
    }
    if (interior) {
      // block (e, neighbour): NS x ns_nb, column-major, leading dimension NS
      double *blk = val + F.blk;
      for (int k = tid; k < NS * ns_nb; k += T) {
        const int i = k % NS, j = k / NS;
        double r = 0.0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
          r = fma(sCo[d][i], sN[sDec[d][i] + NS * j], r);
          r = fma(sCn[d][j], sN[i + NS * sDec[d][j]], r);
        }
        blk[k] = -fma(so, r, pc * sN[k]);
      }
    } else {
#pragma unroll
      for (int m = 0; m < (NS + T - 1) / T; m++) {
        const int i = tid + m * T;
        if (i < NS) {
          double s = so * pc * sO[i];
#pragma unroll
          for (int d = 0; d < 3; d++) s = fma(sCo[d][i], sO[sDec[d][i]], s);
          racc[m] = fma(gval, s, racc[m]);
        }
      }
    }
  }
  if (h1 == h0) return;
  double *dblk = val + boff_diag[e];
#pragma unroll
  for (int m = 0; m < PER; m++) {
    if (tid + m * T >= NP) continue;
    const int i = pair[m] & 255, j = pair[m] >> 8;
    dblk[i + NS * j] += acc[m];
    if (i != j) dblk[j + NS * i] += acd[m];
  }
#pragma unroll
  for (int m = 0; m < (NS + T - 1) / T; m++) {
    const int i = tid + m * T;
    if (i < NS) rhs[roff[e] + i] += racc[m];
  }
}

long long dg_tet_face_table_size() { return 96LL * TT_NS * TT_NS; }

int launch_dg_tet_face_table(cudaStream_t st, double *tab) {
  dg_tet_face_table_kernel<<<96, 256, 0, st>>>(tab);
  GB_CUDA(cudaGetLastError());
  return 1;
}

int launch_dg_tet_faces(cudaStream_t st, int p, int count, const int *ent_el, const int *hf_ptr,
                        const DgHalfFace *hf, const int *el_p, const int *el_nodes, const double *xyz,
                        const double *k_el, const double *D_el, double pen, double g, const double *tab,
                        const long long *boff_diag, const int *roff, double *val, double *rhs) {
  if (count <= 0) return 0;
  GB_CHECK(p >= 1 && p <= GB_DG_PMAX, "DG degree must be 1..4");
#define GB_TT_LAUNCH(PP)                                                                                      \
  dg_tet_faces_kernel<PP><<<count, tt_threads(PP), 0, st>>>(count, ent_el, hf_ptr, hf, el_p, el_nodes, xyz,   \
                                                            k_el, D_el, pen, g, tab, boff_diag, roff, val, rhs)
  switch (p) {
    case 1: GB_TT_LAUNCH(1); break;
    case 2: GB_TT_LAUNCH(2); break;
    case 3: GB_TT_LAUNCH(3); break;
    default: GB_TT_LAUNCH(4); break;
  }
#undef GB_TT_LAUNCH
  GB_CUDA(cudaGetLastError());
  return 1;
}

}  // namespace gbfem
