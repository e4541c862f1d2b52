// DG prism face integrals from moments of the face geometry (FP64): the
// faces between prisms and their Dirichlet faces, all degrees 1..4.
//
// Reference: pdr_conv_diff_comp_fa_stiff_mat_app of the DG weak form
// (pds_conv_diff_weakform_dg.c:232-1140); the form is restated in
// dg_face.cuh.  With n out of side 1, s_1 = 1, s_2 = -1, the point fields
//   F_0 = c a,  (F_1, F_2, F_3) = f a v_1,  (F_4, F_5, F_6) = f a v_2
// (a = |ds| w, v_s = J_s^-1 A_s^T n, f = 1/2 inside, 1 on the boundary) give
//   diagonal block of side o:  K_ij = sum_q s_o f a (g_i phi_j - phi_i g_j) + c a phi_i phi_j,
//   block (1, 2):              K_ij = -N_ij - S_ij,   block (2, 1): K_ji = N_ij - S_ij,
//     N_ij = sum_q f a (g_i phi_j + phi_i g_j),  S_ij = sum_q c a phi_i phi_j,
//   load (boundary):           R_i = gD sum_q (a g_i + c a phi_i).
// The basis is monomial, g = v . grad phi lowers one exponent, and on a face
// all local coordinates are products of a few one-variable functions:
//  - a quadrilateral is an edge of the triangle (vertex weights x_A = 1 - s,
//    x_B = s in both elements) times zeta = +- z, and the rule is a tensor
//    product: sums over z first (per edge point and power of z), then over s
//    against x_A^i x_B^j;
//  - a triangle has zeta = +-1, so a function depends on its zeta exponent
//    through a sign only, and its pairs reduce to pairs of triangle
//    monomials.
// The diagonal share of all faces of an element needs only
// sum_faces s_o F xi^i eta^j zeta^k, so the moments of the faces are added
// before the entries are formed (4 FMA and an add per pair of entries); the
// off-diagonal blocks of a face are formed together, because N and S are
// shared.  p = 3: a quadrilateral takes 460 FP64 warp instructions for both
// blocks and a triangle 450, an element's diagonal share 550, against 3,800,
// 3,000 and 5,600 of the sums over the points (2 nq FMA an entry).  Every
// term keeps its sign pattern (x_A, x_B, xi, eta >= 0), so the error is that
// of an FP64 dot product.  Measured (GB300), all faces: p = 3, 54,000 prisms
// 48.1 -> 5.9 ms; p = 1 / 2 / 4: 12 / 35 / 330 ns an element.  Each entry is written by one thread in a fixed
// order: deterministic.
//
// The split needs the edge of a quadrilateral to be an edge of the triangle
// in both its elements (always so where prisms are stacked in columns); the
// host checks it, and a mesh with a quadrilateral turned by 90 degrees
// between its neighbours keeps the sums over the points (dg_faces.cu).

#include "dg_face.cuh"
#include "gbfem_internal.h"

#include <algorithm>
#include <mutex>

namespace gbfem {

__device__ const double m_fq[GB_DG_PMAX][2][GB_DG_MAXNQF][3] = GB_DG_FQ_INIT;
__device__ const unsigned char m_exp[GB_DG_PMAX][GB_DG_MAXNS][3] = GB_DG_EXP_INIT;
__device__ const int m_ns[GB_DG_PMAX + 1] = GB_DG_NS_INIT;

__host__ __device__ constexpr int fm_tri(int d) { return (d + 1) * (d + 2) / 2; }
__host__ __device__ constexpr int fm_mono(int i, int j) { return (i + j) * (i + j + 1) / 2 + j; }
constexpr int FM_MONO = fm_tri(2 * GB_DG_PMAX);  // monomials of degree <= 8
constexpr int FM_ZP = 2 * GB_DG_PMAX + 1;        // powers of z
constexpr int FM_Q1 = GB_DG_PMAX + 1;            // line points
constexpr int FM_QT = 16;                        // triangle points

// One pair of entries (u, w), u <= w, of a diagonal block: offsets of the
// moments M0, M1, M2, M3 and the coefficients of M1..M3 plus 4
struct DgFaceEntry {
  unsigned short off[4];
  unsigned char coef[3], u, w, pad[3];
};

// Reference tables of a device: powers of the line points Z[rule][n][k],
// edge monomials XE[rule][mono][m], triangle monomials XT[rule][perm][mono][q]
// (perm = 3 i1 + i2: face vertices at the element's triangle vertices 1, 2),
// the diagonal entries per degree and the exponents of the monomials
struct DgFaceTables {
  const double *Z, *XE, *XT;
  const DgFaceEntry *ENT[GB_DG_PMAX + 1];
  const unsigned char *MON;  // [mono][2]
};

static DgFaceTables g_fm[64];
static bool g_fm_ready[64];
static std::mutex g_fm_lock;  // contexts are made and used from several threads

// moments of a diagonal block: M0 [T(2P)][2P+1], M1, M2 [T(2P-1)][2P+1], M3 [T(2P)][2P]
template <int P>
struct FmDiag {
  static constexpr int NS = P == 1 ? 6 : P == 2 ? 18 : P == 3 ? 40 : 75;
  static constexpr int K = 2 * P + 1, T2 = fm_tri(2 * P), T1 = fm_tri(2 * P - 1);
  static constexpr int O1 = T2 * K, O2 = O1 + T1 * K, O3 = O2 + T1 * K, NM = O3 + T2 * (K - 1);
  static constexpr int NT = 2 * T2 + 2 * T1;  // monomial sums of a triangle
};

static int fm_tables(int device, DgFaceTables *out) {
  GB_CHECK(device >= 0 && device < 64, "device index out of range");
  std::lock_guard<std::mutex> hold(g_fm_lock);
  if (!g_fm_ready[device]) {
    static const double FQ[GB_DG_PMAX][2][GB_DG_MAXNQF][3] = GB_DG_FQ_INIT;
    std::vector<double> Z(4 * FM_Q1 * FM_ZP, 0.0), XE(4 * FM_MONO * FM_Q1, 0.0), XT(4 * 9 * FM_MONO * FM_QT, 0.0);
    std::vector<unsigned char> MON(2 * FM_MONO);
    for (int d = 0; d <= 2 * GB_DG_PMAX; d++)
      for (int j = 0; j <= d; j++) {
        MON[2 * fm_mono(d - j, j)] = (unsigned char)(d - j);
        MON[2 * fm_mono(d - j, j) + 1] = (unsigned char)j;
      }
    for (int r = 0; r < 4; r++) {
      const int Q1 = r + 2, nt = GB_DG_NQF[r + 1][0];
      for (int n = 0; n < Q1; n++) {
        const double z = FQ[r][1][n][1], xb = 0.5 + 0.5 * z, xa = 0.5 - 0.5 * z;
        double p = 1.0;
        for (int k = 0; k < FM_ZP; k++, p *= z) Z[(r * FM_Q1 + n) * FM_ZP + k] = p;
        for (int a = 0; a < FM_MONO; a++) {
          double v = 1.0;
          for (int i = 0; i < MON[2 * a]; i++) v *= xa;
          for (int j = 0; j < MON[2 * a + 1]; j++) v *= xb;
          XE[(r * FM_MONO + a) * FM_Q1 + n] = v;
        }
      }
      for (int q = 0; q < nt; q++) {
        const double b[3] = {1.0 - FQ[r][0][q][0] - FQ[r][0][q][1], FQ[r][0][q][0], FQ[r][0][q][1]};
        for (int pm = 0; pm < 9; pm++)
          for (int a = 0; a < FM_MONO; a++) {
            double v = 1.0;
            for (int i = 0; i < MON[2 * a]; i++) v *= b[pm / 3];
            for (int j = 0; j < MON[2 * a + 1]; j++) v *= b[pm % 3];
            XT[((r * 9 + pm) * FM_MONO + a) * FM_QT + q] = v;
          }
      }
    }
    DgFaceTables &T = g_fm[device];
    auto up = [](auto **d, const auto &h) -> int {
      void *p = nullptr;
      GB_CUDA(cudaMalloc(&p, h.size() * sizeof(h[0])));
      GB_CUDA(cudaMemcpy(p, h.data(), h.size() * sizeof(h[0]), cudaMemcpyHostToDevice));
      *d = static_cast<std::remove_reference_t<decltype(**d)> *>(p);
      return 0;
    };
    GB_TRY(up(&T.Z, Z));
    GB_TRY(up(&T.XE, XE));
    GB_TRY(up(&T.XT, XT));
    GB_TRY(up(&T.MON, MON));
    for (int p = 1; p <= GB_DG_PMAX; p++) {
      const int ns = GB_DG_NS[p], K = 2 * p + 1, T2 = fm_tri(2 * p), T1 = fm_tri(2 * p - 1);
      std::vector<DgFaceEntry> E;
      for (int u = 0; u < ns; u++)
        for (int w = u; w < ns; w++) {
          const unsigned char *x = GB_DG_EXP[p - 1][u], *y = GB_DG_EXP[p - 1][w];
          const int i = x[0] + y[0], j = x[1] + y[1], k = x[2] + y[2];
          DgFaceEntry e{};
          e.u = (unsigned char)u;
          e.w = (unsigned char)w;
          for (int d = 0; d < 3; d++) e.coef[d] = (unsigned char)(4 + (int)y[d] - (int)x[d]);
          e.off[0] = (unsigned short)(fm_mono(i, j) * K + k);
          // (a zero coefficient goes with the block's first moment)
          e.off[1] = (unsigned short)(T2 * K + (y[0] != x[0] ? fm_mono(i - 1, j) * K + k : 0));
          e.off[2] = (unsigned short)(T2 * K + T1 * K + (y[1] != x[1] ? fm_mono(i, j - 1) * K + k : 0));
          e.off[3] = (unsigned short)(T2 * K + 2 * T1 * K + (y[2] != x[2] ? fm_mono(i, j) * (K - 1) + k - 1 : 0));
          E.push_back(e);
        }
      GB_TRY(up(&T.ENT[p], E));
    }
    g_fm_ready[device] = true;
  }
  *out = g_fm[device];
  return 0;
}

bool dg_face_moments_cover(const DgFaceRec &r) {
  auto shape = [&](const unsigned char *l) -> int {  // -1 unsuitable, else which rule direction runs along the edge
    if (r.nfv == 3) {
      const int lev = l[0] / 3, a = l[0] % 3, b = l[1] % 3, c = l[2] % 3;
      return l[1] / 3 == lev && l[2] / 3 == lev && a != b && b != c && a != c ? 0 : -1;
    }
    auto edge = [&](int i, int j) { return l[i] / 3 == l[j] / 3 && l[i] % 3 != l[j] % 3; };
    auto vert = [&](int i, int j) { return l[i] / 3 != l[j] / 3 && l[i] % 3 == l[j] % 3; };
    if (edge(0, 1) && edge(3, 2) && vert(0, 3) && vert(1, 2)) return 0;
    if (edge(0, 3) && edge(1, 2) && vert(0, 1) && vert(3, 2)) return 1;
    return -1;
  };
  const int s1 = shape(r.loc1);
  return s1 >= 0 && (r.el2 < 0 || shape(r.loc2) == s1);
}

// ---------------------------------------------------------------- geometry
// The point fields of every face, by groups with the same rule (nq points,
// degree pr, ti 0 triangles, 1 quadrilaterals), all in one launch: geo[f * nq + q]
// of face slot f.  NF faces per CTA: the vertex differences of both sides
// first, then one or two points a thread.  FP64-bound (about 180 instructions a point)
// where there are many faces (162,000: 720 us); a launch a group, each
// waiting for its loads and one long chain a thread, took 34 us at 2,000 prisms
// of p = 2 (68 us for both groups, 31 us in one launch of one point a
// thread) and 46 us each for the eight groups of 8,000 prisms of p = 1..4
// (368 us, 135 us).
constexpr int FG_THREADS = 128;
struct DgFieldGroup {
  int block, first, count, NF, nq, pr, ti;
};
struct DgFieldGroups {
  DgFieldGroup g[8];
};
__global__ void __launch_bounds__(FG_THREADS) dg_face_fields_kernel(
    DgFieldGroups groups, int ngroups, const DgFaceRec *__restrict__ rec, const int *__restrict__ el_nodes,
    const double *__restrict__ xyz, const double *__restrict__ k_el, const double *__restrict__ D_el, double pen,
    double *__restrict__ geo) {
  int gi = 0;
  while (gi + 1 < ngroups && (int)blockIdx.x >= groups.g[gi + 1].block) gi++;
  const int NF = groups.g[gi].NF, nq = groups.g[gi].nq, pr = groups.g[gi].pr, ti = groups.g[gi].ti;
  extern __shared__ double smem[];  // [NF][2][30] differences and tensor, [NF] penalty / sqrt(area)
  const int at = (blockIdx.x - groups.g[gi].block) * NF, nf = min(NF, groups.g[gi].count - at);
  const int first = groups.g[gi].first + at, tid = threadIdx.x;
  double *sPen = smem + 60 * NF;
  for (int t = tid; t < nf * 60; t += FG_THREADS) {
    const DgFaceRec &R = rec[first + t / 60];
    const int r = t % 60, s = r / 30, i = r % 30, e = s ? R.el2 : R.el1;
    double v = 0.0;
    if (e >= 0) {
      if (i < 21) {
        // X1-X0, X4-X3, X2-X0, X5-X3, X3-X0, X4-X1, X5-X2 (see dg_volume.cuh)
        const int g = i / 3, d = i % 3;
        const int hi = g == 0 ? 1 : g == 1 ? 4 : g == 2 ? 2 : g == 3 ? 5 : g - 1;
        const int lo = g == 0 || g == 2 ? 0 : g == 1 || g == 3 ? 3 : g - 4;
        const int *en = el_nodes + 6 * (size_t)e;
        v = xyz[3 * (size_t)en[hi] + d] - xyz[3 * (size_t)en[lo] + d];
      } else {
        const int k = i - 21;
        v = D_el ? D_el[9 * (size_t)e + k] : (k % 4 == 0 ? (k_el ? k_el[e] : 1.0) : 0.0);
      }
    }
    smem[t] = v;
  }
  for (int f = tid; f < nf; f += FG_THREADS) {
    const DgFaceRec &R = rec[first + f];
    v3 V[4];
    for (int i = 0; i < 4; i++) {
      const double *x = xyz + 3 * (size_t)el_nodes[6 * (size_t)R.el1 + R.loc1[i < R.nfv ? i : 0]];
      V[i] = {x[0], x[1], x[2]};
    }
    const int pp = R.el2 >= 0 && R.p2 < R.p1 ? R.p2 : R.p1;
    sPen[f] = pen * pp / sqrt(dg_face_area(V, R.nfv));
  }
  __syncthreads();
  for (int t = tid; t < nf * nq; t += FG_THREADS) {
    const int f = t / nq, q = t - f * nq;
    const DgFaceRec &R = rec[first + f];
    const double s = m_fq[pr - 1][ti][q][0], tt = m_fq[pr - 1][ti][q][1], w = m_fq[pr - 1][ti][q][2];
    v3 n = {0.0, 0.0, 0.0};
    double fa = 0.0;
    double *g = geo + R.geo + q;
    for (int sd = 0; sd < 2; sd++) {
      if (sd == 1 && R.el2 < 0) {
        for (int c = 4; c < 7; c++) g[(size_t)c * nq] = 0.0;
        break;
      }
      const unsigned char *l = sd ? R.loc2 : R.loc1;
      double xi = 0.0, eta = 0.0, zeta;
      if (ti == 0) {
        const double b[3] = {1.0 - s - tt, s, tt};
        for (int i = 0; i < 3; i++) {
          if (l[i] % 3 == 1) xi = b[i];
          if (l[i] % 3 == 2) eta = b[i];
        }
        zeta = l[0] < 3 ? -1.0 : 1.0;
      } else {
        const bool along_s = l[0] / 3 == l[1] / 3;  // the first rule direction runs along the triangle's edge
        const double e = along_s ? s : tt, z = along_s ? tt : s;
        const int A = l[0] % 3, B = (along_s ? l[1] : l[3]) % 3;
        const double xa = 0.5 - 0.5 * e, xb = 0.5 + 0.5 * e;
        xi = A == 1 ? xa : B == 1 ? xb : 0.0;
        eta = A == 2 ? xa : B == 2 ? xb : 0.0;
        zeta = l[0] < 3 ? z : -z;
      }
      const double *B = smem + 60 * f + 30 * sd, *A = B + 21;
      const double lo = 0.5 - 0.5 * zeta, hi = 0.5 + 0.5 * zeta, l1 = 0.5 * xi, l2 = 0.5 * eta, l0 = 0.5 - l1 - l2;
      const v3 ea = {B[0], B[1], B[2]}, eb = {B[3], B[4], B[5]}, fA = {B[6], B[7], B[8]}, fB = {B[9], B[10], B[11]};
      const v3 d0 = {B[12], B[13], B[14]}, d1 = {B[15], B[16], B[17]}, d2 = {B[18], B[19], B[20]};
      const v3 j1 = v3_fma(lo, ea, v3_scale(hi, eb)), j2 = v3_fma(lo, fA, v3_scale(hi, fB)),
               j3 = v3_fma(l0, d0, v3_fma(l1, d1, v3_scale(l2, d2)));
      const v3 c1 = v3_cross(j2, j3), c2 = v3_cross(j3, j1), c3 = v3_cross(j1, j2);
      if (sd == 0) {
        // outward side vector of side 1 (prism_side_vector): -c3, c3, -c2,
        // c1 + c2, -c1
        const v3 ds = R.side1 == 0   ? v3_scale(-1.0, c3)
                      : R.side1 == 1 ? c3
                      : R.side1 == 2 ? v3_scale(-1.0, c2)
                      : R.side1 == 3 ? v3{c1.x + c2.x, c1.y + c2.y, c1.z + c2.z}
                                     : v3_scale(-1.0, c1);
        const double d = sqrt(v3_dot(ds, ds));
        n = v3_scale(1.0 / d, ds);
        const double a = d * w;
        fa = R.el2 >= 0 ? 0.5 * a : a;
        g[0] = sPen[f] * a;
      }
      const double r = fa / v3_dot(j1, c1);
      const v3 an = {A[0] * n.x + A[3] * n.y + A[6] * n.z, A[1] * n.x + A[4] * n.y + A[7] * n.z,
                     A[2] * n.x + A[5] * n.y + A[8] * n.z};
      g[(size_t)(1 + 3 * sd) * nq] = v3_dot(c1, an) * r;
      g[(size_t)(2 + 3 * sd) * nq] = v3_dot(c2, an) * r;
      g[(size_t)(3 + 3 * sd) * nq] = v3_dot(c3, an) * r;
    }
  }
}

// ---------------------------------------------------------- element shares
__device__ __forceinline__ double flip(double v, int neg) {  // the sign on the integer side, not the FP64 pipe
  return __longlong_as_double(__double_as_longlong(v) ^ ((long long)(neg & 1) << 63));
}

// (NaN or infinity, on the integer side.)  Where a derivative of a function is
// identically zero, or the function on the face, its moment is left out, and a field
// that is not finite (a coefficient that is not, a face without an area) would leave
// no trace in the entry; the sums over the points multiply it by zero, which is NaN.
// So it is looked for.
__device__ __forceinline__ int fm_nonfinite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

// How a quadrilateral lies in one of its elements: triangle vertices A, B of
// its edge (x_A = 1 - s, x_B = s), whether zeta runs against the rule.
struct FmQuad {
  int A, B, down, along_s;
  __device__ FmQuad(const unsigned char *l) {
    along_s = l[0] / 3 == l[1] / 3;
    A = l[0] % 3;
    B = (along_s ? l[1] : l[3]) % 3;
    down = l[0] >= 3;
  }
  // xi^i eta^j on the edge as x_A^eA x_B^eB; false: identically zero
  __device__ bool trace(int i, int j, int &eA, int &eB) const {
    const int off = 3 - A - B;  // the vertex not on the edge
    if ((off == 1 && i) || (off == 2 && j)) return false;
    eA = A == 1 ? i : A == 2 ? j : 0;
    eB = B == 1 ? i : B == 2 ? j : 0;
    return true;
  }
};

// Per owner element of degree P: the diagonal share of its faces and the
// boundary load, added to the block and rows the volume kernel wrote.
// Stages: fields to shared memory; line sums of the quadrilaterals and
// monomial sums of the triangles; moments over all faces; entries.
template <int P, int THR>
__global__ void __launch_bounds__(THR) dg_face_diag_kernel(
    int count, const int *__restrict__ ent_el, const int *__restrict__ hf_ptr, const int *__restrict__ hrec,
    const DgFaceRec *__restrict__ rec, const double *__restrict__ geo, DgFaceTables tb, double gval,
    const long long *__restrict__ boff_diag, const int *__restrict__ roff, double *__restrict__ val,
    double *__restrict__ rhs) {
  using D = FmDiag<P>;
  constexpr int NS = D::NS, K = D::K, T1 = D::T1, T2 = D::T2;
  constexpr int QM = FM_Q1, ZS = FM_Q1;  // line points, row stride of the line sums
  constexpr int NZ = 4 * K * QM;
  __shared__ double sF[5][4 * QM * QM];
  __shared__ double sS[3][4 * K * ZS];  // line sums [field][k][m] of the quadrilaterals
  __shared__ double sT[2][D::NT];       // monomial sums of the triangles
  __shared__ double sM[D::NM];
  __shared__ double sC[9];              // the doubles -4 .. 4
  __shared__ DgFaceRec sR[5];
  __shared__ int sOwn[5], sQuad[3], sTri[2], sBad;
  const int tid = threadIdx.x, e = ent_el[blockIdx.x];
  const int h0 = hf_ptr[e], nf = hf_ptr[e + 1] - h0;
  if (nf == 0) return;
  if (tid < 9) sC[tid] = (double)(tid - 4);
  if (tid == 0) sBad = 0;
  if (tid < nf) {
    const int h = hrec[h0 + tid];
    sR[tid] = rec[h >> 1];
    sOwn[tid] = h & 1;
  }
  __syncthreads();
  if (tid == 0) {
    int q = 0, t = 0;
    for (int f = 0; f < nf; f++)
      if (sR[f].nfv == 4)
        sQuad[q++] = f;
      else
        sTri[t++] = f;
    for (; q < 3; q++) sQuad[q] = -1;
    for (; t < 2; t++) sTri[t] = -1;
  }
  // fields of the owner's side with its sign
  int bad = 0;  // 1: a field of any face is not finite, 3: of a Dirichlet face
  for (int f = 0; f < nf; f++) {
    const DgFaceRec &R = sR[f];
    const int pm = R.el2 >= 0 && R.p2 > R.p1 ? R.p2 : R.p1;
    const int nq = R.nfv == 4 ? (pm + 1) * (pm + 1) : (pm == 1 ? 3 : pm == 2 ? 6 : pm == 3 ? 12 : 16);
    const double *g = geo + R.geo;
    const int o = sOwn[f];
    for (int t = tid; t < 4 * nq; t += THR) {
      const int c = t / nq, q = t - c * nq;
      const double v = g[(size_t)(c == 0 ? 0 : c + 3 * o) * nq + q];
      sF[f][t] = c == 0 ? v : flip(v, o);
      if (fm_nonfinite(v)) bad |= R.el2 < 0 ? 3 : 1;
    }
  }
  if (bad) atomicOr(&sBad, bad);
  __syncthreads();
  bad = sBad;
  for (int t = tid; t < 3 * NZ; t += THR) {
    const int qi = t / NZ, f = sQuad[qi];
    if (f < 0) break;  // (the quadrilaterals come first)
    const DgFaceRec &R = sR[f];
    const int pm = R.el2 >= 0 && R.p2 > R.p1 ? R.p2 : R.p1, Q1 = pm + 1;
    const int r = t - qi * NZ, c = r / (K * QM), k = (r / QM) % K, m = r % QM;
    if (m >= Q1) continue;
    const unsigned char *l = sOwn[f] ? R.loc2 : R.loc1;
    const bool along_s = l[0] / 3 == l[1] / 3;
    const double *F = sF[f] + c * Q1 * Q1 + (along_s ? m * Q1 : m), *Z = tb.Z + (size_t)(pm - 1) * FM_Q1 * FM_ZP + k;
    const int st = along_s ? 1 : Q1;
    double a = 0.0;
    for (int n = 0; n < Q1; n++) a = fma(F[n * st], __ldg(Z + n * FM_ZP), a);
    sS[qi][(c * K + k) * ZS + m] = flip(a, (l[0] >= 3) & k);
  }
  for (int t = tid; t < 2 * D::NT; t += THR) {
    const int ti = t / D::NT, f = sTri[ti], r = t - ti * D::NT;
    if (f < 0) {
      sT[ti][r] = 0.0;
      continue;
    }
    const DgFaceRec &R = sR[f];
    const int pm = R.el2 >= 0 && R.p2 > R.p1 ? R.p2 : R.p1, nq = pm == 1 ? 3 : pm == 2 ? 6 : pm == 3 ? 12 : 16;
    const int c = r < T2 ? 0 : r < T2 + T1 ? 1 : r < T2 + 2 * T1 ? 2 : 3;
    const int al = r - (c == 0 ? 0 : c == 1 ? T2 : c == 2 ? T2 + T1 : T2 + 2 * T1);
    const unsigned char *l = sOwn[f] ? R.loc2 : R.loc1;
    const int i1 = l[0] % 3 == 1 ? 0 : l[1] % 3 == 1 ? 1 : 2, i2 = l[0] % 3 == 2 ? 0 : l[1] % 3 == 2 ? 1 : 2;
    const double *X = tb.XT + ((size_t)((pm - 1) * 9 + 3 * i1 + i2) * FM_MONO + al) * FM_QT, *F = sF[f] + c * nq;
    double a = 0.0;
    for (int q = 0; q < nq; q++) a = fma(F[q], __ldg(X + q), a);
    sT[ti][r] = a;
  }
  __syncthreads();
  // moments: field c, monomial al, power k, summed over the faces in order
  // (monomials on an axis before the others, so that the warps whose
  // monomials vanish on two of the three edges skip those edges together)
  for (int t = tid; t < D::NM; t += THR) {
    const int c = t < D::O1 ? 0 : t < D::O2 ? 1 : t < D::O3 ? 2 : 3;
    const int kc = c == 3 ? K - 1 : K, dg = c == 0 || c == 3 ? 2 * P : 2 * P - 1;
    const int r = t - (c == 0 ? 0 : c == 1 ? D::O1 : c == 2 ? D::O2 : D::O3), ia = r / kc, k = r - ia * kc;
    int i, j;
    if (ia <= dg) {
      i = ia;
      j = 0;
    } else if (ia <= 2 * dg) {
      i = 0;
      j = ia - dg;
    } else {
      const int b = ia - 2 * dg - 1;  // both exponents >= 1: (i - 1, j - 1) in graded order
      i = tb.MON[2 * b] + 1;
      j = tb.MON[2 * b + 1] + 1;
    }
    double a = 0.0;
    for (int qi = 0; qi < 3; qi++) {
      const int f = sQuad[qi];
      if (f < 0) break;
      const DgFaceRec &R = sR[f];
      const FmQuad Q(sOwn[f] ? R.loc2 : R.loc1);
      int eA, eB;
      if (!Q.trace(i, j, eA, eB)) continue;
      const int pm = R.el2 >= 0 && R.p2 > R.p1 ? R.p2 : R.p1;
      const double *S = sS[qi] + (c * K + k) * ZS, *X = tb.XE + ((size_t)(pm - 1) * FM_MONO + fm_mono(eA, eB)) * FM_Q1;
      for (int m = 0; m <= pm; m++) a = fma(S[m], __ldg(X + m), a);
    }
    const int ot = (c == 0 ? 0 : c == 1 ? T2 : c == 2 ? T2 + T1 : T2 + 2 * T1) + fm_mono(i, j);
    for (int ti = 0; ti < 2; ti++) {
      const int f = sTri[ti];
      if (f < 0) break;
      const unsigned char *l = sOwn[f] ? sR[f].loc2 : sR[f].loc1;
      a += flip(sT[ti][ot], (l[0] < 3) & k);
    }
    sM[(c == 0 ? 0 : c == 1 ? D::O1 : c == 2 ? D::O2 : D::O3) + fm_mono(i, j) * kc + k] = a;
  }
  // boundary load: R_i = g sum (F . grad phi_i + F_0 phi_i) over the Dirichlet
  // faces (their first neighbour owns them)
  for (int i = tid; i < NS; i += THR) {
    const int a = m_exp[P - 1][i][0], b = m_exp[P - 1][i][1], c = m_exp[P - 1][i][2];
    double s = 0.0;
    bool any = false;
    for (int qi = 0; qi < 3; qi++) {
      const int f = sQuad[qi];
      if (f < 0) break;
      if (sR[f].el2 >= 0) continue;
      any = true;
      const FmQuad Q(sR[f].loc1);
      const double *S = sS[qi], *X = tb.XE + (size_t)(sR[f].p1 - 1) * FM_MONO * FM_Q1;
      int eA, eB;
      auto term = [&](int ii, int jj, int cc, int k, double cf) {
        if (!Q.trace(ii, jj, eA, eB)) return;
        const double *Y = X + fm_mono(eA, eB) * FM_Q1;
        double v = 0.0;
        for (int m = 0; m <= sR[f].p1; m++) v = fma(S[(cc * K + k) * ZS + m], __ldg(Y + m), v);
        s = fma(cf, v, s);
      };
      if (a) term(a - 1, b, 1, c, sC[4 + a]);
      if (b) term(a, b - 1, 2, c, sC[4 + b]);
      if (c) term(a, b, 3, c - 1, sC[4 + c]);
      term(a, b, 0, c, 1.0);
    }
    for (int ti = 0; ti < 2; ti++) {
      const int f = sTri[ti];
      if (f < 0) break;
      if (sR[f].el2 >= 0) continue;
      any = true;
      const double *T = sT[ti];
      const int dn = sR[f].loc1[0] < 3;  // zeta = -1
      double v = T[fm_mono(a, b)];
      if (a) v = fma(sC[4 + a], T[T2 + fm_mono(a - 1, b)], v);
      if (b) v = fma(sC[4 + b], T[T2 + T1 + fm_mono(a, b - 1)], v);
      if (c) v = fma(flip(sC[4 + c], dn), T[T2 + 2 * T1 + fm_mono(a, b)], v);
      s += flip(v, dn & c);
    }
    if (any) {
      double *r = rhs + roff[e] + i;
      *r = bad & 2 ? nan("") : fma(gval, s, *r);
    }
  }
  __syncthreads();
  // entries: rows w, u of columns u, w: S + N and S - N
  double *blk = val + boff_diag[e];
  for (int t = tid; t < NS * (NS + 1) / 2; t += THR) {
    const DgFaceEntry E = tb.ENT[P][t];
    const double S = bad ? nan("") : sM[E.off[0]];
    const double N = fma(sC[E.coef[0]], sM[E.off[1]], fma(sC[E.coef[1]], sM[E.off[2]], sC[E.coef[2]] * sM[E.off[3]]));
    double *lo = blk + E.w + NS * E.u, *up = blk + E.u + NS * E.w;
    if (lo == up) {
      *lo += S;
    } else {
      const double x = *lo, y = *up;
      *lo = x + (S + N);
      *up = y + (S - N);
    }
  }
}

// -------------------------------------------------------- off-diagonal blocks
// Both blocks of every interior face whose larger degree is PM: one CTA a
// face.  Quadrilaterals: line sums, moments W_c (c = 0..6) over x_A^i x_B^j
// and z^k, then E = sum over the triangle parts of the gradients per pair of
// triangle monomials and power, then N = E + c W_3 + c' W_6 and S = W_0 per
// entry.  Triangles: the same with the pair sums over the points directly.
template <int PM, bool QUAD>
struct FmOff {
  static constexpr int Q1 = PM + 1, NQ = QUAD ? Q1 * Q1 : (PM == 1 ? 3 : PM == 2 ? 6 : PM == 3 ? 12 : 16);
  static constexpr int DM = 2 * PM, K = DM + 1, NT = fm_tri(PM);
  // doubles: fields, then (QUAD) line sums, moments, pair sums; (triangles)
  // basis and gradient values of both sides and weighted values of side 2, pair sums
  static constexpr int F = 7 * NQ;
  static constexpr int S = QUAD ? 7 * K * (Q1 | 1) : 0;
  static constexpr int W = QUAD ? fm_tri(DM) * K + 4 * fm_tri(DM - 1) * K + 2 * fm_tri(DM) * (K - 1) + 3 * K : 7 * NT * (NQ | 1);
  static constexpr int E = QUAD ? NT * NT * K : 4 * NT * NT;
  static constexpr int DOUBLES = F + S + W + E + 8;
  static constexpr int INFO = QUAD ? 5 * NT * NT : 0;  // shorts
  static constexpr int BYTES = 8 * DOUBLES + 2 * ((INFO + 3) / 4 * 4);
  static constexpr int THR = PM == 1 ? 32 : PM == 2 ? 64 : 128;
};

template <int PM, bool QUAD>
__global__ void __launch_bounds__(FmOff<PM, QUAD>::THR) dg_face_blocks_kernel(
    const DgFaceRec *__restrict__ rec, const double *__restrict__ geo, DgFaceTables tb, double *__restrict__ val) {
  using D = FmOff<PM, QUAD>;
  constexpr int THR = D::THR, NQ = D::NQ, Q1 = D::Q1;
  extern __shared__ double smem[];
  double *sF = smem, *sC = sF + D::F, *sS = sC + 8, *sW = sS + D::S, *sE = sW + D::W;
  unsigned short *sI = reinterpret_cast<unsigned short *>(sE + D::E);
  __shared__ unsigned char sFn[2][GB_DG_MAXNS][2];  // (triangle monomial, zeta exponent) of each function
  const DgFaceRec R = rec[blockIdx.x];
  const int tid = threadIdx.x, p1 = R.p1, p2 = R.p2, ns1 = m_ns[p1], ns2 = m_ns[p2];
  const int nt1 = fm_tri(p1), nt2 = fm_tri(p2), npair = nt1 * nt2, DD = p1 + p2, K = DD + 1;
  if (tid < 5) sC[tid] = (double)tid;
  for (int t = tid; t < ns1 + ns2; t += THR) {
    const int sd = t >= ns1, u = sd ? t - ns1 : t;
    const unsigned char *x = m_exp[(sd ? p2 : p1) - 1][u];
    sFn[sd][u][0] = (unsigned char)fm_mono(x[0], x[1]);
    sFn[sd][u][1] = x[2];
  }
  int bad = 0;
  for (int t = tid; t < D::F; t += THR) {
    const double v = geo[R.geo + t];
    sF[t] = v;
    if (QUAD) bad |= fm_nonfinite(v);
  }
  const int neg1 = QUAD ? R.loc1[0] >= 3 : R.loc1[0] < 3, neg2 = QUAD ? R.loc2[0] >= 3 : R.loc2[0] < 3;
  // QUAD: row offsets of the moments in sW (the last K doubles: no moment, zero)
  const int TD = fm_tri(DD), TD1 = fm_tri(DD - 1);
  const int o1 = TD * K, o2 = o1 + TD1 * K, o4 = o2 + TD1 * K, o5 = o4 + TD1 * K, o3 = o5 + TD1 * K, o6 = o3 + TD * (K - 1),
            oz = o6 + TD * (K - 1);
  if (QUAD) {
    const FmQuad A(R.loc1), B(R.loc2);
    // per pair of triangle monomials: the moment rows of its five products
    for (int t = tid; t < npair; t += THR) {
      const int x = t / nt2, y = t - x * nt2;
      const int a = tb.MON[2 * x], b = tb.MON[2 * x + 1], a2 = tb.MON[2 * y], b2 = tb.MON[2 * y + 1];
      int eA, eB, fA, fB;
      const bool v2 = B.trace(a2, b2, fA, fB), v1 = A.trace(a, b, eA, eB);
      unsigned short *I = sI + 5 * t;
      I[0] = (unsigned short)(v1 && v2 ? fm_mono(eA + fA, eB + fB) : 0xffff);
      int gA, gB;
      I[1] = (unsigned short)(a && v2 && A.trace(a - 1, b, gA, gB) ? o1 + fm_mono(gA + fA, gB + fB) * K : oz);
      I[2] = (unsigned short)(b && v2 && A.trace(a, b - 1, gA, gB) ? o2 + fm_mono(gA + fA, gB + fB) * K : oz);
      I[3] = (unsigned short)(a2 && v1 && B.trace(a2 - 1, b2, gA, gB) ? o4 + fm_mono(eA + gA, eB + gB) * K : oz);
      I[4] = (unsigned short)(b2 && v1 && B.trace(a2, b2 - 1, gA, gB) ? o5 + fm_mono(eA + gA, eB + gB) * K : oz);
    }
    bad = __syncthreads_or(bad);
    for (int t = tid; t < K; t += THR) sW[oz + t] = bad ? nan("") : 0.0;
    // line sums S[c][k][m]
    constexpr int ZS = Q1 | 1;
    const double *Z = tb.Z + (size_t)(PM - 1) * FM_Q1 * FM_ZP;
    for (int t = tid; t < 7 * K * Q1; t += THR) {
      const int ck = t / Q1, m = t - ck * Q1, c = ck / K, k = ck - c * K;
      const double *F = sF + c * NQ + (A.along_s ? m * Q1 : m);
      const int st = A.along_s ? 1 : Q1;
      double a = 0.0;
#pragma unroll
      for (int n = 0; n < Q1; n++) a = fma(F[n * st], __ldg(Z + n * FM_ZP + k), a);
      sS[ck * ZS + m] = a;
    }
    __syncthreads();
    // moments, in the order of their rows; W_3, W_6 carry the signs of zeta
    const double *XE = tb.XE + (size_t)(PM - 1) * FM_MONO * FM_Q1;
    for (int t = tid; t < oz; t += THR) {
      int c, k, al;
      if (t < o3) {
        const int row = t / K;
        k = t - row * K;
        c = row < TD ? 0 : 1 + (row - TD) / TD1;
        al = row < TD ? row : (row - TD) - (c - 1) * TD1;
        if (c > 2) c++;  // 4, 5
      } else {
        const int row = (t - o3) / (K - 1);
        k = (t - o3) - row * (K - 1);
        c = row < TD ? 3 : 6;
        al = row < TD ? row : row - TD;
      }
      const double *S = sS + (c * K + k) * ZS, *X = XE + al * FM_Q1;
      double a = 0.0;
#pragma unroll
      for (int m = 0; m < Q1; m++) a = fma(S[m], __ldg(X + m), a);
      sW[t] = c == 3 ? flip(a, neg1) : c == 6 ? flip(a, neg2) : a;
    }
    __syncthreads();
    // E[pair][k]
    for (int t = tid; t < npair * K; t += THR) {
      const int pr = t / K, k = t - pr * K, x = pr / nt2, y = pr - x * nt2;
      const unsigned short *I = sI + 5 * pr;
      const double *C1 = sC, *C = sW + k;
      sE[t] = fma(C1[tb.MON[2 * x]], C[I[1]], fma(C1[tb.MON[2 * x + 1]], C[I[2]],
                  fma(C1[tb.MON[2 * y]], C[I[3]], C1[tb.MON[2 * y + 1]] * C[I[4]])));
    }
  } else {
    __syncthreads();
    // values X, weighted tangential gradients U = F . grad per side; side 2's
    // values times F_0, F_3, F_6
    constexpr int QS = NQ | 1;
    double *X1 = sW, *U1 = X1 + D::NT * QS, *X2 = U1 + D::NT * QS, *U2 = X2 + D::NT * QS, *P0 = U2 + D::NT * QS,
           *P3 = P0 + D::NT * QS, *P6 = P3 + D::NT * QS;
    for (int t = tid; t < (nt1 + nt2) * NQ; t += THR) {
      const int r = t / NQ, q = t - r * NQ, sd = r >= nt1, x = sd ? r - nt1 : r;
      const unsigned char *l = sd ? R.loc2 : R.loc1;
      const int i1 = l[0] % 3 == 1 ? 0 : l[1] % 3 == 1 ? 1 : 2, i2 = l[0] % 3 == 2 ? 0 : l[1] % 3 == 2 ? 1 : 2;
      const double *X = tb.XT + (size_t)((PM - 1) * 9 + 3 * i1 + i2) * FM_MONO * FM_QT + q;
      const int a = tb.MON[2 * x], b = tb.MON[2 * x + 1];
      const double v = __ldg(X + x * FM_QT);
      const double da = a ? __ldg(X + fm_mono(a - 1, b) * FM_QT) : 0.0, db = b ? __ldg(X + fm_mono(a, b - 1) * FM_QT) : 0.0;
      const double *F = sF + (1 + 3 * sd) * NQ + q;
      const double u = fma(sC[a] * da, F[0], sC[b] * db * F[NQ]);
      (sd ? X2 : X1)[x * QS + q] = v;
      (sd ? U2 : U1)[x * QS + q] = u;
      if (sd) {
        P0[x * QS + q] = sF[q] * v;
        P3[x * QS + q] = sF[3 * NQ + q] * v;
        P6[x * QS + q] = sF[6 * NQ + q] * v;
      }
    }
    __syncthreads();
    // pair sums: E, then sum F_3, F_6 (with the signs of zeta), F_0
    for (int t = tid; t < 4 * npair; t += THR) {
      const int w = t / npair, pr = t - w * npair, x = pr / nt2, y = pr - x * nt2;
      const double *Xa = X1 + x * QS;
      double a = 0.0;
      if (w == 0) {
        const double *Ua = U1 + x * QS, *Xb = X2 + y * QS, *Ub = U2 + y * QS;
#pragma unroll
        for (int q = 0; q < NQ; q++) a = fma(Ua[q], Xb[q], fma(Xa[q], Ub[q], a));
      } else {
        const double *Pb = (w == 1 ? P3 : w == 2 ? P6 : P0) + y * QS;
#pragma unroll
        for (int q = 0; q < NQ; q++) a = fma(Xa[q], Pb[q], a);
      }
      sE[t] = w == 1 ? flip(a, neg1) : w == 2 ? flip(a, neg2) : a;
    }
  }
  __syncthreads();
  // entries (i, j): function i of side 1, j of side 2
  double *b12 = val + R.blk1, *b21 = val + R.blk2;
  auto entry = [&](int i, int j) {
    const int x = sFn[0][i][0], c = sFn[0][i][1], y = sFn[1][j][0], c2 = sFn[1][j][1], pr = x * nt2 + y, k = c + c2;
    double N, S;
    if (QUAD) {
      const int r = sI[5 * pr];
      N = sE[pr * K + k];
      S = 0.0;
      if (r != 0xffff) {
        const int kd = k > 0 ? k - 1 : 0;
        N = fma(sC[c], sW[o3 + r * (K - 1) + kd], fma(sC[c2], sW[o6 + r * (K - 1) + kd], N));
        S = sW[r * K + k];
      }
    } else {
      N = fma(sC[c], sE[npair + pr], fma(sC[c2], sE[2 * npair + pr], sE[pr]));
      S = sE[3 * npair + pr];
    }
    const int neg = (neg1 & c) ^ (neg2 & c2);
    b12[i + (size_t)ns1 * j] = flip(N + S, neg ^ 1);
    b21[j + (size_t)ns2 * i] = flip(N - S, neg);
  };
  if (PM >= 3) {
    // a warp takes 4 x 8 entries, so that both blocks are written in whole
    // 32-byte sectors
    const int di = tid & 3, dj = (tid >> 2) & 7, ti = (ns1 + 3) >> 2, tj = (ns2 + 7) >> 3;
    for (int t = tid >> 5; t < ti * tj; t += THR >> 5) {
      const int j0 = t / ti, i = 4 * (t - j0 * ti) + di, j = 8 * j0 + dj;
      if (i < ns1 && j < ns2) entry(i, j);
    }
  } else {
    for (int t = tid; t < ns1 * ns2; t += THR) entry(t % ns1, t / ns1);
  }
}

// ------------------------------------------------------------------ launches
// start[b] .. start[b + 1]: the records of rule degree b % 4 + 1, triangles (b < 4) or quadrilaterals
int launch_dg_face_fields(cudaStream_t st, const int *start, const DgFaceRec *rec, const int *el_nodes,
                          const double *xyz, const double *k_el, const double *D_el, double pen, double *geo) {
  // one point a thread up to eight blocks an SM (2,000 prisms of p = 2: 31 us, two points 44;
  // 54,000 of p = 3: 729 and 696)
  long long points = 0;
  for (int b = 0; b < 8; b++) points += (long long)(start[b + 1] - start[b]) * GB_DG_NQF[b % 4 + 1][b / 4];
  const int per = points <= 8LL * 152 * FG_THREADS ? 1 : 2;
  DgFieldGroups G;
  int n = 0, blocks = 0, most = 0;
  for (int b = 7; b >= 0; b--) {  // the longest first
    const int count = start[b + 1] - start[b], nq = GB_DG_NQF[b % 4 + 1][b / 4];
    if (count <= 0) continue;
    const int NF = std::max(1, per * FG_THREADS / nq);
    G.g[n++] = {blocks, start[b], count, NF, nq, b % 4 + 1, b / 4};
    blocks += (count + NF - 1) / NF;
    most = std::max(most, NF);
  }
  if (blocks == 0) return 0;
  dg_face_fields_kernel<<<blocks, FG_THREADS, 61 * most * sizeof(double), st>>>(G, n, rec, el_nodes, xyz, k_el, D_el,
                                                                                pen, geo);
  GB_CUDA(cudaGetLastError());
  return 1;
}

int launch_dg_face_diag(cudaStream_t st, int device, int p, int count, const int *ent_el, const int *hf_ptr,
                        const int *hrec, const DgFaceRec *rec, const double *geo, double g, const long long *boff_diag,
                        const int *roff, double *val, double *rhs, int variant) {
  if (count <= 0) return 0;
  GB_CHECK(p >= 1 && p <= GB_DG_PMAX, "DG degree must be 1..4");
  GB_CHECK(variant >= 0 && variant < 2, "face kernel variant out of range");
  DgFaceTables tb;
  GB_TRY(fm_tables(device, &tb));
#define GB_FM_DIAG(PP, T0, T1)                                                                                   \
  if (variant == 0)                                                                                              \
    dg_face_diag_kernel<PP, T0><<<count, T0, 0, st>>>(count, ent_el, hf_ptr, hrec, rec, geo, tb, g, boff_diag,   \
                                                      roff, val, rhs);                                           \
  else                                                                                                           \
    dg_face_diag_kernel<PP, T1><<<count, T1, 0, st>>>(count, ent_el, hf_ptr, hrec, rec, geo, tb, g, boff_diag,   \
                                                      roff, val, rhs)
  switch (p) {
    case 1: GB_FM_DIAG(1, 32, 64); break;
    case 2: GB_FM_DIAG(2, 64, 128); break;
    case 3: GB_FM_DIAG(3, 128, 256); break;
    default: GB_FM_DIAG(4, 128, 256); break;
  }
#undef GB_FM_DIAG
  GB_CUDA(cudaGetLastError());
  return 1;
}

int launch_dg_face_blocks(cudaStream_t st, int device, int pm, int ti, int count, const DgFaceRec *rec,
                          const double *geo, double *val) {
  if (count <= 0) return 0;
  DgFaceTables tb;
  GB_TRY(fm_tables(device, &tb));
#define GB_FM_OFF(PP, QQ)                                                                                       \
  {                                                                                                             \
    GB_CUDA(cudaFuncSetAttribute(dg_face_blocks_kernel<PP, QQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                                 FmOff<PP, QQ>::BYTES));                                                        \
    dg_face_blocks_kernel<PP, QQ><<<count, FmOff<PP, QQ>::THR, FmOff<PP, QQ>::BYTES, st>>>(rec, geo, tb, val);  \
  }
#define GB_FM_P(PP) \
  if (ti) GB_FM_OFF(PP, true) else GB_FM_OFF(PP, false)
  switch (pm) {
    case 1: GB_FM_P(1) break;
    case 2: GB_FM_P(2) break;
    case 3: GB_FM_P(3) break;
    default: GB_FM_P(4) break;
  }
#undef GB_FM_P
#undef GB_FM_OFF
  GB_CUDA(cudaGetLastError());
  return 1;
}

}  // namespace gbfem
