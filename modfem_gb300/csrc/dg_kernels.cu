// DG prism volume integrals (tensor monomial basis, p = 1..4), FP64.
//
// Reference: apr_num_int_el of apd_dg_prism (aps_dg_prism_intf.c:1239-1728),
// basis and rules as in dg_tables.h; the algorithm (moments of the geometry
// over the rule, then each entry from six moments) is in dg_volume.cuh.
//
// The element's own matrix is its diagonal block in the block-CRS storage
// (dense ns x ns, column-major, offset boff[e]); no other element writes
// there, so no atomics are needed for volume terms.

#include "gbfem_internal.h"
#include "dg_tables.h"
#include "dg_volume.cuh"
#include "prism_std.cuh"

#include <mutex>

namespace gbfem {

static DgDeviceTables g_dg_tables[64];
static bool g_dg_tables_ready[64] = {false};
static std::mutex g_dg_tables_lock;  // contexts are made and used from several threads

// The volume kernel's tables for degree p (layouts in dg_volume.cuh): point
// rule QP, monomials and line-point powers VT, entries ENT (upper triangle row by
// row, then the function of every load-vector moment).
static void host_dg_tables(int p, std::vector<double> &QP, std::vector<double> &VT, std::vector<DgVolEntry> &ENT) {
  const int ns = GB_DG_NS[p], nq = GB_DG_NQ[p], nz = p + 1, nt = nq / nz;
  const int K0 = 2 * p + 1, K1 = 2 * p, K2 = 2 * p - 1;
  const int T0 = dg_tri(2 * p - 2), T1 = dg_tri(2 * p - 1), T2 = dg_tri(2 * p);
  auto mono = [](int i, int j) { return (i + j) * (i + j + 1) / 2 + j; };
  QP.resize((size_t)nq * 4);
  for (int q = 0; q < nq; q++)
    for (int k = 0; k < 4; k++) QP[q * 4 + k] = GB_DG_QP[p - 1][q][k];
  VT.assign((size_t)T2 * nt + nz * K0 + 2 * p * p + 1, 0.0);
  for (int t = 0; t < nt; t++) {
    double pe = 1.0;
    for (int j = 0; j <= 2 * p; j++, pe *= QP[4 * t + 1]) {
      double px = pe;
      for (int i = 0; i + j <= 2 * p; i++, px *= QP[4 * t]) VT[(size_t)mono(i, j) * nt + t] = px;
    }
  }
  for (int n = 0; n < nz; n++) {
    double pz = 1.0;
    for (int k = 0; k < K0; k++, pz *= QP[4 * (size_t)n * nt + 2]) VT[(size_t)T2 * nt + n * K0 + k] = pz;
  }
  for (int i = 0; i <= 2 * p * p; i++) VT[(size_t)T2 * nt + nz * K0 + i] = i;
  ENT.clear();
  for (int u = 0; u < ns; u++)
    for (int w = u; w < ns; w++) {
      const int a = GB_DG_EXP[p - 1][u][0], b = GB_DG_EXP[p - 1][u][1], c = GB_DG_EXP[p - 1][u][2];
      const int a2 = GB_DG_EXP[p - 1][w][0], b2 = GB_DG_EXP[p - 1][w][1], c2 = GB_DG_EXP[p - 1][w][2];
      const int i = a + a2, j = b + b2, k = c + c2;
      DgVolEntry E{};
      E.u = (unsigned char)u;
      E.w = (unsigned char)w;
      auto put = [&](int comp, int coef, long long off) {
        E.coef[comp] = (unsigned char)coef;
        E.off[comp] = (unsigned short)(coef ? off : 0);
      };
      put(0, a * a2, (long long)mono(i - 2, j) * K0 + k);
      put(1, a * b2 + b * a2, (long long)T0 * K0 + mono(i - 1, j - 1) * K0 + k);
      put(2, b * b2, 2ll * T0 * K0 + mono(i, j - 2) * K0 + k);
      put(3, a * c2 + c * a2, 3ll * T0 * K0 + mono(i - 1, j) * K1 + k - 1);
      put(4, b * c2 + c * b2, 3ll * T0 * K0 + T1 * K1 + mono(i, j - 1) * K1 + k - 1);
      put(5, c * c2, 3ll * T0 * K0 + 2ll * T1 * K1 + mono(i, j) * K2 + k - 2);
      ENT.push_back(E);
    }
  for (int r = 0; r < dg_tri(p) * (p + 1); r++) {
    DgVolEntry E{};
    for (int u = 0; u < ns; u++)
      if (mono(GB_DG_EXP[p - 1][u][0], GB_DG_EXP[p - 1][u][1]) == r / (p + 1) && GB_DG_EXP[p - 1][u][2] == r % (p + 1))
        E.u = (unsigned char)u;
    ENT.push_back(E);
  }
}

int dg_tables_for_device(int device, DgDeviceTables **out) {
  GB_CHECK(device >= 0 && device < 64, "device index out of range");
  std::lock_guard<std::mutex> hold(g_dg_tables_lock);
  if (!g_dg_tables_ready[device]) {
    for (int p = 1; p <= GB_DG_PMAX; p++) {
      std::vector<double> QP, VT;
      std::vector<DgVolEntry> ENT;
      host_dg_tables(p, QP, VT, ENT);
      double *qp = nullptr, *vt = nullptr;
      DgVolEntry *en = nullptr;
      GB_CUDA(cudaMalloc(&qp, QP.size() * sizeof(double)));
      GB_CUDA(cudaMalloc(&vt, VT.size() * sizeof(double)));
      GB_CUDA(cudaMalloc(&en, ENT.size() * sizeof(DgVolEntry)));
      GB_CUDA(cudaMemcpy(qp, QP.data(), QP.size() * sizeof(double), cudaMemcpyHostToDevice));
      GB_CUDA(cudaMemcpy(vt, VT.data(), VT.size() * sizeof(double), cudaMemcpyHostToDevice));
      GB_CUDA(cudaMemcpy(en, ENT.data(), ENT.size() * sizeof(DgVolEntry), cudaMemcpyHostToDevice));
      g_dg_tables[device].QP[p] = qp;
      g_dg_tables[device].VT[p] = vt;
      g_dg_tables[device].ENT[p] = en;
    }
    g_dg_tables_ready[device] = true;
  }
  *out = &g_dg_tables[device];
  return 0;
}

// Elements of degree P, NE per CTA: ent_el[i] (0-based), matrix block at
// val + boff[e], rhs rows at rhs + roff[e].  D_el (tensor, 9 per element) or
// k_el (isotropic).
template <int P, int NE>
__global__ void __launch_bounds__(DG_VOL_THREADS) dg_prism_elements_kernel(
    int count, const int *__restrict__ ent_el, const int *__restrict__ el_nodes, const double *__restrict__ xyz,
    const double *__restrict__ k_el, const double *__restrict__ D_el, double f, const double *__restrict__ tab,
    const double *__restrict__ QP, const DgVolEntry *__restrict__ ent, const long long *__restrict__ boff,
    const int *__restrict__ roff, double *__restrict__ val, double *__restrict__ rhs) {
  extern __shared__ double smem[];
  const int first = blockIdx.x * NE;
  const int n = count - first < NE ? count - first : NE;
  dg_prism_volume_tile<P>(
      n, f, tab, QP, ent, smem,
      [&](int el, int i) -> double {
        const int e = ent_el[first + el];
        if (i < 18) return xyz[3 * (size_t)el_nodes[6 * (size_t)e + i / 3] + i % 3];
        i -= 18;
        if (D_el) return D_el[9 * (size_t)e + i];
        return i % 4 == 0 ? (k_el ? k_el[e] : 1.0) : 0.0;
      },
      [&](int el) { return val + boff[ent_el[first + el]]; }, [&](int el) { return rhs + roff[ent_el[first + el]]; });
}

int launch_dg_prism_elements(cudaStream_t st, int device, int p, int count, const int *ent_el, const int *el_nodes,
                             const double *xyz, const double *k_el, const double *D_el, double f,
                             const long long *boff, const int *roff, double *val, double *rhs, int variant) {
  if (count <= 0) return 0;
  GB_CHECK(p >= 1 && p <= GB_DG_PMAX, "DG degree must be 1..4");
  GB_CHECK(variant >= 0 && variant < DG_VOL_VARIANTS, "volume kernel variant out of range");
  DgDeviceTables *tb = nullptr;
  int r = dg_tables_for_device(device, &tb);
  if (r < 0) return r;
#define GB_DG_LAUNCH(PP, VV)                                                                                     \
  {                                                                                                              \
    constexpr int NE_ = dg_vol_elems(PP, VV);                                                                    \
    constexpr int bytes = (int)sizeof(double) * dg_vol_smem(PP, VV);                                             \
    GB_CUDA(cudaFuncSetAttribute(dg_prism_elements_kernel<PP, NE_>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                 bytes));                                                                        \
    dg_prism_elements_kernel<PP, NE_><<<(count + NE_ - 1) / NE_, DG_VOL_THREADS, bytes, st>>>(                   \
        count, ent_el, el_nodes, xyz, k_el, D_el, f, tb->VT[PP], tb->QP[PP], tb->ENT[PP], boff, roff, val, rhs); \
  }
#define GB_DG_P(PP)                     \
  switch (variant) {                    \
    case 0: GB_DG_LAUNCH(PP, 0) break;  \
    case 1: GB_DG_LAUNCH(PP, 1) break;  \
    default: GB_DG_LAUNCH(PP, 2) break; \
  }
  switch (p) {
    case 1: GB_DG_P(1); break;
    case 2: GB_DG_P(2); break;
    case 3: GB_DG_P(3); break;
    default: GB_DG_P(4); break;
  }
#undef GB_DG_P
#undef GB_DG_LAUNCH
  GB_CUDA(cudaGetLastError());
  return 1;
}

}  // namespace gbfem
