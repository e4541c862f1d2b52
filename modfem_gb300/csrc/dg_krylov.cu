// Variable-block CRS products and block Jacobi for the DG matrix, FP64.
//
// Storage (the device form of lad_block, lsd_mkb/lad_block/lah_block.h): block
// row e holds the dofs of element e (roff[e] .. roff[e+1]); its blocks
// bptr[e] .. bptr[e+1] have column elements bcol[k] (ascending, the diagonal
// included) and dense values at val + boff[k], column-major with the row
// block's size as leading dimension (Dia / Aux of las_block_intf.c:362-520).
//
// The block Jacobi preconditioner of the reference (lar_fill_preconditioner_
// block with Block_type 1: an LU factorisation of every diagonal block,
// las_block_intf.c:1224-1330, applied by forward/back substitution) is kept
// here as the explicit inverse of each diagonal block: applying it is then a
// dense block product fused into the SpMV.

#include <type_traits>

#include "dg_spmv.cuh"
#include "dg_tables.h"
#include "gbfem_internal.h"

namespace gbfem {

// Gauss-Jordan inversion with partial pivoting (largest magnitude, first
// row on ties) of the diagonal blocks of one class, each block in the registers
// of a group of GA x GB lanes (lane (a, b): rows a + GA s, columns b + GB u).
// Rows are not exchanged: step k takes its pivot from row r_k of those left
// and exchanges unknown k with right hand side r_k, so that in the end
// inverse[k][r_j] = entry (r_k, j).  The pivot column (f) and row (p) pass
// through shared memory and leave zeros behind; with g_i = f_i / pivot,
// g_r = -1 / pivot and p_k = 1 the whole step is entry (i, j) -= g_i p_j.  n^3 FMA
// a block bound it by the FP64 pipe (p = 3: 2,000 of some 2,330 FP64 warp
// instructions, which hold it for 6.4 ms of 54,000 blocks' 6.7); held in shared memory, three
// loads and a store an FMA, the pipe stood half idle: 13.8 ms.  (21,296 prisms of p = 1..4
// 52, 504, 2,695, 19,765 us, 20,250 tetrahedra 33, 106, 530, 2,042 us; one CTA a
// block in shared memory 581, 1,886, 6,317, 25,931 and 384, 919, 2,030, 4,798 us.)
template <int P>
struct DgInv {
  static constexpr int NS = DgSpmvDims<P>::NS;
  static constexpr int GA = NS > 40 ? 16 : NS > 10 ? 8 : NS > 6 ? 4 : 2;
  static constexpr int GB = NS > 40 ? 8 : NS > 6 ? 4 : 2;
  static constexpr int G = GA * GB, W = G < 32 ? G : 32;    // lanes a block; of those that search the pivot
  static constexpr int R = (NS + GA - 1) / GA, C = (NS + GB - 1) / GB, Q = (NS + W - 1) / W;
  static constexpr int CTA = 128, PER = CTA / G;            // blocks per CTA
};

template <int P>
__global__ void __launch_bounds__(DgInv<P>::CTA, 3) dg_block_inverse_kernel(
    int count, const int *__restrict__ ent_el, const long long *__restrict__ boff_diag, const double *__restrict__ val,
    const long long *__restrict__ dinv_off, double *__restrict__ dinv, int *err) {
  using D = DgInv<P>;
  constexpr int n = D::NS, GA = D::GA, GB = D::GB, G = D::G, W = D::W, R = D::R, C = D::C, Q = D::Q;
  __shared__ double sf[D::PER][n], sg[D::PER][R * GA], sp[D::PER][C * GB];
  __shared__ int srow[D::PER][n], sstep[D::PER][n];
  const int grp = threadIdx.x / G, l = threadIdx.x % G, a = l % GA, b = l / GA, lw = threadIdx.x % W;
  const unsigned mask = W == 32 ? ~0u : ((1u << (W & 31)) - 1u) << ((threadIdx.x & 31) / W * W);
  const int idx = blockIdx.x * D::PER + grp;
  const int e = ent_el[min(idx, count - 1)];  // a group beyond the last block computes along and writes nothing
  double *f = sf[grp], *g = sg[grp], *p = sp[grp];
  auto sync = [] {
    if (G <= 32)
      __syncwarp();
    else
      __syncthreads();
  };
  const double *src = val + boff_diag[e];
  double A[R][C];
#pragma unroll
  for (int s = 0; s < R; s++)
#pragma unroll
    for (int u = 0; u < C; u++) {
      const int i = a + GA * s, j = b + GB * u;
      A[s][u] = i < n && j < n ? src[i + n * j] : 0.0;
    }
  for (int i = l; i < R * GA; i += G) g[i] = 0.0;
  for (int j = l; j < C * GB; j += G) p[j] = 0.0;
  unsigned used = 0;  // bit q: row lw + W q has been a pivot row
  bool singular = false;
#pragma unroll 1
  for (int k = 0; k < n; k++) {
    const int ku = b == k % GB ? k / GB : -1;
#pragma unroll
    for (int s = 0; s < R; s++) {
#pragma unroll
      for (int u = 0; u < C; u++)
        if (u == ku) {
          if (a + GA * s < n) f[a + GA * s] = A[s][u];
          A[s][u] = 0.0;
        }
    }
    sync();
    // every warp of the group finds the same pivot row: magnitudes as
    // integers (a NaN is never chosen), a zero column has none
    double fv[Q];
    unsigned long long best = 0;
    int r = n;
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = lw + W * q;
      fv[q] = i < n ? f[i] : 0.0;
      const unsigned long long v = (unsigned long long)__double_as_longlong(fv[q]) & 0x7fffffffffffffffull;
      if (!(used >> q & 1u) && v > best && v <= 0x7ff0000000000000ull) {
        best = v;
        r = i;
      }
    }
    const unsigned hi = __reduce_max_sync(mask, (unsigned)(best >> 32));
    const unsigned lo = __reduce_max_sync(mask, (unsigned)(best >> 32) == hi ? (unsigned)best : 0u);
    r = __reduce_min_sync(mask, best == ((unsigned long long)hi << 32 | lo) ? r : n);
    if (r >= n) {  // singular diagonal block (the same for the whole group)
      singular = true;
      r = 0;
    }
    if (r % W == lw) used |= 1u << (r / W);
    const double pinv = 1.0 / f[r];
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = lw + W * q;
      if (i < n && l < W) g[i] = i == r ? -pinv : fv[q] * pinv;
    }
    const int rs = a == r % GA ? r / GA : -1;
#pragma unroll
    for (int s = 0; s < R; s++) {
#pragma unroll
      for (int u = 0; u < C; u++)
        if (s == rs) {
          const int j = b + GB * u;
          if (j < n) p[j] = j == k ? 1.0 : A[s][u];
          A[s][u] = 0.0;
        }
    }
    if (l == 0) {
      srow[grp][k] = r;
      sstep[grp][r] = k;
    }
    sync();
    double gi[R], pj[C];
#pragma unroll
    for (int s = 0; s < R; s++) gi[s] = -g[a + GA * s];
#pragma unroll
    for (int u = 0; u < C; u++) pj[u] = p[b + GB * u];
#pragma unroll
    for (int s = 0; s < R; s++)
#pragma unroll
      for (int u = 0; u < C; u++) A[s][u] = fma(gi[s], pj[u], A[s][u]);
  }
  if (idx >= count) return;
  if (singular) {
    if (l == 0) atomicExch(err, 3);
    return;
  }
  double *dst = dinv + dinv_off[e];
#pragma unroll
  for (int s = 0; s < R; s++) {
    const int i = a + GA * s;
    if (i >= n) continue;
    const int row = sstep[grp][i];
#pragma unroll
    for (int u = 0; u < C; u++) {
      const int j = b + GB * u;
      if (j < n) dst[row + n * srow[grp][j]] = A[s][u];
    }
  }
}

int launch_dg_block_inverse(cudaStream_t st, int cls, int count, const int *ent_el, const long long *boff_diag,
                            const double *val, const long long *dinv_off, double *dinv, int *err) {
  if (count <= 0) return 0;
#define GB_INV(PP)                                                                                             \
  dg_block_inverse_kernel<PP><<<(count + DgInv<PP>::PER - 1) / DgInv<PP>::PER, DgInv<PP>::CTA, 0, st>>>(       \
      count, ent_el, boff_diag, val, dinv_off, dinv, err);
  switch (cls) {
    case 1: GB_INV(1) break;
    case 2: GB_INV(2) break;
    case 3: GB_INV(3) break;
    case 4: GB_INV(4) break;
    case 5: GB_INV(5) break;
    case 6: GB_INV(6) break;
    case 7: GB_INV(7) break;
    case 8: GB_INV(8) break;
    default: GB_CHECK(false, "DG block class must be 1..8 (prisms 1..4, tetrahedra 5..8)");
  }
#undef GB_INV
  GB_CUDA(cudaGetLastError());
  return 1;
}

template <int P, typename VT>
__global__ void __launch_bounds__(DGS_THREADS) dg_block_spmv_kernel(
    int mode, int count, const int *__restrict__ ent_el, const int *__restrict__ roff,
    const long long *__restrict__ row_val, const long long *__restrict__ cx_off, const int *__restrict__ colx,
    const VT *__restrict__ val, const long long *__restrict__ dinv_off, const VT *__restrict__ dinv,
    const double *__restrict__ x, const double *__restrict__ b, double *__restrict__ out) {
  __shared__ VT sv[DGS_ROWS][DgSpmvDims<P>::NS];
  dg_block_row_spmv<P, VT>(mode, count, ent_el, roff, row_val, cx_off, colx, val, dinv_off, dinv, x, b, out, sv);
}

// one CTA a block row (small systems)
template <int P>
__global__ void __launch_bounds__(DGS_THREADS) dg_block_spmv_wide_kernel(
    int mode, const int *__restrict__ ent_el, const int *__restrict__ roff, const long long *__restrict__ row_val,
    const long long *__restrict__ cx_off, const int *__restrict__ colx, const double *__restrict__ val,
    const long long *__restrict__ dinv_off, const double *__restrict__ dinv, const double *__restrict__ x,
    const double *__restrict__ b, double *__restrict__ out) {
  dg_block_row_wide<P>(mode, ent_el[blockIdx.x], roff, row_val, cx_off, colx, val, dinv_off, dinv, x, b, out);
}

// Residual out = b - A x with the products and sums carried in two FP64
// words per row (error-free transformations: the exact product error from an
// FMA, Knuth's TwoSum, the errors summed in a second word and added once at
// the end: the compensated dot product "Dot2" of Ogita, Rump and Oishi,
// SIAM J. Sci. Comput. 26, 2005).  The result is as accurate as if computed
// in twice the working precision, then rounded: iterative refinement driven
// by it reaches a forward error near FP64 rounding whatever the FP64 residual
// floor of a badly scaled system.  Same lane layout as dg_block_row_spmv.
template <int P>
__global__ void __launch_bounds__(DGS_THREADS) dg_block_residual_dd_kernel(
    int count, const int *__restrict__ ent_el, const int *__restrict__ roff, const long long *__restrict__ row_val,
    const long long *__restrict__ cx_off, const int *__restrict__ colx, const double *__restrict__ val,
    const double *__restrict__ x, const double *__restrict__ b, double *__restrict__ out) {
  constexpr int NS = DgSpmvDims<P>::NS;
  constexpr int S = (NS + DGS_LANES - 1) / DGS_LANES;
  const int grp = threadIdx.x / DGS_LANES, g = threadIdx.x % DGS_LANES;
  const int idx = blockIdx.x * DGS_ROWS + grp;
  if (idx >= count) return;
  const int e = ent_el[idx];
  const int r0 = roff[e];
  double hi[S], lo[S];
#pragma unroll
  for (int s = 0; s < S; s++) {
    const int i = g + DGS_LANES * s;
    hi[s] = b && i < NS ? b[r0 + i] : 0.0;
    lo[s] = 0.0;
  }
  const double *A = val + row_val[e] + g;
  const int *cx = colx + cx_off[e];
  const int nct = (int)(cx_off[e + 1] - cx_off[e]);
  for (int t = 0; t < nct; t++) {
    const double xv = -x[cx[t]];
    const double *col = A + (size_t)t * NS;
#pragma unroll
    for (int s = 0; s < S; s++) {
      if (g + DGS_LANES * s >= NS) continue;
      const double a = col[DGS_LANES * s];
      const double p = a * xv;
      const double ep = fma(a, xv, -p);  // exact: a xv = p + ep
      const double sum = hi[s] + p;      // TwoSum(hi, p)
      const double bb = sum - hi[s];
      const double es = (hi[s] - (sum - bb)) + (p - bb);
      hi[s] = sum;
      lo[s] += ep + es;
    }
  }
#pragma unroll
  for (int s = 0; s < S; s++) {
    const int i = g + DGS_LANES * s;
    if (i < NS) out[r0 + i] = hi[s] + lo[s];
  }
}

int launch_dg_block_residual_dd(cudaStream_t st, int p, int count, const int *ent_el, const int *roff,
                                const long long *row_val, const long long *cx_off, const int *colx,
                                const double *val, const double *x, const double *b, double *out) {
  if (count <= 0) return 0;
  GB_CHECK(p >= 1 && p <= 2 * GB_DG_PMAX, "DG block class must be 1..8 (prisms 1..4, tetrahedra 5..8)");
  const int grid = (count + DGS_ROWS - 1) / DGS_ROWS;
#define GB_DGR_LAUNCH(PP)                                                                               \
  dg_block_residual_dd_kernel<PP><<<grid, DGS_THREADS, 0, st>>>(count, ent_el, roff, row_val, cx_off, colx, \
                                                                val, x, b, out)
  switch (p) {
    case 1: GB_DGR_LAUNCH(1); break;
    case 2: GB_DGR_LAUNCH(2); break;
    case 3: GB_DGR_LAUNCH(3); break;
    case 4: GB_DGR_LAUNCH(4); break;
    case 5: GB_DGR_LAUNCH(5); break;
    case 6: GB_DGR_LAUNCH(6); break;
    case 7: GB_DGR_LAUNCH(7); break;
    default: GB_DGR_LAUNCH(8); break;
  }
#undef GB_DGR_LAUNCH
  GB_CUDA(cudaGetLastError());
  return 1;
}

__global__ void to_float_kernel(long long n, const double *__restrict__ a, float *__restrict__ b) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

__global__ void to_dw_kernel(long long n, const double *__restrict__ a, dw *__restrict__ b) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = dw_from_double(a[i]);
}

int launch_to_dw(cudaStream_t st, long long n, const double *a, void *b) {
  if (n <= 0) return 0;
  to_dw_kernel<<<152 * 8, 256, 0, st>>>(n, a, reinterpret_cast<dw *>(b));
  GB_CUDA(cudaGetLastError());
  return 1;
}

int launch_to_float(cudaStream_t st, long long n, const double *a, float *b) {
  if (n <= 0) return 0;
  to_float_kernel<<<152 * 8, 256, 0, st>>>(n, a, b);
  GB_CUDA(cudaGetLastError());
  return 1;
}

template <typename VT>
static int launch_dg_block_spmv_t(cudaStream_t st, int mode, int p, int count, const int *ent_el, const int *roff,
                                  const long long *row_val, const long long *cx_off, const int *colx, const VT *val,
                                  const long long *dinv_off, const VT *dinv, const double *x, const double *b,
                                  double *out, int longest = 0) {
  if (count <= 0) return 0;
  GB_CHECK(mode >= 0 && mode <= 2, "bad block SpMV mode");
  GB_CHECK(p >= 1 && p <= 2 * GB_DG_PMAX, "DG block class must be 1..8 (prisms 1..4, tetrahedra 5..8)");
  GB_CHECK(mode == 2 || (dinv && dinv_off), "block SpMV needs the inverted diagonal blocks");
  const int grid = (count + DGS_ROWS - 1) / DGS_ROWS;
#define GB_DGS_LAUNCH(PP)                                                                                      \
  if constexpr (std::is_same<VT, double>::value) {                                                             \
    if (count <= dgs_wide_max(PP, longest)) {                                                                   \
      dg_block_spmv_wide_kernel<PP><<<count, DGS_THREADS, 0, st>>>(mode, ent_el, roff, row_val, cx_off, colx,  \
                                                                   val, dinv_off, dinv, x, b, out);            \
      break;                                                                                                   \
    }                                                                                                          \
  }                                                                                                            \
  dg_block_spmv_kernel<PP, VT><<<grid, DGS_THREADS, 0, st>>>(mode, count, ent_el, roff, row_val, cx_off, colx, \
                                                             val, dinv_off, dinv, x, b, out)
  switch (p) {
    case 1: GB_DGS_LAUNCH(1); break;
    case 2: GB_DGS_LAUNCH(2); break;
    case 3: GB_DGS_LAUNCH(3); break;
    case 4: GB_DGS_LAUNCH(4); break;
    case 5: GB_DGS_LAUNCH(5); break;
    case 6: GB_DGS_LAUNCH(6); break;
    case 7: GB_DGS_LAUNCH(7); break;
    default: GB_DGS_LAUNCH(8); break;
  }
#undef GB_DGS_LAUNCH
  GB_CUDA(cudaGetLastError());
  return 1;
}

int launch_dg_block_spmv(cudaStream_t st, int mode, int p, int count, const int *ent_el, const int *roff,
                         const long long *row_val, const long long *cx_off, const int *colx, const double *val,
                         const long long *dinv_off, const double *dinv, const double *x, const double *b,
                         double *out, int longest) {
  return launch_dg_block_spmv_t<double>(st, mode, p, count, ent_el, roff, row_val, cx_off, colx, val, dinv_off,
                                        dinv, x, b, out, longest);
}

int launch_dg_block_spmv32(cudaStream_t st, int mode, int p, int count, const int *ent_el, const int *roff,
                           const long long *row_val, const long long *cx_off, const int *colx, const float *val,
                           const long long *dinv_off, const float *dinv, const double *x, const double *b,
                           double *out) {
  return launch_dg_block_spmv_t<float>(st, mode, p, count, ent_el, roff, row_val, cx_off, colx, val, dinv_off,
                                       dinv, x, b, out);
}

int launch_dg_block_spmv_dw(cudaStream_t st, int mode, int p, int count, const int *ent_el, const int *roff,
                           const long long *row_val, const long long *cx_off, const int *colx, const void *val,
                           const long long *dinv_off, const void *dinv, const double *x, const double *b,
                           double *out) {
  return launch_dg_block_spmv_t<dw>(st, mode, p, count, ent_el, roff, row_val, cx_off, colx,
                                    reinterpret_cast<const dw *>(val), dinv_off, reinterpret_cast<const dw *>(dinv),
                                    x, b, out);
}

}  // namespace gbfem
