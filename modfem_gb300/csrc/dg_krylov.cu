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
// index on ties) of the diagonal blocks of one class, each block held in
// shared memory by a group of G threads: a warp up to 40 functions (p = 3: 17
// blocks per SM, no CTA barriers), four warps for 75.  n^3 FMA a block bound
// it by the FP64 pipe (p = 3: 2,000 of 2,400 FP64 warp instructions); the
// pivot search compares bit patterns on the integer pipe.  54,000 blocks of
// 40: 16.1 ms with 256 threads and five barriers a step, 13.8 ms so.
template <int P>
struct DgInv {
  static constexpr int NS = DgSpmvDims<P>::NS;
  static constexpr int G = NS > 40 ? 128 : 32;            // threads per block
  static constexpr int CTA = 128, PER = CTA / G;          // blocks per CTA
  static constexpr int SZ = NS * NS + 2 * NS + (NS + 1) / 2 + 1;  // doubles per block
  static constexpr int BYTES = 8 * SZ * PER;
};

template <int P>
__global__ void __launch_bounds__(DgInv<P>::CTA) dg_block_inverse_kernel(
    int count, const int *__restrict__ ent_el, const long long *__restrict__ boff_diag, const double *__restrict__ val,
    const long long *__restrict__ dinv_off, double *__restrict__ dinv, int *err) {
  using D = DgInv<P>;
  constexpr int n = D::NS, G = D::G;
  extern __shared__ double smem[];
  const int grp = threadIdx.x / G, l = threadIdx.x % G, lane = threadIdx.x % 32;
  const int idx = blockIdx.x * D::PER + grp;
  if (idx >= count) return;  // whole warps (or the whole CTA)
  const int e = ent_el[idx];
  double *a = smem + (size_t)grp * D::SZ, *fcol = a + n * n, *prow = fcol + n;
  int *piv = reinterpret_cast<int *>(prow + n);
  auto sync = [] {
    if (G == 32)
      __syncwarp();
    else
      __syncthreads();
  };
  const double *src = val + boff_diag[e];
  for (int t = l; t < n * n; t += G) a[t] = src[t];
  sync();
  for (int k = 0; k < n; k++) {
    // every warp of the group finds the same pivot row: magnitudes as
    // integers (a NaN is never chosen), a zero column has none
    long long best = 0;
    int r = n;
    for (int i = k + lane; i < n; i += 32) {
      const long long v = __double_as_longlong(a[i + n * k]) & 0x7fffffffffffffffll;
      if (v > best && v <= 0x7ff0000000000000ll) {
        best = v;
        r = i;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, r, o);
      if (ov > best || (ov == best && oi < r)) {
        best = ov;
        r = oi;
      }
    }
    if (r >= n) {  // singular diagonal block (uniform across the group)
      if (l == 0) atomicExch(err, 3);
      return;
    }
    if (l == 0) piv[k] = r;
    const double pinv = 1.0 / a[r + n * k];
    // column k with rows k and r exchanged
    for (int i = l; i < n; i += G) fcol[i] = a[(i == r ? k : i) + n * k];
    sync();
    for (int j = l; j < n; j += G) {
      const double x = j == k ? pinv : a[r + n * j] * pinv;
      a[r + n * j] = a[k + n * j];
      a[k + n * j] = x;
      prow[j] = x;
    }
    sync();
    for (int t = l; t < n * n; t += G) {
      const int j = t / n, i = t - j * n;
      if (i == k) continue;
      a[t] = j == k ? -fcol[i] * pinv : fma(-fcol[i], prow[j], a[t]);
    }
    sync();
  }
  // undo the row interchanges as column interchanges, last first
  for (int k = n - 1; k >= 0; k--) {
    const int r = piv[k];
    if (r != k)
      for (int i = l; i < n; i += G) {
        const double t = a[i + n * k];
        a[i + n * k] = a[i + n * r];
        a[i + n * r] = t;
      }
    sync();
  }
  double *dst = dinv + dinv_off[e];
  for (int t = l; t < n * n; t += G) dst[t] = a[t];
}

int launch_dg_block_inverse(cudaStream_t st, int cls, int count, const int *ent_el, const long long *boff_diag,
                            const double *val, const long long *dinv_off, double *dinv, int *err) {
  if (count <= 0) return 0;
#define GB_INV(PP)                                                                                              \
  {                                                                                                             \
    using D = DgInv<PP>;                                                                                        \
    GB_CUDA(cudaFuncSetAttribute(dg_block_inverse_kernel<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize,      \
                                 D::BYTES));                                                                    \
    dg_block_inverse_kernel<PP><<<(count + D::PER - 1) / D::PER, D::CTA, D::BYTES, st>>>(count, ent_el,         \
                                                                                         boff_diag, val,        \
                                                                                         dinv_off, dinv, err);  \
  }
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
                                  double *out) {
  if (count <= 0) return 0;
  GB_CHECK(mode >= 0 && mode <= 2, "bad block SpMV mode");
  GB_CHECK(p >= 1 && p <= 2 * GB_DG_PMAX, "DG block class must be 1..8 (prisms 1..4, tetrahedra 5..8)");
  GB_CHECK(mode == 2 || (dinv && dinv_off), "block SpMV needs the inverted diagonal blocks");
  const int grid = (count + DGS_ROWS - 1) / DGS_ROWS;
#define GB_DGS_LAUNCH(PP)                                                                                      \
  if constexpr (std::is_same<VT, double>::value) {                                                             \
    if (count <= dgs_wide_max(PP)) {                                                                            \
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
                         double *out) {
  return launch_dg_block_spmv_t<double>(st, mode, p, count, ent_el, roff, row_val, cx_off, colx, val, dinv_off,
                                        dinv, x, b, out);
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
