// Block-row SpMV of the DG variable-block storage (device code shared by the
// plain kernels and the serving engine's slot kernels).
#pragma once

#include "dword.cuh"
#include "gmres_step.cuh"

namespace gbfem {

// One 8-lane group per block row (32 block rows per CTA), launched per
// degree class so that the row block size NS is a compile-time constant:
// lane g accumulates rows g, g+8, ... (40 rows = 5 full slots for p = 3, 75 =
// 10 slots of which the last is 3/8 full for p = 4).  On GB300 the SpMV is
// bound by the FP64 pipe as much as by HBM (one FMA per 8-byte value against
// ~0.6 T FMA/s), so lanes must not idle: a warp per row would leave 24 of 64
// lane slots empty for NS = 40.
//
// The blocks of a row are consecutive and column-major with leading dimension
// NS, so the whole block row is one NS x nct column-major matrix starting at
// the row's first block; colx lists the dof index of each of its nct columns.
// One flat loop over the columns (instead of blocks, then columns) keeps the
// four groups of a warp in step when their neighbours differ in degree; the
// rows of a class are ordered by nct for the same reason.  With a
// preconditioner the group's rows go through shared memory into the product
// with the inverted diagonal block.  The arithmetic type VT is double, float
// (inner solves of iterative refinement) or dw (double words on the FP32
// pipes: the FP64 pipe bounds the double form at ~5 TB/s of values, below
// HBM; the double-word form is bound by HBM).
constexpr int DGS_LANES = 8;
constexpr int DGS_THREADS = 256;
constexpr int DGS_ROWS = DGS_THREADS / DGS_LANES;

__device__ __forceinline__ double dgs_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float dgs_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ dw dgs_fma(dw a, dw b, dw c) { return t_fma(a, b, c); }
// vector entries into the arithmetic type and results back to FP64
template <typename VT>
__device__ __forceinline__ VT dgs_in(double v) {
  return (VT)v;
}
template <>
__device__ __forceinline__ dw dgs_in<dw>(double v) {
  return dw_from_double(v);
}
__device__ __forceinline__ double dgs_out(double v) { return v; }
__device__ __forceinline__ double dgs_out(float v) { return (double)v; }
__device__ __forceinline__ double dgs_out(dw v) { return dw_to_double(v); }

// P: block class, 1..4 tensor-basis prisms of degree P (6, 18, 40, 75
// functions), 5..8 complete-basis tetrahedra of degree P - 4 (4, 10, 20, 35)
template <int P>
struct DgSpmvDims {
  static constexpr int NS = P == 1 ? 6 : P == 2 ? 18 : P == 3 ? 40 : P == 4 ? 75
                          : P == 5 ? 4 : P == 6 ? 10 : P == 7 ? 20 : 35;
};

// The body of the block SpMV for the block rows of one CTA (blockDim.x ==
// DGS_THREADS); sv: DGS_ROWS x NS values of shared memory.  VT is the type of
// the stored matrix and of the arithmetic (double, or float for the inner
// solves of iterative refinement); vectors are FP64 either way.
template <int P, typename VT = double>
__device__ __forceinline__ void dg_block_row_spmv(
    int mode, int count, const int *__restrict__ ent_el, const int *__restrict__ roff,
    const long long *__restrict__ row_val, const long long *__restrict__ cx_off, const int *__restrict__ colx,
    const VT *__restrict__ val, const long long *__restrict__ dinv_off, const VT *__restrict__ dinv,
    const double *__restrict__ x, const double *__restrict__ b, double *__restrict__ out,
    VT (*sv)[DgSpmvDims<P>::NS]) {
  constexpr int NS = DgSpmvDims<P>::NS;
  constexpr int S = (NS + DGS_LANES - 1) / DGS_LANES;
  const int grp = threadIdx.x / DGS_LANES, g = threadIdx.x % DGS_LANES;
  const int idx = blockIdx.x * DGS_ROWS + grp;
  const bool active = idx < count;
  const int e = active ? ent_el[idx] : 0;
  const int r0 = roff[e];
  VT acc[S];
#pragma unroll
  for (int s = 0; s < S; s++) acc[s] = VT(0);
  if (active) {
    const VT *A = val + row_val[e] + g;
    const int *cx = colx + cx_off[e];
    const int nct = (int)(cx_off[e + 1] - cx_off[e]);
    int t = 0;
    for (; t + 2 <= nct; t += 2) {
      const VT x0 = dgs_in<VT>(x[cx[t]]), x1 = dgs_in<VT>(x[cx[t + 1]]);
      const VT *col0 = A + (size_t)t * NS, *col1 = col0 + NS;
#pragma unroll
      for (int s = 0; s < S; s++)
        if (g + DGS_LANES * s < NS) acc[s] = dgs_fma(col1[DGS_LANES * s], x1, dgs_fma(col0[DGS_LANES * s], x0, acc[s]));
    }
    if (t < nct) {
      const VT x0 = dgs_in<VT>(x[cx[t]]);
      const VT *col0 = A + (size_t)t * NS;
#pragma unroll
      for (int s = 0; s < S; s++)
        if (g + DGS_LANES * s < NS) acc[s] = dgs_fma(col0[DGS_LANES * s], x0, acc[s]);
    }
  }
  if (mode != 1) {
#pragma unroll
    for (int s = 0; s < S; s++) {
      const int i = g + DGS_LANES * s;
      acc[s] = (b && active && i < NS ? dgs_in<VT>(b[r0 + i]) : VT(0)) - acc[s];
    }
  }
  if (mode == 2) {
    if (active) {
#pragma unroll
      for (int s = 0; s < S; s++) {
        const int i = g + DGS_LANES * s;
        if (i < NS) out[r0 + i] = dgs_out(acc[s]);
      }
    }
    return;
  }
#pragma unroll
  for (int s = 0; s < S; s++) {
    const int i = g + DGS_LANES * s;
    if (i < NS) sv[grp][i] = acc[s];
  }
  __syncwarp();
  if (!active) return;
  const VT *D = dinv + dinv_off[e] + g;
  VT o[S];
#pragma unroll
  for (int s = 0; s < S; s++) o[s] = VT(0);
  for (int j = 0; j < NS; j++) {
    const VT t = sv[grp][j];
    const VT *col = D + (size_t)j * NS;
#pragma unroll
    for (int s = 0; s < S; s++)
      if (g + DGS_LANES * s < NS) o[s] = dgs_fma(col[DGS_LANES * s], t, o[s]);
  }
#pragma unroll
  for (int s = 0; s < S; s++) {
    const int i = g + DGS_LANES * s;
    if (i < NS) out[r0 + i] = dgs_out(o[s]);
  }
}

// One block row by a whole CTA of DGS_THREADS threads, for systems too small to
// fill the chip with eight-lane groups (250 prisms of degree 2 are 8 CTAs of
// them, and a group walks a row's 104 columns alone): the columns are split
// over C = 256 / NS groups of NS threads (a thread a row), four or eight loads
// in flight, the partial sums added pairwise, then the same for the inverted
// diagonal block.  The order depends on the class only.
template <int P>
struct DgWide {
  static constexpr int NS = DgSpmvDims<P>::NS, C = DGS_THREADS / NS;
  static constexpr int U = NS >= 35 ? 8 : 4;  // loads in flight
};
// Block rows of a class up to which the CTA form is the faster one (measured
// crossovers; us a product, CTA form against groups of eight lanes):
//   prisms  p = 1: 432 rows 10.7 / 11.1, 1,024 18 / 12;   p = 2: 2,000 23 / 37, 6,750 67 / 68
//           p = 3: 2,000 63 / 200, 11,664 290 / 275;      p = 4: 2,000 183 / 863, 11,664 939 / 1,033
//   tetrahedra p = 1: never;                              p = 2: 1,296 16 / 18, 2,058 21 / 18
//           p = 3: 2,058 25 / 38, 6,000 61 / 64;          p = 4: 2,058 52 / 134, 10,368 211 / 197
// (the groups' time stays flat until they fill the chip: they walk a row's
// columns one or two at a time).  In meshes of mixed degrees the rows of the low
// classes are longer and the groups' walk with them, so the limit grows with
// the class's longest row over that of a uniform mesh (6 or 5 blocks of its own).
// Degrees 1..4 mixed, rows a class: prisms p = 1 2,048 22 / 97, 6,912 55 / 100, 16,384
// 124 / 103 (limit 6,400); p = 2..4 16,384 183 / 246, 335 / 419, 653 / 1,000; tetrahedra
// p = 1 1,500 15 / 40, 6,144 46 / 38 (4,480); p = 2 6,144 38 / 68, 15,972 90 / 75 (5,376).
__host__ __device__ constexpr int dgs_wide_max(int cls, int longest = 0) {
  constexpr int base[9] = {0, 512, 6656, 10000, 13000, 512, 1536, 6144, 8192};
  constexpr int own[9] = {1, 36, 108, 240, 450, 20, 50, 100, 175};
  if (cls == 5 && longest < 2 * own[5]) return 0;
  return longest <= own[cls] ? base[cls] : (int)((long long)base[cls] * longest / own[cls]);
}
template <int P>
__device__ __forceinline__ double dg_wide_product(const double *__restrict__ A, int nct, const int *__restrict__ cx,
                                                  const double *x, double *red) {
  constexpr int NS = DgWide<P>::NS, C = DgWide<P>::C, U = DgWide<P>::U;
  const int i = threadIdx.x % NS, g = threadIdx.x / NS;
  double acc = 0.0;
  if (g < C)
    for (int t = g; t < nct; t += U * C) {
      double a[U], v[U];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (t + u * C < nct) {
          a[u] = A[(size_t)(t + u * C) * NS + i];
          v[u] = x[cx ? cx[t + u * C] : t + u * C];
        }
#pragma unroll
      for (int u = 0; u < U; u++)
        if (t + u * C < nct) acc = fma(a[u], v[u], acc);
    }
  if (g < C) red[g * NS + i] = acc;
  __syncthreads();
  return threadIdx.x < NS ? gm_pairs<C>(red + threadIdx.x, NS) : 0.0;
}
// (mode and arguments as dg_block_row_spmv; block row of element e)
template <int P>
__device__ __forceinline__ void dg_block_row_wide(int mode, int e, const int *__restrict__ roff,
                                                  const long long *__restrict__ row_val,
                                                  const long long *__restrict__ cx_off, const int *__restrict__ colx,
                                                  const double *__restrict__ val,
                                                  const long long *__restrict__ dinv_off,
                                                  const double *__restrict__ dinv, const double *__restrict__ x,
                                                  const double *__restrict__ b, double *__restrict__ out) {
  constexpr int NS = DgWide<P>::NS;
  __shared__ double red[DGS_THREADS], y[NS];
  const int r0 = roff[e], tid = threadIdx.x;
  const long long c0 = cx_off[e];
  double s = dg_wide_product<P>(val + row_val[e], (int)(cx_off[e + 1] - c0), colx + c0, x, red);
  if (tid < NS && mode != 1) s = (b ? b[r0 + tid] : 0.0) - s;
  if (mode == 2) {
    if (tid < NS) out[r0 + tid] = s;
    return;
  }
  if (tid < NS) y[tid] = s;
  __syncthreads();
  s = dg_wide_product<P>(dinv + dinv_off[e], NS, nullptr, y, red);
  if (tid < NS) out[r0 + tid] = s;
}

}  // namespace gbfem
