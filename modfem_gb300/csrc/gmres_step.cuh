// Device pieces of a restarted-GMRES step shared by the library's solver
// (gmres_dev.cu) and the serving engine (serve.cu): warp and block sums of the
// Gram-Schmidt dot products, the combination of Krylov vectors, and the step's
// scalar logic.  Krylov vectors after the first are stored unnormalised with a
// scale each (V_k = sc_k W_k).
#pragma once

namespace gbfem {

// Sums of eight values over a warp: afterwards lane l holds the sum of value
// l / 4.  Each exchange halves the values a lane keeps: 9 adds instead of 40.
__device__ __forceinline__ double gm_warp_sums(double (&t)[8], int lane) {
#pragma unroll
  for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int u = 0; u < h; u++) {
      const double send = up ? t[u] : t[u + h], keep = up ? t[u + h] : t[u];
      t[u] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double v = t[0];
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

// pairwise sum of N shared values at stride `st` (short chain of dependent adds)
template <int N>
__device__ __forceinline__ double gm_pairs(const double *p, int st) {
  if constexpr (N == 1)
    return p[0];
  else
    return gm_pairs<N / 2>(p, st) + gm_pairs<N - N / 2>(p + (N / 2) * st, st);
}

// Column sums k <= j of `rows` rows of block partials (leading dimension ld) by
// a block of T threads, in an order that depends on the sizes only: out[k] in
// shared memory.  Lanes take consecutive k of one row, groups of lanes the
// rows in turn, eight rows in flight.
template <int T>
__device__ __forceinline__ void gm_sum_dots(const double *partial, int rows, int ld, int j, double *out) {
  __shared__ double red[T];
  const int tid = threadIdx.x;
  for (int kb = 0; kb <= j; kb += 32) {
    const int nk = min(32, j + 1 - kb), kw = nk <= 8 ? 8 : nk <= 16 ? 16 : 32, G = T / kw, k = tid % kw, g = tid / kw;
    const double *p = partial + kb + k;
    double v = 0.0;
    for (int r = g; r < rows; r += 8 * G) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; u++) x[u] = k < nk && r + u * G < rows ? __ldg(p + (size_t)(r + u * G) * ld) : 0.0;
      v += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
    }
    for (int o = kw; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) < kw) red[(tid >> 5) * 32 + (tid & 31)] = v;
    __syncthreads();
    if (tid < nk) out[kb + tid] = gm_pairs<T / 32>(red + tid, 32);
    __syncthreads();
  }
}

// sum_k c[k] V_k[i], U vectors' loads in flight, two accumulators (an FP64 FMA
// waits long for the one before it).  An incomplete group's FMAs are predicated:
// in the small systems that take U = 32 a branch around every four of them costs
// more than it saves (9,261 rows: 0.7 us a step).
template <int U>
__device__ __forceinline__ double gm_combine(const double *V, long long n, const double *c, int nk, long long i) {
  double a0 = 0.0, a1 = 0.0;
  const double *v = V + i;
  for (int k = 0; k < nk; k += U) {
    double x[U];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (k + u < nk) x[u] = __ldg(v + (size_t)(k + u) * n);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (k + u < nk) {
        if (u & 1)
          a1 = fma(c[k + u], x[u], a1);
        else
          a0 = fma(c[k + u], x[u], a0);
      }
  }
  return a0 + a1;
}

// out[q] = sum_k c[k] V_k[i + q T], q < R: R rows' chains of FMAs side by side and
// 4 R loads in flight
template <int R>
__device__ __forceinline__ void gm_combine_rows(const double *V, long long n, const double *c, int nk, long long i,
                                                int T, double (&out)[R]) {
  const double *v = V + i;
#pragma unroll
  for (int q = 0; q < R; q++) out[q] = 0.0;
  int k = 0;
  for (; k + 4 <= nk; k += 4, v += 4 * n) {
    double x[4][R];
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int q = 0; q < R; q++) x[u][q] = __ldg(v + u * n + q * T);
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int q = 0; q < R; q++) out[q] = fma(c[k + u], x[u][q], out[q]);
  }
  for (; k < nk; k++, v += n)
#pragma unroll
    for (int q = 0; q < R; q++) out[q] = fma(c[k], __ldg(v + q * T), out[q]);
}

// The step's logic for step j (one block of T threads): |w| from the norm
// partials, the earlier rotations applied to the Hessenberg column (the chain
// c_{k+1} = rc_k h_{k+1} - rs_k c_k composes affine maps by a warp scan, 5 steps
// per 32 rotations: an FP64 operation takes tens of cycles), the new rotation,
// the residual estimate and the decision (next step, or end of the cycle,
// where the block also solves R y = s by columns).  Thread 0 calls
// decide(resid, hn): it stores the caller's state and returns whether the cycle
// ends.
struct GmStep {
  int m, ng, nstride;   // Krylov dimension; norm partials and their stride
  const double *npart;
  double *H, *cs, *sn, *s, *y, *hcol, *sc;
};
template <int T, int MMAX, class Decide>
__device__ __forceinline__ void gm_step_logic(const GmStep &a, int j, Decide decide) {
  __shared__ double col[MMAX + 2];
  __shared__ double sh[T / 32];
  __shared__ int s_done;
  const int tid = threadIdx.x, ld = a.m + 1;
  double v = 0.0;
  for (int b = tid; b < a.ng; b += 4 * T) {
    double x[4];
#pragma unroll
    for (int u = 0; u < 4; u++) x[u] = b + u * T < a.ng ? a.npart[(size_t)(b + u * T) * a.nstride] : 0.0;
    v += (x[0] + x[1]) + (x[2] + x[3]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((tid & 31) == 0) sh[tid >> 5] = v;
  __syncthreads();
  if (tid < 32) {
    double *H = a.H + (size_t)j * ld;
    double c = a.hcol[0];
    for (int k0 = 0; k0 < j; k0 += 32) {
      const int k = k0 + tid;
      const double rc = k < j ? a.cs[k] : 1.0, rs = k < j ? a.sn[k] : 0.0, hk = k < j ? a.hcol[k + 1] : 0.0;
      double A = k < j ? -rs : 1.0, B = rc * hk;  // (identity beyond the last rotation)
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double A1 = __shfl_up_sync(0xffffffffu, A, o), B1 = __shfl_up_sync(0xffffffffu, B, o);
        if (tid >= o) {
          B = fma(A, B1, B);
          A *= A1;
        }
      }
      const double next = fma(A, c, B);  // c_{k+1}
      double prev = __shfl_up_sync(0xffffffffu, next, 1);
      if (tid == 0) prev = c;
      if (k < j) H[k] = fma(rc, prev, rs * hk);
      c = __shfl_sync(0xffffffffu, next, 31);
    }
    if (tid == 0) {
      const double h2 = gm_pairs<T / 32>(sh, 1), hn = sqrt(h2);
      const double rr = hypot(c, hn), cj = c / rr, sj = hn / rr;
      H[j] = rr;
      H[j + 1] = 0.0;
      a.cs[j] = cj;
      a.sn[j] = sj;
      const double s0 = a.s[j], s1 = -sj * s0, resid = fabs(s1);
      a.s[j] = cj * s0;
      a.s[j + 1] = s1;
      a.sc[j + 1] = 1.0 / hn;
      s_done = decide(resid, hn);
    }
  }
  __syncthreads();
  if (!s_done) return;
  // y = R^-1 s by columns, then scaled to the stored W_k
  if (j < 32) {
    // one warp, lane i holds row i: R's columns and the reciprocals of its
    // diagonal loaded at once, then a product, a shuffle and an FMA a column
    if (tid >= 32) return;
    double R[32], y = tid <= j ? a.s[tid] : 0.0;
#pragma unroll
    for (int k = 0; k < 32; k++) R[k] = k <= j && tid <= k ? a.H[(size_t)k * ld + tid] : 0.0;
    const double rd = tid <= j ? 1.0 / a.H[(size_t)tid * ld + tid] : 0.0;
#pragma unroll
    for (int k = 31; k >= 0; k--) {
      if (k > j) continue;
      const double yk = __shfl_sync(0xffffffffu, y * rd, k);
      y = tid == k ? yk : fma(-R[k], yk, y);
    }
    if (tid <= j) a.y[tid] = y * a.sc[tid];
    return;
  }
  for (int k = tid; k <= j; k += T) col[k] = a.s[k];
  __syncthreads();
  for (int k = j; k >= 0; k--) {
    const double *Hk = a.H + (size_t)k * ld;
    if (tid == 0) col[k] = col[k] / Hk[k];
    __syncthreads();
    const double yk = col[k];
    for (int i = tid; i < k; i += T) col[i] -= Hk[i] * yk;
    __syncthreads();
  }
  for (int k = tid; k <= j; k += T) a.y[k] = col[k] * a.sc[k];
}

}  // namespace gbfem
