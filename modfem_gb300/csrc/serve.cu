// Serving engine: independent FE problems (std linear or DG prisms) arriving
// over time are integrated, assembled and solved on one GPU with continuous
// batching.  No counterpart in the reference (ModFEM solves one problem per
// process); the per-request numerics are the library's own
// (gbfem_assemble / gbfem_dg_assemble, GMRES with Jacobi / block Jacobi).
//
// Pipeline:
//  * two lanes, std and DG requests, each with its own FIFO admission queue,
//    slot quota, CUDA stream (std at the highest priority, DG at the lowest),
//    step graph and state readback, polled independently: a std request
//    never waits for a DG request's FP64-bound block SpMVs, nor behind DG
//    requests in the queue;
//  * admission: FIFO per lane; a request starts when its lane has a free slot
//    (half of max_active, or more while the other lane has nobody waiting)
//    and its estimated device footprint fits in the shared HBM budget
//    (replaced by the measured footprint once it is built).  Std requests of
//    GBFEM_SERVE_OPT_SOLO_DOFS dofs or more never enter the engine's lanes:
//    they are admitted on the budget alone;
//  * preparation (worker threads, one CUDA stream each, std requests' at a
//    high priority, solo-sized ones' at the highest; solo-sized std
//    requests taken first, then the other
//    std ones, then DG): upload, structure (built on the device for std
//    requests), integrate + assemble, preconditioner; overlaps with
//    the solves running.  Solo-sized requests are then solved by one of eight
//    solo threads, alone on their stream, with the device-resident GMRES of
//    gbfem_solve;
//  * solve (engine thread, one stream per lane): every step of a lane
//    advances each of its active requests by one GMRES iteration with
//    batched kernels over all of them - one CRS SpMV launch for all std
//    requests, one launch per degree class for each DG request, and one
//    launch each for the Gram-Schmidt dot products, the orthogonalisation and
//    the scalar GMRES logic (Hessenberg column, Givens rotations, convergence
//    test, restart and the small triangular solve, one block a request), so a
//    step needs no host round trip per request; the host reads the requests'
//    phases every few steps to retire finished ones and admit new ones
//    between steps.  What a step does for a request depends on its phase:
//    residual at a restart, Arnoldi step, or update of x at the end of a
//    cycle (a cycle of m Arnoldi steps takes m + 2 engine steps).
//
// Assembly is deterministic (the gather scatter for std requests, one
// owning thread per block entry for DG) and every request's reductions are
// partitioned by its own size only and summed in a fixed order, so its result
// does not depend on which other requests share the steps: a request gives
// the same bits alone and in a mix.
//
// The kernel sequence of a lane's step depends only on its set of active
// requests (their state lives on the device): it is launched kernel by kernel
// after a change of that set, and once the set has stood for some polls it is
// captured as a CUDA graph and replayed every step (a capture costs as much as
// dozens of steps' launches; in a burst the set changes every few steps).

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "dg_spmv.cuh"
#include "dg_tables.h"
#include "gbfem_internal.h"
#include "gmres_step.cuh"

namespace gbfem {

constexpr int SRV_MAXSLOTS = 64;
constexpr int SRV_MMAX = 64;              // largest Krylov dimension of a served request
constexpr int SRV_PART = SRV_MMAX + 2;    // per reduction block: dots 0..m, norm at SRV_MMAX + 1
constexpr int SRV_T = 256;
constexpr int SRV_SPMV_LANES = 8;         // a prism row's 21 entries: three rounds
constexpr int SRV_SPMV_ROWS = SRV_T / SRV_SPMV_LANES;
constexpr int SRV_RED = 160;              // reduction blocks of a request at most
// Entries per reduction block of a request of n unknowns: one a thread (the step
// of a small request is memory latency) until the blocks are SRV_RED, since
// every block of the orthogonalisation sums the partials of all.  By the
// request's size only, so its sums are the same in every mix.
constexpr int srv_chunk(int n) { return SRV_T * ((n + SRV_T * SRV_RED - 1) / (SRV_T * SRV_RED)); }

enum { PH_RESTART = 0, PH_ARNOLDI = 1, PH_DONE = 2, PH_UPDATE = 3 };

// host-written description of an active request
struct SrvDesc {
  int kind;  // 0 std CRS (point Jacobi), 1 DG blocks (block Jacobi)
  int n, m, max_iter;
  double tol_rel, tol_abs;
  const int *row_ptr, *col_ind;
  const double *val, *dinv;
  const int *roff, *colx;
  const long long *row_val, *cx_off, *dinv_off;
  const double *dgval, *dgdinv;
  const double *b;
  double *x, *V, *tmp, *H, *cs, *sn, *s, *y, *hcol, *sc;
  int red_first, red_nb, chunk;
};

// device-written GMRES state of a request
struct SrvState {
  int phase, j, it, done_cols, final_flag, pad[3];
  double beta0, resid;
};

// CRS rows of the std requests: restart residual tmp = dinv (b - A x), or
// W_{j+1} = dinv A W_j in an Arnoldi step.
__global__ void __launch_bounds__(SRV_T) srv_crs_spmv(const int2 *map, const SrvDesc *dd, const SrvState *ss) {
  const int2 mp = map[blockIdx.x];
  const SrvDesc &D = dd[mp.x];
  const SrvState &S = ss[mp.x];
  const bool restart = S.phase == PH_RESTART;
  if (!restart && S.phase != PH_ARNOLDI) return;  // uniform over the block
  const int lane = threadIdx.x & (SRV_SPMV_LANES - 1);
  const long long r = (long long)mp.y + threadIdx.x / SRV_SPMV_LANES;
  const bool valid = r < D.n;
  const double *x = restart ? D.x : D.V + (size_t)S.j * D.n;
  double *out = restart ? D.tmp : D.V + (size_t)(S.j + 1) * D.n;
  const int lo = valid ? D.row_ptr[r] : 0, hi = valid ? D.row_ptr[r + 1] : 0;
  double s = 0.0;
  for (int k = lo + lane; k < hi; k += 4 * SRV_SPMV_LANES) {  // up to 32 entries of a row in flight
    double a[4], xv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int q = k + u * SRV_SPMV_LANES;
      a[u] = q < hi ? D.val[q] : 0.0;
      xv[u] = q < hi ? x[D.col_ind[q]] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (k + u * SRV_SPMV_LANES < hi) s = fma(a[u], xv[u], s);
  }
#pragma unroll
  for (int o = SRV_SPMV_LANES / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, SRV_SPMV_LANES);
  if (valid && lane == 0) out[r] = restart ? (D.b[r] - s) * D.dinv[r] : D.dinv[r] * s;
}

// the block rows of degree P of one DG request (the same two forms); WIDE:
// one CTA a block row
template <int P, bool WIDE>
__global__ void __launch_bounds__(DGS_THREADS) srv_dg_spmv(int slot, int count, const int *ent_el,
                                                           const SrvDesc *dd, const SrvState *ss) {
  const SrvDesc &D = dd[slot];
  const SrvState &S = ss[slot];
  const bool restart = S.phase == PH_RESTART;
  if (!restart && S.phase != PH_ARNOLDI) return;
  const double *x = restart ? D.x : D.V + (size_t)S.j * D.n, *b = restart ? D.b : nullptr;
  double *out = restart ? D.tmp : D.V + (size_t)(S.j + 1) * D.n;
  if constexpr (WIDE) {
    dg_block_row_wide<P>(restart ? 0 : 1, ent_el[blockIdx.x], D.roff, D.row_val, D.cx_off, D.colx, D.dgval,
                         D.dinv_off, D.dgdinv, x, b, out);
  } else {
    __shared__ double sv[DGS_ROWS][DgSpmvDims<P>::NS];
    dg_block_row_spmv<P>(restart ? 0 : 1, count, ent_el, D.roff, D.row_val, D.cx_off, D.colx, D.dgval, D.dinv_off,
                         D.dgdinv, x, b, out, sv);
  }
}

// Block partials of <W_k, W_{j+1}>, k <= j, or of <tmp, tmp> at a restart:
// sixteen vectors at a time, so that a small request (one row a thread) waits
// for memory once per sixteen.
__global__ void __launch_bounds__(SRV_T) srv_dots(const int2 *map, const SrvDesc *dd, const SrvState *ss,
                                                  double *partial) {
  constexpr int W = SRV_T / 32, KP = SRV_MMAX;
  __shared__ double part[W][KP];
  const int2 mp = map[blockIdx.x];
  const SrvDesc &D = dd[mp.x];
  const SrvState &S = ss[mp.x];
  const bool restart = S.phase == PH_RESTART;
  if (!restart && S.phase != PH_ARNOLDI) return;
  const int j = restart ? 0 : S.j, l = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long n = D.n, end = min(n, (long long)mp.y + D.chunk);
  const double *w = restart ? D.tmp : D.V + (size_t)(j + 1) * n, *V = restart ? D.tmp : D.V;
  for (int k0 = 0; k0 <= j; k0 += 16) {
    double t[2][8];
#pragma unroll
    for (int u = 0; u < 16; u++) t[u / 8][u % 8] = 0.0;
    for (long long i = mp.y + threadIdx.x; i < end; i += SRV_T) {
      const double wi = w[i];
      double x[16];
#pragma unroll
      for (int u = 0; u < 16; u++)
        if (k0 + u <= j) x[u] = V[(size_t)(k0 + u) * n + i];
#pragma unroll
      for (int u = 0; u < 16; u++)
        if (k0 + u <= j) t[u / 8][u % 8] = fma(x[u], wi, t[u / 8][u % 8]);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (k0 + 8 * h > j) break;
      const double d = gm_warp_sums(t[h], l);
      if ((l & 3) == 0) part[warp][k0 + 8 * h + (l >> 2)] = d;
    }
  }
  __syncthreads();
  double *out = partial + (size_t)(D.red_first + mp.y / D.chunk) * SRV_PART;
  for (int k = threadIdx.x; k <= j; k += SRV_T) out[k] = gm_pairs<W>(&part[0][k], KP);
}

// Arnoldi step: h_k = sc_k sc_j <W_k, W_{j+1}>, W_{j+1} = sc_j W_{j+1} - sum_k h_k
// sc_k W_k and the block partials of its squared norm.  Restart: V_0 = tmp /
// |tmp|.  End of a cycle: x += sum_k y_k W_k.
__global__ void __launch_bounds__(SRV_T) srv_orthogonalize(const int2 *map, const SrvDesc *dd, const SrvState *ss,
                                                           double *partial) {
  constexpr int W = SRV_T / 32;
  __shared__ double coef[SRV_MMAX + 1], sh[W];
  const int2 mp = map[blockIdx.x];
  const SrvDesc &D = dd[mp.x];
  const SrvState &S = ss[mp.x];
  const int phase = S.phase;
  if (phase == PH_DONE) return;
  const long long n = D.n, end = min(n, (long long)mp.y + D.chunk);
  double *part = partial + (size_t)D.red_first * SRV_PART;
  if (phase == PH_UPDATE) {
    const int done = S.done_cols;
    for (int k = threadIdx.x; k < done; k += SRV_T) coef[k] = D.y[k];
    __syncthreads();
    for (long long i = mp.y + threadIdx.x; i < end; i += SRV_T) D.x[i] += gm_combine<16>(D.V, n, coef, done, i);
    return;
  }
  const int j = phase == PH_RESTART ? 0 : S.j;
  gm_sum_dots<SRV_T>(part, D.red_nb, SRV_PART, j, coef);
  if (phase == PH_RESTART) {
    const double inv = 1.0 / sqrt(coef[0]);
    for (long long i = mp.y + threadIdx.x; i < end; i += SRV_T) D.V[i] = D.tmp[i] * inv;
    return;
  }
  const double scj = D.sc[j];
  for (int k = threadIdx.x; k <= j; k += SRV_T) {
    const double sk = D.sc[k], h = sk * (scj * coef[k]);
    if (mp.y == 0) D.hcol[k] = h;
    coef[k] = h * sk;
  }
  __syncthreads();
  double *w = D.V + (size_t)(j + 1) * n, s = 0.0;
  for (long long i = mp.y + threadIdx.x; i < end; i += SRV_T) {
    const double wi = fma(scj, w[i], -gm_combine<16>(D.V, n, coef, j + 1, i));
    w[i] = wi;
    s = fma(wi, wi, s);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) part[(size_t)(mp.y / D.chunk) * SRV_PART + SRV_MMAX + 1] = gm_pairs<W>(sh, 1);
}

// The scalar logic, one block a request: the restart test
// (lss_mkb_core.c:2377-2400, as gbfem_solve), the Arnoldi column, or the
// end of a cycle's update.
constexpr int SRV_LOGIC_T = 128;
__global__ void __launch_bounds__(SRV_LOGIC_T) srv_logic(const int *act, const SrvDesc *dd, SrvState *ss,
                                                         const double *partial) {
  __shared__ double tot[1];
  const int slot = act[blockIdx.x];
  const SrvDesc &D = dd[slot];
  SrvState &S = ss[slot];
  const int phase = S.phase;
  const double *part = partial + (size_t)D.red_first * SRV_PART;
  if (phase == PH_ARNOLDI) {
    const int j = S.j;
    const GmStep g = {D.m, D.red_nb, SRV_PART, part + SRV_MMAX + 1, D.H, D.cs, D.sn, D.s, D.y, D.hcol, D.sc};
    gm_step_logic<SRV_LOGIC_T, SRV_MMAX>(g, j, [&](double resid, double) -> int {
      const int it = S.it + 1;
      S.it = it;
      S.resid = resid;
      const bool conv = resid < D.tol_abs || resid / S.beta0 < D.tol_rel;
      const bool end = j == D.m - 1 || it >= D.max_iter || conv;
      if (end) {
        S.done_cols = j + 1;
        S.final_flag = (conv || it >= D.max_iter) ? 1 : 0;
        S.phase = PH_UPDATE;
      } else {
        S.j = j + 1;
      }
      return end;
    });
  } else if (phase == PH_RESTART) {
    gm_sum_dots<SRV_LOGIC_T>(part, D.red_nb, SRV_PART, 0, tot);
    if (threadIdx.x != 0) return;
    const double rn = sqrt(tot[0]);
    if (S.beta0 < 0) S.beta0 = rn;
    S.resid = rn;
    if (rn < D.tol_abs || (S.beta0 > 0 && rn / S.beta0 < D.tol_rel) || S.it >= D.max_iter) {
      S.phase = PH_DONE;
      return;
    }
    D.s[0] = rn;
    for (int i = 1; i <= D.m; i++) D.s[i] = 0.0;
    D.sc[0] = 1.0;  // V_0 is stored normalised
    S.j = 0;
    S.done_cols = 0;
    S.phase = PH_ARNOLDI;
  } else if (phase == PH_UPDATE && threadIdx.x == 0) {
    S.phase = S.final_flag ? PH_DONE : PH_RESTART;
  }
}

}  // namespace gbfem

using gbfem::DevBuf;
using gbfem::SrvDesc;
using gbfem::SrvState;

namespace {

double now_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

const int kNs[5] = {0, 6, 18, 40, 75};

struct SrvRequest {
  long long id = 0;
  int kind = 0, p = 1, krylov = 30, max_iter = 1000;
  double tol = 1e-8, f = 1.0, g = 0.0, pen = 10.0;
  int nno = 0, nel = 0, nbf = 0, nfa = 0;
  std::vector<double> xyz, k;
  std::vector<int> el, bf_el, bf_side, fa_type, fa_bc, fa_el, fa_side, fa_nodes;
  long long footprint = 0, charged = 0;
  double t_submit = 0, t_admit = 0, t_ready = 0, t_start = 0, t_done = 0;
  int status = 0;  // 0 queued, 1 preparing, 2 ready, 3 solving, 4 done, -1 failed, -2 cancelled
  bool cancel = false;  // cancellation asked while preparing or solving
  bool solo = false;    // large std request: solved alone by a solo thread
  bool solo_admit = false;  // admitted as a solo request, outside the lane's slots
  std::string err;
  gbfem_ctx ctx = nullptr;
  DevBuf<double> kry;
  int n = 0, slot = -1;
  std::vector<double> x;
  int iters = 0;
  double rel = 0.0;
};

using ReqPtr = std::shared_ptr<SrvRequest>;

}  // namespace

// What a request's context and Krylov space will hold (a std request's sliced-ELL
// copy only when it is solved alone); the rounded part covers the small arrays
// and the basis tables of the face configurations.  ntri of the nfa faces are triangles.
long long gbfem_serve_footprint_impl(int kind, int p, int nno, int nel, int nbf, int nfa, int ntri, int krylov) {
  const long long m1 = krylov + 1;
  long long b = 24LL * nno + 24LL * nel + 8LL * nel + 16LL * nbf + (3LL << 18);
  if (kind == 0) {
    const long long n = nno, nnz = 27LL * nno;  // prism meshes hold about 21 entries per row
    b += 12LL * nnz + 4LL * (n + 1) + 4LL * nno + 168LL * nel;                // CRS, tables
    b += 336LL * nel + 28LL * nel + 4LL * (n + 2) + (112LL + 4) * nbf;        // gather scatter: local matrices, incidence, face lists
    b += 8LL * n * (m1 + 4) + 8LL * m1 * m1 + 8LL * 152 * (m1 + 8);           // Krylov
    b += 12LL * nnz + 4LL * n;                                                // sliced-ELL copy
  } else {
    const long long ns = kNs[p], n = ns * nel, blocks = nel + 2LL * nfa;
    b += 8LL * ns * ns * blocks + 8LL * ns * ns * nel + (4LL * ns + 12) * blocks + 64LL * nel;
    // half-faces, face records, point fields (7 doubles a point)
    b += (96 + 8 + (long long)sizeof(gbfem::DgFaceRec)) * nfa;
    b += 56LL * (GB_DG_NQF[p][0] * (long long)ntri + GB_DG_NQF[p][1] * (long long)(nfa - ntri));
    b += 8LL * n * (m1 + 4) + 8LL * m1 * m1;
  }
  return b;
}

// One lane of the engine: the active requests of one kind and what their
// batched steps need.
struct SrvLane {
  cudaStream_t stream = nullptr;
  cudaEvent_t done = nullptr;  // recorded after a poll's steps and state readback
  bool busy = false, changed = false;
  std::deque<ReqPtr> waitq;    // admission queue of this kind
  int held = 0;                // admitted and not yet retired
  std::vector<int> act;        // slots
  DevBuf<int2> d_map_vec, d_map_crs;
  DevBuf<int> d_act;
  DevBuf<double> d_partial;
  SrvState *h_state = nullptr;  // pinned readback of the last poll
  int n_vec = 0, n_crs = 0;
  cudaGraphExec_t graph = nullptr;  // of the current set, once it has stood
  int graph_kernels = 0, polls = 0;  // polls since the set changed
};

struct gbfem_server_s {
  int device = 0;
  long long budget = 0, in_use = 0, peak_in_use = 0;
  int max_active = 0;
  std::mutex mu;
  std::condition_variable cv_engine, cv_prep, cv_done, cv_solo;
  std::deque<ReqPtr> prepq, readyq;
  // prepared solo requests, solved by the solo threads (so that a long solve
  // does not hold a preparation worker)
  std::deque<ReqPtr> soloq;
  std::vector<std::thread> solo_workers;
  std::map<long long, ReqPtr> reqs;
  long long next_id = 0;
  int n_preparing = 0, n_active = 0;
  bool stop = false;
  std::vector<std::thread> workers;
  std::thread engine;
  // Contexts and Krylov spaces of finished requests wait here for the next
  // request of their kind: a new context's stream, events and some thirty
  // device allocations cost more than a small request's work, and each
  // cudaFree synchronises the device.  At most SRV_IDLE of a kind and an
  // eighth of the HBM budget; not charged to it, but freed as soon as an
  // admission needs the room, and with the server.
  struct Idle {
    int key = 0, nno = 0, nel = 0;  // key: kind, or 2 for solo-sized std requests (another stream priority)
    gbfem_ctx ctx = nullptr;
    DevBuf<double> kry;
    long long bytes = 0;
  };
  std::deque<Idle> idle;  // oldest first
  long long idle_bytes = 0;
  // the others are freed by the reaper thread (a cudaFree on the engine
  // thread would hold every lane until all GPU work drained)
  struct Reaped {
    gbfem_ctx ctx;
    double *kry;
    long long bytes;
  };
  std::deque<Reaped> reapq;
  long long reap_bytes = 0;  // held until the reaper has freed them
  std::condition_variable cv_reap;
  bool reap_stop = false;
  std::thread reaper;
  // engine-owned
  SrvLane lanes[2];  // 0: std requests, 1: DG requests
  ReqPtr slots[gbfem::SRV_MAXSLOTS];
  DevBuf<SrvDesc> d_desc;
  DevBuf<SrvState> d_state;
  SrvState *h_init = nullptr;  // pinned: initial states of newly started requests
  SrvDesc *h_desc = nullptr;
  long long steps = 0, launches = 0;
  int peak_active = 0;
  int steps_per_poll = 4;
  int inject_prep_failures = 0;  // GBFEM_SERVE_OPT_FAIL_PREPARATIONS
  int solo_dofs = 40000;         // GBFEM_SERVE_OPT_SOLO_DOFS
  int std_precedence = 1;        // GBFEM_SERVE_OPT_STD_PRECEDENCE
  std::atomic<int> n_solo{0};    // solo requests admitted and not finished
  int prio_std = 0;              // stream priority of std requests' contexts
  int prio_solo = 0;             // of solo-sized std requests' contexts (the greatest)
  std::string fatal;
};

namespace {

constexpr int SRV_IDLE = 8;
constexpr int SRV_CAPTURE_POLLS = 16;  // polls of one set before its step is captured

int idle_key(const SrvRequest &r) { return r.kind == 0 && r.solo_admit ? 2 : r.kind; }

void queue_reap(gbfem_server s, const gbfem_server_s::Idle &i) {  // caller holds s->mu
  s->reapq.push_back({i.ctx, i.kry.p, i.bytes});
  s->reap_bytes += i.bytes;
  s->cv_reap.notify_one();
}

void drop_oldest_idle(gbfem_server s) {  // caller holds s->mu
  s->idle_bytes -= s->idle.front().bytes;
  queue_reap(s, s->idle.front());
  s->idle.pop_front();
}

// Whether `bytes` more fit in the HBM budget (idle contexts give way, but not
// for a request that would have to wait all the same); a request larger than the
// budget runs alone.  What the reaper has still to free counts: it admits again
// afterwards.
bool fits(gbfem_server s, long long bytes) {  // caller holds s->mu
  if (s->in_use > 0 && s->in_use + bytes > s->budget) return false;
  while (!s->idle.empty() && s->in_use + s->idle_bytes + bytes > s->budget) drop_oldest_idle(s);
  return s->in_use + s->reap_bytes + bytes <= s->budget || s->in_use + s->reap_bytes == 0;
}

// A finished request's context and Krylov space (no device work of it may be
// in flight) are kept for another request; a failed one's go to the reaper.
void reap(gbfem_server s, SrvRequest &r, bool reusable = true) {
  gbfem_server_s::Idle i;
  i.key = idle_key(r);
  i.nno = r.nno;
  i.nel = r.nel;
  i.ctx = r.ctx;
  i.kry = r.kry;
  r.ctx = nullptr;
  r.kry = DevBuf<double>();  // ownership has passed
  if (!i.ctx && !i.kry.p) return;
  std::lock_guard<std::mutex> lk(s->mu);
  i.bytes = gbfem_device_bytes(i.ctx) + (long long)i.kry.bytes();
  if (i.ctx && reusable && !s->stop) {
    int same = 0;
    for (const auto &o : s->idle) same += o.key == i.key;
    while (!s->idle.empty() && same >= SRV_IDLE) {
      // the oldest of this kind makes room
      auto o = std::find_if(s->idle.begin(), s->idle.end(), [&](const gbfem_server_s::Idle &q) { return q.key == i.key; });
      std::swap(*o, s->idle.front());
      drop_oldest_idle(s);
      same--;
    }
    if (s->idle_bytes + i.bytes <= s->budget / 8 &&
        s->in_use - r.charged + s->reap_bytes + s->idle_bytes + i.bytes <= s->budget) {  // (its charge ends with it)
      s->idle_bytes += i.bytes;
      s->idle.push_back(i);
      return;
    }
  }
  queue_reap(s, i);
}

// An idle context for the request, of its own mesh size if there is one (its
// buffers then fit as they are).  What it holds is charged beside the estimate
// (buffers only grow, so the two together bound what it will hold) until the
// preparation puts the measured footprint in their place, or, for a request solved
// alone, until it is done.
bool take_idle(gbfem_server s, SrvRequest &r) {
  std::lock_guard<std::mutex> lk(s->mu);
  const int key = idle_key(r);
  auto best = s->idle.end();
  for (auto it = s->idle.begin(); it != s->idle.end(); ++it) {
    if (it->key != key) continue;
    best = it;
    if (it->nno == r.nno && it->nel == r.nel) break;
  }
  if (best == s->idle.end()) return false;
  r.ctx = best->ctx;
  r.kry = best->kry;
  s->idle_bytes -= best->bytes;
  s->in_use += best->bytes;
  r.charged += best->bytes;
  s->peak_in_use = std::max(s->peak_in_use, s->in_use);
  s->idle.erase(best);
  return true;
}

// A lane may hold half of max_active requests, or more while the other lane
// has nobody waiting; the HBM budget is shared.
void try_admit(gbfem_server s) {  // caller holds s->mu
  const int share = std::max(1, s->max_active / 2);
  // std requests of at least solo_dofs dofs (one per vertex) are solved by
  // their preparation worker on their own stream, not in the engine's
  // lanes: they take no lane slot, only their share of the HBM budget
  if (s->solo_dofs > 0) {
    auto &q = s->lanes[0].waitq;
    for (auto it = q.begin(); it != q.end();) {
      ReqPtr r = *it;
      if (r->nno < s->solo_dofs) {
        ++it;
        continue;
      }
      if (!fits(s, r->footprint)) break;
      it = q.erase(it);
      r->solo_admit = true;
      s->n_solo++;
      s->in_use += r->footprint;
      r->charged = r->footprint;
      s->peak_in_use = std::max(s->peak_in_use, s->in_use);
      r->status = 1;
      r->t_admit = now_s();
      s->n_preparing++;
      s->prepq.push_back(r);
      s->cv_prep.notify_one();
    }
  }
  for (int L = 0; L < 2; L++) {
    SrvLane &ln = s->lanes[L], &other = s->lanes[1 - L];
    while (!ln.waitq.empty()) {
      ReqPtr r = ln.waitq.front();
      if (ln.held + other.held >= s->max_active) break;
      if (ln.held >= share && !other.waitq.empty()) break;
      if (!fits(s, r->footprint)) break;
      ln.waitq.pop_front();
      ln.held++;
      s->in_use += r->footprint;
      r->charged = r->footprint;
      s->peak_in_use = std::max(s->peak_in_use, s->in_use);
      r->status = 1;
      r->t_admit = now_s();
      s->n_preparing++;
      s->prepq.push_back(r);
      s->cv_prep.notify_one();
    }
  }
}

void reaper_loop(gbfem_server s) {
  cudaSetDevice(s->device);
  std::unique_lock<std::mutex> lk(s->mu);
  for (;;) {
    s->cv_reap.wait(lk, [&] { return s->reap_stop || !s->reapq.empty(); });
    if (s->reapq.empty()) return;  // stop, and nothing left
    const auto item = s->reapq.front();
    s->reapq.pop_front();
    lk.unlock();
    if (item.ctx) gbfem_destroy(item.ctx);
    if (item.kry) cudaFree(item.kry);
    lk.lock();
    s->reap_bytes -= item.bytes;
    try_admit(s);
  }
}

int prepare(gbfem_server s, SrvRequest &r) {
  {
    // host-side fault injection: this preparation fails as a device
    // allocation would, before any device work
    std::lock_guard<std::mutex> lk(s->mu);
    if (s->inject_prep_failures > 0) {
      s->inject_prep_failures--;
      gbfem::set_error("injected allocation failure (GBFEM_SERVE_OPT_FAIL_PREPARATIONS)");
      return -1;
    }
  }
  // std requests' preparation and solo solves at the std lane's priority:
  // the DG lane's long block SpMVs (lowest priority) do not hold them up
  int rc = 0;
  if (!take_idle(s, r) &&
      (rc = gbfem::create_context(&r.ctx, s->device, r.kind == 0 ? (r.solo_admit ? s->prio_solo : s->prio_std) : 0)) < 0)
    return rc;
  gbfem_ctx c = r.ctx;
  std::vector<int> fid, fbc;
  if (r.kind == 0) {
    fbc.assign(r.nbf, 1);
    rc = gbfem_set_mesh(c, r.nno, r.xyz.data(), r.nel, GBFEM_PRISM, r.el.data(), r.nbf, nullptr, r.bf_el.data(),
                        r.bf_side.data(), fbc.data());
  } else {
    rc = gbfem_set_mesh(c, r.nno, r.xyz.data(), r.nel, GBFEM_PRISM, r.el.data(), 0, nullptr, nullptr, nullptr,
                        nullptr);
  }
  if (rc < 0) return rc;
  rc = gbfem_set_coefficients(c, r.k.data(), nullptr, r.f, r.g, 1.0e7);
  if (rc < 0) return rc;
  if (r.kind == 0) {
    int nd = 0;
    long long nnz = 0;
    // structure on the device
    if ((rc = gbfem_build_structure_device(c, &nd, &nnz)) < 0) return rc;
    // the gather scatter: the same summation order every time (no element
    // colouring needed), so a request's matrix (and result) does not depend
    // on when it runs
    if ((rc = gbfem_assemble(c, GBFEM_SCATTER_GATHER)) < 0) return rc;
    r.n = nd;
    {
      std::lock_guard<std::mutex> lk(s->mu);
      r.solo = r.solo_admit || (s->solo_dofs > 0 && nd >= s->solo_dofs);
    }
    if (r.solo) {
      // solved by the preparation worker with the device-resident GMRES
      if (cudaStreamSynchronize(c->stream) != cudaSuccess) {
        gbfem::set_error("preparation failed on the device");
        return -1;
      }
      return 0;
    }
    if ((rc = c->dinv.alloc(nd)) < 0) return rc;
    if ((rc = gbfem::launch_jacobi_diag(c->stream, nd, c->row_ptr.p, c->col_ind.p, c->val.p, c->dinv.p)) < 0)
      return rc;
  } else {
    std::vector<int> pe(r.nel, r.p);
    if ((rc = gbfem_dg_set_degrees(c, pe.data())) < 0) return rc;
    if ((rc = gbfem_dg_set_faces(c, r.nfa, r.fa_type.data(), r.fa_bc.data(), r.fa_el.data(), r.fa_side.data(),
                                 r.fa_nodes.data())) < 0)
      return rc;
    if ((rc = gbfem_dg_set_penalty(c, r.pen)) < 0) return rc;
    int nd = 0;
    long long nv = 0;
    if ((rc = gbfem_dg_build_structure(c, &nd, &nv)) < 0) return rc;
    if ((rc = gbfem_dg_assemble(c)) < 0) return rc;
    r.n = nd;
    if ((rc = c->dg_dinv.alloc((size_t)c->dg_ninv)) < 0) return rc;
    cudaMemsetAsync(c->err.p, 0, sizeof(int), c->stream);
    if ((rc = gbfem::dg_invert_diagonal(c)) < 0) return rc;
    int herr = 0;
    cudaMemcpyAsync(&herr, c->err.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess || herr != 0) {
      gbfem::set_error("DG block Jacobi: singular diagonal block");
      return -2;
    }
  }
  // Krylov workspace: x, tmp, V (m+1 columns), H, cs, sn, s, y, hcol, sc
  const long long n = r.n, m1 = r.krylov + 1;
  if ((rc = r.kry.alloc((size_t)(n * (m1 + 2) + m1 * m1 + 6 * (m1 + 1)))) < 0) return rc;
  if (cudaMemsetAsync(r.kry.p, 0, r.kry.bytes(), c->stream) != cudaSuccess) return -1;
  if (cudaStreamSynchronize(c->stream) != cudaSuccess) {
    gbfem::set_error("preparation failed on the device");
    return -1;
  }
  return 0;
}

void prep_worker(gbfem_server s) {
  cudaSetDevice(s->device);
  for (;;) {
    ReqPtr r;
    {
      std::unique_lock<std::mutex> lk(s->mu);
      s->cv_prep.wait(lk, [&] { return s->stop || !s->prepq.empty(); });
      if (s->prepq.empty()) return;
      // solo-sized std requests first (the longest latency-bound path:
      // preparation, then a device GMRES of hundreds of iterations), then
      // the other std requests (short preparation, latency-bound solve),
      // then DG, each in admission order
      auto it = std::find_if(s->prepq.begin(), s->prepq.end(), [](const ReqPtr &q) { return q->solo_admit; });
      if (it == s->prepq.end())
        it = std::find_if(s->prepq.begin(), s->prepq.end(), [](const ReqPtr &q) { return q->kind == 0; });
      if (it == s->prepq.end()) it = s->prepq.begin();
      r = *it;
      s->prepq.erase(it);
    }
    const int rc = prepare(s, *r);
    std::unique_lock<std::mutex> lk(s->mu);
    s->n_preparing--;
    r->t_ready = now_s();
    if (rc < 0 || r->cancel) {
      r->status = rc < 0 ? -1 : -2;
      r->err = rc < 0 ? gbfem_last_error() : "cancelled";
      lk.unlock();
      reap(s, *r, rc >= 0);
      lk.lock();
      s->in_use -= r->charged;
      r->charged = 0;
      r->t_done = now_s();
      if (!r->solo_admit) s->lanes[r->kind].held--;
      if (r->solo_admit) s->n_solo--;
      try_admit(s);
      s->cv_done.notify_all();
      continue;
    }
    if (r->solo) {
      // a large std request: solved by a solo thread on its own stream
      r->status = 3;
      s->soloq.push_back(r);
      s->cv_solo.notify_one();
      continue;
    }
    // replace the estimate by what the request holds
    const long long actual = gbfem_device_bytes(r->ctx) + (long long)r->kry.bytes();
    s->in_use += actual - r->charged;
    r->charged = actual;
    s->peak_in_use = std::max(s->peak_in_use, s->in_use);
    r->status = 2;
    s->readyq.push_back(r);
    s->cv_engine.notify_one();
    try_admit(s);
  }
}

// Solo requests (large std): gbfem_solve's device GMRES on the request's own
// stream and restart-cycle graph, beside the engine's batched lanes; the
// estimate (which includes the Krylov space and the sliced-ELL copy) stays charged until done.
void solo_worker(gbfem_server s) {
  cudaSetDevice(s->device);
  for (;;) {
    ReqPtr r;
    bool skip = false;
    {
      std::unique_lock<std::mutex> lk(s->mu);
      s->cv_solo.wait(lk, [&] { return s->stop || !s->soloq.empty(); });
      if (s->soloq.empty()) return;
      r = s->soloq.front();
      s->soloq.pop_front();
      s->n_active++;
      r->t_start = now_s();
      skip = r->cancel;
    }
    r->x.assign(r->n, 0.0);
    double res = 0.0, rel = 0.0;
    // (cancelled while queued here: not solved)
    const int it = skip ? 0
                        : gbfem::gmres_device_std(r->ctx, r->krylov, r->max_iter, r->tol, 1, r->x.data(), &res,
                                                       &rel);
    const std::string err = it < 0 ? std::string(gbfem_last_error()) : std::string();
    reap(s, *r, it >= 0);
    std::lock_guard<std::mutex> lk(s->mu);
    r->iters = it < 0 ? 0 : it;
    r->rel = rel;
    s->in_use -= r->charged;
    r->charged = 0;
    r->status = it < 0 ? -1 : (r->cancel ? -2 : 4);
    if (it < 0) r->err = err;
    if (r->cancel && it >= 0) r->err = "cancelled";
    r->t_done = now_s();
    s->n_active--;
    if (!r->solo_admit) s->lanes[r->kind].held--;
    if (r->solo_admit) s->n_solo--;
    try_admit(s);
    s->cv_done.notify_all();
  }
}

void fill_desc(SrvDesc &d, SrvRequest &r) {
  memset(&d, 0, sizeof(d));
  gbfem_ctx c = r.ctx;
  const long long n = r.n, m1 = r.krylov + 1;
  d.kind = r.kind;
  d.n = r.n;
  d.m = r.krylov;
  d.max_iter = r.max_iter;
  d.tol_rel = r.tol < 1e-12 ? 1e-12 : r.tol;
  d.tol_abs = 1e-12;
  if (r.kind == 0) {
    d.row_ptr = c->row_ptr.p;
    d.col_ind = c->col_ind.p;
    d.val = c->val.p;
    d.dinv = c->dinv.p;
    d.b = c->rhs.p;
  } else {
    d.roff = c->dg_roff_d.p;
    d.colx = c->dg_colx_d.p;
    d.row_val = c->dg_row_val_d.p;
    d.cx_off = c->dg_cx_off_d.p;
    d.dinv_off = c->dg_dinv_off_d.p;
    d.dgval = c->dg_val.p;
    d.dgdinv = c->dg_dinv.p;
    d.b = c->dg_rhs.p;
  }
  double *w = r.kry.p;
  d.x = w;
  d.tmp = w + n;
  d.V = w + 2 * n;
  d.H = d.V + n * m1;
  d.cs = d.H + m1 * m1;
  d.sn = d.cs + (m1 + 1);
  d.s = d.sn + (m1 + 1);
  d.y = d.s + (m1 + 1);
  d.hcol = d.y + (m1 + 1);
  d.sc = d.hcol + (m1 + 1);
}

// rebuild a lane's block maps and its requests' descriptors after its
// active set changed (the lane is idle: nothing of it is in flight)
int rebuild(gbfem_server s, SrvLane &ln, int L) {
  std::vector<int2> mv, mc;
  int red = 0;
  ln.act.clear();
  for (int i = 0; i < gbfem::SRV_MAXSLOTS; i++) {
    if (!s->slots[i] || s->slots[i]->kind != L) continue;
    SrvRequest &r = *s->slots[i];
    ln.act.push_back(i);
    SrvDesc &d = s->h_desc[i];
    d.chunk = gbfem::srv_chunk(r.n);
    const int nb = (r.n + d.chunk - 1) / d.chunk;
    d.red_first = red;
    d.red_nb = nb;
    red += nb;
    for (int b = 0; b < nb; b++) mv.push_back(make_int2(i, b * d.chunk));
    if (r.kind == 0)
      for (int r0 = 0; r0 < r.n; r0 += gbfem::SRV_SPMV_ROWS) mc.push_back(make_int2(i, r0));
  }
  ln.n_vec = (int)mv.size();
  ln.n_crs = (int)mc.size();
  if (ln.d_map_vec.alloc(std::max<size_t>(mv.size(), 1)) < 0 || ln.d_map_crs.alloc(std::max<size_t>(mc.size(), 1)) < 0 ||
      ln.d_act.alloc(std::max<size_t>(ln.act.size(), 1)) < 0 ||
      ln.d_partial.alloc((size_t)std::max(red, 1) * gbfem::SRV_PART) < 0)
    return -1;
  if (!mv.empty())
    GB_CUDA(cudaMemcpyAsync(ln.d_map_vec.p, mv.data(), mv.size() * sizeof(int2), cudaMemcpyHostToDevice, ln.stream));
  if (!mc.empty())
    GB_CUDA(cudaMemcpyAsync(ln.d_map_crs.p, mc.data(), mc.size() * sizeof(int2), cudaMemcpyHostToDevice, ln.stream));
  if (!ln.act.empty())
    GB_CUDA(cudaMemcpyAsync(ln.d_act.p, ln.act.data(), ln.act.size() * sizeof(int), cudaMemcpyHostToDevice, ln.stream));
  // only this lane's descriptors: the other lane's kernels read theirs meanwhile
  for (int i : ln.act)
    GB_CUDA(cudaMemcpyAsync(s->d_desc.p + i, s->h_desc + i, sizeof(SrvDesc), cudaMemcpyHostToDevice, ln.stream));
  // the host copies (maps, descriptors) are rewritten by the next rebuild
  GB_CUDA(cudaStreamSynchronize(ln.stream));
  return 0;
}

int step(gbfem_server s, SrvLane &ln) {
  using namespace gbfem;
  cudaStream_t st = ln.stream;
  const int2 *mv = ln.d_map_vec.p;
  SrvDesc *dd = s->d_desc.p;
  SrvState *ss = s->d_state.p;
  double *part = ln.d_partial.p;
  int L = 0;
  if (ln.n_crs) {
    srv_crs_spmv<<<ln.n_crs, SRV_T, 0, st>>>(ln.d_map_crs.p, dd, ss);
    L++;
  }
  for (int i : ln.act) {
    SrvRequest &r = *s->slots[i];
    if (r.kind != 1) continue;
    for (int p = 1; p <= 4; p++) {
      const int cnt = (int)r.ctx->dg_list[p].n;
      if (!r.ctx->dg_list[p].p || cnt == 0) continue;
      const int grid = (cnt + DGS_ROWS - 1) / DGS_ROWS;
      const int *lst = r.ctx->dg_list[p].p;
#define GB_SRV_DG(PP)                                                             \
  if (cnt <= dgs_wide_max(PP))                                                    \
    srv_dg_spmv<PP, true><<<cnt, DGS_THREADS, 0, st>>>(i, cnt, lst, dd, ss);      \
  else                                                                            \
    srv_dg_spmv<PP, false><<<grid, DGS_THREADS, 0, st>>>(i, cnt, lst, dd, ss)
      switch (p) {
        case 1: GB_SRV_DG(1); break;
        case 2: GB_SRV_DG(2); break;
        case 3: GB_SRV_DG(3); break;
        default: GB_SRV_DG(4); break;
      }
#undef GB_SRV_DG
      L++;
    }
  }
  srv_dots<<<ln.n_vec, SRV_T, 0, st>>>(mv, dd, ss, part);
  srv_orthogonalize<<<ln.n_vec, SRV_T, 0, st>>>(mv, dd, ss, part);
  srv_logic<<<(int)ln.act.size(), SRV_LOGIC_T, 0, st>>>(ln.d_act.p, dd, ss, part);
  L += 3;
  GB_CUDA(cudaGetLastError());
  return L;
}

void drop_graph(SrvLane &ln) {
  if (ln.graph) cudaGraphExecDestroy(ln.graph);
  ln.graph = nullptr;
  ln.polls = 0;
}

// capture a lane's step for its current active set
int capture(gbfem_server s, SrvLane &ln) {
  GB_CUDA(cudaStreamBeginCapture(ln.stream, cudaStreamCaptureModeThreadLocal));
  const int L = step(s, ln);
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(ln.stream, &g);
  if (L < 0) return L;
  GB_CUDA(e);
  const cudaError_t ei = cudaGraphInstantiate(&ln.graph, g, 0);
  cudaGraphDestroy(g);
  GB_CUDA(ei);
  ln.graph_kernels = L;
  return 0;
}

// A finished (or cancelled) request leaves its slot; the lane is idle here
// (its last poll completed), so nothing of it is in flight.
void retire(gbfem_server s, SrvLane &ln, int i, bool cancelled = false) {
  ReqPtr r = s->slots[i];
  const SrvState &S = ln.h_state[i];
  if (!cancelled) {
    r->x.resize(r->n);
    cudaMemcpyAsync(r->x.data(), r->kry.p, (size_t)r->n * sizeof(double), cudaMemcpyDeviceToHost, ln.stream);
    cudaStreamSynchronize(ln.stream);
    r->iters = S.it;
    r->rel = S.beta0 > 0 ? S.resid / S.beta0 : 0.0;
  }
  reap(s, *r);
  s->slots[i].reset();
  std::lock_guard<std::mutex> lk(s->mu);
  s->in_use -= r->charged;
  r->charged = 0;
  r->status = cancelled ? -2 : 4;
  if (cancelled) r->err = "cancelled";
  r->t_done = now_s();
  s->n_active--;
  ln.held--;
  try_admit(s);
  s->cv_done.notify_all();
}

void engine_fail(gbfem_server s, const std::string &msg) {
  std::lock_guard<std::mutex> lk(s->mu);
  s->fatal = msg;
  s->stop = true;
  s->cv_done.notify_all();
}

void engine_loop(gbfem_server s) {
  cudaSetDevice(s->device);
  double last_progress = 0.0;
  for (;;) {
    {
      std::unique_lock<std::mutex> lk(s->mu);
      const bool idle = s->lanes[0].act.empty() && s->lanes[1].act.empty() && !s->lanes[0].busy &&
                        !s->lanes[1].busy;
      if (idle && s->readyq.empty()) {
        s->cv_engine.wait(lk, [&] { return s->stop || !s->readyq.empty(); });
        if (s->stop && s->readyq.empty()) return;
      }
      while (!s->readyq.empty()) {
        int i = 0;
        while (i < gbfem::SRV_MAXSLOTS && s->slots[i]) i++;
        if (i == gbfem::SRV_MAXSLOTS) break;
        ReqPtr r = s->readyq.front();
        s->readyq.pop_front();
        SrvLane &ln = s->lanes[r->kind];
        r->slot = i;
        r->status = 3;
        r->t_start = now_s();
        s->slots[i] = r;
        s->n_active++;
        fill_desc(s->h_desc[i], *r);
        SrvState init;
        memset(&init, 0, sizeof(init));
        init.phase = gbfem::PH_RESTART;
        init.beta0 = -1.0;
        s->h_init[i] = init;
        // behind the lane's work in flight (which does not touch slot i)
        cudaMemcpyAsync(s->d_state.p + i, s->h_init + i, sizeof(SrvState), cudaMemcpyHostToDevice, ln.stream);
        ln.changed = true;
      }
      s->peak_active = std::max(s->peak_active, s->n_active);
    }
    bool progressed = false;
    for (int L = 0; L < 2; L++) {
      SrvLane &ln = s->lanes[L];
      if (ln.busy) {
        const cudaError_t q = cudaEventQuery(ln.done);
        if (q == cudaErrorNotReady) continue;
        if (q != cudaSuccess) {
          engine_fail(s, std::string("serving step failed: ") + cudaGetErrorString(q));
          return;
        }
        ln.busy = false;
        progressed = true;
        for (int i : std::vector<int>(ln.act)) {
          bool cancelled;
          {
            std::lock_guard<std::mutex> lk(s->mu);
            cancelled = s->slots[i]->cancel;
          }
          if (ln.h_state[i].phase == gbfem::PH_DONE || cancelled) {
            retire(s, ln, i, cancelled);
            ln.changed = true;
          }
        }
      }
      if (ln.changed) {
        drop_graph(ln);
        if (rebuild(s, ln, L) < 0) {
          engine_fail(s, gbfem_last_error());
          return;
        }
        ln.changed = false;
      }
      if (ln.act.empty()) continue;
      // std precedence: no new DG steps while a solo request is in flight
      if (L == 1 && s->std_precedence && s->n_solo.load() > 0) continue;
      // several steps per poll: a finished request's kernels are no-ops until
      // it is retired, so the extra steps only cost their launch
      if (!ln.graph && ++ln.polls > SRV_CAPTURE_POLLS && capture(s, ln) < 0) {
        engine_fail(s, gbfem_last_error());
        return;
      }
      bool ok = true;
      for (int k = 0; k < s->steps_per_poll && ok; k++) {
        int launched = ln.graph_kernels;
        if (ln.graph)
          ok = cudaGraphLaunch(ln.graph, ln.stream) == cudaSuccess;
        else
          ok = (launched = step(s, ln)) >= 0;
        s->steps++;
        s->launches += launched;
      }
      if (!ok ||
          cudaMemcpyAsync(ln.h_state, s->d_state.p, sizeof(SrvState) * gbfem::SRV_MAXSLOTS, cudaMemcpyDeviceToHost,
                          ln.stream) != cudaSuccess ||
          cudaEventRecord(ln.done, ln.stream) != cudaSuccess) {
        engine_fail(s, std::string("serving step failed: ") + cudaGetErrorString(cudaGetLastError()));
        return;
      }
      ln.busy = true;
      progressed = true;
    }
    // a poll's steps take some tens of microseconds for small requests: spin
    // for the first 200 us without progress (a sleep of 20 us lasts 70 and
    // more), then sleep between looks
    const double t = now_s();
    if (progressed)
      last_progress = t;
    else if (t - last_progress < 200e-6)
      std::this_thread::yield();
    else
      std::this_thread::sleep_for(std::chrono::microseconds(20));
  }
}

}  // namespace

extern "C" {

long long gbfem_serve_footprint(const gbfem_serve_request *q) {
  if (!q) return -2;
  int ntri = 0;
  for (int f = 0; q->kind == GBFEM_SERVE_DG && q->fa_type && f < q->nfa; f++) ntri += q->fa_type[f] == 3;
  return gbfem_serve_footprint_impl(q->kind, q->dg_p, q->nno, q->nel, q->nbf, q->nfa, ntri, q->krylov);
}

int gbfem_server_create(gbfem_server *out, int device, long long hbm_budget, int max_active, int prep_threads) {
  GB_CHECK(out, "null server pointer");
  GB_CHECK(max_active >= 1 && max_active <= gbfem::SRV_MAXSLOTS, "max_active must be 1..64");
  GB_CHECK(prep_threads >= 1 && prep_threads <= 16, "prep_threads must be 1..16");
  GB_CUDA(cudaSetDevice(device));
  gbfem_server s = new gbfem_server_s();
  s->device = device;
  s->max_active = max_active;
  if (hbm_budget <= 0) {
    size_t fr = 0, tot = 0;
    cudaMemGetInfo(&fr, &tot);
    hbm_budget = (long long)(0.85 * (double)fr);
  }
  s->budget = hbm_budget;
  bool ok = s->d_desc.alloc(gbfem::SRV_MAXSLOTS) >= 0 && s->d_state.alloc(gbfem::SRV_MAXSLOTS) >= 0 &&
            cudaHostAlloc(&s->h_init, sizeof(SrvState) * gbfem::SRV_MAXSLOTS, cudaHostAllocPortable) == cudaSuccess &&
            cudaHostAlloc(&s->h_desc, sizeof(SrvDesc) * gbfem::SRV_MAXSLOTS, cudaHostAllocPortable) == cudaSuccess;
  // the std lane's short steps get a high stream priority (below only the
  // solo-sized std requests' streams), the DG lane's long FP64-bound SpMVs
  // the lowest: when both lanes have work queued the block scheduler starts
  // std blocks first
  int prio_least = 0, prio_greatest = 0;
  cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest);
  // solo-sized std requests above every other stream, the other std work
  // (preparations, the std lane) next, the DG lane last (greatest is the
  // numerically smallest priority)
  s->prio_solo = prio_greatest;
  s->prio_std = prio_greatest < prio_least ? prio_greatest + 1 : prio_greatest;
  for (int L = 0; L < 2 && ok; L++) {
    SrvLane &ln = s->lanes[L];
    ok = cudaStreamCreateWithPriority(&ln.stream, cudaStreamNonBlocking, L == 0 ? s->prio_std : prio_least) ==
             cudaSuccess &&
         cudaEventCreateWithFlags(&ln.done, cudaEventDisableTiming) == cudaSuccess &&
         cudaHostAlloc(&ln.h_state, sizeof(SrvState) * gbfem::SRV_MAXSLOTS, cudaHostAllocPortable) == cudaSuccess;
    if (ok) memset(ln.h_state, 0, sizeof(SrvState) * gbfem::SRV_MAXSLOTS);
  }
  if (!ok) {
    gbfem::set_error("server allocation failed");
    for (SrvLane &ln : s->lanes) {
      if (ln.h_state) cudaFreeHost(ln.h_state);
      if (ln.done) cudaEventDestroy(ln.done);
      if (ln.stream) cudaStreamDestroy(ln.stream);
    }
    if (s->h_init) cudaFreeHost(s->h_init);
    if (s->h_desc) cudaFreeHost(s->h_desc);
    delete s;
    return -1;
  }
  memset(s->h_init, 0, sizeof(SrvState) * gbfem::SRV_MAXSLOTS);
  memset(s->h_desc, 0, sizeof(SrvDesc) * gbfem::SRV_MAXSLOTS);
  cudaMemset(s->d_state.p, 0, sizeof(SrvState) * gbfem::SRV_MAXSLOTS);
  for (int i = 0; i < prep_threads; i++) s->workers.emplace_back(prep_worker, s);
  for (int i = 0; i < 8; i++) s->solo_workers.emplace_back(solo_worker, s);
  s->engine = std::thread(engine_loop, s);
  s->reaper = std::thread(reaper_loop, s);
  *out = s;
  return 0;
}

int gbfem_server_destroy(gbfem_server s) {
  if (!s) return 0;
  {
    std::lock_guard<std::mutex> lk(s->mu);
    s->stop = true;
    for (SrvLane &ln : s->lanes) ln.waitq.clear();
  }
  s->cv_prep.notify_all();
  s->cv_engine.notify_all();
  for (auto &t : s->workers) t.join();
  // the solo threads solve what is queued for them, then return
  s->cv_solo.notify_all();
  for (auto &t : s->solo_workers) t.join();
  // the engine finishes the requests it holds, then returns
  if (s->engine.joinable()) s->engine.join();
  {
    std::lock_guard<std::mutex> lk(s->mu);
    while (!s->idle.empty()) drop_oldest_idle(s);
    s->reap_stop = true;
  }
  s->cv_reap.notify_all();
  if (s->reaper.joinable()) s->reaper.join();  // after freeing what was queued
  cudaSetDevice(s->device);
  for (auto &kv : s->reqs) {
    if (kv.second->ctx) gbfem_destroy(kv.second->ctx);
    kv.second->kry.release();
  }
  for (auto &r : s->readyq) {
    if (r->ctx) gbfem_destroy(r->ctx);
    r->kry.release();
  }
  for (SrvLane &ln : s->lanes) {
    if (ln.stream) cudaStreamSynchronize(ln.stream);
    if (ln.graph) cudaGraphExecDestroy(ln.graph);
    ln.d_map_vec.release();
    ln.d_map_crs.release();
    ln.d_act.release();
    ln.d_partial.release();
    if (ln.h_state) cudaFreeHost(ln.h_state);
    if (ln.done) cudaEventDestroy(ln.done);
    if (ln.stream) cudaStreamDestroy(ln.stream);
  }
  s->d_desc.release();
  s->d_state.release();
  if (s->h_init) cudaFreeHost(s->h_init);
  if (s->h_desc) cudaFreeHost(s->h_desc);
  delete s;
  return 0;
}

long long gbfem_server_submit(gbfem_server s, const gbfem_serve_request *q) {
  GB_CHECK(s && q, "null argument");
  GB_CHECK(q->kind == GBFEM_SERVE_STD || q->kind == GBFEM_SERVE_DG, "kind must be GBFEM_SERVE_STD or _DG");
  GB_CHECK(q->nno > 0 && q->nel > 0 && q->node_xyz && q->el_nodes && q->k_el, "empty request");
  GB_CHECK(q->krylov >= 1 && q->krylov <= gbfem::SRV_MMAX, "krylov must be 1..64 for served requests");
  GB_CHECK(q->max_iter >= 1, "max_iter must be positive");
  if (q->kind == GBFEM_SERVE_DG) {
    GB_CHECK(q->dg_p >= 1 && q->dg_p <= 4, "DG degree must be 1..4");
    GB_CHECK(q->nfa > 0 && q->fa_type && q->fa_bc && q->fa_el && q->fa_side && q->fa_nodes, "DG needs a face table");
  } else {
    GB_CHECK(q->nbf == 0 || (q->bf_el && q->bf_side), "boundary face arrays missing");
  }
  auto r = std::make_shared<SrvRequest>();
  r->kind = q->kind;
  r->p = q->dg_p;
  r->krylov = q->krylov;
  r->max_iter = q->max_iter;
  r->tol = q->tol_rel;
  r->f = q->f;
  r->g = q->g;
  r->pen = q->dg_penalty > 0 ? q->dg_penalty : 10.0;
  r->nno = q->nno;
  r->nel = q->nel;
  r->xyz.assign(q->node_xyz, q->node_xyz + 3 * (size_t)q->nno);
  r->el.assign(q->el_nodes, q->el_nodes + 6 * (size_t)q->nel);
  r->k.assign(q->k_el, q->k_el + q->nel);
  if (q->kind == GBFEM_SERVE_STD) {
    r->nbf = q->nbf;
    r->bf_el.assign(q->bf_el, q->bf_el + q->nbf);
    r->bf_side.assign(q->bf_side, q->bf_side + q->nbf);
  } else {
    r->nfa = q->nfa;
    r->fa_type.assign(q->fa_type, q->fa_type + q->nfa);
    r->fa_bc.assign(q->fa_bc, q->fa_bc + q->nfa);
    r->fa_el.assign(q->fa_el, q->fa_el + 2 * (size_t)q->nfa);
    r->fa_side.assign(q->fa_side, q->fa_side + q->nfa);
    r->fa_nodes.assign(q->fa_nodes, q->fa_nodes + 4 * (size_t)q->nfa);
  }
  r->footprint = gbfem_serve_footprint(q);
  std::lock_guard<std::mutex> lk(s->mu);
  GB_CHECK(!s->stop, "server is stopping");
  GB_CHECK(s->fatal.empty(), s->fatal.c_str());
  r->id = s->next_id++;
  r->t_submit = now_s();
  s->reqs[r->id] = r;
  s->lanes[r->kind].waitq.push_back(r);
  try_admit(s);
  return r->id;
}

int gbfem_server_wait(gbfem_server s, long long id, double timeout_s) {
  GB_CHECK(s, "null server");
  std::unique_lock<std::mutex> lk(s->mu);
  auto it = s->reqs.find(id);
  GB_CHECK(it != s->reqs.end(), "unknown request id");
  ReqPtr r = it->second;
  auto pred = [&] { return r->status == 4 || r->status < 0 || !s->fatal.empty(); };
  if (timeout_s < 0)
    s->cv_done.wait(lk, pred);
  else if (!s->cv_done.wait_for(lk, std::chrono::duration<double>(timeout_s), pred))
    return 0;
  if (!s->fatal.empty()) {
    gbfem::set_error(s->fatal);
    return -1;
  }
  if (r->status < 0) {
    gbfem::set_error("request failed: " + r->err);
    return -2;
  }
  return 1;
}

int gbfem_server_result(gbfem_server s, long long id, double *x, long long nx, int *iters, double *rel_res,
                        double *times) {
  GB_CHECK(s, "null server");
  std::lock_guard<std::mutex> lk(s->mu);
  auto it = s->reqs.find(id);
  GB_CHECK(it != s->reqs.end(), "unknown request id");
  SrvRequest &r = *it->second;
  GB_CHECK(r.status == 4, "request not finished");
  if (x) {
    GB_CHECK(nx >= (long long)r.x.size(), "solution buffer too small");
    memcpy(x, r.x.data(), r.x.size() * sizeof(double));
  }
  if (iters) *iters = r.iters;
  if (rel_res) *rel_res = r.rel;
  if (times) {
    times[0] = r.t_admit - r.t_submit;  // queued for admission
    times[1] = r.t_ready - r.t_admit;   // upload, structure, integrate + assemble, preconditioner
    times[2] = r.t_start - r.t_ready;   // waiting for an engine slot
    times[3] = r.t_done - r.t_start;    // batched GMRES
    times[4] = r.t_done - r.t_submit;   // latency
  }
  return (int)r.x.size();
}

int gbfem_server_cancel(gbfem_server s, long long id) {
  GB_CHECK(s, "null server");
  std::lock_guard<std::mutex> lk(s->mu);
  auto it = s->reqs.find(id);
  GB_CHECK(it != s->reqs.end(), "unknown request id");
  ReqPtr r = it->second;
  if (r->status == 4 || r->status < 0) return 1;  // finished, failed or cancelled already
  if (r->status == 0) {  // queued: leaves the queue now
    auto &q = s->lanes[r->kind].waitq;
    q.erase(std::remove(q.begin(), q.end(), r), q.end());
  } else if (r->status == 2) {  // prepared, waiting for an engine slot: freed now
    s->readyq.erase(std::remove(s->readyq.begin(), s->readyq.end(), r), s->readyq.end());
    if (r->ctx) gbfem_destroy(r->ctx);
    r->ctx = nullptr;
    r->kry.release();
    s->in_use -= r->charged;
    r->charged = 0;
    if (!r->solo_admit) s->lanes[r->kind].held--;
    try_admit(s);
  } else {  // preparing or solving: its worker or the engine retires it
    r->cancel = true;
    return 0;
  }
  r->status = -2;
  r->err = "cancelled";
  r->t_done = now_s();
  s->cv_done.notify_all();
  return 0;
}

int gbfem_server_release(gbfem_server s, long long id) {
  GB_CHECK(s, "null server");
  std::lock_guard<std::mutex> lk(s->mu);
  auto it = s->reqs.find(id);
  GB_CHECK(it != s->reqs.end(), "unknown request id");
  GB_CHECK(it->second->status == 4 || it->second->status < 0, "request not finished");
  s->reqs.erase(it);
  return 0;
}

int gbfem_server_set_option(gbfem_server s, int option, long long value) {
  GB_CHECK(s, "null server");
  if (option == GBFEM_SERVE_OPT_STEPS_PER_POLL) {
    GB_CHECK(value >= 1 && value <= 64, "steps per poll must be 1..64");
    std::lock_guard<std::mutex> lk(s->mu);
    s->steps_per_poll = (int)value;
    return 0;
  }
  if (option == GBFEM_SERVE_OPT_SOLO_DOFS) {
    GB_CHECK(value >= 0 && value <= 2000000000LL, "solo threshold out of range");
    std::lock_guard<std::mutex> lk(s->mu);
    s->solo_dofs = (int)value;
    return 0;
  }
  if (option == GBFEM_SERVE_OPT_STD_PRECEDENCE) {
    GB_CHECK(value == 0 || value == 1, "std precedence is 0 or 1");
    std::lock_guard<std::mutex> lk(s->mu);
    s->std_precedence = (int)value;
    return 0;
  }
  if (option == GBFEM_SERVE_OPT_FAIL_PREPARATIONS) {
    GB_CHECK(value >= 0 && value <= 1000000, "injected failure count out of range");
    std::lock_guard<std::mutex> lk(s->mu);
    s->inject_prep_failures = (int)value;
    return 0;
  }
  gbfem::set_error("unknown server option");
  return -2;
}

int gbfem_server_stats(gbfem_server s, long long *st) {
  GB_CHECK(s && st, "null argument");
  std::lock_guard<std::mutex> lk(s->mu);
  st[0] = s->steps;
  st[1] = s->launches;
  st[2] = s->peak_active;
  st[3] = s->peak_in_use;
  st[4] = s->budget;
  st[5] = s->in_use;
  st[6] = (long long)(s->lanes[0].waitq.size() + s->lanes[1].waitq.size());
  st[7] = s->n_active;
  return 0;
}

}  // extern "C"
