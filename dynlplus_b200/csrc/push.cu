// Residual push with device-resident frontiers: the work behind FusedPush.run (dynlp/kernels.py:396-433)
// with the round semantics of the synchronous push (dynlp/solvers.py:100-125).
//
// A round moves the residual of every frontier row u into its score and onto its neighbours:
//   d_u = R[u,:] / diag[u];  Z[u,:] += d_u;  R[u,:] = 0;  R[v,:] += w_uv d_u for every live entry (u, v)
// and the next frontier is the set of rows the round touched that still violate
// |R[v,c]| > eps[c] * diag[v] for some column c.
//
// Rounds are synchronous: every frontier row's residual is taken before any push of the round
// lands, so the sequence of frontiers is the one the synchronous push defines (up to the order of
// the floating-point atomic sums), not a schedule-dependent relaxation. Each round has two phases:
//   push_scatter  one group of G lanes per frontier row streams the row's entries, adds w * d
//                 into the neighbours' residual rows and records first touches in a bitmap; the
//                 touched rows go to a list through warp-aggregated appends (one atomic per warp);
//   push_sift     one thread per touched row clears its bit, tests the row and, when it violates,
//                 takes its residual for the next round at a slot reserved by a warp-aggregated
//                 append: the next frontier's scaled residuals d are stored compactly (D), so the
//                 scatter reads them as rows and no take races a push.
// Counters live in a control block on the device with two copies of the frontier and touched
// counts; the round of one parity resets the copies the other parity fills next, so the rounds chain
// without the host. k_push_whole runs all rounds in one cooperative launch with a grid barrier after
// each phase; k_push_scatter and k_push_sift are the phases as launches, for the host-driven loop.
// The frontiers are short (thousands of rows, tens at the end), so a round is bound by latency: the
// dependent reads of one row and its two barriers. The round cap and the host's cancel word are
// checked where a round would take residuals, once for the whole grid, so a stopped run never leaves
// a taken residual unpushed: R stays the residual of Z.
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace dlp {

constexpr int kPushThreads = 256;
// Lanes per frontier row. Eight: the graphs of the workloads have mean degrees of 8 to 32, and a
// row's entries are streamed in ceil(degree / 8) warp-uniform steps.
constexpr int kPushGroup = 8;

// Entries of a lane in flight, and columns of a row in flight where one thread has the row.
constexpr int kPushFly = 4;
constexpr int kPushCols = 4;

enum { kRunning = 0, kConverged = 1, kCapped = 2, kCancelled = 3 };

struct PushCtl {
  int32_t rounds;      // rounds whose scatter ran
  int32_t max_rounds;
  int32_t status;      // kRunning, kConverged, kCapped, kCancelled
  int32_t allow;       // the round's sift may take rows (1), or minus the status that ends the run
  int32_t fcnt[2];     // frontier size for the round of each parity
  int32_t tcnt[2];     // touched rows of the round of each parity
  unsigned long long edges;          // stored entries streamed (the reference's edge visits)
  unsigned long long frontier_rows;  // sum of the frontier sizes of the rounds run
  unsigned long long touched_rows;   // sum of the touched-list sizes
  GridBar bar;                       // k_push_whole
  double eps[33];
};

template <typename T>
struct PushArgs {
  const int32_t *rbeg, *rend, *col;
  const void *w;
  const T *diag;
  T *Z;
  int64_t ldz;
  T *R;
  int64_t ldr;
  int32_t C;
  const double *eps;
  int32_t *front;    // frontier rows (n)
  T *D;              // their scaled residuals, C per row (n x C)
  int32_t *touched;  // touched rows (n)
  uint32_t *bits;    // first-touch bitmap (ceil(n / 32) words; zero between rounds)
  PushCtl *ctl;
  const int32_t *cancel;
};

// R, Z, D and the lists change within a k_push_whole launch, so they are read through L2 (__ldcg).
// The entries of a row are read one per lane of its group and then added CL lanes per entry, a lane for
// every CL-th column: the adds to a neighbour's row are one run of bytes, one line where a lane per entry
// touched a line per column (a run of 14 rounds at 17 columns, n = 60,000: 803 -> 434 us; of 11 at 9, n = 1M:
// 417 -> 363). Rows of one and two columns have as many lanes (n = 1M, all rows pushed in six rounds, fp32: 2,502 ->
// 2,268 and 2,846 -> 2,614).
template <typename TW, typename T, int CMAX>
__device__ __forceinline__ void push_scatter(const PushArgs<T> &a, int p, int nf) {
  PushCtl *ctl = a.ctl;
  const TW *__restrict__ w = (const TW *)a.w;
  constexpr int G = kPushGroup, CL = CMAX <= 2 ? CMAX : CMAX <= 4 ? 4 : 8, DC = (CMAX + CL - 1) / CL, ES = G / CL;
  const int lane = lane_id();
  const int gl = lane % G, g0 = lane - gl;  // lane within the row's group
  const int cl = gl % CL, sub = gl / CL;
  constexpr int kGroups = 32 / G;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long stride = (((long long)gridDim.x * blockDim.x) >> 5) * kGroups;
  unsigned long long my_edges = 0;
  uint32_t walked = 0;
  for (long long base = warp * kGroups; base < nf; base += stride) {  // warp-uniform bounds
    const long long g = base + lane / G;
    const bool valid = g < nf;
    int beg = 0, end = 0;
    T d[DC];
#pragma unroll
    for (int k = 0; k < DC; ++k) d[k] = T(0);
    if (valid) {
      const int u = __ldcg(a.front + g);
      beg = a.rbeg[u];
      end = a.rend[u];
      bar_announce(&ctl->bar, end - beg, walked);
      const T *dr = a.D + g * a.C;
#pragma unroll
      for (int k = 0; k < DC; ++k)
        if (cl + k * CL < a.C) d[k] = __ldcg(dr + cl + k * CL);
      if (gl == 0) my_edges += (unsigned long long)(end - beg);
    }
    int trips = valid ? (end - beg + G - 1) / G : 0;
    trips = __reduce_max_sync(0xffffffffu, trips);
    for (int t = 0; t < trips; t += kPushFly) {
      int32_t v[kPushFly];
      T wv[kPushFly];
      unsigned first[kPushFly];
#pragma unroll
      for (int u = 0; u < kPushFly; ++u) {
        const int j = beg + gl + (t + u) * G;
        v[u] = j < end ? a.col[j] : 0;
        wv[u] = j < end ? cvt<T>(w[j]) : T(0);
      }
#pragma unroll
      for (int u = 0; u < kPushFly; ++u) {
        if (t + u >= trips) break;
#pragma unroll
        for (int e = 0; e < CL; ++e) {
          const int src = g0 + e * ES + sub;
          const int32_t ve = __shfl_sync(0xffffffffu, v[u], src);
          const T we = __shfl_sync(0xffffffffu, wv[u], src);
          if (we != T(0)) {  // inert entries (deleted edges, edges leaving the solved set) carry nothing
            T *r = a.R + (long long)ve * a.ldr + cl;
#pragma unroll
            for (int k = 0; k < DC; ++k)
              if (cl + k * CL < a.C) atomic_add(r + k * CL, we * d[k]);
          }
        }
      }
      bool fresh[kPushFly];
#pragma unroll
      for (int u = 0; u < kPushFly; ++u) {
        const uint32_t bit = 1u << (v[u] & 31);
        fresh[u] = wv[u] != T(0) && (atomicOr(a.bits + (v[u] >> 5), bit) & bit) == 0u;
      }
      int total = 0;
#pragma unroll
      for (int u = 0; u < kPushFly; ++u) {
        first[u] = __ballot_sync(0xffffffffu, fresh[u]);
        total += __popc(first[u]);
      }
      if (total) {  // warp-uniform
        int at = lane == 0 ? atomicAdd(&ctl->tcnt[p], total) : 0;
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int u = 0; u < kPushFly; ++u) {
          if (fresh[u]) a.touched[at + __popc(first[u] & ((1u << lane) - 1u))] = v[u];
          at += __popc(first[u]);
        }
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) my_edges += __shfl_xor_sync(0xffffffffu, my_edges, off);
  if (lane == 0 && my_edges) atomicAdd(&ctl->edges, my_edges);
}

// The take of one row: d = R[v,:] / diag[v] stored at D[slot,:]; Z[v,:] += d; R[v,:] = 0.
template <typename T>
__device__ __forceinline__ void take_row(const PushArgs<T> &a, int32_t v, int slot, T dv) {
  T *r = a.R + (long long)v * a.ldr;
  T *z = a.Z + (long long)v * a.ldz;
  T *dd = a.D + (long long)slot * a.C;
  for (int c0 = 0; c0 < a.C; c0 += kPushCols) {
    T x[kPushCols], y[kPushCols];
#pragma unroll
    for (int i = 0; i < kPushCols; ++i) {
      x[i] = c0 + i < a.C ? __ldcg(r + c0 + i) : T(0);
      y[i] = c0 + i < a.C ? __ldcg(z + c0 + i) : T(0);
    }
#pragma unroll
    for (int i = 0; i < kPushCols; ++i) {
      if (c0 + i < a.C) {
        const T q = x[i] / dv;
        dd[c0 + i] = q;
        z[c0 + i] = y[i] + q;
        r[c0 + i] = T(0);
      }
    }
  }
}

// allow: 1, or minus the status that ends the run before rows are taken.
template <typename T>
__device__ __forceinline__ void push_sift(const PushArgs<T> &a, int p, int nt, int allow) {
  PushCtl *ctl = a.ctl;
  const int q = p ^ 1;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long b = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); b < nt; b += stride) {
    const long long i = b + (threadIdx.x & 31);
    bool viol = false;
    int32_t v = 0;
    T dv = T(1);
    if (i < nt) {
      v = __ldcg(a.touched + i);
      atomicAnd(a.bits + (v >> 5), ~(1u << (v & 31)));
      dv = a.diag[v];
      const T *r = a.R + (long long)v * a.ldr;
      // in the working precision, as the synchronous push compares (dynlp/solvers.py:105-106)
      for (int c0 = 0; c0 < a.C; c0 += kPushCols) {
        T x[kPushCols];
#pragma unroll
        for (int i = 0; i < kPushCols; ++i) x[i] = c0 + i < a.C ? __ldcg(r + c0 + i) : T(0);
#pragma unroll
        for (int i = 0; i < kPushCols; ++i) viol |= c0 + i < a.C && fabs(x[i]) > (T)a.eps[c0 + i] * dv;
      }
    }
    if (allow < 0) {
      if (viol) ctl->status = -allow;  // a violating row is left for a round that will not run
      continue;
    }
    const int slot = warp_reserve(viol, &ctl->fcnt[q]);
    if (viol) {
      a.front[slot] = v;
      take_row(a, v, slot, dv);
    }
  }
}

template <typename TW, typename T, int CMAX>
__global__ void __launch_bounds__(kPushThreads) k_push_scatter(PushArgs<T> a, int p) {
  PushCtl *ctl = a.ctl;
  const int q = p ^ 1;
  const int nf = ctl->fcnt[p];
  const int status = ctl->status;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->fcnt[q] = 0;  // this round's sift fills the next frontier
    ctl->tcnt[q] = 0;  // and the next round's scatter the next touched list
    if (status != kRunning || nf == 0) {
      if (status == kRunning) ctl->status = kConverged;
    } else {
      ctl->rounds += 1;
      ctl->frontier_rows += (unsigned long long)nf;
      // one decision for the whole round: its sift takes rows in every block or in none
      ctl->allow = read_cancel(a.cancel) ? -kCancelled : (ctl->rounds < ctl->max_rounds ? 1 : -kCapped);
    }
  }
  if (status != kRunning || nf == 0) return;
  push_scatter<TW, T, CMAX>(a, p, nf);
}

template <typename T>
__global__ void __launch_bounds__(kPushThreads) k_push_sift(PushArgs<T> a, int p) {
  PushCtl *ctl = a.ctl;
  const int nt = ctl->tcnt[p];
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->touched_rows += (unsigned long long)nt;
  push_sift(a, p, nt, ctl->allow);
}

// The first round's take: the candidate rows cand[0..nc) become the frontier of parity 0.
template <typename T>
__global__ void __launch_bounds__(kPushThreads) k_push_seed(PushArgs<T> a, const int32_t *__restrict__ cand, int nc) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nc) return;
  const int32_t u = cand[g];
  a.front[g] = u;
  take_row(a, u, (int)g, a.diag[u]);
}

// The whole run in one cooperative launch: the seed's take, then rounds of scatter, barrier, sift, barrier
// until the frontier is empty or the run stops. As two launches a round in a graph's loop, 17 rounds took
// 320 us at n = 60,000 (2 fp64 columns, mean degree 16); in one launch, with both phases as they are now, the
// whole call of 15 rounds takes 280.
template <typename TW, typename T, int CMAX>
__global__ void __launch_bounds__(kPushThreads) k_push_whole(PushArgs<T> a, const int32_t *__restrict__ cand, int nc,
                                                             int words) {
  PushCtl *ctl = a.ctl;
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const bool lead = t0 == 0;
  uint32_t target = 0;
  for (long long i = t0; i < words; i += stride) a.bits[i] = 0u;
  for (long long g = t0; g < nc; g += stride) {
    const int32_t u = cand[g];
    a.front[g] = u;
    take_row(a, u, (int)g, a.diag[u]);
  }
  if (!grid_barrier(&ctl->bar, target)) return;
  unsigned long long rows = 0, touched = 0;
  int rounds = 0;
  for (int p = 0;; p ^= 1) {
    const int nf = __ldcg(&ctl->fcnt[p]);
    if (nf == 0 || __ldcg(&ctl->status) != kRunning) break;
    ++rounds;
    rows += (unsigned long long)nf;
    if (lead) {
      ctl->fcnt[p ^ 1] = 0;  // this round's sift fills the next frontier
      ctl->tcnt[p ^ 1] = 0;  // and the next round's scatter the next touched list
      // one decision for the whole round: its sift takes rows in every block or in none
      ctl->allow = read_cancel(a.cancel) ? -kCancelled : (rounds < ctl->max_rounds ? 1 : -kCapped);
    }
    push_scatter<TW, T, CMAX>(a, p, nf);
    if (!grid_barrier(&ctl->bar, target)) return;
    const int nt = __ldcg(&ctl->tcnt[p]);
    touched += (unsigned long long)nt;
    push_sift(a, p, nt, __ldcg(&ctl->allow));
    if (!grid_barrier(&ctl->bar, target)) return;
  }
  if (lead) {
    ctl->rounds = rounds;
    ctl->frontier_rows = rows;
    ctl->touched_rows = touched;
    if (__ldcg(&ctl->status) == kRunning) ctl->status = kConverged;
  }
}

// ---- host side ----------------------------------------------------------------------------------
static size_t al256(size_t x) { return (x + 255) / 256 * 256; }

struct PushWs {
  PushCtl *ctl;
  int32_t *front, *touched;
  uint32_t *bits;
  void *D;
};

static size_t push_ws_bytes(int32_t n, int32_t C, size_t elem) {
  const size_t nn = (size_t)(n > 0 ? n : 1), cc = (size_t)(C > 0 ? C : 1);
  return al256(sizeof(PushCtl)) + 2 * al256(sizeof(int32_t) * nn) +
         al256(sizeof(uint32_t) * ((nn + 31) / 32)) + al256(elem * nn * cc);
}

static PushWs carve_push(void *ws, int32_t n) {
  const size_t nn = (size_t)(n > 0 ? n : 1);
  char *p = (char *)ws;
  PushWs W;
  W.ctl = (PushCtl *)p;
  p += al256(sizeof(PushCtl));
  W.front = (int32_t *)p;
  p += al256(sizeof(int32_t) * nn);
  W.touched = (int32_t *)p;
  p += al256(sizeof(int32_t) * nn);
  W.bits = (uint32_t *)p;
  p += al256(sizeof(uint32_t) * ((nn + 31) / 32));
  W.D = p;
  return W;
}

struct PushProblem {
  const int32_t *rbeg, *rend, *col;
  const void *w;
  int w_dtype;
  int32_t n, C;
  const void *diag;
  void *Z;
  int64_t ldz;
  void *R;
  int64_t ldr;
  int dtype;
};

template <typename T>
static PushArgs<T> push_args(const PushProblem &q, const PushWs &W, const int32_t *cancel) {
  PushArgs<T> a;
  a.rbeg = q.rbeg;
  a.rend = q.rend;
  a.col = q.col;
  a.w = q.w;
  a.diag = (const T *)q.diag;
  a.Z = (T *)q.Z;
  a.ldz = q.ldz;
  a.R = (T *)q.R;
  a.ldr = q.ldr;
  a.C = q.C;
  a.eps = W.ctl->eps;
  a.front = W.front;
  a.D = (T *)W.D;
  a.touched = W.touched;
  a.bits = W.bits;
  a.ctl = W.ctl;
  a.cancel = cancel;
  return a;
}

// Blocks per SM of k_push_whole: with more, the barriers cost more than the phases gain (n = 60,000, 4 and 17
// columns, us a run: 215 and 440 with one, 216 and 434 with two, 250 and 563 with four; n = 1M, 9 columns:
// 401, 363, 451).
constexpr int kPushPerSm = 2;
// From so many candidates on the rounds are launched: their phases then want more blocks in flight than a barrier can
// join cheaply (n = 1M, fp64, us, launched / one launch: 1M candidates, 1 column 15,100 / 22,200, 5 columns 28,500 /
// 36,300, 17 columns 81,800 / 88,300; 333,000, 1 column 8,040 / 9,990; n = 200,000, all, 1 column 4,620 / 4,700;
// but 100,000 of 1M 404 / 344).
constexpr int kPushLaunchRows = 200000;

// What is launched: one round of parity p (its two phases), or the whole run (p < 0).
struct PushLaunch {
  int p, ncand, words;
  const int32_t *cand;
  cudaStream_t s;
};

template <typename TW, typename T, int CMAX>
static int launch_push_t(const PushArgs<T> &a, const PushLaunch &l) {
  if (l.p >= 0) {
    const int grid = sm_count() * 8;
    k_push_scatter<TW, T, CMAX><<<grid, kPushThreads, 0, l.s>>>(a, l.p);
    k_push_sift<T><<<grid, kPushThreads, 0, l.s>>>(a, l.p);
    return check_launch(2);
  }
  static const int per = [] {
    int k = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_push_whole<TW, T, CMAX>, kPushThreads, 0) !=
        cudaSuccess)
      (void)cudaGetLastError();
    return k;
  }();
  if (per < 1) return DLP_ERR_CUDA;
  PushArgs<T> args_a = a;
  const int32_t *cand = l.cand;
  int nc = l.ncand, words = l.words;
  void *args[] = {(void *)&args_a, (void *)&cand, (void *)&nc, (void *)&words};
  return launch_any_grid((const void *)k_push_whole<TW, T, CMAX>, sm_count() * std::min(per, kPushPerSm), kPushThreads, args,
                         0, l.s);
}

template <typename TW, typename T>
static int launch_push_c(const PushProblem &q, const PushArgs<T> &a, const PushLaunch &l) {
  if (q.C == 1) return launch_push_t<TW, T, 1>(a, l);
  if (q.C == 2) return launch_push_t<TW, T, 2>(a, l);
  if (q.C <= 4) return launch_push_t<TW, T, 4>(a, l);
  if (q.C <= 12) return launch_push_t<TW, T, 12>(a, l);
  if (q.C <= 20) return launch_push_t<TW, T, 20>(a, l);
  if (q.C <= 33) return launch_push_t<TW, T, 33>(a, l);
  return DLP_ERR_INVALID;
}

static int launch_push(const PushProblem &q, const PushWs &W, const int32_t *cancel, const PushLaunch &l) {
  if (q.dtype == DLP_F32 && q.w_dtype == DLP_F32)
    return launch_push_c<float, float>(q, push_args<float>(q, W, cancel), l);
  if (q.dtype == DLP_F64 && q.w_dtype == DLP_F32)
    return launch_push_c<float, double>(q, push_args<double>(q, W, cancel), l);
  if (q.dtype == DLP_F64 && q.w_dtype == DLP_F64)
    return launch_push_c<double, double>(q, push_args<double>(q, W, cancel), l);
  return DLP_ERR_DTYPE;
}

static int launch_seed(const PushProblem &q, const PushWs &W, const int32_t *cand, int nc, cudaStream_t s) {
  const int grid = ceil_div_i(nc, kPushThreads);
  if (q.dtype == DLP_F32)
    k_push_seed<float><<<grid, kPushThreads, 0, s>>>(push_args<float>(q, W, nullptr), cand, nc);
  else
    k_push_seed<double><<<grid, kPushThreads, 0, s>>>(push_args<double>(q, W, nullptr), cand, nc);
  return check_launch();
}

}  // namespace dlp

using namespace dlp;

extern "C" {

size_t dlp_fused_push_workspace_bytes(int32_t n, int32_t C) { return push_ws_bytes(n, C, sizeof(double)); }

int dlp_fused_push(const int32_t *rbeg, const int32_t *rend, const int32_t *col, const void *w, int w_dtype,
                   int32_t n, int32_t C, const void *diag, void *Z, int64_t ldz, void *R, int64_t ldr, int dtype,
                   const double *eps, const int32_t *cand, int32_t ncand, int32_t max_rounds, int32_t check_every,
                   int32_t use_graph, void *ws, size_t ws_bytes, int32_t *rounds_out, int32_t *converged_out,
                   unsigned long long *edges_out, dlp_stream_t stream) {
  if (n < 0 || C <= 0 || C > 33 || ldz < C || ldr < C || ncand < 0 || ncand > n || !eps) return DLP_ERR_INVALID;
  if (!(dtype == DLP_F32 && w_dtype == DLP_F32) && !(dtype == DLP_F64 && (w_dtype == DLP_F32 || w_dtype == DLP_F64)))
    return DLP_ERR_DTYPE;
  if (!ws || ws_bytes < push_ws_bytes(n, C, sizeof(double))) return DLP_ERR_WORKSPACE;
  if (rounds_out) *rounds_out = 0;
  if (converged_out) *converged_out = 1;
  if (edges_out) *edges_out = 0;
  if (ncand == 0) return DLP_OK;
  if (!rbeg || !rend || !col || !w || !diag || !Z || !R || !cand) return DLP_ERR_INVALID;
  if (converged_out) *converged_out = 0;
  if (max_rounds <= 0) return DLP_ERR_CAP;
  cudaStream_t s = (cudaStream_t)stream;
  PushProblem q{rbeg, rend, col, w, w_dtype, n, C, diag, Z, ldz, R, ldr, dtype};
  PushWs W = carve_push(ws, n);
  const int32_t *cancel = cancel_word();
  PushCtl h{};
  h.max_rounds = max_rounds;
  h.fcnt[0] = ncand;
  memcpy(h.eps, eps, sizeof(double) * (size_t)C);
  DLP_CUDA(cudaMemcpyAsync(W.ctl, &h, sizeof(h), cudaMemcpyHostToDevice, s));
  const int words = (int)(((long long)n + 31) / 32);
  PushCtl out{};
  if (use_graph && ncand < kPushLaunchRows) {
    DLP_TRY(launch_push(q, W, cancel, PushLaunch{-1, ncand, words, cand, s}));
  } else {
    DLP_CUDA(cudaMemsetAsync(W.bits, 0, sizeof(uint32_t) * (size_t)words, s));
    DLP_TRY(launch_seed(q, W, cand, ncand, s));
    const int every = check_every > 0 ? check_every : 8;
    for (long long r = 0; r <= (long long)max_rounds + 1; r += 2 * ((every + 1) / 2)) {
      for (int i = 0; i < (every + 1) / 2; ++i) {
        DLP_TRY(launch_push(q, W, cancel, PushLaunch{0, 0, 0, nullptr, s}));
        DLP_TRY(launch_push(q, W, cancel, PushLaunch{1, 0, 0, nullptr, s}));
      }
      DLP_CUDA(cudaMemcpyAsync(&out, W.ctl, sizeof(out), cudaMemcpyDeviceToHost, s));
      DLP_CUDA(cudaStreamSynchronize(s));
      if (out.status != kRunning) break;
    }
  }
  DLP_CUDA(cudaMemcpyAsync(&out, W.ctl, sizeof(out), cudaMemcpyDeviceToHost, s));
  DLP_CUDA(cudaStreamSynchronize(s));
  // a wait ran out in a block, or the loop ended without a decision
  if (out.bar.abort || out.status == kRunning) return DLP_ERR_DEVICE;
  if (rounds_out) *rounds_out = out.rounds;
  if (converged_out) *converged_out = out.status == kConverged ? 1 : 0;
  if (edges_out) *edges_out = out.edges;
  if (out.status == kCapped) return DLP_ERR_CAP;
  if (out.status == kCancelled) return DLP_ERR_CANCELLED;
  return DLP_OK;
}

int dlp_fused_push_counts(const void *ws, unsigned long long *out, dlp_stream_t stream) {
  if (!ws || !out) return DLP_ERR_INVALID;
  PushCtl c{};
  cudaStream_t s = (cudaStream_t)stream;
  DLP_CUDA(cudaMemcpyAsync(&c, ws, sizeof(c), cudaMemcpyDeviceToHost, s));
  DLP_CUDA(cudaStreamSynchronize(s));
  out[0] = (unsigned long long)c.rounds;
  out[1] = c.frontier_rows;
  out[2] = c.touched_rows;
  out[3] = c.edges;
  return DLP_OK;
}

}  // extern "C"
