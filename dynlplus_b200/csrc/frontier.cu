// DynLP's frontier Jacobi with its round loop on the device (dynlp/solvers.py:213-241): one
// cooperative launch runs the rounds
//   1. every frontier row's new value from the values before the round (k_jacobi's formula and
//      summation order), kept in Y; rows that move by more than delta go to the update list;
//   2. the update list's rows take their new values; they and their neighbours, each once, are the
//      next frontier;
// with a grid barrier after each part. What bounds it: a round of a small frontier is a chain of
// dependent loads (row range, column, score) and the two barriers, no bandwidth; the host loop it
// replaces spent some 20 launches and three host reads per round on the same work.
// Measured on B200 (vertex arrivals, n = 20,000, degree 10, one column, five batches of some 350
// rounds each): see the figures at k_frontier_rounds.
#include "gather.cuh"

namespace dlp {

constexpr int kFrThreads = 256;
constexpr int kFrChunk = 8192;  // rounds per launch: the host loop regains control between launches

// Counts rotate over three slots so that a round clears the slot the next one fills while the third
// is still being read.
struct FrCtl {
  GridBar bar;
  int32_t fcnt[3], ucnt[3];  // frontier rows and changed rows of round r at slot r mod 3
  int32_t round, status;     // rounds run; 1: converged
  unsigned long long edges;  // stored entries visited (frontier rows, and changed rows when marking)
};

template <class T>
struct FrArgs {
  const int32_t *rbeg, *rend, *col;
  const typename T::TW *w;
  int32_t n, C;
  typename T::TX *X;
  int64_t ldx;
  const typename T::TX *rhs;
  int64_t ldr;
  const typename T::TX *diag;
  double delta;
  int32_t *front[2];   // the frontier of round r: front[r & 1]
  int32_t *upd;        // positions in the frontier of the rows that changed
  int32_t *stamp;      // r + 1 once the row joined the frontier of round r + 1
  typename T::TX *Y;   // new values, one row per frontier position
  FrCtl *ctl;
  int32_t max_rounds;
  int G, LV, NV;
};

// 256 threads, one to two blocks per SM (frontier_grid): more blocks make the barriers slower, and a
// frontier seldom fills more. Arrivals n = 20,000, degree 10, one column, some 1,760 rounds in all:
// 411 ms with a host loop.
template <class T, int VW, int VPL>
__global__ void __launch_bounds__(kFrThreads) k_frontier_rounds(FrArgs<T> p) {
  using TA = typename T::TA;
  using TX = typename T::TX;
  FrCtl *ctl = p.ctl;
  const int lane = threadIdx.x & 31;
  const int G = p.G, LV = p.LV, NV = p.NV;
  const int gl = lane & (G - 1);
  const int cl = gl & (LV - 1);
  const int es = gl / LV;
  const int ES = G / LV;
  const int gpw = 32 / G;
  const int gbase = lane & ~(G - 1);
  const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << gbase);
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int r0 = __ldcg(&ctl->round);
  uint32_t bar = 0;
  unsigned long long edges = 0;
  int done = 0, status = 0;
  for (; done < p.max_rounds; ++done) {
    const int rd = r0 + done, s = rd % 3, sn = (rd + 1) % 3;
    const int nf = __ldcg(&ctl->fcnt[s]);
    if (nf == 0) {
      status = 1;
      break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctl->fcnt[(rd + 2) % 3] = 0;
      ctl->ucnt[sn] = 0;
    }
    const int32_t *front = p.front[rd & 1];
    for (long long g0 = warp * gpw; g0 < nf; g0 += nwarps * gpw) {
      const long long gi = g0 + lane / G;
      const bool valid = gi < nf;
      const int r = valid ? __ldcg(front + gi) : 0;
      const int beg = valid ? p.rbeg[r] : 0;
      const int end = valid ? p.rend[r] : 0;
      TA acc[VPL][VW];
      gather_row<typename T::TW, TX, TA, VW, VPL, gather_batch_wide<TA, VW, VPL>(), kRowVec, true>(
          p.col, p.w, p.X, p.ldx, beg, end, es, ES, cl, LV, NV, G, acc);
      bool ch = false;
      if (valid && es == 0) {
        const TA inv = TA(1) / cvt<TA>(p.diag[r]);
#pragma unroll
        for (int k = 0; k < VPL; ++k) {
          const int vi = cl + k * LV;
          if (vi < NV) {
#pragma unroll
            for (int i = 0; i < VW; ++i) {
              const int c = vi * VW + i;
              if (c < p.C) {
                const TA yv = (cvt<TA>(p.rhs[(long long)r * p.ldr + c]) + acc[k][i]) * inv;
                p.Y[gi * p.C + c] = cvt<TX>(yv);
                ch |= fabs(yv - cvt<TA>(__ldcg(p.X + (long long)r * p.ldx + c))) > (TA)p.delta;
              }
            }
          }
        }
      }
      const bool any = (__ballot_sync(0xffffffffu, ch) & gmask) != 0;
      if (valid && gl == 0) edges += (unsigned long long)(end - beg);
      const int slot = warp_reserve(valid && gl == 0 && any, &ctl->ucnt[s]);
      if (slot >= 0) p.upd[slot] = (int32_t)gi;
    }
    if (!grid_barrier(&ctl->bar, bar)) return;
    const int nu = __ldcg(&ctl->ucnt[s]);
    if (nu == 0) {
      ++done;
      status = 1;
      break;
    }
    // eight lanes per changed row; entry 0 is the row itself
    int32_t *next = p.front[(rd + 1) & 1];
    for (long long g0 = warp * 4; g0 < nu; g0 += nwarps * 4) {
      const long long i = g0 + (lane >> 3);
      const bool valid = i < nu;
      const int gi = valid ? __ldcg(p.upd + i) : 0;
      const int r = valid ? __ldcg(front + gi) : 0;
      const int beg = valid ? p.rbeg[r] : 0, end = valid ? p.rend[r] : 0;
      if (valid)
        for (int c = lane & 7; c < p.C; c += 8)
          p.X[(long long)r * p.ldx + c] = __ldcg(p.Y + (long long)gi * p.C + c);
      if (valid && (lane & 7) == 0) edges += (unsigned long long)(end - beg);
      const int trips = __reduce_max_sync(0xffffffffu, valid ? (end - beg + 1 + 7) >> 3 : 0);
      for (int t = 0; t < trips; ++t) {
        const int j = beg - 1 + (lane & 7) + 8 * t;
        bool first = false;
        int v = 0;
        if (valid && j < end) {
          v = j < beg ? r : p.col[j];
          first = __ldcg(p.stamp + v) != rd + 1 && atomicExch(p.stamp + v, rd + 1) != rd + 1;
        }
        const int slot = warp_reserve(first, &ctl->fcnt[sn]);
        if (slot >= 0) next[slot] = v;
      }
    }
    if (!grid_barrier(&ctl->bar, bar)) return;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) edges += __shfl_xor_sync(0xffffffffu, edges, off);
  if (lane == 0 && edges) atomicAdd(&ctl->edges, edges);
  // every block has read ctl->round: it passed a barrier, or done is 0 and the value stays
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (done) ctl->round = r0 + done;
    ctl->status = status;
  }
}

__global__ void k_frontier_seed(const int32_t *__restrict__ seed, int32_t ns, FrCtl *ctl, int32_t *front) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) ctl->fcnt[0] = ns;
  if (i < ns) front[i] = seed[i];
}

static size_t fr_align(size_t x) { return (x + 255) / 256 * 256; }

static size_t fr_bytes(int32_t n, int32_t C, size_t es) {
  const size_t nn = (size_t)(n > 0 ? n : 1);
  return fr_align(sizeof(FrCtl)) + 4 * fr_align(4 * nn) + fr_align(es * nn * (size_t)C);
}

template <class T>
struct FrRun {
  FrArgs<T> a;
  cudaStream_t s;
  template <int VW, int VPL>
  int launch() {
    static const int per = [] {
      int k = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_frontier_rounds<T, VW, VPL>, kFrThreads, 0) != cudaSuccess)
        (void)cudaGetLastError();
      return k;
    }();
    if (per < 1) return DLP_ERR_CUDA;
    // enough blocks for half of the rows at once, at most two per SM
    const long long want = ((long long)a.n * a.G / 2 + kFrThreads - 1) / kFrThreads;
    const int cap = sm_count() * std::min(per, 2);
    const int grid = (int)std::max(1LL, std::min(want, (long long)cap));
    void *args[] = {(void *)&a};
    DLP_CUDA(cudaLaunchCooperativeKernel((const void *)k_frontier_rounds<T, VW, VPL>, dim3(grid), dim3(kFrThreads), args,
                                         0, s));
    return check_launch();
  }
  template <int VW>
  int launch_vpl(int VPL) {
    switch (VPL) {
      case 1: return launch<VW, 1>();
      case 2: return launch<VW, 2>();
      case 3: return launch<VW, 3>();
      case 4: return launch<VW, 4>();
      case 8: return launch<VW, 8>();
      default: return DLP_ERR_INVALID;
    }
  }
};

template <class T>
static int run_frontier(const int32_t *rbeg, const int32_t *rend, const int32_t *col, const void *w, int32_t n,
                        int32_t C, void *X, int64_t ldx, const void *rhs, int64_t ldr, const void *diag, double delta,
                        const int32_t *seed, int32_t nseed, int32_t max_rounds, int32_t group, double avg_deg, void *ws,
                        int32_t *rounds_out, unsigned long long *edges_out, cudaStream_t s) {
  using TX = typename T::TX;
  Layout L;
  DLP_TRY(choose_layout(C, sizeof(TX), X, ldx, group, avg_deg, &L));
  const size_t nn = (size_t)n;
  char *q = (char *)ws;
  auto take = [&](size_t b) {
    char *r = q;
    q += fr_align(b);
    return r;
  };
  FrRun<T> R;
  R.s = s;
  FrArgs<T> &a = R.a;
  a = FrArgs<T>{};
  a.rbeg = rbeg;
  a.rend = rend;
  a.col = col;
  a.w = (const typename T::TW *)w;
  a.n = n;
  a.C = C;
  a.X = (TX *)X;
  a.ldx = ldx;
  a.rhs = (const TX *)rhs;
  a.ldr = ldr;
  a.diag = (const TX *)diag;
  a.delta = delta;
  a.ctl = (FrCtl *)take(sizeof(FrCtl));
  a.stamp = (int32_t *)take(4 * nn);
  a.front[0] = (int32_t *)take(4 * nn);
  a.front[1] = (int32_t *)take(4 * nn);
  a.upd = (int32_t *)take(4 * nn);
  a.Y = (TX *)take(sizeof(TX) * nn * (size_t)C);
  a.G = L.G;
  a.LV = L.LV;
  a.NV = L.NV;
  DLP_CUDA(cudaMemsetAsync(a.ctl, 0, fr_align(sizeof(FrCtl)) + 4 * nn, s));  // control block and stamps
  k_frontier_seed<<<ceil_div_i(nseed, 256), 256, 0, s>>>(seed, nseed, a.ctl, a.front[0]);
  DLP_TRY(check_launch());
  FrCtl h{};
  while (h.round < max_rounds) {
    a.max_rounds = std::min(kFrChunk, max_rounds - h.round);
    if (h.round > 0) DLP_CUDA(cudaMemsetAsync(&a.ctl->bar, 0, sizeof(GridBar), s));
    DLP_TRY(L.VW == 1 ? R.template launch_vpl<1>(L.VPL) : R.template launch_vpl<16 / sizeof(TX)>(L.VPL));
    DLP_CUDA(cudaMemcpyAsync(&h, a.ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
    DLP_CUDA(cudaStreamSynchronize(s));
    if (h.bar.abort) return DLP_ERR_DEVICE;
    if (h.status) break;
  }
  if (rounds_out) *rounds_out = h.round;
  if (edges_out) *edges_out = h.edges;
  return DLP_OK;
}

}  // namespace dlp

using namespace dlp;

extern "C" {

size_t dlp_frontier_solve_workspace_bytes(int32_t n, int32_t C, int dtype) {
  return fr_bytes(n, C > 0 ? C : 1, dtype == DLP_F64 ? 8 : 4);
}

int dlp_frontier_solve(const int32_t *rbeg, const int32_t *rend, const int32_t *col, const void *w, int w_dtype,
                       int32_t n, int32_t C, void *X, int64_t ldx, const void *rhs, int64_t ldr, const void *diag,
                       int dtype, double delta, const int32_t *seed, int32_t nseed, int32_t max_rounds, int32_t group,
                       double avg_deg, void *ws, size_t ws_bytes, int32_t *rounds_out, unsigned long long *edges_out,
                       dlp_stream_t stream) {
  if (rounds_out) *rounds_out = 0;
  if (edges_out) *edges_out = 0;
  if (n < 0 || C <= 0 || nseed < 0 || nseed > n || ldx < C || ldr < C) return DLP_ERR_INVALID;
  if (nseed == 0 || max_rounds <= 0) return DLP_OK;
  if (!rbeg || !rend || !col || !w || !X || !rhs || !diag || !seed) return DLP_ERR_INVALID;
  if (!ws || ws_bytes < dlp_frontier_solve_workspace_bytes(n, C, dtype)) return DLP_ERR_WORKSPACE;
#define DLP_FR_ARGS rbeg, rend, col, w, n, C, X, ldx, rhs, ldr, diag, delta, seed, nseed, max_rounds, group, avg_deg, \
                    ws, rounds_out, edges_out, (cudaStream_t)stream
  if (w_dtype == DLP_F32 && dtype == DLP_F32) return run_frontier<T_F32>(DLP_FR_ARGS);
  if (w_dtype == DLP_F64 && dtype == DLP_F64) return run_frontier<T_F64>(DLP_FR_ARGS);
  if (w_dtype == DLP_F32 && dtype == DLP_F64) return run_frontier<T_W32X64>(DLP_FR_ARGS);
#undef DLP_FR_ARGS
  return DLP_ERR_DTYPE;
}

}  // extern "C"
