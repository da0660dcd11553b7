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
// rounds each): host loop 411 ms; lists 33 ms of kernel time (18.6 us a round); without lists, below
// kFrDenseRows rows, 10 ms.
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
    uint32_t walked = 0;
    for (long long g0 = warp * gpw; g0 < nf; g0 += nwarps * gpw) {
      const long long gi = g0 + lane / G;
      const bool valid = gi < nf;
      const int r = valid ? __ldcg(front + gi) : 0;
      const int beg = valid ? p.rbeg[r] : 0;
      const int end = valid ? p.rend[r] : 0;
      bar_announce(&ctl->bar, end - beg, walked);
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
    walked = 0;
    for (long long g0 = warp * 4; g0 < nu; g0 += nwarps * 4) {
      const long long i = g0 + (lane >> 3);
      const bool valid = i < nu;
      const int gi = valid ? __ldcg(p.upd + i) : 0;
      const int r = valid ? __ldcg(front + gi) : 0;
      const int beg = valid ? p.rbeg[r] : 0, end = valid ? p.rend[r] : 0;
      bar_announce(&ctl->bar, end - beg, walked);
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

// The same rounds for systems small enough that looking at every row's mark is cheaper than keeping lists:
// a lane group owns its rows, X is kept in two buffers that the rounds read and write in turn (so a round
// needs one barrier, not two), and joining a frontier is a plain store of the round's number to the row's
// mark of the next round's parity. The number of blocks with a changed row travels with the barrier's
// arrival count, one counter per parity. A round is then a mark load, the gather of active rows and the
// barrier.
struct FrDenseCtl {
  unsigned long long bar[2];  // arrivals (low 32 bits) and arrivals with a change (high) of each parity
  int32_t abort, round, status, pad;
  unsigned long long edges;
};

template <class T>
struct FrDense {
  const int32_t *rbeg, *rend, *col;
  const typename T::TW *w;
  int32_t n, C, rows;
  typename T::TX *X[2];  // the caller's X and the second buffer
  int64_t ldx[2];
  const typename T::TX *rhs;
  int64_t ldr;
  const typename T::TX *diag;
  double delta;
  int32_t *mark[2];  // mark[r & 1][v] == r + 1: v is in the frontier of round r
  FrDenseCtl *ctl;
  int32_t max_rounds;
  int G, LV;
};
constexpr int kFrDenseThreads = 512;

template <class T, int VW>
__global__ void __launch_bounds__(kFrDenseThreads, 1) k_frontier_dense(FrDense<T> p) {
  using TA = typename T::TA;
  using TX = typename T::TX;
  constexpr int NT = kFrDenseThreads;
  FrDenseCtl *ctl = p.ctl;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int G = p.G, LV = p.LV, ES = G / LV, gpw = 32 / G;
  const int gl = lane & (G - 1), cl = gl & (LV - 1), es = gl / LV;
  const bool on = cl * VW < p.C;
  const unsigned gmask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << (lane & ~(G - 1));
  const int row0 = blockIdx.x * p.rows, nr = max(0, min(p.rows, p.n - row0));
  extern __shared__ uint8_t s_moved[];  // per row: it changed in the round before (its old buffer is stale)
  __shared__ int s_any, s_go;
  for (int i = threadIdx.x; i < nr; i += NT) s_moved[i] = 0;
  const int r0 = __ldcg(&ctl->round);
  unsigned long long edges = 0;
  unsigned long long seen[2] = {0, 0};  // each parity's count after its last round (zero at the launch)
  int done = 0, status = 0;
  for (; done < p.max_rounds; ++done) {
    const int rd = r0 + done;
    const TX *X = p.X[rd & 1];
    TX *Xn = p.X[(rd + 1) & 1];
    const int64_t ldx = p.ldx[rd & 1], ldn = p.ldx[(rd + 1) & 1];
    const int32_t *mark = p.mark[rd & 1];
    int32_t *next = p.mark[(rd + 1) & 1];
    if (threadIdx.x == 0) s_any = 0;
    __syncthreads();
    for (int g0 = wid * gpw; g0 < nr; g0 += (NT / 32) * gpw) {
      const int i = g0 + lane / G;
      const bool valid = i < nr;
      const long long r = row0 + i;
      const bool act = valid && __ldcg(mark + r) == rd + 1;
      const bool stale = valid && s_moved[i] != 0;
      if (!__any_sync(0xffffffffu, act || stale)) continue;
      const int beg = act ? p.rbeg[r] : 0, end = act ? p.rend[r] : 0;
      TA acc[VW];
#pragma unroll
      for (int k = 0; k < VW; ++k) acc[k] = TA(0);
      // the row's own values and right-hand side, in flight with the gather
      TX xo[VW], xn[VW], rh[VW];
      const bool own = valid && es == 0 && (act || stale);
#pragma unroll
      for (int k = 0; k < VW; ++k) {
        const int c = cl * VW + k;
        xo[k] = own && c < p.C ? __ldcg(X + r * ldx + c) : TX(0);
        rh[k] = own && act && c < p.C ? p.rhs[r * p.ldr + c] : TX(0);
      }
      const TA inv = own && act ? TA(1) / cvt<TA>(p.diag[r]) : TA(0);
      constexpr int U = VW == 1 ? 8 : 4;  // entries in flight per lane
      for (int j0 = beg + es; j0 < end && on; j0 += U * ES) {
        int v[U];
        TA wv[U];
        TX x[U][VW];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int j = j0 + u * ES;
          v[u] = j < end ? p.col[j] : -1;
          wv[u] = j < end ? cvt<TA>(p.w[j]) : TA(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
          for (int k = 0; k < VW; ++k) x[u][k] = TX(0);
          if (v[u] >= 0) {
            if constexpr (VW > 1) load_vec_coherent<TX, VW, TX>(X + (long long)v[u] * ldx + cl * VW, x[u]);
            else x[u][0] = __ldcg(X + (long long)v[u] * ldx + cl);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int k = 0; k < VW; ++k) acc[k] = fmaa(wv[u], cvt<TA>(x[u][k]), acc[k]);
      }
      for (int off = LV; off < G; off <<= 1) {
#pragma unroll
        for (int k = 0; k < VW; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], off);
      }
      bool ch = false;
#pragma unroll
      for (int k = 0; k < VW; ++k) {
        const TA yv = (cvt<TA>(rh[k]) + acc[k]) * inv;
        xn[k] = cvt<TX>(yv);
        ch |= own && act && cl * VW + k < p.C && fabs(yv - cvt<TA>(xo[k])) > (TA)p.delta;
      }
      const bool any = (__ballot_sync(0xffffffffu, ch) & gmask) != 0;  // the row changed (any of its lanes)
      if (valid && es == 0 && (any || stale)) {
#pragma unroll
        for (int k = 0; k < VW; ++k)
          if (cl * VW + k < p.C) __stcg(Xn + r * ldn + cl * VW + k, any ? xn[k] : xo[k]);
      }
      if (gl == 0 && act) edges += (unsigned long long)(end - beg);
      if (any && gl == 0) {
        edges += (unsigned long long)(end - beg);
        s_any = 1;
      }
      if (any) {  // the row and its stored neighbours are the next frontier
        for (int j = beg + gl; j < end; j += G) __stcg(next + p.col[j], rd + 2);
        if (gl == 0) __stcg(next + r, rd + 2);
      }
      if (valid && gl == 0) s_moved[i] = any;
    }
    // the barrier, with this block's word on whether any row changed
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long *bar = &ctl->bar[rd & 1];
      const unsigned long long was = seen[rd & 1];
      __threadfence();
      atomicAdd(bar, 1ull + (s_any ? 1ull << 32 : 0ull));
      int spins = 0, go = 0;
      unsigned long long v = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
        if ((uint32_t)v - (uint32_t)was >= gridDim.x) break;
        if ((++spins & 1023) == 0) {
          if (*(volatile int32_t *)&ctl->abort) go = -1;
          if (spins >= kBarSpins) {
            atomicExch(&ctl->abort, 1);
            go = -1;
          }
          if (go < 0) break;
        }
      }
      __threadfence();
      seen[rd & 1] = v;
      s_go = go < 0 ? -1 : (uint32_t)(v >> 32) != (uint32_t)(was >> 32);
    }
    __syncthreads();
    if (s_go < 0) return;
    if (s_go == 0) {  // nothing changed in this round
      ++done;
      status = 1;
      break;
    }
  }
  // the newest values are those the next round would read; the other buffer takes them too (the result is
  // in the caller's X, and a further launch starts from equal buffers)
  const int rd = r0 + done;
  const TX *src = p.X[rd & 1];
  TX *dst = p.X[(rd + 1) & 1];
  const int64_t lds = p.ldx[rd & 1], ldd = p.ldx[(rd + 1) & 1];
  for (int i = threadIdx.x; i < nr * p.C; i += NT) {
    const long long r = row0 + i / p.C;
    const int c = i % p.C;
    __stcg(dst + r * ldd + c, __ldcg(src + r * lds + c));
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) edges += __shfl_xor_sync(0xffffffffu, edges, off);
  if (lane == 0 && edges) atomicAdd(&ctl->edges, edges);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->round = rd;
    ctl->status = status;
  }
}

__global__ void k_frontier_marks(const int32_t *__restrict__ seed, int32_t ns, int32_t *mark) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ns) mark[seed[i]] = 1;
}

__global__ void k_frontier_seed(const int32_t *__restrict__ seed, int32_t ns, FrCtl *ctl, int32_t *front) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) ctl->fcnt[0] = ns;
  if (i < ns) front[i] = seed[i];
}

static size_t fr_align(size_t x) { return (x + 255) / 256 * 256; }

static size_t fr_bytes(int32_t n, int32_t C, size_t es) {
  const size_t nn = (size_t)(n > 0 ? n : 1);
  // the dense form's second buffer is padded by up to three columns
  return fr_align(sizeof(FrCtl)) + 4 * fr_align(4 * nn) + fr_align(es * nn * (size_t)(C + 3));
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
    return launch_any_grid((const void *)k_frontier_rounds<T, VW, VPL>, grid, kFrThreads, args, 0, s);
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

// Whether the rounds run without lists: up to kFrDenseRows rows, and the gather layout's entry slots leave
// room for one lane per vector of a row.
constexpr int kFrDenseRows = 300000;

template <class T, int VW>
static int launch_dense(FrDense<T> &a, cudaStream_t s) {
  void *args[] = {(void *)&a};
  const int grid = (a.n + a.rows - 1) / a.rows;
  return launch_cooperative((const void *)k_frontier_dense<T, VW>, grid, kFrDenseThreads, args, (size_t)a.rows, s);
}

template <class T>
static int run_dense(FrDense<T> &a, int VW, const int32_t *seed, int32_t nseed, int32_t max_rounds, char *marks,
                     int32_t *rounds_out, unsigned long long *edges_out, cudaStream_t s) {
  using TX = typename T::TX;
  DLP_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(FrDenseCtl), s));
  const size_t mb = fr_align(4 * (size_t)a.n);
  DLP_CUDA(cudaMemsetAsync(marks, 0, 2 * mb, s));
  a.mark[0] = (int32_t *)marks;
  a.mark[1] = (int32_t *)(marks + mb);
  k_frontier_marks<<<ceil_div_i(nseed, 256), 256, 0, s>>>(seed, nseed, a.mark[0]);
  DLP_TRY(check_launch());
  DLP_CUDA(cudaMemcpy2DAsync(a.X[1], a.ldx[1] * sizeof(TX), a.X[0], a.ldx[0] * sizeof(TX), a.C * sizeof(TX), a.n,
                             cudaMemcpyDeviceToDevice, s));
  FrDenseCtl h{};
  while (h.round < max_rounds) {
    a.max_rounds = std::min(kFrChunk, max_rounds - h.round);
    if (h.round > 0) DLP_CUDA(cudaMemsetAsync(a.ctl->bar, 0, sizeof(a.ctl->bar), s));
    if (VW == 1) DLP_TRY((launch_dense<T, 1>(a, s)));
    else DLP_TRY((launch_dense<T, 16 / sizeof(TX)>(a, s)));
    DLP_CUDA(cudaMemcpyAsync(&h, a.ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
    DLP_CUDA(cudaStreamSynchronize(s));
    if (h.abort) return DLP_ERR_DEVICE;
    if (h.status) break;
  }
  if (rounds_out) *rounds_out = h.round;
  if (edges_out) *edges_out = h.edges;
  return DLP_OK;
}

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
  {
    const int LV = next_pow2(L.NV), ES = L.G / L.LV;
    if (n <= kFrDenseRows && LV * ES <= 32) {
      FrDense<T> d{};
      d.rbeg = rbeg;
      d.rend = rend;
      d.col = col;
      d.w = (const typename T::TW *)w;
      d.n = n;
      d.C = C;
      d.rows = std::max((n + sm_count() - 1) / sm_count(), 8);
      d.rhs = (const TX *)rhs;
      d.ldr = ldr;
      d.diag = (const TX *)diag;
      d.delta = delta;
      d.G = LV * ES;
      d.LV = LV;
      d.ctl = (FrDenseCtl *)take(sizeof(FrCtl) > sizeof(FrDenseCtl) ? sizeof(FrCtl) : sizeof(FrDenseCtl));
      char *marks = take(4 * nn);
      take(4 * nn);
      take(4 * nn);
      take(4 * nn);
      d.X[0] = (TX *)X;
      d.ldx[0] = ldx;
      d.X[1] = (TX *)take(sizeof(TX) * nn * (size_t)(C + 3));
      d.ldx[1] = (int64_t)L.NV * L.VW;
      const int st = run_dense<T>(d, L.VW, seed, nseed, max_rounds, marks, rounds_out, edges_out, s);
      if (st != kNotLaunched) return st;  // else the lists, on as many blocks as the device holds
      q = (char *)ws;
    }
  }
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
