// Connected components (dynlp/cc.py:8-23) as a lock-free union-find: every edge hooks the larger
// of its two roots under the smaller one with atomicCAS, finds use path halving, and a final pass
// compresses every vertex to its root. Because a root is only ever hooked under a smaller id, the
// root of each component is its minimum vertex id, whatever the schedule: the result is the
// reference's canonical labelling before its rank relabel (cc.py:22), bit-exact.
#include <algorithm>

#include "common.cuh"

namespace dlp {

int compact_roots(const int32_t *parent, int32_t n, int32_t *pos, int32_t *count, void *ws, size_t ws_bytes,
                  cudaStream_t s);
int compact_masked_roots(const int32_t *parent, const uint8_t *mask, int32_t n, int32_t *pos, int32_t *count,
                         void *ws, size_t ws_bytes, cudaStream_t s);
int compact_positions(const uint8_t *flag, int32_t n, int32_t *pos, int32_t *count, void *ws, size_t ws_bytes,
                      cudaStream_t s);
size_t compact_ws_bytes(int32_t n);

constexpr int kCcThreads = 256;
constexpr int kMaxSteps = 1 << 26;  // bound on any chase / retry loop (far above any path length)

__global__ void k_cc_init(int32_t *parent, int32_t n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) parent[i] = (int32_t)i;
}

// Root of x with path halving. parent[] only ever decreases, so stale reads are safe.
__device__ __forceinline__ int32_t find_root(volatile int32_t *parent, int32_t x, int32_t *err) {
  int32_t cur = parent[x];
  if (cur == x) return x;
  int32_t prev = x;
  int steps = 0;
  int32_t next;
  while (cur > (next = parent[cur])) {
    parent[prev] = next;
    prev = cur;
    cur = next;
    if (++steps > kMaxSteps) {
      if (err) atomicExch(err, DLP_ERR_DEVICE);
      break;
    }
  }
  return cur;
}

__device__ __forceinline__ void unite(int32_t *parent_, int32_t a, int32_t b, int32_t *err) {
  volatile int32_t *parent = parent_;
  int32_t ra = find_root(parent, a, err), rb = find_root(parent, b, err);
  int steps = 0;
  while (ra != rb) {
    if (ra < rb) {
      const int32_t t = ra;
      ra = rb;
      rb = t;
    }
    // hook ra (larger) under rb (smaller)
    const int32_t ret = atomicCAS(parent_ + ra, ra, rb);
    if (ret == ra) break;
    ra = ret;  // ra was hooked meanwhile: climb from its new parent
    if (++steps > kMaxSteps) {
      if (err) atomicExch(err, DLP_ERR_DEVICE);
      break;
    }
  }
}

__global__ void __launch_bounds__(kCcThreads)
    k_cc_edges(int32_t n, const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, int64_t m,
               int32_t *parent, int32_t *err) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (long long)gridDim.x * blockDim.x) {
    const int32_t a = rows[i], b = cols[i];
    if ((unsigned)a >= (unsigned)n || (unsigned)b >= (unsigned)n) {
      if (err) atomicExch(err, DLP_ERR_DEVICE);
      continue;
    }
    if (a != b) unite(parent, a, b, err);
  }
}

// The edge list's components in rounds, one cooperative launch: every edge whose ends have different roots
// offers the smaller root to the larger one (atomicMin: the smallest offer of the round stands, an edge whose
// offer did not is seen again in the next round), then every vertex is pointed at its root. Ends with a
// round that saw no such edge, or after kCcRounds with one pass of unions. The offers spread over the larger
// roots and no thread retries, where the lock-free unions (k_cc_edges) of a forming giant component meet on a
// few roots and chase chains that change under them: n = 2M, 1.5M edges (a giant component of half the
// vertices) 850 -> 188 us; n = 1M, 4M edges 390 -> 260.
struct CcCtl {
  GridBar bar;
  int32_t open[2];  // the round of each parity saw an edge between two roots
};
constexpr int kCcRoundThreads = 1024;
__device__ __forceinline__ int32_t ld_l1(const int32_t *p) {
  int32_t v;
  asm volatile("ld.global.ca.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Rounds before the edges still open are joined by the lock-free unions. A giant component has formed by then and its
// many edges are closed; the unions of the rest meet on no common root, while further rounds would read every edge
// again for them (us, 4 / 5 / 6 / 64 rounds: 800,000 vertices of degree 1.26, the slowest of five graphs, 356 / 174 /
// 177 / 176; 2M in a path in random order 314 / 333 / 358 / 543, the unions alone 298; a grid of 2M in random order
// 812 / 740 / 454 / 489, the unions alone 2,124).
constexpr int kCcRounds = 5;
constexpr int32_t kCcLost = -DLP_ERR_DEVICE;  // *err of a lost wait (an edge's end out of range: DLP_ERR_DEVICE)
// Where the rounds are used: half a million edges on, a mean degree above 1.25, where a giant component forms, and up
// to 12M vertices, whose parents the L2 holds beside the edges that pass through. Elsewhere the unions are done sooner
// (whole calls, us, unions / rounds: n = 2M, degree 0.8, 148 / 218; 4M, 1.05, 285 / 377; 8M, 1.2, 571 / 674; 30M, 1.5,
// 2,793 / 3,708; 60M, 4, 9,449 / 17,529; inside: n = 1M, degree 1.33, 226 / 199; 2M, 1.5, 878 / 269; 4M, 4, 1,504 / 561;
// 8M, 1.5, 1,183 / 763; 8M, 10, 3,026 / 1,390; 16M, 1.5, 1,236 / 1,440; 16M, 10, 4,535 / 2,735).
constexpr int64_t kCcRoundEdges = 500000;
constexpr int32_t kCcRoundRows = 12000000;
__global__ void __launch_bounds__(kCcRoundThreads, 2)
    k_cc_rounds(int32_t n, const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, long long m,
                int32_t *parent, int32_t *err, CcCtl *ctl) {
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  uint32_t target = 0;
  auto barrier = [&]() -> bool {
    if (grid_barrier(&ctl->bar, target)) return true;
    if (threadIdx.x == 0) atomicExch(err, kCcLost);
    return false;
  };
  for (long long v = t0; v < n; v += step) parent[v] = (int32_t)v;
  if (!barrier()) return;
  for (int round = 0;; ++round) {
    bool open = false;
    for (long long i = t0; i < m; i += step) {
      const int32_t a = rows[i], b = cols[i];
      if ((unsigned)a >= (unsigned)n || (unsigned)b >= (unsigned)n) {
        if (round == 0) atomicExch(err, DLP_ERR_DEVICE);
        continue;
      }
      const int32_t ra = __ldcg(parent + a), rb = __ldcg(parent + b);
      if (ra == rb) continue;
      open = true;
      const int32_t hi = max(ra, rb), lo = min(ra, rb);
      if (round < kCcRounds) {
        if (__ldcg(parent + hi) > lo) atomicMin(parent + hi, lo);  // most offers to a large root come too late
      } else {
        unite(parent, a, b, err);  // exact in one pass
      }
    }
    if (t0 == 0) ctl->open[(round + 1) & 1] = 0;
    if (__syncthreads_or(open) && threadIdx.x == 0) atomicExch(&ctl->open[round & 1], 1);
    if (!barrier()) return;
    if (__ldcg(&ctl->open[round & 1]) == 0) return;
    for (long long v = t0; v < n; v += step) {
      // climbed through the L1: a giant component's root is read by all its vertices, and from L2 every read
      // of it goes to the same place. Lines are as of this phase's start or newer (the barrier dropped older
      // ones), and an older parent is a valid ancestor; a climb that ends below the root leaves its edges
      // open, so another round follows.
      int32_t r = (int32_t)v, q = ld_l1(parent + r);
      for (int k = 0; q != r && k < kMaxSteps; ++k) {
        r = q;
        q = ld_l1(parent + r);
      }
      __stcg(parent + v, r);
    }
    if (!barrier()) return;
    if (round >= kCcRounds) return;
  }
}

// Graph form, in the sampling-then-skip order of Afforest (Sutton, Ben-Nun, Barak, IPDPS 2018):
//   1. kCcSample rounds: every vertex hooks its k-th live in-mask neighbour, then compress;
//   2. the most frequent root L among a fixed sample of vertices is taken as the big component;
//   3. the rows of every vertex outside L are hooked in full (both directions, so an edge whose
//      other end lies in L is still seen); rows of L are skipped, except for their sink entries
//      until L is joined to the sink.
// Any edge skipped in 3 has both ends in L, so the partition is the full one; and since every hook
// puts a larger root under a smaller one, each root is still its component's minimum vertex id.
constexpr int kCcSample = 2;
constexpr int kCcModeSample = 1024;

template <typename TW>
__device__ __forceinline__ bool live(const TW *w, int j) {
  return !w || cvt<float>(w[j]) != 0.0f;
}

// Sampling round k: every vertex of the mask hooks its k-th live in-mask neighbour (CSR order).
// One neighbour per round with a compression in between keeps every find one or two hops long.
template <typename TW>
__global__ void __launch_bounds__(kCcThreads)
    k_cc_sample(int32_t n, int k, const int32_t *__restrict__ rbeg, const int32_t *__restrict__ rend,
                const int32_t *__restrict__ col, const TW *__restrict__ w, const uint8_t *__restrict__ vmask,
                int32_t *parent, int32_t *err) {
  for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < n;
       u += (long long)gridDim.x * blockDim.x) {
    if (vmask && !vmask[u]) continue;
    const int end = rend[u];
    int seen = 0;
    for (int j = rbeg[u]; j < end; ++j) {
      if (!live(w, j)) continue;
      const int32_t v = col[j];
      if ((unsigned)v >= (unsigned)n) {
        if (err) atomicExch(err, DLP_ERR_DEVICE);
        continue;
      }
      if (vmask && !vmask[v]) continue;
      if (seen++ == k) {
        unite(parent, (int32_t)u, v, err);
        break;
      }
    }
  }
}

// One block: the most frequent root among kCcModeSample in-mask vertices spread over [0, n)
// (ties: the smaller root); -1 when no sampled vertex is in the mask. scratch[1] = 0 (L not yet
// joined to the sink).
__global__ void __launch_bounds__(kCcModeSample) k_cc_big(int32_t n, const uint8_t *__restrict__ vmask,
                                                          const int32_t *__restrict__ parent, int32_t *scratch) {
  __shared__ int32_t root[kCcModeSample];
  __shared__ unsigned long long best;
  const int k = threadIdx.x;
  const int S = n < kCcModeSample ? n : kCcModeSample;
  int32_t r = -1;
  if (k < S) {
    const int32_t i = (int32_t)(((long long)k * n) / S);
    if (!vmask || vmask[i]) r = parent[i];
  }
  root[k] = r;
  if (k == 0) best = 0ull;
  __syncthreads();
  if (r >= 0) {
    unsigned cnt = 0;
    for (int j = 0; j < S; ++j) cnt += root[j] == r;
    // larger count first, then smaller root
    const unsigned long long key = ((unsigned long long)cnt << 32) | (0xffffffffu - (unsigned)r);
    atomicMax(&best, key);
  }
  __syncthreads();
  if (k == 0) {
    scratch[0] = best ? (int32_t)(0xffffffffu - (unsigned)(best & 0xffffffffu)) : -1;
    scratch[1] = 0;
  }
}

// 8 lanes per row; sink vertex id = n. With scratch == NULL every row is hooked in full (entry
// (u, v) once, from the smaller end).
template <typename TW>
__global__ void __launch_bounds__(kCcThreads)
    k_cc_graph(int32_t n, const int32_t *__restrict__ rbeg, const int32_t *__restrict__ rend,
               const int32_t *__restrict__ col, const TW *__restrict__ w, const uint8_t *__restrict__ vmask,
               const uint8_t *__restrict__ sink, int32_t *parent, int32_t *err, int32_t *scratch) {
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const int32_t big = scratch ? scratch[0] : -1;
  volatile int32_t *grounded = scratch ? scratch + 1 : nullptr;
  for (long long t = t0; t < (long long)n * 8; t += stride) {
    const int32_t u = (int32_t)(t >> 3);
    const int l = (int)(t & 7);
    if (vmask && !vmask[u]) continue;
    const bool inL = big >= 0 && ((volatile int32_t *)parent)[u] == big;
    if (inL && (!sink || *grounded)) continue;
    const int beg = rbeg[u], end = rend[u];
    for (int j = beg + l; j < end; j += 8) {
      if (!live(w, j)) continue;
      const int32_t v = col[j];
      if ((unsigned)v >= (unsigned)n) {
        if (err) atomicExch(err, DLP_ERR_DEVICE);
        continue;
      }
      if (!vmask || vmask[v]) {
        // skipped rows (L) are covered from the other end; without a sample pass the mirror
        // entry (v, u) covers the pair once
        if (!inL && (scratch || u < v)) unite(parent, u, v, err);
      } else if (sink && sink[v]) {
        unite(parent, u, n, err);
        if (inL) *grounded = 1;
      }
    }
  }
}

__global__ void k_cc_compress(int32_t *parent_, int32_t n, int32_t *err) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  volatile int32_t *parent = parent_;
  int32_t x = parent[i];
  int steps = 0;
  while (true) {
    const int32_t p = parent[x];
    if (p == x) break;
    x = p;
    if (++steps > kMaxSteps) {
      if (err) atomicExch(err, DLP_ERR_DEVICE);
      break;
    }
  }
  parent[i] = x;
}

__global__ void k_cc_gather_rank(const int32_t *__restrict__ parent, int32_t n, int32_t *label) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t p = parent[i];
  if (p != (int32_t)i) label[i] = label[p];
}

// ------------------------------------------------------------------------------------------------
// Grounded set by reachability: the vertices of the mask whose component (live in-mask entries)
// holds an entry to a sink vertex outside the mask -- the set {u : parent[u] == parent[n]} of the
// graph form above, found by bottom-up sweeps instead of a full union-find: an unreached vertex of
// the mask joins as soon as one of its live entries leads to a sink vertex or to a reached vertex.
// Marks are read and written in place, so one sweep carries a mark along many hops; a sweep that
// marks nothing ends it (the reached set is then closed under adjacency, i.e. whole components).
// ------------------------------------------------------------------------------------------------
// The whole grounding in one cooperative launch: bottom-up sweeps until one reaches nothing new (at most
// kReachMaxSweeps), the union-find over the rows they left where they do not settle (long chains), and the
// membership update, with a grid barrier where a launch boundary or a host read was. A settled graph takes
// four sweeps; launch by launch, each batch of sweeps ended in a host read in the middle of the patch.
// Bound by the first sweep's row scans (n = 1M, degree 10: 183 us in all) and, below, by the sweeps' number
// and barriers (n = 3,000: 26 us, in place of four launches, two clears and a host read; 60,000: 33). One
// thread per row: 4 or 8 lanes a row, or several entries in flight, scan sooner than the marks spread in place
// and need more sweeps (60,000: 41 to 68 us; 250,000: 61 -> 67 to 134).
// info: [0] vertices of vmask or sink, [1] vertices of vmask left ungrounded, [2] sweeps run (negative:
// the union-find finished), [3] a barrier's wait ran out.
constexpr int kGroundThreads = 1024;
constexpr int kReachMaxSweeps = 32;  // then the union-find finishes the job
template <typename TW>
__global__ void __launch_bounds__(kGroundThreads, 2)
    k_ground_whole(int32_t n, const int32_t *__restrict__ rbeg, const int32_t *__restrict__ rend,
                   const int32_t *__restrict__ col, const TW *__restrict__ w, const uint8_t *__restrict__ vmask,
                   const uint8_t *__restrict__ sink, volatile uint8_t *reached, int32_t *flags, int32_t *parent,
                   uint8_t *umask, uint8_t *in_t, int32_t *count, int32_t *err, int32_t *info, GridBar *bar) {
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  const bool first = t0 == 0;
  uint32_t target = 0;
  auto barrier = [&]() -> bool {
    if (grid_barrier(bar, target)) return true;
    if (threadIdx.x == 0) atomicExch(info + 3, 1);
    return false;
  };
  int sweeps = 0;
  uint32_t walked;
  bool settled = false;
  while (!settled && sweeps < kReachMaxSweeps) {  // flags and reached were cleared before the launch
    bool any = false;
    walked = 0;
    for (long long u = t0; u < n; u += step) {
      if ((vmask && !vmask[u]) || reached[u]) continue;
      const int beg = rbeg[u], end = rend[u];
      bar_announce(bar, end - beg, walked);
      for (int j = beg; j < end; ++j) {
        if (!live(w, j)) continue;
        const int32_t v = col[j];
        if ((unsigned)v >= (unsigned)n) {
          if (err) atomicExch(err, DLP_ERR_DEVICE);
          continue;
        }
        const bool inm = !vmask || vmask[v];
        if (inm ? reached[v] != 0 : (sink && sink[v])) {
          reached[u] = 1;
          any = true;
          break;
        }
      }
    }
    if (__syncthreads_or(any) && threadIdx.x == 0) atomicAdd(flags + sweeps, 1);
    if (!barrier()) return;
    settled = __ldcg(flags + sweeps) == 0;
    ++sweeps;
  }
  // The union-find over what the sweeps left. Every vertex next to the sink was reached by the first sweep, so the sink
  // itself has no part in it: the reached vertices, all of one component, stand as one, r0, the smallest of them, and
  // only the rows of the others are walked, both directions of an edge (one alone leaves a path in order as one long
  // chain: n = 60,000 0.5 -> 4.6 ms). n = 1M, one labelled vertex, us, every row / these: a grid 1,500 / 1,210, in random
  // order 2,720 / 2,150; a path 1,190 / 880. (The smallest is kept as the largest n - v, of words cleared to zero.)
  int32_t *least = flags + kReachMaxSweeps;
  int32_t r0 = n;
  if (!settled) {
    int near = 0;
    for (long long v = t0; v < n; v += step) {
      parent[v] = (int32_t)v;
      if (reached[v]) near = max(near, (int)(n - v));
    }
    near = __reduce_max_sync(0xffffffffu, near);
    if ((threadIdx.x & 31) == 0 && near) atomicMax(least, near);
    if (!barrier()) return;
    r0 = n - __ldcg(least);
    walked = 0;
    for (long long u = t0; u < n; u += step) {
      if ((vmask && !vmask[u]) || reached[u]) continue;
      bar_announce(bar, rend[u] - rbeg[u], walked);
      for (int j = rbeg[u]; j < rend[u]; ++j) {
        if (!live(w, j)) continue;
        const int32_t v = col[j];
        if ((unsigned)v >= (unsigned)n || (vmask && !vmask[v])) continue;  // out of range: flagged by the sweeps
        unite(parent, (int32_t)u, reached[v] ? r0 : v, err);
      }
    }
    if (!barrier()) return;
  }
  // without a reached vertex there is no root to share (r0 is n)
  const int32_t root = settled || r0 >= n ? -1 : find_root(parent, r0, err);
  int changes = 0, active = 0, lost = 0;
  for (long long v = t0; v < n; v += step) {
    const bool m = !vmask || vmask[v];
    const bool nu = m && (reached[v] != 0 || (!settled && find_root(parent, (int32_t)v, err) == root));
    const bool ch = nu != (umask[v] != 0);
    umask[v] = nu ? 1 : 0;
    in_t[v] = ch ? 1 : 0;
    changes += ch;
    active += (m ? 1 : 0) + (sink && sink[v] ? 1 : 0);
    lost += m && !nu;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    changes += __shfl_xor_sync(0xffffffffu, changes, off);
    active += __shfl_xor_sync(0xffffffffu, active, off);
    lost += __shfl_xor_sync(0xffffffffu, lost, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (changes) atomicAdd(count, changes);
    if (active) atomicAdd(info, active);
    if (lost) atomicAdd(info + 1, lost);
  }
  if (first) info[2] = settled ? sweeps : -sweeps;
}

// ------------------------------------------------------------------------------------------------
// Felzenszwalb-Huttenlocher merging in Boruvka rounds (dynlp/cc.py:37-73) in one cooperative launch. A
// component is named by its smallest vertex (the order of the reference's ranks), so no round renumbers.
// A round: every component's lightest outgoing edge (ordered-float atomicMin), the smallest component on
// the other side among its ties, the merge test, the unions, then internal dissimilarity, size and
// grounding folded into the new roots and the vertices relabelled; six grid barriers. Bound by them (some
// 15 us a round); the tensor operations it replaces took 25 launches and three host reads a round (vertex
// arrivals, n = 20,000, 40 rounds in five batches: 25 ms of 45).
// ------------------------------------------------------------------------------------------------
struct FhCtl {
  GridBar bar;
  int32_t ext[2], ok[2];  // this round saw an outgoing edge / a permitted merge, by the round's parity
  int32_t bad;            // an edge's end outside [-m, m): nothing is merged
};

__device__ __forceinline__ uint32_t float_order(float x) {  // monotone in the float's order (x + 0: both zeros are equal)
  const uint32_t b = __float_as_uint(__fadd_rn(x, 0.f));
  return b & 0x80000000u ? ~b : b | 0x80000000u;
}

constexpr int kFhThreads = 512;
__global__ void __launch_bounds__(kFhThreads, 1)
    k_fh_components(int32_t m, long long E, const int32_t *__restrict__ rows, const int32_t *__restrict__ cols,
                    const float *__restrict__ d, float k, const float *__restrict__ ground, int32_t *parent,
                    int32_t *lab, float *internal, int32_t *size, int32_t *grounded, uint32_t *best, float *bestd,
                    int32_t *nb, int32_t *err, FhCtl *ctl) {
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  uint32_t target = 0;
  auto barrier = [&]() -> bool {
    if (grid_barrier(&ctl->bar, target)) return true;
    if (threadIdx.x == 0) atomicExch(err, DLP_ERR_DEVICE);
    return false;
  };
  for (long long v = t0; v < m; v += step) {
    parent[v] = lab[v] = (int32_t)v;
    internal[v] = 0.f;
    size[v] = 1;
    grounded[v] = ground && ground[v] != 0.f;
    best[v] = 0xffffffffu;
    nb[v] = m;
  }
  bool wrong = false;
  for (long long e = t0; e < E; e += step)
    wrong |= rows[e] < -m || rows[e] >= m || cols[e] < -m || cols[e] >= m;
  if (wrong) {
    atomicExch(err, DLP_ERR_INVALID);
    atomicExch(&ctl->bad, 1);
  }
  if (!barrier()) return;
  if (__ldcg(&ctl->bad)) return;
  // the component of an edge's end (a negative one counts from the last vertex, as an index does)
  auto component = [&](int32_t v) { return __ldcg(lab + (v < 0 ? v + m : v)); };
  bool fh = true;
  for (int round = 0;; ++round) {
    const int p = round & 1;
    // the lightest outgoing edge of every component (of the ungrounded ones once fh is over)
    bool any = false;
    for (long long e = t0; e < E; e += step) {
      const int32_t cu = component(rows[e]), cv = component(cols[e]);
      if (cu == cv || (!fh && __ldcg(grounded + cu))) continue;
      any = true;
      atomicMin(best + cu, float_order(d[e]));
    }
    if (__syncthreads_or(any) && threadIdx.x == 0) atomicExch(&ctl->ext[p], 1);
    if (t0 == 0) ctl->ext[p ^ 1] = ctl->ok[p ^ 1] = 0;
    if (!barrier()) return;
    if (__ldcg(&ctl->ext[p]) == 0) break;
    for (long long e = t0; e < E; e += step) {
      const int32_t cu = component(rows[e]), cv = component(cols[e]);
      if (cu == cv || (!fh && __ldcg(grounded + cu))) continue;
      if (float_order(d[e]) == __ldcg(best + cu)) {
        atomicMin(nb + cu, cv);
        __stcg(bestd + cu, d[e]);  // ties store the same value
      }
    }
    if (!barrier()) return;
    any = false;
    for (long long c = t0; c < m; c += step) {
      const int32_t t = __ldcg(nb + c);
      if (t >= m) continue;
      if (fh) {
        const float a = __fadd_rn(__ldcg(internal + c), __fmul_rn(__frcp_rn((float)__ldcg(size + c)), k));
        const float b = __fadd_rn(__ldcg(internal + t), __fmul_rn(__frcp_rn((float)__ldcg(size + t)), k));
        if (!(__ldcg(bestd + c) <= fminf(a, b))) {
          __stcg(nb + c, m);  // not permitted
          continue;
        }
      }
      any = true;
    }
    if (__syncthreads_or(any) && threadIdx.x == 0) atomicExch(&ctl->ok[p], 1);
    if (!barrier()) return;
    if (__ldcg(&ctl->ok[p]) == 0) {  // only under fh: a component with an outgoing edge always merges after
      if (!ground) break;
      fh = false;
      for (long long c = t0; c < m; c += step) {
        best[c] = 0xffffffffu;
        nb[c] = m;
      }
      if (!barrier()) return;
      continue;
    }
    for (long long c = t0; c < m; c += step) {
      const int32_t t = __ldcg(nb + c);
      if (t < m) unite(parent, (int32_t)c, t, err);
    }
    if (!barrier()) return;
    for (long long c = t0; c < m; c += step) {
      const int32_t v = __ldcg(lab + c);  // before this round's relabelling: c is a component if v == c
      if (v == (int32_t)c) {
        const int32_t r = find_root(parent, (int32_t)c, err);
        if (r != (int32_t)c) {
          atomicMax((int *)internal + r, __float_as_int(__ldcg(internal + c)));  // non-negative: ordered as ints
          atomicAdd(size + r, __ldcg(size + c));
          if (__ldcg(grounded + c)) atomicExch(grounded + r, 1);
        }
        if (__ldcg(nb + c) < m) {
          atomicMax((int *)internal + r, __float_as_int(fmaxf(__ldcg(bestd + c), 0.f)));
          __stcg(nb + c, m);
        }
        __stcg(best + c, 0xffffffffu);
      }
      __stcg(bestd + c, 0.f);
    }
    if (!barrier()) return;
    for (long long v = t0; v < m; v += step) __stcg(lab + v, find_root(parent, __ldcg(lab + v), err));
    if (!barrier()) return;
  }
}

// label[lpos[v]] = rank[parent[v]] for every masked v: the rank of its component's minimum id,
// written at the vertex's place among the masked vertices.
__global__ void k_cc_mask_gather(int32_t n, const int32_t *__restrict__ parent, const uint8_t *__restrict__ vmask,
                                 const int32_t *__restrict__ rank, const int32_t *__restrict__ lpos, int32_t *label) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n && vmask[v]) label[lpos[v]] = rank[parent[v]];
}

// ------------------------------------------------------------------------------------------------
// Components of a graph that changes by small batches between calls (warm start). The masked
// subgraph of the workloads is one giant component plus a few tiny ones, so instead of Afforest's
// sampling rounds the giant component is found by a breadth-first search from the root the previous
// call found for its most frequent component: top-down levels (8 lanes per frontier vertex,
// first-touch bits, warp-aggregated appends) while the frontier is small, then bottom-up sweeps over
// the bitmap. Every reached vertex is connected to the seed, so the reached set R is one connected
// set whatever the seed; its vertices start under R's minimum id, and the union-find then hooks the
// rows outside R in full (k_cc_graph with R as the skipped component). The result is the exact
// minimum-id labelling of dlp_cc_graph; a poor seed (a vertex cut off by the batch) only leaves more
// rows to the union-find. No host read: the schedule of levels is fixed and levels past the end of
// the search return at once.
// ------------------------------------------------------------------------------------------------
constexpr int kWarmDown = 7;  // top-down levels at most
constexpr int kWarmUp = 4;    // bottom-up sweeps at most
// control words: [0] seed, then R's root (k_cc_graph's skipped root), [1] sink flag of k_cc_graph
// (unused: no sink), [2] bottom-up switch, [3] minimum reached id, [4 + l] frontier size of level l
enum { kWSeed = 0, kWUp = 2, kWMin = 3, kWCnt = 4 };

__global__ void k_warm_seed(int32_t n, const uint8_t *__restrict__ vmask, uint32_t *bits, int32_t *front0,
                            int32_t *ctl) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int32_t sd = ctl[kWSeed];
  ctl[1] = 0;
  ctl[kWUp] = 0;
  ctl[kWMin] = 0x7fffffff;
  for (int l = 0; l <= kWarmDown; ++l) ctl[kWCnt + l] = 0;
  if (sd >= 0 && sd < n && (!vmask || vmask[sd])) {
    bits[sd >> 5] |= 1u << (sd & 31);
    front0[0] = sd;
    ctl[kWCnt] = 1;
  }
}

template <typename TW>
__global__ void __launch_bounds__(kCcThreads)
    k_bfs_down(int32_t n, const int32_t *__restrict__ rbeg, const int32_t *__restrict__ rend,
               const int32_t *__restrict__ col, const TW *__restrict__ w, const uint8_t *__restrict__ vmask,
               uint32_t *bits, const int32_t *__restrict__ front_in, int32_t *front_out, int32_t *ctl, int level,
               int cap) {
  constexpr int G = 8, kGroups = 32 / G;
  const int nf = ctl[kWCnt + level];
  if (nf == 0) return;
  if (nf > cap) {  // a large frontier: the bottom-up sweeps take over from the bitmap
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl[kWUp] = 1;
    return;
  }
  const int lane = lane_id(), gl = lane % G;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long stride = (((long long)gridDim.x * blockDim.x) >> 5) * kGroups;
  for (long long base = warp * kGroups; base < nf; base += stride) {  // warp-uniform bounds
    const long long g = base + lane / G;
    int beg = 0, end = 0;
    if (g < nf) {
      const int32_t u = front_in[g];
      beg = rbeg[u];
      end = rend[u];
    }
    const int trips = __reduce_max_sync(0xffffffffu, (end - beg + G - 1) / G);
    for (int t = 0; t < trips; ++t) {
      const int j = beg + gl + t * G;
      bool fresh = false;
      int32_t v = 0;
      if (j < end && live(w, j)) {
        v = col[j];
        if ((unsigned)v < (unsigned)n && (!vmask || vmask[v])) {
          const uint32_t bit = 1u << (v & 31);
          fresh = (atomicOr(bits + (v >> 5), bit) & bit) == 0u;
        }
      }
      warp_append(fresh, v, front_out, ctl + kWCnt + level + 1);
    }
  }
}

// Bottom-up sweep: an unreached vertex of the mask joins when one of its live in-mask entries
// leads to a reached vertex (bits read and written in place, so a sweep carries marks many hops).
template <typename TW>
__global__ void __launch_bounds__(kCcThreads)
    k_bfs_up(int32_t n, const int32_t *__restrict__ rbeg, const int32_t *__restrict__ rend,
             const int32_t *__restrict__ col, const TW *__restrict__ w, const uint8_t *__restrict__ vmask,
             uint32_t *bits_, const int32_t *ctl) {
  if (!ctl[kWUp] && !ctl[kWCnt + kWarmDown]) return;  // the top-down levels finished the search
  volatile uint32_t *bits = bits_;
  for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < n;
       u += (long long)gridDim.x * blockDim.x) {
    if (vmask && !vmask[u]) continue;
    const uint32_t ub = 1u << (u & 31);
    if (bits[u >> 5] & ub) continue;
    const int end = rend[u];
    for (int j = rbeg[u]; j < end; ++j) {
      if (!live(w, j)) continue;
      const int32_t v = col[j];
      if ((unsigned)v >= (unsigned)n || (vmask && !vmask[v])) continue;
      if (bits[v >> 5] & (1u << (v & 31))) {
        atomicOr(bits_ + (u >> 5), ub);
        break;
      }
    }
  }
}

// Smallest reached id: the first set bit of each word, then a minimum.
__global__ void k_warm_min(int32_t n, const uint32_t *__restrict__ bits, int32_t *ctl) {
  const long long wd = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int32_t m = 0x7fffffff;
  if (wd < ((long long)n + 31) / 32 && bits[wd]) m = (int32_t)(wd * 32 + __ffs(bits[wd]) - 1);
  m = __reduce_min_sync(0xffffffffu, m);
  if (lane_id() == 0 && m != 0x7fffffff) atomicMin(ctl + kWMin, m);
}

// parent[v] = R's minimum id for the reached vertices, v otherwise (parent[n] = n, the unused sink);
// control word 0 becomes R's root for k_cc_graph (-1 when nothing was reached).
__global__ void k_warm_parent(int32_t n, const uint32_t *__restrict__ bits, int32_t *parent, int32_t *ctl) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t m = ctl[kWMin];
  if (v < n) parent[v] = (bits[v >> 5] >> (v & 31)) & 1u ? m : (int32_t)v;
  else if (v == n) parent[v] = (int32_t)n;
  if (v == 0) ctl[kWSeed] = m == 0x7fffffff ? -1 : m;
}

static int grid_persist(long long work) {
  long long blocks = (work + kCcThreads - 1) / kCcThreads;
  const long long cap = (long long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  return (int)(blocks < 1 ? 1 : blocks);
}

}  // namespace dlp

using namespace dlp;

extern "C" {

int dlp_cc_edges(int32_t n, const int32_t *rows, const int32_t *cols, int64_t m, int32_t *parent, int32_t *err,
                 dlp_stream_t stream) {
  if (n < 0 || m < 0 || (n > 0 && !parent) || (m > 0 && (!rows || !cols))) return DLP_ERR_INVALID;
  if (n == 0) return DLP_OK;
  cudaStream_t s = (cudaStream_t)stream;
  k_cc_init<<<ceil_div_i(n, kCcThreads), kCcThreads, 0, s>>>(parent, n);
  if (m > 0) k_cc_edges<<<grid_persist(m), kCcThreads, 0, s>>>(n, rows, cols, m, parent, err);
  k_cc_compress<<<ceil_div_i(n, kCcThreads), kCcThreads, 0, s>>>(parent, n, err);
  return check_launch(m > 0 ? 3 : 2);
}

size_t dlp_cc_edges_workspace_bytes(void) { return 256; }

int dlp_cc_edges_ws(int32_t n, const int32_t *rows, const int32_t *cols, int64_t m, int32_t *parent, int32_t *err,
                    void *ws, size_t ws_bytes, dlp_stream_t stream) {
  if (!ws || ws_bytes < dlp_cc_edges_workspace_bytes() || !err) return DLP_ERR_WORKSPACE;
  if (n <= 0 || n > kCcRoundRows || m < kCcRoundEdges || 8 * m <= 5 * (int64_t)n) return dlp_cc_edges(n, rows, cols, m, parent, err, stream);
  if (!parent || !rows || !cols) return DLP_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  CcCtl *ctl = (CcCtl *)ws;
  DLP_CUDA(cudaMemsetAsync(ctl, 0, sizeof(CcCtl), s));
  static const int per = [] {
    int k = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_cc_rounds, kCcRoundThreads, 0) != cudaSuccess)
      (void)cudaGetLastError();
    return k;
  }();
  if (per < 1) return DLP_ERR_CUDA;
  long long mm = m;
  void *args[] = {(void *)&n, (void *)&rows, (void *)&cols, (void *)&mm, (void *)&parent, (void *)&err, (void *)&ctl};
  const int grid = (int)std::min((long long)sm_count() * per, (std::max((long long)n, mm) + kCcRoundThreads - 1) / kCcRoundThreads);
  return launch_any_grid((const void *)k_cc_rounds, grid, kCcRoundThreads, args, 0, s);
}

size_t dlp_cc_graph_workspace_bytes(void) { return 256; }

int dlp_cc_graph(int32_t n, const int32_t *rbeg, const int32_t *rend, const int32_t *col, const void *w,
                 int w_dtype, const uint8_t *vmask, const uint8_t *sink, int32_t *parent, int32_t *err, void *ws,
                 size_t ws_bytes, dlp_stream_t stream) {
  if (n < 0 || !parent) return DLP_ERR_INVALID;
  if (ws && ws_bytes < dlp_cc_graph_workspace_bytes()) return DLP_ERR_WORKSPACE;
  if (n > 0 && (!rbeg || !rend || !col)) return DLP_ERR_INVALID;
  if (w && w_dtype != DLP_F32 && w_dtype != DLP_F64 && w_dtype != DLP_BF16) return DLP_ERR_DTYPE;
  cudaStream_t s = (cudaStream_t)stream;
  int32_t *scratch = (int32_t *)ws;
  int launches = 2;
  k_cc_init<<<ceil_div_i((long long)n + 1, kCcThreads), kCcThreads, 0, s>>>(parent, n + 1);
  if (n > 0) {
    const int grid = grid_persist((long long)n * 8);
    const int grid1 = grid_persist(n);
#define DLP_CC_PASSES(TW)                                                                                      \
  if (scratch) {                                                                                               \
    for (int k = 0; k < kCcSample; ++k) {                                                                     \
      k_cc_sample<TW><<<grid1, kCcThreads, 0, s>>>(n, k, rbeg, rend, col, (const TW *)w, vmask, parent, err);   \
      k_cc_compress<<<ceil_div_i(n, kCcThreads), kCcThreads, 0, s>>>(parent, n, err);                         \
    }                                                                                                          \
    k_cc_big<<<1, kCcModeSample, 0, s>>>(n, vmask, parent, scratch);                                           \
    launches += 2 * kCcSample + 1;                                                                             \
  }                                                                                                            \
  k_cc_graph<TW><<<grid, kCcThreads, 0, s>>>(n, rbeg, rend, col, (const TW *)w, vmask, sink, parent, err, scratch); \
  launches += 1;
    if (!w || w_dtype == DLP_F32) {
      DLP_CC_PASSES(float)
    } else if (w_dtype == DLP_F64) {
      DLP_CC_PASSES(double)
    } else {
      DLP_CC_PASSES(bf16)
    }
#undef DLP_CC_PASSES
  }
  k_cc_compress<<<ceil_div_i((long long)n + 1, kCcThreads), kCcThreads, 0, s>>>(parent, n + 1, err);
  return check_launch(launches);
}

static size_t warm_ws_layout(int32_t n, size_t *off_bits, size_t *off_f0, size_t *off_f1) {
  const size_t nn = (size_t)(n > 0 ? n : 1);
  size_t b = 256;  // control words
  *off_bits = b;
  b += ((nn + 31) / 32 * 4 + 255) / 256 * 256;
  *off_f0 = b;
  b += (nn * 4 + 255) / 256 * 256;
  *off_f1 = b;
  return b + (nn * 4 + 255) / 256 * 256;
}


static size_t reach_ws_layout(int32_t n, size_t *off_flags, size_t *off_parent, size_t *off_cc) {
  size_t b = ((size_t)n + 255) / 256 * 256;  // reached
  *off_flags = b;
  b += 256;                                  // one flag per sweep (kReachMaxSweeps ints)
  *off_parent = b;
  b += ((size_t)n + 1 + 63) / 64 * 256;      // parent of the fallback (n + 1 ints)
  *off_cc = b;
  return b + 256;                            // dlp_ground_reach's info words
}

size_t dlp_cc_graph_warm_workspace_bytes(int32_t n) {
  size_t a, b, c;
  return warm_ws_layout(n, &a, &b, &c);
}

int dlp_cc_graph_warm(int32_t n, const int32_t *rbeg, const int32_t *rend, const int32_t *col, const void *w,
                      int w_dtype, const uint8_t *vmask, int32_t *parent, int32_t *err, void *ws, size_t ws_bytes,
                      dlp_stream_t stream) {
  if (n < 0 || !parent) return DLP_ERR_INVALID;
  if (n > 0 && (!rbeg || !rend || !col)) return DLP_ERR_INVALID;
  if (w && w_dtype != DLP_F32 && w_dtype != DLP_F64 && w_dtype != DLP_BF16) return DLP_ERR_DTYPE;
  size_t off_bits, off_f0, off_f1;
  if (!ws || ws_bytes < warm_ws_layout(n, &off_bits, &off_f0, &off_f1)) return DLP_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    k_cc_init<<<1, kCcThreads, 0, s>>>(parent, 1);
    return check_launch();
  }
  char *base = (char *)ws;
  int32_t *ctl = (int32_t *)base;
  uint32_t *bits = (uint32_t *)(base + off_bits);
  int32_t *front[2] = {(int32_t *)(base + off_f0), (int32_t *)(base + off_f1)};
  DLP_CUDA(cudaMemsetAsync(bits, 0, ((size_t)n + 31) / 32 * 4, s));
  k_warm_seed<<<1, 32, 0, s>>>(n, vmask, bits, front[0], ctl);
  const int cap = std::max(n / 16, 1024);
  const int grid = grid_persist((long long)n * 8);
  const int grid1 = grid_persist(n);
#define DLP_WARM_PASSES(TW)                                                                                       \
  for (int l = 0; l < kWarmDown; ++l)                                                                            \
    k_bfs_down<TW><<<grid, kCcThreads, 0, s>>>(n, rbeg, rend, col, (const TW *)w, vmask, bits, front[l & 1],      \
                                               front[(l + 1) & 1], ctl, l, cap);                                  \
  for (int u = 0; u < kWarmUp; ++u)                                                                              \
    k_bfs_up<TW><<<grid1, kCcThreads, 0, s>>>(n, rbeg, rend, col, (const TW *)w, vmask, bits, ctl);               \
  k_warm_min<<<ceil_div_i(((long long)n + 31) / 32, kCcThreads), kCcThreads, 0, s>>>(n, bits, ctl);              \
  k_warm_parent<<<ceil_div_i((long long)n + 1, kCcThreads), kCcThreads, 0, s>>>(n, bits, parent, ctl);           \
  k_cc_graph<TW><<<grid, kCcThreads, 0, s>>>(n, rbeg, rend, col, (const TW *)w, vmask, nullptr, parent, err, ctl);
  if (!w || w_dtype == DLP_F32) {
    DLP_WARM_PASSES(float)
  } else if (w_dtype == DLP_F64) {
    DLP_WARM_PASSES(double)
  } else {
    DLP_WARM_PASSES(bf16)
  }
#undef DLP_WARM_PASSES
  k_cc_compress<<<ceil_div_i((long long)n + 1, kCcThreads), kCcThreads, 0, s>>>(parent, n + 1, err);
  k_cc_big<<<1, kCcModeSample, 0, s>>>(n, vmask, parent, ctl);  // the next call's seed
  return check_launch(kWarmDown + kWarmUp + 6);
}

size_t dlp_ground_reach_workspace_bytes(int32_t n) {
  size_t a, b, c;
  return reach_ws_layout(n < 0 ? 0 : n, &a, &b, &c);
}

int dlp_ground_reach_async(int32_t n, const int32_t *rbeg, const int32_t *rend, const int32_t *col, const void *w,
                           int w_dtype, const uint8_t *vmask, const uint8_t *sink, uint8_t *umask, uint8_t *in_t,
                           int32_t *count, int32_t *err, int32_t *info, void *ws, size_t ws_bytes,
                           dlp_stream_t stream) {
  if (n < 0 || !info || (n > 0 && (!rbeg || !rend || !col || !umask || !in_t || !count))) return DLP_ERR_INVALID;
  if (w && w_dtype != DLP_F32 && w_dtype != DLP_F64 && w_dtype != DLP_BF16) return DLP_ERR_DTYPE;
  size_t off_flags, off_parent, off_cc;
  if (!ws || ws_bytes < reach_ws_layout(n, &off_flags, &off_parent, &off_cc)) return DLP_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  DLP_CUDA(cudaMemsetAsync(info, 0, 4 * sizeof(int32_t), s));
  if (n == 0) return DLP_OK;
  char *base = (char *)ws;
  uint8_t *reached = (uint8_t *)base;
  int32_t *flags = (int32_t *)(base + off_flags);
  int32_t *parent = (int32_t *)(base + off_parent);
  GridBar *bar = (GridBar *)(flags + kReachMaxSweeps + 1);  // in the flags' 256 bytes, after r0's word
  static_assert((kReachMaxSweeps + 1) * sizeof(int32_t) + sizeof(GridBar) <= 256, "flags and barrier share a line of 256 bytes");
  DLP_CUDA(cudaMemsetAsync(reached, 0, off_flags + 256, s));  // reached, the flags and the barrier
  auto launch = [&](auto kern, auto *wp) -> int {
    static const int per = [&] {
      int k = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, kern, kGroundThreads, 0) != cudaSuccess) (void)cudaGetLastError();
      return k;
    }();
    if (per < 1) return DLP_ERR_CUDA;
    const int grid = std::max(1, std::min(ceil_div_i(n, kGroundThreads), sm_count() * per));
    void *args[] = {(void *)&n,     (void *)&rbeg,  (void *)&rend,   (void *)&col,   (void *)&wp,   (void *)&vmask,
                    (void *)&sink,  (void *)&reached, (void *)&flags, (void *)&parent, (void *)&umask, (void *)&in_t,
                    (void *)&count, (void *)&err,   (void *)&info,   (void *)&bar};
    return launch_any_grid((const void *)kern, grid, kGroundThreads, args, 0, s);
  };
  if (!w || w_dtype == DLP_F32) return launch(k_ground_whole<float>, (const float *)w);
  if (w_dtype == DLP_F64) return launch(k_ground_whole<double>, (const double *)w);
  return launch(k_ground_whole<bf16>, (const bf16 *)w);
}

int dlp_ground_reach(int32_t n, const int32_t *rbeg, const int32_t *rend, const int32_t *col, const void *w,
                     int w_dtype, const uint8_t *vmask, const uint8_t *sink, uint8_t *umask, uint8_t *in_t,
                     int32_t *count, int32_t *err, int32_t *sweeps_out, void *ws, size_t ws_bytes,
                     dlp_stream_t stream) {
  if (sweeps_out) *sweeps_out = 0;
  size_t off_flags, off_parent, off_cc;
  if (n >= 0 && (!ws || ws_bytes < reach_ws_layout(n, &off_flags, &off_parent, &off_cc))) return DLP_ERR_WORKSPACE;
  int32_t *info = n >= 0 ? (int32_t *)((char *)ws + off_cc) : nullptr;
  DLP_TRY(dlp_ground_reach_async(n, rbeg, rend, col, w, w_dtype, vmask, sink, umask, in_t, count, err, info, ws,
                                 ws_bytes, stream));
  int32_t h[4] = {0, 0, 0, 0};
  DLP_CUDA(cudaMemcpyAsync(h, info, sizeof(h), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  DLP_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
  if (sweeps_out) *sweeps_out = h[2];
  return h[3] ? DLP_ERR_DEVICE : DLP_OK;
}

static size_t fh_vec(int32_t m) { return ((size_t)(m > 0 ? m : 1) * 4 + 255) / 256 * 256; }

size_t dlp_fh_components_workspace_bytes(int32_t m) { return 7 * fh_vec(m) + 256; }

int dlp_fh_components(int32_t m, int64_t E, const int32_t *rows, const int32_t *cols, const float *d, double k,
                      const float *ground, int32_t *root, int32_t *err, void *ws, size_t ws_bytes, dlp_stream_t stream) {
  if (m < 0 || E < 0 || (m > 0 && !root) || (E > 0 && (!rows || !cols || !d)) || !err) return DLP_ERR_INVALID;
  if (!ws || ws_bytes < dlp_fh_components_workspace_bytes(m)) return DLP_ERR_WORKSPACE;
  if (m == 0) return DLP_OK;
  cudaStream_t s = (cudaStream_t)stream;
  char *p = (char *)ws;
  auto take = [&]() {
    char *q = p;
    p += fh_vec(m);
    return q;
  };
  int32_t *lab = (int32_t *)take();
  float *internal = (float *)take();
  int32_t *size = (int32_t *)take(), *grounded = (int32_t *)take();
  uint32_t *best = (uint32_t *)take();
  float *bestd = (float *)take();
  int32_t *nb = (int32_t *)take();
  FhCtl *ctl = (FhCtl *)p;
  DLP_CUDA(cudaMemsetAsync(ctl, 0, sizeof(FhCtl), s));
  long long EE = E;
  float kf = (float)k;
  void *args[] = {(void *)&m,        (void *)&EE,   (void *)&rows,     (void *)&cols, (void *)&d,     (void *)&kf,
                  (void *)&ground,   (void *)&root, (void *)&lab,      (void *)&internal, (void *)&size,
                  (void *)&grounded, (void *)&best, (void *)&bestd,    (void *)&nb,   (void *)&err,   (void *)&ctl};
  const int grid = (int)std::max(1LL, std::min((long long)sm_count(), (std::max((long long)m, EE) + kFhThreads - 1) / kFhThreads));
  DLP_TRY(launch_any_grid((const void *)k_fh_components, grid, kFhThreads, args, 0, s));
  // root[v] is the parent after the last unions: relabelled to the component's smallest vertex
  DLP_CUDA(cudaMemcpyAsync(root, lab, sizeof(int32_t) * (size_t)m, cudaMemcpyDeviceToDevice, s));
  return DLP_OK;
}

size_t dlp_cc_mask_labels_workspace_bytes(int32_t n) {
  const size_t v = ((size_t)(n > 0 ? n : 1) * sizeof(int32_t) + 255) / 256 * 256;
  return 2 * v + compact_ws_bytes(n);
}

int dlp_cc_mask_labels(int32_t n, const int32_t *parent, const uint8_t *vmask, int32_t *label, int32_t *n_comp,
                       int32_t *n_masked, void *ws, size_t ws_bytes, dlp_stream_t stream) {
  if (n < 0 || !n_comp || !n_masked || (n > 0 && (!parent || !vmask || !label))) return DLP_ERR_INVALID;
  if (!ws || ws_bytes < dlp_cc_mask_labels_workspace_bytes(n)) return DLP_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t v = ((size_t)(n > 0 ? n : 1) * sizeof(int32_t) + 255) / 256 * 256;
  int32_t *rank = (int32_t *)ws;
  int32_t *lpos = (int32_t *)((char *)ws + v);
  void *cws = (char *)ws + 2 * v;
  const size_t cbytes = ws_bytes - 2 * v;
  DLP_TRY(compact_masked_roots(parent, vmask, n, rank, n_comp, cws, cbytes, s));
  DLP_TRY(compact_positions(vmask, n, lpos, n_masked, cws, cbytes, s));
  if (n > 0) k_cc_mask_gather<<<ceil_div_i(n, kCcThreads), kCcThreads, 0, s>>>(n, parent, vmask, rank, lpos, label);
  return check_launch(n > 0 ? 1 : 0);
}

int dlp_cc_relabel(int32_t n, const int32_t *parent, int32_t *label, int32_t *n_comp, void *ws, size_t ws_bytes,
                   dlp_stream_t stream) {
  if (n < 0 || (n > 0 && (!parent || !label)) || !n_comp) return DLP_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  // label[root] = rank of the root among roots; then every vertex copies its root's rank.
  DLP_TRY(compact_roots(parent, n, label, n_comp, ws, ws_bytes, s));
  if (n > 0) k_cc_gather_rank<<<ceil_div_i(n, kCcThreads), kCcThreads, 0, s>>>(parent, n, label);
  return check_launch(n > 0 ? 1 : 0);
}

}  // extern "C"
