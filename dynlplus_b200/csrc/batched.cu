// Many independent harmonic solves in one launch sequence: block PCG over a concatenated
// (block-diagonal) CSR where every instance keeps its own CG scalars and stop state, so each
// instance follows the iterates it would follow alone.
//
// Rows are cut into tiles that never straddle two instances. Every kernel walks the tile list;
// reductions go tile -> instance in a fixed order (tile partials, then the instance's tiles), so an
// instance's sums do not depend on what else is in the batch. Instances stop independently
// (relative residual and/or the reference's violation rule, a true-residual recheck, patience,
// iteration cap) and stopped instances are skipped by the next iterations. Per iteration four launches: apply
// (SpMM + pAp), update (alpha from the instance's tiles, R, rz, norms), instance reduce (beta, stop),
// direction (Z, P); a fifth for alpha where an instance may have many tiles. The host queues check_every iterations between reads: the launches cost less than
// the kernels take, and a graph of them had to be captured again for every new batch (a millisecond each).
#include <algorithm>

#include "gather.cuh"

namespace dlp {

struct BCtl {
  int32_t *done, *iters, *stall, *stopped, *sel;  // per instance
  double *best, *viol, *relres;                    // per instance
  double *alpha, *beta, *rz, *eps, *epsinv, *rhsn;  // per instance x C
  double *tp1, *tp2, *tpv;                          // tile partials
  int32_t *counts;                                  // [running, proposed]
};

struct BTiles {
  const int32_t *tinst, *tbeg, *tend;  // per tile
  const int32_t *toff;                 // tiles of instance i: [toff[i], toff[i+1])
  int32_t ntiles, ninst;
};

struct BParams {
  int32_t mode, patience, max_iter;
  double target;
};

static size_t a256(size_t x) { return (x + 255) / 256 * 256; }

static size_t bctl_bytes(int32_t B, int32_t T, int32_t C) {
  return 5 * a256(4 * (size_t)B) + 3 * a256(8 * (size_t)B) + 6 * a256(8 * (size_t)B * C) + a256(8 * (size_t)T * C) +
         a256(16 * (size_t)T * C) + a256(8 * (size_t)T) + a256(8);
}

static BCtl carve_b(void *ws, int32_t B, int32_t T, int32_t C) {
  char *p = (char *)ws;
  BCtl c;
  int32_t **ip[5] = {&c.done, &c.iters, &c.stall, &c.stopped, &c.sel};
  for (auto q : ip) {
    *q = (int32_t *)p;
    p += a256(4 * (size_t)B);
  }
  double **dp[3] = {&c.best, &c.viol, &c.relres};
  for (auto q : dp) {
    *q = (double *)p;
    p += a256(8 * (size_t)B);
  }
  double **cp[6] = {&c.alpha, &c.beta, &c.rz, &c.eps, &c.epsinv, &c.rhsn};
  for (auto q : cp) {
    *q = (double *)p;
    p += a256(8 * (size_t)B * C);
  }
  c.tp1 = (double *)p;
  p += a256(8 * (size_t)T * C);
  c.tp2 = (double *)p;
  p += a256(16 * (size_t)T * C);
  c.tpv = (double *)p;
  p += a256(8 * (size_t)T);
  c.counts = (int32_t *)p;
  return c;
}

// whether phase ph works on an instance: 0 running ones, 1 proposed stops, 2 and 3 all (the start)
__device__ __forceinline__ bool b_on(int ph, int done) { return ph >= 2 || done == ph; }

__global__ void k_b_count(int32_t B, BCtl c) {
  __shared__ int s_run, s_prop;
  if (threadIdx.x == 0) s_run = s_prop = 0;
  __syncthreads();
  int run = 0, prop = 0;
  for (int i = threadIdx.x; i < B; i += blockDim.x) {
    const int d = c.done[i];
    run += d == 0;
    prop += d == 1;
  }
  if (run) atomicAdd(&s_run, run);
  if (prop) atomicAdd(&s_prop, prop);
  __syncthreads();
  if (threadIdx.x == 0) {
    c.counts[0] = s_run;
    c.counts[1] = s_prop;
  }
}

__global__ void k_b_init(int32_t B, int32_t C, const double *__restrict__ eps, const double *__restrict__ rhsn, BCtl c) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B) c.done[i] = c.iters[i] = c.stall[i] = c.stopped[i] = c.sel[i] = 0;
  if (i < (long long)B * C) {
    c.rz[i] = 0.0;
    c.eps[i] = eps[i];
    c.epsinv[i] = 1.0 / eps[i];
    c.rhsn[i] = rhsn[i];
  }
}

template <class T>
struct BApply {
  const int32_t *indptr, *col;
  const typename T::TW *w;
  int32_t C;
  const typename T::TX *P;
  int64_t ldp;
  const typename T::TV *diag;
  typename T::TY *AP;
  int64_t ldap;
  BTiles tl;
  BCtl c;
  int G, LV, NV;
};

// ROW as in gather_row: fp64 rows of 9-10 values (three loads), fp32 rows of 8 (one) or 12 (two) held whole by one
// lane; the own row then comes and AP goes whole too (its rows padded alike, checked by the launcher).
// Measured on B200 (16 systems, 200,000 rows, 3.2M entries, 9 fp64 columns): 91 -> 62 us.
template <class T, int VW, int VPL, int ROW = kRowVec>
__global__ void __launch_bounds__(kThreads) k_b_apply(BApply<T> p) {
  using TA = typename T::TA;
  __shared__ double sm[kThreads / 32][64];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int G = p.G, LV = p.LV, NV = p.NV;
  const int gl = lane & (G - 1);
  const int cl = gl & (LV - 1);
  const int es = gl / LV;
  const int ES = G / LV;
  const int rpb = kThreads / G;  // rows per block pass
  for (int t = blockIdx.x; t < p.tl.ntiles; t += gridDim.x) {
    const int inst = p.tl.tinst[t];
    if (p.c.done[inst] != 0) continue;  // uniform over the block
    double dot[VPL][VW];
#pragma unroll
    for (int k = 0; k < VPL; ++k)
#pragma unroll
      for (int i = 0; i < VW; ++i) dot[k][i] = 0.0;
    const int tb = p.tl.tbeg[t], te = p.tl.tend[t];
    for (int r0 = tb; r0 < te; r0 += rpb) {
      const int r = r0 + (int)(threadIdx.x / G);
      const bool valid = r < te;
      const int beg = valid ? p.indptr[r] : 0, end = valid ? p.indptr[r + 1] : 0;
      TA acc[VPL][VW];
      gather_row<typename T::TW, typename T::TX, TA, VW, VPL,
                 (ROW == kRow12F ? 2 : ROW == kRowVec ? gather_batch_wide<TA, VW, VPL>() : 4), ROW>(
          p.col, p.w, p.P, p.ldp, beg, end, es, ES, cl, LV, NV, G, acc);
      if (valid && es == 0) {
        const TA d = cvt<TA>(p.diag[r]);
        if constexpr (ROW == kRow10D) {
          double raw[5][2], ap[10];
          const bool hi = load_row10d((const double *)p.P + (long long)r * p.ldp, raw);
#pragma unroll
          for (int c = 0; c < 10; ++c) {
            const double pv = row10_col(raw, hi, c);
            ap[c] = d * pv - acc[c / 2][c % 2];
            if (c < p.C) dot[c / 2][c % 2] += pv * ap[c];
          }
          store_row10d<true>((double *)p.AP + (long long)r * p.ldap, ap);
        } else if constexpr (ROW == kRow8F || ROW == kRow12F) {
          float raw[VPL][4], ap[VPL][4];
          bool hi = false;
          if constexpr (ROW == kRow8F) load_row8((const float *)p.P + (long long)r * p.ldp, raw);
          else hi = load_row12((const float *)p.P + (long long)r * p.ldp, raw);
#pragma unroll
          for (int c = 0; c < 4 * VPL; ++c) {
            float pv;
            if constexpr (ROW == kRow8F) pv = raw[c / 4][c % 4];
            else pv = row12_col(raw, hi, c);
            const float x = d * pv - acc[c / 4][c % 4];
            ap[c / 4][c % 4] = x;
            if (c < p.C) dot[c / 4][c % 4] += (double)pv * (double)x;
          }
          if constexpr (ROW == kRow8F) store_row8((float *)p.AP + (long long)r * p.ldap, ap);
          else store_row12((float *)p.AP + (long long)r * p.ldap, ap);
        } else {
#pragma unroll
          for (int k = 0; k < VPL; ++k) {
            const int vi = cl + k * LV;
            if (vi < NV) {
#pragma unroll
              for (int i = 0; i < VW; ++i) {
                const int cc = vi * VW + i;
                if (cc < p.C) {
                  const TA pv = cvt<TA>(p.P[(long long)r * p.ldp + cc]);
                  const TA ap = d * pv - acc[k][i];
                  p.AP[(long long)r * p.ldap + cc] = cvt<typename T::TY>(ap);
                  dot[k][i] += (double)pv * (double)ap;
                }
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < VPL; ++k)
#pragma unroll
      for (int i = 0; i < VW; ++i)
        for (int off = LV; off < 32; off <<= 1) dot[k][i] += __shfl_xor_sync(0xffffffffu, dot[k][i], off);
    if (lane < LV) {
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int vi = lane + k * LV;
        if (vi < NV) {
#pragma unroll
          for (int i = 0; i < VW; ++i) {
            const int cc = vi * VW + i;
            if (cc < p.C) sm[wid][cc] = dot[k][i];
          }
        }
      }
    }
    __syncthreads();
    for (int cc = threadIdx.x; cc < p.C; cc += blockDim.x) {
      double s = 0.0;
      for (int w = 0; w < kThreads / 32; ++w) s += sm[w][cc];
      p.c.tp1[(long long)t * p.C + cc] = s;
    }
    __syncthreads();
  }
}

// R = rhs - (diag Z - W Z) on the rows of the phase's instances, accumulated in fp64 for fp32 rows too
template <class T, int VW, int VPL>
__global__ void __launch_bounds__(kThreads)
    k_b_residual(int phase, BApply<T> p, const typename T::TX *__restrict__ rhs, int64_t ldrhs) {
  using TA = typename T::TA;
  const int lane = threadIdx.x & 31;
  const int G = p.G, LV = p.LV, NV = p.NV;
  const int gl = lane & (G - 1), cl = gl & (LV - 1), es = gl / LV, ES = G / LV;
  const int rpb = kThreads / G;
  for (int t = blockIdx.x; t < p.tl.ntiles; t += gridDim.x) {
    if (!b_on(phase, p.c.done[p.tl.tinst[t]])) continue;
    const int te = p.tl.tend[t];
    for (int r0 = p.tl.tbeg[t]; r0 < te; r0 += rpb) {
      const int r = r0 + (int)(threadIdx.x / G);
      const bool valid = r < te;
      const int beg = valid ? p.indptr[r] : 0, end = valid ? p.indptr[r + 1] : 0;
      TA acc[VPL][VW];
      gather_row<typename T::TW, typename T::TX, TA, VW, VPL>(p.col, p.w, p.P, p.ldp, beg, end, es, ES, cl, LV, NV, G,
                                                                acc);
      if (valid && es == 0) {
        const TA d = cvt<TA>(p.diag[r]);
#pragma unroll
        for (int k = 0; k < VPL; ++k) {
          const int vi = cl + k * LV;
          if (vi < NV) {
#pragma unroll
            for (int i = 0; i < VW; ++i) {
              const int cc = vi * VW + i;
              if (cc < p.C)
                p.AP[(long long)r * p.ldap + cc] = (typename T::TY)(
                    cvt<TA>(rhs[(long long)r * ldrhs + cc]) - d * cvt<TA>(p.P[(long long)r * p.ldp + cc]) + acc[k][i]);
            }
          }
        }
      }
    }
  }
}

// Element sweeps of a tile: thread t owns column t mod C of rows t / C, t / C + 256 / C, ... of the tile, four rows
// in flight, so its sums are scalars and consecutive threads touch consecutive elements.
constexpr int kBThreads = 256;
constexpr int kBUnroll = 4;

// pAp over an instance's tiles (a fixed order) and its alpha, for one column, by a warp
__device__ __forceinline__ double b_fold_alpha(const BCtl &c, int t0, int nt, int C, int x, double rz) {
  const double s = warp_strided_reduce(c.tp1 + (long long)t0 * C + x, C, nt, false);
  const double al = s > 0.0 ? rz / s : 0.0;
  return isfinite(al) && fabs(al) < 1e30 ? al : 0.0;
}

// Up to kBFoldTiles tiles every block of an instance folds its tiles' pAp for itself, which spares a launch; beyond,
// where those reads grow with the tiles squared, a block per instance does it once (one system, fp32, a solve in us,
// folded by all / once: 5 columns, 957 tiles 2,901 / 2,960, 1,914: 5,309 / 5,304, 7,654: 33,179 / 31,183; 9 columns
// 4,853 / 4,908, 10,027 / 9,850, 52,857 / 46,829).
constexpr int kBFoldTiles = 1024;
__global__ void k_b_alpha(int32_t C, BTiles tl, BCtl c) {
  const int inst = blockIdx.x, t0 = tl.toff[inst], nt = tl.toff[inst + 1] - t0;
  if (nt <= kBFoldTiles || !b_on(0, c.done[inst])) return;
  for (int x = threadIdx.x >> 5; x < C; x += blockDim.x >> 5) {
    const double al = b_fold_alpha(c, t0, nt, C, x, c.rz[(long long)inst * C + x]);
    if (lane_id() == 0) c.alpha[(long long)inst * C + x] = al;
  }
}

// Phase 0: alpha of the tile's instance from its tiles' pAp (every block of the instance folds them in the same
// order, or k_b_alpha has; its first tile's block keeps it, and whether the instance is in this iteration, for the
// direction sweep), R -= alpha AP; then, as phase 1 (a true residual after a proposed stop) and phase 2 (the start), the
// tile's sums of R^2 / diag and R^2 and the largest violation. Phase 3: as 2, R copied from AP (the
// right-hand side of a zero start). Measured with the direction sweep on the same systems: 57 -> 20 us.
template <typename TS>
__global__ void __launch_bounds__(kBThreads) k_b_update(int phase, int32_t C, TS *R, int64_t ldr,
                                                        const TS *__restrict__ AP, int64_t ldap,
                                                        const TS *__restrict__ diag, BTiles tl, BCtl c) {
  __shared__ double s_a[kBThreads], s_b[kBThreads], s_v[kBThreads / 32], s_al[64];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int RB = kBThreads / C, q = tid / C, cc = tid - q * C;
  const bool on = q < RB;
  for (int t = blockIdx.x; t < tl.ntiles; t += gridDim.x) {
    const int inst = tl.tinst[t], t0 = tl.toff[inst], nt = tl.toff[inst + 1] - t0;
    const bool act = b_on(phase, c.done[inst]);
    if (phase == 0 && t == t0 && tid == 0) c.sel[inst] = act;
    if (!act) continue;
    if (phase == 0) {
      for (int x = wid; x < C; x += kBThreads / 32) {
        const long long k = (long long)inst * C + x;
        const double al = nt > kBFoldTiles ? c.alpha[k] : b_fold_alpha(c, t0, nt, C, x, c.rz[k]);
        if (lane == 0) {
          s_al[x] = al;
          if (t == t0 && nt <= kBFoldTiles) c.alpha[k] = al;
        }
      }
      __syncthreads();
    }
    double rz = 0.0, ss = 0.0, vmax = 0.0;
    if (on) {
      const TS al = phase == 0 ? (TS)s_al[cc] : TS(0);
      const double ei = c.epsinv[(long long)inst * C + cc];
      const int te = tl.tend[t];
      for (int r = tl.tbeg[t] + q; r < te; r += kBUnroll * RB) {
        TS rv[kBUnroll], av[kBUnroll], dv[kBUnroll];
#pragma unroll
        for (int u = 0; u < kBUnroll; ++u) {
          const long long rr = r + u * RB;
          const bool ok = rr < te;
          rv[u] = ok && phase != 3 ? R[rr * ldr + cc] : TS(0);
          av[u] = ok && (phase == 0 || phase == 3) ? AP[rr * ldap + cc] : TS(0);
          dv[u] = ok ? diag[rr] : TS(1);
        }
#pragma unroll
        for (int u = 0; u < kBUnroll; ++u) {
          const long long rr = r + u * RB;
          if (rr >= te) continue;
          TS x = rv[u];
          if (phase == 0) x = x - al * av[u];
          if (phase == 3) x = av[u];
          if (phase == 0 || phase == 3) R[rr * ldr + cc] = x;
          const double r64 = (double)x, r2 = r64 * r64, dinv = __drcp_rn((double)dv[u]);
          rz += r2 * dinv;
          ss += r2;
          vmax = fmax(vmax, isfinite(r64) ? fabs(r64) * dinv * ei : INFINITY);
        }
      }
    }
    s_a[tid] = rz;
    s_b[tid] = ss;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, off));
    if (lane == 0) s_v[wid] = vmax;
    __syncthreads();
    for (int x = wid; x < C; x += kBThreads / 32) {
      double a = 0.0, b = 0.0;
      for (int k = lane; k < RB; k += 32) {
        a += s_a[k * C + x];
        b += s_b[k * C + x];
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
      }
      if (lane == 0) {
        c.tp2[((long long)t * C + x) * 2 + 0] = a;
        c.tp2[((long long)t * C + x) * 2 + 1] = b;
      }
    }
    if (tid == 0) {
      double v = 0.0;
      for (int w = 0; w < kBThreads / 32; ++w) v = fmax(v, s_v[w]);
      c.tpv[t] = v;
    }
    __syncthreads();
  }
}

// one block per instance: beta, norms, stop decision
__global__ void k_b_beta(int phase, int32_t C, BTiles tl, BCtl c, BParams bp) {
  const int inst = blockIdx.x;
  if (threadIdx.x == 0) c.stopped[inst] = 0;
  if (!b_on(phase, c.done[inst])) return;
  const int t0 = tl.toff[inst], nt = tl.toff[inst + 1] - t0;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ double s_rel, s_v;
  if (threadIdx.x == 0) s_rel = 0.0;
  __syncthreads();
  for (int cc = wid; cc < C; cc += blockDim.x >> 5) {
    const double a = warp_strided_reduce(c.tp2 + ((long long)t0 * C + cc) * 2 + 0, (long long)C * 2, nt, false);
    const double b = warp_strided_reduce(c.tp2 + ((long long)t0 * C + cc) * 2 + 1, (long long)C * 2, nt, false);
    if (lane == 0) {
      const long long k = (long long)inst * C + cc;
      const double rzo = c.rz[k];
      const double be = (phase != 2 && rzo > 0.0) ? a / rzo : 0.0;
      c.beta[k] = isfinite(be) && fabs(be) < 1e30 ? be : 0.0;
      c.rz[k] = a;
      const double rel = c.rhsn[k] > 0.0 ? sqrt(b) / c.rhsn[k] : sqrt(b);
      atomicMax((unsigned long long *)&s_rel, __double_as_longlong(isfinite(rel) ? rel : INFINITY));
    }
  }
  if (wid == 0) {
    const double v = warp_strided_reduce(c.tpv + t0, 1, nt, true);
    if (lane == 0) s_v = v;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  const double v = s_v, rel = s_rel;
  c.viol[inst] = v;
  c.relres[inst] = rel;
  double m = 0.0;
  if (bp.mode & 1) m = fmax(m, v);
  if (bp.mode & 2) m = fmax(m, bp.target > 0.0 ? rel / bp.target : rel);
  const bool bad = !isfinite(m);
  const bool conv = m <= 1.0;
  int d = c.done[inst];
  if (phase == 0) c.iters[inst] += 1;
  if (bad) {
    d = 4;
  } else if (phase == 2) {
    c.best[inst] = m;
    c.stall[inst] = 0;
    d = conv ? 5 : 0;
  } else if (phase == 0 && conv) {
    d = 1;
  } else if (phase == 1 && conv) {
    d = 5;
  } else {
    if (m < 0.9 * c.best[inst]) {
      c.best[inst] = m;
      c.stall[inst] = 0;
    } else {
      c.stall[inst] += 1;
    }
    if (c.stall[inst] >= bp.patience) d = 2;
    else if (phase == 1) d = 0;
  }
  if (d == 0 && c.iters[inst] >= bp.max_iter) d = 3;
  if (phase == 0 && d != 0) c.stopped[inst] = 1;
  if (phase == 1 && d == 0) c.stopped[inst] = 2;  // resumed: direction from the true residual
  c.done[inst] = d;
}

// mode 0: Z += alpha P, P = R/diag + beta P (P only while running); mode 1: P update for resumed
// instances; mode 2: P = R/diag for all; mode 4: as 2, and Z = 0
template <typename TS>
__global__ void __launch_bounds__(kBThreads) k_b_dir(int mode, int32_t C, TS *Z, int64_t ldz, TS *P, int64_t ldp,
                                                     const TS *__restrict__ R, int64_t ldr,
                                                     const TS *__restrict__ diag, BTiles tl, BCtl c) {
  const int tid = threadIdx.x, RB = kBThreads / C, q = tid / C, cc = tid - q * C;
  if (q >= RB) return;
  for (int t = blockIdx.x; t < tl.ntiles; t += gridDim.x) {
    const int inst = tl.tinst[t];
    const bool act = mode == 0 ? c.sel[inst] != 0 : mode == 1 ? c.stopped[inst] == 2 : true;
    if (!act) continue;
    const bool upd = mode != 0 || c.done[inst] == 0, init = mode >= 2;
    const TS al = mode == 0 ? (TS)c.alpha[(long long)inst * C + cc] : TS(0);
    const TS be = init ? TS(0) : (TS)c.beta[(long long)inst * C + cc];
    const int te = tl.tend[t];
    for (int r = tl.tbeg[t] + q; r < te; r += kBUnroll * RB) {
      TS pv[kBUnroll], zv[kBUnroll], rv[kBUnroll], dv[kBUnroll];
#pragma unroll
      for (int u = 0; u < kBUnroll; ++u) {
        const long long rr = r + u * RB;
        const bool ok = rr < te;
        pv[u] = ok && !init ? P[rr * ldp + cc] : TS(0);
        zv[u] = ok && mode == 0 ? Z[rr * ldz + cc] : TS(0);
        rv[u] = ok && upd ? R[rr * ldr + cc] : TS(0);
        dv[u] = ok && upd ? diag[rr] : TS(1);
      }
#pragma unroll
      for (int u = 0; u < kBUnroll; ++u) {
        const long long rr = r + u * RB;
        if (rr >= te) continue;
        if (mode == 0) Z[rr * ldz + cc] = zv[u] + al * pv[u];
        if (mode == 4) Z[rr * ldz + cc] = TS(0);
        if (upd) {
          const TS y = rv[u] / dv[u];
          P[rr * ldp + cc] = init ? y : y + be * pv[u];
        }
      }
    }
  }
}

struct BProblem {
  const int32_t *indptr, *col;
  const float *w;
  int32_t N, C;
  const void *diag, *rhs;
  int64_t ldrhs;
  void *Z;
  int64_t ldz;
  void *R;
  int64_t ldr;
  void *P;
  int64_t ldp;
  void *AP;
  int64_t ldap;
  int dtype;
  int group;
};

// Mean degree the gather layout is chosen for: a fixed one, so that an instance's sums do not depend on the degrees of
// the others in its batch. fp32 rows take four entry slots: with two, a row's chains of rounded additions are twice as
// long, which the corrections' scores show (24 systems of degree 8 to 24 to 1e-6, four seeds, mean of the largest
// errors 4.97e-8 against 4.69e-8; degree 64 2.75e-8 against 1.52e-8; 15.1 ms against 15.4). fp64 rows take two (48
// systems 10.7 ms against 11.5).
constexpr double kBDegree32 = 16.0, kBDegree64 = 8.0;

template <class T>
static int b_launch_apply(const BProblem &q, const BTiles &tl, const BCtl &c, cudaStream_t s) {
  using TX = typename T::TX;
  Layout L;
  constexpr bool f32 = sizeof(TX) == 4;
  DLP_TRY(choose_layout(q.C, sizeof(TX), q.P, q.ldp, q.group, f32 ? kBDegree32 : kBDegree64, &L));
  auto rows = [&](const void *p, int64_t ld, int align, int width) {
    return (uintptr_t)p % align == 0 && (ld * (int64_t)sizeof(TX)) % align == 0 && ld >= width;
  };
  const bool r10 = !f32 && L.VW == 2 && L.NV == 5 && rows(q.AP, q.ldap, 16, 10);
  const bool r8 = f32 && L.VW == 4 && L.NV == 2 && L.LV == 1 && rows(q.P, q.ldp, 32, 8) && rows(q.AP, q.ldap, 32, 8);
  const bool r12 = f32 && L.VW == 4 && L.NV == 3 && L.LV == 1 && rows(q.AP, q.ldap, 16, 12);
  if (r10) {  // one lane holds the whole row (run_spmm's layout)
    L.G /= L.LV;
    L.LV = 1;
  }
  BApply<T> a{q.indptr, q.col, (const typename T::TW *)q.w, q.C, (const TX *)q.P, q.ldp,
              (const typename T::TV *)q.diag, (typename T::TY *)q.AP, q.ldap, tl, c, L.G, L.LV, L.NV};
  const int grid = std::min(tl.ntiles, sm_count() * 8);
  constexpr int VWV = 16 / sizeof(TX);
  if constexpr (!f32) {
    if (r10) {
      k_b_apply<T, 2, 5, kRow10D><<<grid, kThreads, 0, s>>>(a);
      return check_launch();
    }
  } else {
    if (r8) {
      k_b_apply<T, 4, 2, kRow8F><<<grid, kThreads, 0, s>>>(a);
      return check_launch();
    }
    if (r12) {
      k_b_apply<T, 4, 3, kRow12F><<<grid, kThreads, 0, s>>>(a);
      return check_launch();
    }
  }
#define DLP_BAPPLY(VW_)                                                       \
  switch (L.VPL) {                                                            \
    case 1: k_b_apply<T, VW_, 1><<<grid, kThreads, 0, s>>>(a); break;        \
    case 2: k_b_apply<T, VW_, 2><<<grid, kThreads, 0, s>>>(a); break;        \
    case 3: k_b_apply<T, VW_, 3><<<grid, kThreads, 0, s>>>(a); break;        \
    case 4: k_b_apply<T, VW_, 4><<<grid, kThreads, 0, s>>>(a); break;        \
    default: return DLP_ERR_INVALID;                                          \
  }
  if (L.VW == 1) {
    DLP_BAPPLY(1)
  } else {
    DLP_BAPPLY(VWV)
  }
#undef DLP_BAPPLY
  return check_launch();
}

template <class T>
static int b_launch_residual(int phase, const BProblem &q, const BTiles &tl, const BCtl &c, cudaStream_t s) {
  using TX = typename T::TX;
  Layout L;
  DLP_TRY(choose_layout(q.C, sizeof(TX), q.Z, q.ldz, q.group, kBDegree64, &L));  // (fp64 sums)
  BApply<T> a{q.indptr, q.col, (const typename T::TW *)q.w, q.C, (const TX *)q.Z, q.ldz,
              (const typename T::TV *)q.diag, (typename T::TY *)q.R, q.ldr, tl, c, L.G, L.LV, L.NV};
  const int grid = std::min(tl.ntiles, sm_count() * 8);
  constexpr int VWV = 16 / sizeof(TX);
  const TX *rhs = (const TX *)q.rhs;
#define DLP_BRES(VW_)                                                                              \
  switch (L.VPL) {                                                                                 \
    case 1: k_b_residual<T, VW_, 1><<<grid, kThreads, 0, s>>>(phase, a, rhs, q.ldrhs); break;      \
    case 2: k_b_residual<T, VW_, 2><<<grid, kThreads, 0, s>>>(phase, a, rhs, q.ldrhs); break;      \
    case 3: k_b_residual<T, VW_, 3><<<grid, kThreads, 0, s>>>(phase, a, rhs, q.ldrhs); break;      \
    case 4: k_b_residual<T, VW_, 4><<<grid, kThreads, 0, s>>>(phase, a, rhs, q.ldrhs); break;      \
    default: return DLP_ERR_INVALID;                                                               \
  }
  if (L.VW == 1) {
    DLP_BRES(1)
  } else {
    DLP_BRES(VWV)
  }
#undef DLP_BRES
  return check_launch();
}

template <typename TS>
static int b_update(int phase, const BProblem &q, const BTiles &tl, const BCtl &c, cudaStream_t s) {
  const bool src = phase == 3;
  k_b_update<TS><<<std::min(tl.ntiles, sm_count() * 8), kBThreads, 0, s>>>(
      phase, q.C, (TS *)q.R, q.ldr, (const TS *)(src ? q.rhs : q.AP), src ? q.ldrhs : q.ldap, (const TS *)q.diag, tl, c);
  return check_launch();
}

template <typename TS>
static int b_dir(int mode, const BProblem &q, const BTiles &tl, const BCtl &c, cudaStream_t s) {
  k_b_dir<TS><<<std::min(tl.ntiles, sm_count() * 8), kBThreads, 0, s>>>(mode, q.C, (TS *)q.Z, q.ldz, (TS *)q.P, q.ldp,
                                                                       (const TS *)q.R, q.ldr, (const TS *)q.diag, tl, c);
  return check_launch();
}

template <typename TS>
static int b_iteration(const BProblem &q, const BTiles &tl, const BCtl &c, const BParams &bp, cudaStream_t s) {
  if (q.dtype == DLP_F32) DLP_TRY(b_launch_apply<T_F32>(q, tl, c, s));
  else DLP_TRY(b_launch_apply<T_W32X64>(q, tl, c, s));
  if (tl.ntiles > kBFoldTiles) {
    k_b_alpha<<<tl.ninst, 256, 0, s>>>(q.C, tl, c);
    DLP_TRY(check_launch());
  }
  DLP_TRY(b_update<TS>(0, q, tl, c, s));
  k_b_beta<<<tl.ninst, 256, 0, s>>>(0, q.C, tl, c, bp);
  DLP_TRY(check_launch());
  return b_dir<TS>(0, q, tl, c, s);
}

// the true residual, its statistics, the decision and the directions of phase 1 (proposed stops) or 2 (the start)
template <typename TS>
static int b_phase(int phase, const BProblem &q, const BTiles &tl, const BCtl &c, const BParams &bp, cudaStream_t s) {
  using TR = Types<float, TS, TS, TS, double>;  // fp64 accumulation in both precisions
  DLP_TRY(b_launch_residual<TR>(phase, q, tl, c, s));
  DLP_TRY(b_update<TS>(phase, q, tl, c, s));
  k_b_beta<<<tl.ninst, 256, 0, s>>>(phase, q.C, tl, c, bp);
  DLP_TRY(check_launch());
  return b_dir<TS>(phase, q, tl, c, s);
}

// the start from Z = 0: the residual is the right-hand side
template <typename TS>
static int b_zero_start(const BProblem &q, const BTiles &tl, const BCtl &c, const BParams &bp, cudaStream_t s) {
  DLP_TRY(b_update<TS>(3, q, tl, c, s));
  k_b_beta<<<tl.ninst, 256, 0, s>>>(2, q.C, tl, c, bp);
  DLP_TRY(check_launch());
  return b_dir<TS>(4, q, tl, c, s);
}

template <typename TS>
static int b_solve(const BProblem &q, const BTiles &tl, const BCtl &c, const BParams &bp, int k, bool zero,
                   cudaStream_t s) {
  DLP_TRY(zero ? b_zero_start<TS>(q, tl, c, bp, s) : b_phase<TS>(2, q, tl, c, bp, s));
  int32_t counts[2] = {0, 0};
  for (int guard = 0; guard < (1 << 30); ++guard) {
    k_b_count<<<1, 1024, 0, s>>>(tl.ninst, c);
    DLP_TRY(check_launch());
    DLP_CUDA(cudaMemcpyAsync(counts, c.counts, sizeof(counts), cudaMemcpyDeviceToHost, s));
    DLP_CUDA(cudaStreamSynchronize(s));
    if (counts[1] > 0) {  // proposed stops: confirm on the true residual, resume the others
      DLP_TRY(b_phase<TS>(1, q, tl, c, bp, s));
      if (counts[0] == 0) continue;
    } else if (counts[0] == 0) {
      break;
    }
    for (int i = 0; i < k; ++i) DLP_TRY(b_iteration<TS>(q, tl, c, bp, s));
  }
  return DLP_OK;
}

}  // namespace dlp

using namespace dlp;

extern "C" {

size_t dlp_pcg_batched_workspace_bytes(int32_t ninst, int32_t ntiles, int32_t C) {
  return bctl_bytes(ninst > 0 ? ninst : 1, ntiles > 0 ? ntiles : 1, C > 0 ? C : 1);
}

int dlp_pcg_batched(const int32_t *indptr, const int32_t *col, const float *w, int32_t N, int32_t C, const void *diag,
                    const void *rhs, int64_t ldrhs, void *Z, int64_t ldz, void *R, int64_t ldr, void *P, int64_t ldp,
                    void *AP, int64_t ldap, int dtype, int32_t ninst, int32_t ntiles, const int32_t *tile_inst,
                    const int32_t *tile_beg, const int32_t *tile_end, const int32_t *inst_tiles,
                    const double *eps_dev, const double *rhs_norm_dev, double target_relres, int32_t mode,
                    int32_t max_iter, int32_t patience, int32_t check_every, int32_t use_graph, int32_t group,
                    double avg_deg, void *ws, size_t ws_bytes, int32_t *iters_out, int32_t *status_out,
                    double *relres_out, dlp_stream_t stream) {
  if (N < 0 || C <= 0 || C > 64 || ninst <= 0 || ntiles <= 0 || ldz < C || ldr < C || ldp < C || ldap < C ||
      ldrhs < C)
    return DLP_ERR_INVALID;
  if (mode < 1 || mode > 7 || (mode & 3) == 0 || !eps_dev || !rhs_norm_dev || !tile_inst || !tile_beg || !tile_end || !inst_tiles)
    return DLP_ERR_INVALID;
  if (!(dtype == DLP_F32 || dtype == DLP_F64)) return DLP_ERR_DTYPE;
  if (!ws || ws_bytes < dlp_pcg_batched_workspace_bytes(ninst, ntiles, C)) return DLP_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  BCtl c = carve_b(ws, ninst, ntiles, C);
  BTiles tl{tile_inst, tile_beg, tile_end, inst_tiles, ntiles, ninst};
  BParams bp{mode, patience > 0 ? patience : 400, max_iter, target_relres};
  BProblem q{indptr, col, w, N, C, diag, rhs, ldrhs, Z, ldz, R, ldr, P, ldp, AP, ldap, dtype, group};
  const size_t iB = 4 * (size_t)ninst;
  (void)use_graph;  // the host drives the loop either way
  (void)avg_deg;    // (kBDegree32, kBDegree64)
  k_b_init<<<ceil_div_i((long long)ninst * C, 256), 256, 0, s>>>(ninst, C, eps_dev, rhs_norm_dev, c);
  DLP_TRY(check_launch());
  bp.mode = mode & 3;
  const bool zero = (mode & 4) != 0;
  const int k = check_every > 0 ? check_every : 8;
  if (dtype == DLP_F32) DLP_TRY(b_solve<float>(q, tl, c, bp, k, zero, s));
  else DLP_TRY(b_solve<double>(q, tl, c, bp, k, zero, s));
  if (iters_out) DLP_CUDA(cudaMemcpyAsync(iters_out, c.iters, iB, cudaMemcpyDeviceToHost, s));
  if (status_out) DLP_CUDA(cudaMemcpyAsync(status_out, c.done, iB, cudaMemcpyDeviceToHost, s));
  if (relres_out) DLP_CUDA(cudaMemcpyAsync(relres_out, c.relres, 8 * (size_t)ninst, cudaMemcpyDeviceToHost, s));
  DLP_CUDA(cudaStreamSynchronize(s));
  return DLP_OK;
}

// ---- the batch's own vectors -----------------------------------------------------------------------
}  // extern "C"

namespace dlp {

// instance of entry (or row) i: the last k with off[k] <= i
__device__ __forceinline__ int b_find(const int32_t *off, int B, long long i) {
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// concatenated CSRs made one block-diagonal CSR in place: rows' pointers by the entries before their instance, columns by
// its rows
__global__ void k_b_offsets(int32_t B, const int32_t *__restrict__ row_off, const int32_t *__restrict__ nnz_off, int32_t N,
                            long long nnz, int32_t *indptr, int32_t *col) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) indptr[i + 1] += nnz_off[b_find(row_off, B, i)];
  if (i < nnz) col[i] += row_off[b_find(nnz_off, B, i)];
}

// per tile and column: sum of squares and largest magnitude
template <typename TS>
__global__ void __launch_bounds__(kBThreads) k_b_tile_stats(int32_t C, const TS *__restrict__ X, int64_t ldx, BTiles tl,
                                                            double *part) {
  __shared__ double s_a[kBThreads], s_m[kBThreads];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int RB = kBThreads / C, q = tid / C, cc = tid - q * C;
  for (int t = blockIdx.x; t < tl.ntiles; t += gridDim.x) {
    double a = 0.0, m = 0.0;
    if (q < RB)
      for (int r = tl.tbeg[t] + q; r < tl.tend[t]; r += RB) {
        const double x = (double)X[(long long)r * ldx + cc];
        a += x * x;
        m = fmax(m, fabs(x));
      }
    s_a[tid] = a;
    s_m[tid] = m;
    __syncthreads();
    for (int x = wid; x < C; x += kBThreads / 32) {
      double u = 0.0, v = 0.0;
      for (int k = lane; k < RB; k += 32) {
        u += s_a[k * C + x];
        v = fmax(v, s_m[k * C + x]);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, off);
        v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
      }
      if (lane == 0) {
        part[((long long)t * C + x) * 2] = u;
        part[((long long)t * C + x) * 2 + 1] = v;
      }
    }
    __syncthreads();
  }
}

__global__ void k_b_inst_stats(int32_t C, BTiles tl, const double *__restrict__ part, double *out) {
  const int inst = blockIdx.x, t0 = tl.toff[inst], nt = tl.toff[inst + 1] - t0;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int x = wid; x < 2 * C; x += blockDim.x >> 5) {  // sums of squares, then magnitudes
    const int cc = x < C ? x : x - C, k = x < C ? 0 : 1;
    const double v = warp_strided_reduce(part + ((long long)t0 * C + cc) * 2 + k, 2LL * C, nt, k == 1);
    if (lane == 0) out[(long long)inst * 2 * C + x] = v;
  }
}

// mode 0: Y (fp32) = X / scale; mode 1: Y (fp64) += X (fp32) * scale; scale per instance and column (0: untouched)
__global__ void __launch_bounds__(kBThreads) k_b_scale(int mode, int32_t C, const void *X, int64_t ldx,
                                                       const double *__restrict__ scale, void *Y, int64_t ldy, BTiles tl) {
  const int tid = threadIdx.x, RB = kBThreads / C, q = tid / C, cc = tid - q * C;
  if (q >= RB) return;
  for (int t = blockIdx.x; t < tl.ntiles; t += gridDim.x) {
    const double sc = scale[(long long)tl.tinst[t] * C + cc];
    if (sc == 0.0) continue;
    for (int r = tl.tbeg[t] + q; r < tl.tend[t]; r += RB) {
      if (mode == 0)
        ((float *)Y)[(long long)r * ldy + cc] = (float)(((const double *)X)[(long long)r * ldx + cc] / sc);
      else
        ((double *)Y)[(long long)r * ldy + cc] += (double)((const float *)X)[(long long)r * ldx + cc] * sc;
    }
  }
}

}  // namespace dlp

extern "C" {

int dlp_batch_offsets(int32_t ninst, const int32_t *row_off, const int32_t *nnz_off, int32_t N, int64_t nnz,
                      int32_t *indptr, int32_t *col, dlp_stream_t stream) {
  if (ninst <= 0 || N < 0 || nnz < 0 || !row_off || !nnz_off || !indptr || (nnz > 0 && !col)) return DLP_ERR_INVALID;
  const long long m = std::max((long long)N, (long long)nnz);
  if (m == 0) return DLP_OK;
  k_b_offsets<<<ceil_div_i(m, 256), 256, 0, (cudaStream_t)stream>>>(ninst, row_off, nnz_off, N, nnz, indptr, col);
  return check_launch();
}

size_t dlp_batch_colstats_workspace_bytes(int32_t ntiles, int32_t C) {
  return sizeof(double) * 2 * (size_t)(ntiles > 0 ? ntiles : 1) * (size_t)(C > 0 ? C : 1);
}

int dlp_batch_colstats(int32_t C, const void *X, int64_t ldx, int dtype, int32_t ninst, int32_t ntiles,
                       const int32_t *tile_inst, const int32_t *tile_beg, const int32_t *tile_end,
                       const int32_t *inst_tiles, double *out, void *ws, size_t ws_bytes, dlp_stream_t stream) {
  if (C <= 0 || C > 64 || ninst <= 0 || ntiles < 0 || ldx < C || !inst_tiles || !out) return DLP_ERR_INVALID;
  if (ntiles > 0 && (!X || !tile_inst || !tile_beg || !tile_end)) return DLP_ERR_INVALID;
  if (dtype != DLP_F32 && dtype != DLP_F64) return DLP_ERR_DTYPE;
  if (!ws || ws_bytes < dlp_batch_colstats_workspace_bytes(ntiles, C)) return DLP_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  BTiles tl{tile_inst, tile_beg, tile_end, inst_tiles, ntiles, ninst};
  const int grid = std::min(ntiles, sm_count() * 8);
  if (ntiles > 0) {
    if (dtype == DLP_F32) k_b_tile_stats<float><<<grid, kBThreads, 0, s>>>(C, (const float *)X, ldx, tl, (double *)ws);
    else k_b_tile_stats<double><<<grid, kBThreads, 0, s>>>(C, (const double *)X, ldx, tl, (double *)ws);
    DLP_TRY(check_launch());
  }
  k_b_inst_stats<<<ninst, 256, 0, s>>>(C, tl, (const double *)ws, out);
  return check_launch();
}

int dlp_batch_scale(int32_t mode, int32_t C, const void *X, int64_t ldx, const double *scale, void *Y, int64_t ldy,
                    int32_t ninst, int32_t ntiles, const int32_t *tile_inst, const int32_t *tile_beg,
                    const int32_t *tile_end, dlp_stream_t stream) {
  if (mode < 0 || mode > 1 || C <= 0 || C > 64 || ntiles < 0 || ldx < C || ldy < C || !scale) return DLP_ERR_INVALID;
  if (ntiles == 0) return DLP_OK;
  if (!X || !Y || !tile_inst || !tile_beg || !tile_end) return DLP_ERR_INVALID;
  BTiles tl{tile_inst, tile_beg, tile_end, nullptr, ntiles, ninst};
  k_b_scale<<<std::min(ntiles, sm_count() * 8), kBThreads, 0, (cudaStream_t)stream>>>(mode, C, X, ldx, scale, Y, ldy, tl);
  return check_launch();
}

}  // extern "C"
