// The whole Jacobi-PCG solve in one launch, for systems whose iteration is bound by latency rather than
// by bytes (whole_fits in pcg.cu): the start, every iteration, the recheck of a proposed stop on the true
// residual and the stop rules run in one resident grid, one block per SM. Included by pcg.cu.
//
// A block owns a run of rows and keeps its part of the system in shared memory: the CSR entries, the
// diagonal, R, Z, AP and its rows of P. Only the direction P (the true residual: Z) is read across blocks,
// through L2. Per iteration:
//   (a) AP = diag P - W P, pAp;   all-to-all sum, alpha
//   (b) R -= alpha AP, rz, ||R||^2, violation;   all-to-all sum, stop decision, beta
//   (c) Z += alpha P, P = R / diag + beta P;   barrier
// What bounds it: the three grid barriers (some 3,000 cycles each on this chip: a store or an atomic takes about
// 1,000 to be seen by another SM's load); at n = 30,000 and 5 columns waiting warps there are four times those
// waiting for loads, with the L1 18% busy. Towards the largest systems the gathers count (about one line per two
// cycles and SM, whatever a lane takes of it), so the rows are spread over every SM and a lane gathers 32 bytes in
// one access where the rows allow. Each block folds all blocks' partial sums itself, in the same order: the same
// bits everywhere, so each takes the same decision and none has to publish it. (Words of value and tag that every
// block polls for every other, one trip instead of three, measured 8,000 cycles at 148 blocks: the polls of all
// blocks meet on the same lines.) All waits are bounded.
#pragma once

namespace dlp {

constexpr int kWholeMaxC = 64;
constexpr int kWholeThreads = 512;
constexpr int kWholeWarps = kWholeThreads / 32;
constexpr int kWholeBlocks = 160;           // most blocks of a launch (one per SM)
constexpr int kWholeSmem = 190 * 1024;      // dynamic shared memory of a block

template <class T>
struct WholeArgs {
  const int32_t *rbeg, *rend, *col;
  const typename T::TW *w;
  int32_t n, C, rows;  // rows: per block
  const typename T::TX *diag, *rhs;
  int64_t ldrhs;
  typename T::TX *Z;
  int64_t ldz;
  typename T::TX *R;
  int64_t ldr;
  typename T::TX *P;
  int64_t ldp;
  PcgBufs B;
  GridBar *bar;
  int G, LV;  // lanes per row; those that share an entry's row of X, VW values each
  int zero, confirm;  // start from Z = 0; recheck a proposed stop on the true residual
};

// VW values of a row of X through L2 (rows other blocks wrote in this launch): 32 bytes in one access.
template <class TX, int VW>
__device__ __forceinline__ void load_gathered(const TX *x, TX (&v)[VW]) {
  if constexpr (sizeof(TX) == 4 && VW == 8) {
    asm volatile("ld.relaxed.gpu.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(x));
  } else if constexpr (sizeof(TX) == 8 && VW == 4) {
    asm volatile("ld.relaxed.gpu.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(x));
  } else if constexpr (VW > 1) {
    load_vec_coherent<TX, VW, TX>(x, v);
  } else {
    v[0] = __ldcg(x);
  }
}

// One lane's VW columns of W X over its entries of a row (every lane of the warp calls this: it
// shuffles): col and w from shared or global memory, lanes of LV hold the row's vectors, edge slots
// es, es + ES, ... the entries.
template <class TW, class TX, int VW>
__device__ __forceinline__ void whole_gather(const int32_t *col, const TW *w, const TX *X, int64_t ldx, int beg, int end,
                                             int es, int ES, int LV, int G, TX (&acc)[VW]) {
  constexpr int U = VW * (int)sizeof(TX) <= 16 ? 8 : 4;
  // two sums per lane, of every other entry: shorter chains of rounded additions (the fp32 residual of a recheck
  // is no coarser than the launched kernels', which have more entry slots: with one sum a solve of 8 columns to
  // 1e-6, n = 60,000, failed its rechecks that theirs passed)
  TX odd[VW];
#pragma unroll
  for (int i = 0; i < VW; ++i) acc[i] = odd[i] = TX(0);
  for (int j0 = beg + es; j0 < end; j0 += U * ES) {
    TX t[U][VW], wv[U];
    int v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * ES;
      v[u] = j < end ? col[j] : -1;
      wv[u] = j < end ? cvt<TX>(w[j]) : TX(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int i = 0; i < VW; ++i) t[u][i] = TX(0);
      if (v[u] >= 0) load_gathered<TX, VW>(X + (long long)v[u] * ldx, t[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < VW; ++i) {
        if (u & 1) odd[i] = fmaa(wv[u], t[u][i], odd[i]);
        else acc[i] = fmaa(wv[u], t[u][i], acc[i]);
      }
  }
#pragma unroll
  for (int i = 0; i < VW; ++i) acc[i] += odd[i];
  for (int off = LV; off < G; off <<= 1) {
#pragma unroll
    for (int i = 0; i < VW; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
  }
}

// Measured on B200 (SBM, degree 16, us per iteration, graph loop -> this launch): n = 3,000: 1 / 5 / 9 fp32
// columns 26.6 / 24.3 / 28.1 -> 10.0 / 10.9 / 13.0; n = 30,000: 28.7 / 27.0 / 32.2 -> 14.0 / 15.4 / 22.6;
// n = 100,000: 37.3 / 34.4 -> 22.3 / 25.6; fp64, 5 columns, n = 3,000 / 30,000: 31.4 / 35.3 -> 11.6 / 23.5.
// A solve's fixed part (start, upload, host read) stays at about 100 us.
template <class T, int VW>
__global__ void __launch_bounds__(kWholeThreads, 1) k_pcg_whole(WholeArgs<T> p) {
  using TW = typename T::TW;
  using TX = typename T::TX;
  constexpr int NT = kWholeThreads, NW = kWholeWarps;
  const PcgBufs &B = p.B;
  const int C = p.C, nb = (int)gridDim.x;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int G = p.G, LV = p.LV, ES = G / LV, gpw = 32 / G;
  const int gl = lane & (G - 1), cl = gl & (LV - 1), es = gl / LV;
  const bool on = cl * VW < C;  // the lane holds columns (LV is a power of two)
  const int row0 = blockIdx.x * p.rows;
  const int nr = max(0, min(p.rows, p.n - row0));

  __shared__ double s_v[3][NT];
  __shared__ double s_red[2 * kWholeMaxC + 2];
  __shared__ double s_rz[kWholeMaxC], s_rzprev[kWholeMaxC], s_rel;
  __shared__ double s_be[kWholeMaxC], s_irn[kWholeMaxC];  // beta; 1 / ||rhs|| (1 where it is zero)
  __shared__ int s_bad, s_lo, s_hi;
  extern __shared__ __align__(16) char dyn[];
  // the block's rows of R, Z, AP, P (C values each), 1 / diag, diag, row ranges, then the CSR entries
  TX *R = (TX *)dyn;
  TX *Z = R + (size_t)p.rows * C;
  TX *AP = Z + (size_t)p.rows * C;
  TX *P = AP + (size_t)p.rows * C;
  double *dinv = (double *)(((uintptr_t)(P + (size_t)p.rows * C) + 15) & ~(uintptr_t)15);
  TX *dg = (TX *)(dinv + p.rows);
  int32_t *rb = (int32_t *)(dg + p.rows), *re = rb + p.rows;
  char *ent = (char *)(((uintptr_t)(re + p.rows) + 15) & ~(uintptr_t)15);

  if (tid < C) s_irn[tid] = B.rhsn[tid] > 0.0 ? 1.0 / B.rhsn[tid] : 1.0;
  if (tid == 0) {
    s_lo = 0x7fffffff;
    s_hi = 0;
  }
  __syncthreads();
  for (int i = tid; i < nr; i += NT) {
    const int b = p.rbeg[row0 + i], e = p.rend[row0 + i];
    rb[i] = b;
    re[i] = e;
    const TX d = p.diag[row0 + i];
    dg[i] = d;
    dinv[i] = __drcp_rn((double)d);  // correctly rounded: the value of 1.0 / d
    if (b < e) {
      atomicMin(&s_lo, b);
      atomicMax(&s_hi, e);
    }
  }
  __syncthreads();
  // the entries come along when the rows' span of slots fits what is left of the block's memory
  const int lo = s_lo, span = max(0, s_hi - s_lo);
  const long long room = (long long)kWholeSmem - (ent - dyn);
  const bool local = (long long)span * (long long)(sizeof(TW) + 4) <= room;
  TW *lw = (TW *)ent;
  int32_t *lc = (int32_t *)(lw + span);
  if (local) {
    for (int i = tid; i < span; i += NT) {
      lc[i] = p.col[lo + i];
      lw[i] = p.w[lo + i];
    }
    for (int i = tid; i < nr; i += NT) {
      const int b = rb[i], e = re[i];
      rb[i] = b < e ? b - lo : 0;
      re[i] = b < e ? e - lo : 0;
    }
  }
  const int32_t *cols = local ? lc : p.col;
  const TW *ws = local ? lw : p.w;

  // element sweeps: thread tid owns column tc of the block's rows tr, tr + RS, ...
  const int RS = NT / C, tr = tid / C, tc = tid - tr * C;
  const bool el = tr < RS;
  const double einv = el ? B.epsinv[tc] : 0.0;
  // the control block's inputs (uploaded before the launch)
  const int mode = B.ctl->mode, patience = B.ctl->patience, max_iter = B.ctl->max_iter;
  const double tgt = B.ctl->target;
  double best = 0.0, viol = 0.0, relres = 0.0;
  int iters = 0, stall = 0, done = 0;
  double *part1 = B.part1, *part2 = B.part2;
  uint32_t target = 0;

  // Every block's stores before the barrier are visible through L2 after it; false when a wait ran out.
  auto barrier = [&]() -> bool {
    if (grid_barrier(p.bar, target)) return true;
    if (tid == 0) atomicExch(&B.ctl->lost, 1);
    return false;
  };
  // Sum over all blocks of NO outputs, per-thread values in s_v: outputs 0..C-1 from s_v[0], C..2C-1 from
  // s_v[1], 2C the maximum of s_v[2], 2C + 1 block 0's read of the cancel word. One warp per output, block
  // sums and then the blocks in fixed orders; the results are in s_red (alpha: rz / sum instead of the sum).
  const int used = min(nr, RS);  // row slots of the element sweeps that hold values
  auto exchange = [&](int NO, double *part, bool alpha = false) -> bool {
    __syncthreads();
    for (int o = wid; o < NO; o += NW) {
      double v = 0.0;
      if (o < 2 * C) {
        const double *src = s_v[o < C ? 0 : 1] + (o < C ? o : o - C);
        for (int k = lane; k < used; k += 32) v += src[k * C];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      } else {
        for (int k = lane; k < used * C; k += 32) v = fmax(v, s_v[2][k]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
      }
      if (lane == 0) __stcg(part + (size_t)o * nb + blockIdx.x, v);
    }
    if (NO > 2 * C && blockIdx.x == 0 && tid == 0)
      __stcg(part + (size_t)(2 * C + 1) * nb, (double)read_cancel(B.cancel));
    if (!barrier()) return false;
    if (NO > 2 * C && wid == NW - 1 && lane == 0) s_red[2 * C + 1] = __ldcg(part + (size_t)(2 * C + 1) * nb);
    for (int o = wid; o < NO; o += NW) {
      double x[kWholeBlocks / 32];
#pragma unroll
      for (int u = 0; u < kWholeBlocks / 32; ++u)
        x[u] = u * 32 + lane < nb ? __ldcg(part + (size_t)o * nb + u * 32 + lane) : 0.0;
      const bool sum = o < 2 * C;
      double v = x[0];
#pragma unroll
      for (int u = 1; u < kWholeBlocks / 32; ++u) v = sum ? v + x[u] : fmax(v, x[u]);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, v, off);
        v = sum ? v + y : fmax(v, y);
      }
      if (lane == 0) {
        if (alpha) {
          v = v > 0.0 ? s_rz[o] / v : 0.0;
          v = isfinite(v) && fabs(v) < 1e30 ? v : 0.0;
        }
        s_red[o] = v;
      }
    }
    __syncthreads();
    return true;
  };
  // the stop decision of finish_sweep from s_red (phase 0 an iteration, 1 a recheck, 2 the start);
  // every thread of every block computes the same values
  auto decide = [&](int phase) {
    if (wid == 0) {  // one column per lane; the largest ratio, and whether a sum of squares is not finite
      double rel = 0.0;
      bool bad = false;
      for (int c = lane; c < C; c += 32) {
        const double b = s_red[C + c];
        bad = bad || !isfinite(b);
        rel = fmax(rel, sqrt(b) * s_irn[c]);
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) rel = fmax(rel, __shfl_xor_sync(0xffffffffu, rel, off));
      bad = __any_sync(0xffffffffu, bad);
      if (lane == 0) {
        s_rel = rel;
        s_bad = bad;
      }
    } else if (wid == 1) {
      for (int c = lane; c < C; c += 32) {
        const double a = s_red[c], den = phase == 1 ? s_rzprev[c] : s_rz[c];
        const double be = (phase < 2 && den > 0.0) ? a / den : 0.0;
        s_be[c] = isfinite(be) && fabs(be) < 1e30 ? be : 0.0;
        if (phase == 0) s_rzprev[c] = den;
        s_rz[c] = a;
      }
    }
    __syncthreads();
    const bool bad = s_bad != 0;
    viol = s_red[2 * C];
    relres = s_rel;
    double m = 0.0;
    if (mode & 1) m = fmax(m, viol);
    if (mode & 2) m = fmax(m, tgt > 0.0 ? relres / tgt : relres);
    const bool conv = m <= 1.0 && !bad;
    if (phase == 0) iters += 1;
    if (phase == 2) {
      best = m;
      stall = 0;
      done = conv ? 5 : 0;
    } else if (conv) {
      done = phase == 0 ? 1 : 5;
    } else {
      if (m < 0.9 * best) {
        best = m;
        stall = 0;
      } else {
        stall += 1;
      }
      done = stall >= patience ? 2 : 0;
    }
    if (done == 0 && iters >= max_iter) done = 3;
    if (done == 0 && s_red[2 * C + 1] != 0.0) done = 6;
    if (bad) done = 4;
  };
  // W X of the block's rows, X = the P buffer (which holds Z for a true residual)
  auto apply = [&](auto epilogue) {
    for (int g0 = wid * gpw; g0 < nr; g0 += NW * gpw) {
      const int r = g0 + lane / G;
      const bool valid = r < nr;
      TX acc[VW];
      whole_gather<TW, TX, VW>(cols, ws, p.P + cl * VW, p.ldp, valid && on ? rb[r] : 0, valid && on ? re[r] : 0, es, ES, LV,
                               G, acc);
      if (valid && es == 0) {
#pragma unroll
        for (int i = 0; i < VW; ++i)
          if (cl * VW + i < C) epilogue(r, cl * VW + i, acc[i]);
      }
    }
  };
  // rz, ||R||^2 and the violation of the block's R, per thread
  auto stats = [&] {
    double rz = 0.0, ss = 0.0, vm = 0.0;
    if (el)
      for (int r = tr; r < nr; r += RS) {
        const double r64 = (double)R[r * C + tc], r2 = r64 * r64, di = dinv[r];
        rz += r2 * di;
        ss += r2;
        vm = fmax(vm, fabs(r64) * di);
      }
    s_v[0][tid] = rz;
    s_v[1][tid] = ss;
    s_v[2][tid] = vm * einv;
  };

  // the start: R = rhs - A Z (rhs from Z = 0), P = R / diag
  if (el)
    for (int r = tr; r < nr; r += RS) {
      const long long g = row0 + r;
      Z[r * C + tc] = p.zero ? TX(0) : p.Z[g * p.ldz + tc];
      R[r * C + tc] = p.rhs[g * p.ldrhs + tc];
    }
  // R = rhs - (diag Z - W Z), Z gathered from the P buffer; false when a wait ran out
  auto true_residual = [&]() -> bool {
    if (el)
      for (int r = tr; r < nr; r += RS) __stcg(p.P + (long long)(row0 + r) * p.ldp + tc, Z[r * C + tc]);
    if (!barrier()) return false;
    apply([&](int r, int c, TX a) {
      R[r * C + c] = p.rhs[(long long)(row0 + r) * p.ldrhs + c] - (dg[r] * Z[r * C + c] - a);
    });
    return barrier();  // the buffer is P's again
  };
  __syncthreads();
  if (!p.zero && !true_residual()) return;
  if (el)
    for (int r = tr; r < nr; r += RS) {
      const TX y = R[r * C + tc] / dg[r];
      P[r * C + tc] = y;
      __stcg(p.P + (long long)(row0 + r) * p.ldp + tc, y);
    }
  stats();
  if (!exchange(2 * C + 1, part2)) return;
  decide(2);
  if (done == 0 && !barrier()) return;

  while (done == 0) {
    // (a)
    apply([&](int r, int c, TX a) { AP[r * C + c] = dg[r] * P[r * C + c] - a; });
    __syncthreads();
    double pap = 0.0;
    if (el)
      for (int r = tr; r < nr; r += RS) pap += (double)P[r * C + tc] * (double)AP[r * C + tc];
    s_v[0][tid] = pap;
    if (!exchange(C, part1, true)) return;
    // (b)
    const TX al = el ? (TX)s_red[tc] : TX(0);
    if (el)
      for (int r = tr; r < nr; r += RS) R[r * C + tc] = R[r * C + tc] - al * AP[r * C + tc];
    stats();
    if (!exchange(2 * C + 1, part2)) return;
    decide(0);
    // (c) Z, and the next direction while the solve runs
    const TX be = el ? (TX)s_be[tc] : TX(0);
    if (el)
      for (int r = tr; r < nr; r += RS) {
        const TX pv = P[r * C + tc];
        Z[r * C + tc] = Z[r * C + tc] + al * pv;
        if (done == 0) {
          const TX pn = R[r * C + tc] / dg[r] + be * pv;
          P[r * C + tc] = pn;
          __stcg(p.P + (long long)(row0 + r) * p.ldp + tc, pn);
        }
      }
    if (done == 0 && !barrier()) return;
    if (done == 1 && !p.confirm) done = 5;  // the caller confirms the stop on a residual of its own
    if (done == 1) {
      // a proposed stop: the true residual decides (dynlp/solvers.py:85-89); a failed recheck goes on
      // from it with the reference's beta
      if (!true_residual()) return;
      stats();
      if (!exchange(2 * C + 1, part2)) return;
      decide(1);
      const TX bt = el ? (TX)s_be[tc] : TX(0);
      if (done == 0) {
        if (el)
          for (int r = tr; r < nr; r += RS) {
            const TX pn = R[r * C + tc] / dg[r] + bt * P[r * C + tc];
            P[r * C + tc] = pn;
            __stcg(p.P + (long long)(row0 + r) * p.ldp + tc, pn);
          }
        if (!barrier()) return;
      }
    }
  }
  if (el)
    for (int r = tr; r < nr; r += RS) {
      p.Z[(long long)(row0 + r) * p.ldz + tc] = Z[r * C + tc];
      p.R[(long long)(row0 + r) * p.ldr + tc] = R[r * C + tc];
    }
  if (blockIdx.x == 0 && tid == 0) {
    PcgCtl *ctl = B.ctl;
    ctl->iters = iters;
    ctl->stall = stall;
    ctl->bad = done == 4;
    ctl->best = best;
    ctl->viol = viol;
    ctl->relres = relres;
    ctl->done = done;
  }
}

}  // namespace dlp
