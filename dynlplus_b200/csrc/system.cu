// The grounded system of one batch (Stream._build, dynlp/stream.py:142-177) from a symmetric CSR: grounding,
// the U x U filter in CSR order, label weights, diagonal and right-hand sides.
//
// plan: the masks, the grounding (dlp_ground_reach_async), each row's kept entries and two scans (local ids and
// entry positions); the host reads the two sizes and allocates; fill: one pass over the rows writes everything.
// Bound by that pass (columns, weights and marks of every entry, 16 bytes with the outputs) at large sizes and
// by launches at small ones: some fifteen instead of about a hundred tensor operations with eleven host reads
// (degree 16, the whole call: n = 100,000 1.61 -> 0.28 ms; n = 5,000 1.21 -> 0.26 ms).
#include <type_traits>

#include "common.cuh"

namespace dlp {

int exclusive_scan_i32(const int32_t *in, int32_t n, int32_t *out, void *ws, size_t ws_bytes, cudaStream_t s);
size_t compact_ws_bytes(int32_t n);

constexpr int kSysThreads = 256;

// the masks, and whether a labelled vertex's class is outside [-K, K) (negative: from the end)
__global__ void k_sys_masks(int32_t n, const uint8_t *__restrict__ active, const uint8_t *__restrict__ labeled,
                            const int32_t *__restrict__ y, int32_t K, uint8_t *vmask, uint8_t *sink, uint8_t *umask,
                            int32_t *bad) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  const bool a = active[v] != 0, l = labeled[v] != 0;
  vmask[v] = a && !l;
  sink[v] = a && l;
  umask[v] = 0;
  if (a && l && (y[v] < -K || y[v] >= K)) atomicExch(bad, 1);
}

// cnt[u] = entries of row u within U (0 outside), flag[u] = u in U; eight lanes per row
__global__ void k_sys_count(int32_t n, const int32_t *__restrict__ indptr, const int32_t *__restrict__ col,
                            const uint8_t *__restrict__ umask, int32_t *flag, int32_t *cnt) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long u = t >> 3;
  const bool in = u < n && umask[u] != 0;
  int c = 0;
  if (in)
    for (int j = indptr[u] + (int)(t & 7); j < indptr[u + 1]; j += 8) {
      const int32_t v = col[j];
      c += (unsigned)v < (unsigned)n && umask[v] != 0;
    }
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
  if (u < n && (t & 7) == 0) {
    flag[u] = in ? 1 : 0;
    cnt[u] = c;
  }
}

__global__ void k_sys_sizes(int32_t n, const int32_t *loc, const int32_t *pos, int32_t *counts) {
  counts[0] = loc[n];
  counts[1] = pos[n];
}

struct SysOut {
  int64_t *U;
  int32_t *indptr, *col;
  void *w;
  double *B, *s, *diag, *rhs, *rhsh;        // fp64
  float *B32, *s32, *diag32, *rhs32, *rhsh32;  // fp32 copies (NULL: none)
};

// A kept weight as it is stored: bf16 by way of fp32, as the tensor library rounds fp64.
template <typename TO, typename TW>
__device__ __forceinline__ TO stored_weight(TW x) {
  if constexpr (std::is_same<TO, bf16>::value) return __float2bfloat16_rn((float)x);
  else return (TO)x;
}

// Eight lanes per row of U: kept entries in stored order (ranked by ballot), the row sum of the stored weights,
// label weights, which stay as they come, added in stored order by the group's first lane (few neighbours are
// labelled).
template <typename TW, typename TO>
__global__ void __launch_bounds__(kSysThreads)
    k_sys_fill(int32_t n, const int32_t *__restrict__ indptr, const int32_t *__restrict__ col, const TW *__restrict__ w,
               const uint8_t *__restrict__ umask, const uint8_t *__restrict__ sink, const int32_t *__restrict__ y,
               int32_t K, double eta, double prior, int32_t C, int32_t col0, const int32_t *__restrict__ loc,
               const int32_t *__restrict__ pos, SysOut o) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long u = t >> 3;
  const int l = (int)(t & 7), lane = threadIdx.x & 31, g0 = lane & ~7;
  const bool in = u < n && umask[u] != 0;
  const int beg = in ? indptr[u] : 0, end = in ? indptr[u + 1] : 0;
  const long long r = in ? loc[u] : 0;
  int at = in ? pos[u] : 0;
  double *B = o.B + r * K;
  if (in) {
    for (int c = l; c < K; c += 8) B[c] = 0.0;
    if (l == 0) {
      o.U[r] = u;
      o.indptr[r] = at;
    }
  }
  __syncwarp();
  double sum = 0.0;
  const int trips = __reduce_max_sync(0xffffffffu, (end - beg + 7) >> 3);
  for (int k = 0; k < trips; ++k) {
    const int j = beg + k * 8 + l;
    const bool have = j < end;
    const int32_t v = have ? col[j] : -1;
    const bool ok = have && (unsigned)v < (unsigned)n;
    const bool keep = ok && umask[v] != 0, lab = ok && sink[v] != 0;
    const double wv = keep || lab ? (double)w[j] : 0.0;
    const unsigned kb = __ballot_sync(0xffffffffu, keep) >> g0 & 0xffu;
    unsigned lb = __ballot_sync(0xffffffffu, lab) >> g0 & 0xffu;
    if (keep) {
      const int q = at + __popc(kb & ((1u << l) - 1u));
      o.col[q] = loc[v];
      const TO x = stored_weight<TO>(w[j]);
      ((TO *)o.w)[q] = x;
      sum += cvt<double>(x);
    }
    at += __popc(kb);
    // labelled neighbours one after another (warp-uniform trip count)
    const int nl = __reduce_max_sync(0xffffffffu, __popc(lb));
    for (int i = 0; i < nl; ++i) {
      const int src = lb ? __ffs(lb) - 1 : 0;
      const double x = __shfl_sync(0xffffffffu, wv, g0 + src);
      const int32_t vv = __shfl_sync(0xffffffffu, v, g0 + src);
      if (lb && l == 0) {
        int32_t c = y[vv];
        if (c < 0) c += K;  // as an index from the end
        if ((unsigned)c < (unsigned)K) B[c] += x;  // the plan reported any other
      }
      lb &= lb - 1;
    }
  }
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  __syncwarp();
  if (!in) return;
  double s = 0.0;
  for (int c = 0; c < K; ++c) s += B[c];
  s += eta;
  const double d = s + sum;
  if (l == 0) {
    o.s[r] = s;
    o.diag[r] = d;
    if (o.s32) {
      o.s32[r] = (float)s;
      o.diag32[r] = (float)d;
    }
  }
  for (int c = l; c <= C; c += 8) {
    const double x = c < C ? B[col0 + c] + eta * prior : d;
    o.rhsh[r * (C + 1) + c] = x;
    if (c < C) o.rhs[r * C + c] = x;
    if (o.rhsh32) {
      o.rhsh32[r * (C + 1) + c] = (float)x;
      if (c < C) o.rhs32[r * C + c] = (float)x;
    }
  }
  if (o.B32)
    for (int c = l; c < K; c += 8) o.B32[r * K + c] = (float)B[c];
}

static size_t sys_al(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace dlp

using namespace dlp;

extern "C" {

size_t dlp_build_system_workspace_bytes(int32_t n) {
  const size_t nn = (size_t)(n > 0 ? n : 1);
  return 2 * sys_al(4 * nn) + sys_al(nn) + std::max(sys_al(compact_ws_bytes(n)), sys_al(dlp_ground_reach_workspace_bytes(n))) +
         2 * sys_al(nn);
}

int dlp_build_system_plan(int32_t n, const int32_t *indptr, const int32_t *col, const uint8_t *active,
                          const uint8_t *labeled, const int32_t *y, int32_t K, uint8_t *umask, uint8_t *sink, int32_t *loc, int32_t *pos,
                          int32_t *counts, void *ws, size_t ws_bytes, dlp_stream_t stream) {
  if (n <= 0 || K <= 0 || !indptr || !active || !labeled || !y || !umask || !sink || !loc || !pos || !counts) return DLP_ERR_INVALID;
  if (!col) return DLP_ERR_INVALID;
  if (!ws || ws_bytes < dlp_build_system_workspace_bytes(n)) return DLP_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t nn = (size_t)n;
  char *p = (char *)ws;
  int32_t *flag = (int32_t *)p, *cnt = (int32_t *)(p + sys_al(4 * nn));
  uint8_t *vmask = (uint8_t *)(p + 2 * sys_al(4 * nn)), *in_t = vmask + sys_al(nn);
  char *sub = (char *)in_t + sys_al(nn);
  const size_t sub_bytes = ws_bytes - (size_t)(sub - p);
  DLP_CUDA(cudaMemsetAsync(counts, 0, 9 * sizeof(int32_t), s));
  k_sys_masks<<<ceil_div_i(n, kSysThreads), kSysThreads, 0, s>>>(n, active, labeled, y, K, vmask, sink, umask, counts + 8);
  DLP_TRY(check_launch());
  // counts: [0] rows, [1] entries, [2] membership changes, [3] a column out of range, [4..7] grounding info,
  // [8] a class out of range
  DLP_TRY(dlp_ground_reach_async(n, indptr, indptr + 1, col, nullptr, DLP_F32, vmask, sink, umask, in_t, counts + 2,
                                 counts + 3, counts + 4, sub, sub_bytes, stream));
  k_sys_count<<<ceil_div_i(8LL * n, kSysThreads), kSysThreads, 0, s>>>(n, indptr, col, umask, flag, cnt);
  DLP_TRY(check_launch());
  DLP_TRY(exclusive_scan_i32(flag, n, loc, sub, sub_bytes, s));
  DLP_TRY(exclusive_scan_i32(cnt, n, pos, sub, sub_bytes, s));
  k_sys_sizes<<<1, 1, 0, s>>>(n, loc, pos, counts);
  return check_launch();
}

int dlp_build_system_fill(int32_t n, const int32_t *indptr, const int32_t *col, const void *w, int w_dtype,
                          const uint8_t *umask, const uint8_t *sink, const int32_t *y, int32_t K, double eta,
                          double prior, int32_t C, int32_t col0, const int32_t *loc, const int32_t *pos, int32_t n_u,
                          int64_t *U, int32_t *indptr_out, int32_t *col_out, void *w_out, int w_out_dtype, double *B,
                          double *s_, double *diag, double *rhs, double *rhsh, float *B32, float *s32, float *diag32,
                          float *rhs32, float *rhsh32, dlp_stream_t stream) {
  if (n <= 0 || n_u < 0 || K <= 0 || C <= 0 || col0 < 0 || col0 + C > K) return DLP_ERR_INVALID;
  if (!indptr || !col || !w || !umask || !sink || !y || !loc || !pos || !indptr_out) return DLP_ERR_INVALID;
  if ((w_dtype != DLP_F32 && w_dtype != DLP_F64) ||
      (w_out_dtype != DLP_F32 && w_out_dtype != DLP_F64 && w_out_dtype != DLP_BF16))
    return DLP_ERR_DTYPE;
  cudaStream_t s = (cudaStream_t)stream;
  // the last row pointer (the scan's total)
  DLP_CUDA(cudaMemcpyAsync(indptr_out + n_u, pos + n, sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
  if (n_u == 0) return DLP_OK;
  if (!U || !B || !s_ || !diag || !rhs || !rhsh) return DLP_ERR_INVALID;
  SysOut o{U, indptr_out, col_out, w_out, B, s_, diag, rhs, rhsh, B32, s32, diag32, rhs32, rhsh32};
  const int grid = ceil_div_i(8LL * n, kSysThreads);
#define DLP_SYS_FILL(TW, TO)                                                                                        \
  k_sys_fill<TW, TO><<<grid, kSysThreads, 0, s>>>(n, indptr, col, (const TW *)w, umask, sink, y, K, eta, prior, C, col0, \
                                                  loc, pos, o)
  if (w_dtype == DLP_F32) {
    if (w_out_dtype == DLP_F32) DLP_SYS_FILL(float, float);
    else if (w_out_dtype == DLP_F64) DLP_SYS_FILL(float, double);
    else DLP_SYS_FILL(float, bf16);
  } else {
    if (w_out_dtype == DLP_F32) DLP_SYS_FILL(double, float);
    else if (w_out_dtype == DLP_F64) DLP_SYS_FILL(double, double);
    else DLP_SYS_FILL(double, bf16);
  }
#undef DLP_SYS_FILL
  return check_launch();
}

}  // extern "C"
