"""Many independent harmonic solves in one launch sequence (no reference counterpart).

`BatchedSystems` concatenates grounded systems with the same column count into one block-
diagonal CSR, cuts the rows into tiles aligned to instance boundaries, and `solve` runs the
batched block PCG of libdlp (`dlp_pcg_batched`): every instance keeps its own CG scalars and stop
state, so its iterates are the ones it would have alone. DynLP+'s h column (A h = diag) rides
along. `autotune` picks the lane group and tile size of the batch by timing the apply kernel.

`solve_many(systems, ...)` groups arbitrary systems by column count and returns each one's
scores; the serving loop uses it to batch fresh-solve requests.
"""
from __future__ import annotations

import ctypes as ct
import time

import numpy as np
import torch

from . import _lib, kernels
from .backend import CSR, code, ld, ptr, stream, workspace
from .solvers import padded_empty

_TUNE: dict = {}


class BatchedSystems:
    def __init__(self, systems, tile_rows=1024, dtype=torch.float64, with_h=True):
        assert systems, "no systems"
        C = systems[0].C
        assert all(s.C == C for s in systems), "one column count per batch"
        self.systems, self.C, self.dtype = systems, C, dtype
        self.Ch = C + (1 if with_h else 0)
        dev = systems[0].diag.device
        self.dev = dev
        sizes = [s.n_u for s in systems]
        self.offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        N = int(self.offsets[-1])
        self.N = N
        nnzs = [s.W.nnz for s in systems]
        self.nnz = int(sum(nnzs))
        # concatenated as they are; one kernel then shifts the row pointers and columns of each block
        self.indptr = torch.cat([torch.zeros(1, dtype=torch.int32, device=dev)] + [s.W.indptr[1:].to(torch.int32) for s in systems])
        self.col = torch.cat([s.W.indices.to(torch.int32) for s in systems])
        self.w = torch.cat([s.W.data.float() for s in systems])
        B = len(systems)
        offs = np.zeros(2 * (B + 1), dtype=np.int32)
        offs[: B + 1] = self.offsets
        offs[B + 2:] = np.cumsum(nnzs)
        offs = torch.from_numpy(offs).to(dev)
        _lib.call("dlp_batch_offsets", B, ptr(offs), ptr(offs[B + 1:]), N, self.nnz, ptr(self.indptr), ptr(self.col),
                  stream())
        s64 = [s.astype(torch.float64) for s in systems]
        self.diag64 = torch.cat([s.diag for s in s64])
        self.diag = self.diag64.to(dtype)
        # from each system's own rhs and diag (its [rhs | diag] copy does not follow a replaced right-hand side)
        self.rhs64 = torch.empty((N, self.Ch), dtype=torch.float64, device=dev)
        self.rhs64[:, :self.C] = torch.cat([s.rhs for s in s64])  # (into the columns directly: a copy per system)
        if with_h:
            self.rhs64[:, self.C] = self.diag64
        self.rhs = self.rhs64.to(dtype)
        self.set_tiles(tile_rows)

    def set_tiles(self, tile_rows):
        """Cut every instance into tiles of up to tile_rows rows, fewer for small instances (some 128 tiles of at
        least 128 rows, up to 128 * tile_rows rows; beyond, the tiles' number grows): the batch then has enough
        tiles to fill the chip, and the cut depends on the instance alone, so it gets the same sums in every batch."""
        self.tile_rows = tile_rows
        sizes = np.diff(self.offsets)
        tr = np.full(sizes.shape[0], int(tile_rows), dtype=np.int64)
        want = np.maximum(128, 2 ** np.ceil(np.log2(np.maximum(sizes, 1) / 128.0)).astype(np.int64).clip(0, 62))
        tr = np.minimum(tr, want)
        count = -(-sizes // tr)
        toff = np.concatenate([[0], np.cumsum(count)])
        inst = np.repeat(np.arange(sizes.shape[0]), count)
        beg = self.offsets[inst] + (np.arange(inst.shape[0]) - toff[inst]) * tr[inst]
        end = np.minimum(beg + tr[inst], self.offsets[inst + 1])
        self.ntiles = int(inst.shape[0])
        m = max(self.ntiles, 1)
        host = np.zeros(3 * m + toff.shape[0], dtype=np.int32)  # one upload for the four arrays
        host[: self.ntiles], host[m: m + self.ntiles], host[2 * m: 2 * m + self.ntiles] = inst, beg, end
        host[3 * m:] = toff
        t = torch.from_numpy(host).to(self.dev)
        self.tinst, self.tbeg, self.tend, self.toff = t[: self.ntiles], t[m: m + self.ntiles], t[2 * m: 2 * m + self.ntiles], t[3 * m:]

    def col_stats(self, X):
        """(sums of squares, largest magnitudes) per instance and column of X (N x C), device B x C each."""
        B, C = len(self.systems), X.shape[1]
        out = torch.empty((B, 2, C), dtype=torch.float64, device=self.dev)
        ws = workspace("batch_stats").get(_lib.lib().dlp_batch_colstats_workspace_bytes(self.ntiles, C))
        _lib.call("dlp_batch_colstats", C, ptr(X), ld(X), code(X), B, self.ntiles, ptr(self.tinst), ptr(self.tbeg),
                  ptr(self.tend), ptr(self.toff), ptr(out), ptr(ws), ws.numel(), stream())
        return out

    def scale_rows(self, mode, X, scale, Y):
        """mode 0: Y = X / scale (fp32 of fp64); mode 1: Y += X * scale; scale per instance and column, zero: untouched."""
        _lib.call("dlp_batch_scale", mode, X.shape[1], ptr(X), ld(X), ptr(scale), ptr(Y), ld(Y), len(self.systems), self.ntiles,
                  ptr(self.tinst), ptr(self.tbeg), ptr(self.tend), stream())

    def csr(self) -> CSR:
        return CSR(self.w, self.col, self.indptr, (self.N, self.N))

    def autotune(self, candidates=((1, 512), (2, 512), (2, 1024), (4, 1024), (2, 2048)), reps=3):
        """Pick (edge lanes per row, tile rows) by timing the batch's SpMM on each candidate; cached
        per (rows, entries, columns)."""
        key = (self.N, self.nnz, self.Ch, self.dtype)
        if key in _TUNE:
            self.group, tr = _TUNE[key]
            self.set_tiles(tr)
            return self.group, tr
        X = padded_empty(self.N, self.Ch, self.dtype, self.dev, 1.0)
        best, arg = float("inf"), (0, self.tile_rows)
        for g, tr in candidates:
            self.set_tiles(tr)
            W = self.csr()
            Y = torch.empty((self.N, self.Ch), dtype=self.dtype, device=self.dev)
            kernels.spmm_axpy(W, X, a=self.diag, b=-1.0, out=Y, group=g)
            torch.cuda.current_stream().synchronize()
            t = time.perf_counter()
            for _ in range(reps):
                kernels.spmm_axpy(W, X, a=self.diag, b=-1.0, out=Y, group=g)
            torch.cuda.current_stream().synchronize()
            dt = (time.perf_counter() - t) / reps
            if dt < best:
                best, arg = dt, (g, tr)
        self.group = arg[0]
        self.set_tiles(arg[1])
        _TUNE[key] = arg
        return arg

    def solve(self, target_relres=1e-6, eps=None, max_iter=100_000, patience=400, check_every=8, use_graph=True,
              group=None, Z0=None, inst_targets=None):
        """Solve every instance; returns (Z (N x Ch), iters, status, relres) with per-instance arrays."""
        B, Ch, N, dev, dt = len(self.systems), self.Ch, self.N, self.dev, self.dtype
        Z = padded_empty(N, Ch, dt, dev)
        if Z0 is not None:
            Z.copy_(Z0)
        R = torch.empty((N, Ch), dtype=dt, device=dev)
        P = padded_empty(N, Ch, dt, dev, 0.0)
        AP = padded_empty(N, Ch, dt, dev)  # rows padded like P's: the apply writes them whole
        # per-instance column norms of the right-hand side (fp64); the h column only needs a loose solve
        rn = self.col_stats(self.rhs)[:, 0].sqrt()
        if Ch > self.C:
            rn[:, self.C:] *= 1e3
        rn = torch.where(rn > 0, rn, torch.ones_like(rn))
        if inst_targets is not None:  # instance i stops at ||R_c|| <= inst_targets[i] ||rhs_c||
            t = torch.as_tensor(np.asarray(inst_targets, dtype=np.float64) / target_relres, device=dev)
            rn = rn * t[:, None]
        rn = rn.contiguous()
        mode = 2 if Z0 is not None else 6  # from zero: no residual to compute
        epsd = torch.full((B, Ch), 1e300, dtype=torch.float64, device=dev)
        if eps is not None:
            mode |= 1
            epsd[:] = torch.as_tensor(eps, dtype=torch.float64, device=dev)
        ws = workspace("batched").get(_lib.lib().dlp_pcg_batched_workspace_bytes(B, self.ntiles, Ch))
        iters = (ct.c_int32 * B)()
        status = (ct.c_int32 * B)()
        rel = (ct.c_double * B)()
        g = self.group if group is None and hasattr(self, "group") else (group or 0)
        _lib.call("dlp_pcg_batched", ptr(self.indptr), ptr(self.col), ptr(self.w), N, Ch, ptr(self.diag), ptr(self.rhs),
                  ld(self.rhs), ptr(Z), ld(Z), ptr(R), ld(R), ptr(P), ld(P), ptr(AP), ld(AP), code(Z), B, self.ntiles,
                  ptr(self.tinst), ptr(self.tbeg), ptr(self.tend), ptr(self.toff), ptr(epsd), ptr(rn),
                  float(target_relres), mode, int(max_iter), int(patience), int(check_every), int(bool(use_graph)),
                  int(g), self.nnz / max(N, 1), ptr(ws), ws.numel(), iters, status, rel, stream())
        return Z, np.array(iters), np.array(status), np.array(rel)

    def split(self, Z):
        """Per-instance score blocks (views)."""
        return [Z[a:b, : self.C] for a, b in zip(self.offsets[:-1], self.offsets[1:])]


def solve_many(systems, target_relres=1e-6, dtype=torch.float64, tile_rows=1024, autotune=False):
    """Solve independent systems in batches grouped by column count; returns F per system (in order)
    and per-system (iterations, status, relative residual)."""
    out = [None] * len(systems)
    info = [None] * len(systems)
    by_c: dict = {}
    for i, s in enumerate(systems):
        by_c.setdefault(s.C, []).append(i)
    for C, idx in by_c.items():
        bs = BatchedSystems([systems[i] for i in idx], tile_rows=tile_rows, dtype=dtype)
        if autotune:
            bs.autotune()
        Z, it, stt, rel = bs.solve(target_relres=target_relres)
        for j, F in zip(idx, bs.split(Z)):
            out[j] = F
        for k, j in enumerate(idx):
            info[j] = (int(it[k]), int(stt[k]), float(rel[k]))
    return out, info


def solve_many_mixed(systems, target_relres=1e-6, tile_rows=1024, rounds=6, autotune=False, inner=1e-4):
    """solve_many in mixed precision: the batched PCG sweeps run in fp32 and the accuracy is won back
    by refinement against the fp64 residual (dynlp/solvers.py:322-337 applied to the batch): after a
    solve from zero, every round computes R = rhs - A Z in fp64 for all instances at once, stops when
    every instance's relative residual meets the target, and otherwise solves A D = R / scale in fp32
    and adds D * scale. The scale (column maxima of R) and the correction's target are each
    instance's own, so an instance's result does not depend on the others in its batch (autotune: the
    rows-per-warp and tile shape of the fp32 sweeps picked by BatchedSystems.autotune; inner: the
    smallest relative residual asked of one fp32 solve). Returns F per system and (iterations,
    status, relative residual) per system."""
    out, info = [None] * len(systems), [None] * len(systems)
    by_c: dict = {}
    for i, s in enumerate(systems):
        by_c.setdefault(s.C, []).append(i)
    for C, idx in by_c.items():
        group = [systems[i] for i in idx]
        bs = BatchedSystems(group, tile_rows=tile_rows, dtype=torch.float32)
        if autotune:
            bs.autotune()
        dev, N, Ch, B = bs.dev, bs.N, bs.Ch, len(group)
        diag64, rhs64 = bs.diag64, bs.rhs64
        A = CSR(bs.w, bs.col, bs.indptr, (N, N))
        spans = list(zip(bs.offsets[:-1], bs.offsets[1:]))
        rhs_n = bs.col_stats(rhs64)[:, 0, :C].sqrt()
        rhs_n = torch.where(rhs_n > 0, rhs_n, torch.ones_like(rhs_n))
        Z64 = padded_empty(N, Ch, torch.float64, dev, 0.0)
        # the fp32 solves aim no lower than `inner`: below their precision floor (about 1e-6 of
        # ||rhs|| on these systems, lower for some) a solve only stalls until its patience runs out
        Zf, it, _, _ = bs.solve(target_relres=max(target_relres, inner))
        Z64.copy_(Zf)
        iters = it.astype(np.int64)
        rel = np.zeros(B)
        rhs32 = torch.empty((N, Ch), dtype=torch.float32, device=dev)
        for rnd in range(rounds + 1):
            R64 = kernels.spmm_axpy(A, Z64, a=diag64, alpha=-1.0, b=1.0, rhs=rhs64, out=padded_empty(N, Ch, torch.float64, dev))
            st = bs.col_stats(R64)
            rel_d = (st[:, 0, :C].sqrt() / rhs_n).amax(dim=1)
            rel = rel_d.cpu().numpy()
            if (rel <= target_relres).all() or rnd == rounds:
                break
            sc = torch.where(st[:, 1] > 0, st[:, 1], torch.ones_like(st[:, 1])).contiguous()
            bs.scale_rows(0, R64, sc, rhs32)
            bs.rhs = rhs32
            # each instance's correction brings its residual to a fifth of the target, or by `inner`
            # when that is further than one fp32 solve safely resolves (another round follows)
            need = [max(0.2 * target_relres / max(r, 1e-300), inner) for r in rel]
            D, it2, _, _ = bs.solve(target_relres=target_relres, inst_targets=need)
            # a converged instance keeps its scores (same as alone)
            bs.scale_rows(1, D, torch.where(rel_d[:, None] > target_relres, sc, torch.zeros_like(sc)).contiguous(), Z64)
            iters += np.where(rel > target_relres, it2, 0)
        for k, j in enumerate(idx):
            a, b = spans[k]
            out[j] = Z64[a:b, :C]
            info[j] = (int(iters[k]), 5 if rel[k] <= target_relres else 2, float(rel[k]))
    return out, info
