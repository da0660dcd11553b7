"""What the fast paths take besides plain calls: layouts, types, limits and inputs that are refused."""
import dataclasses

import numpy as np
import pytest
import torch

from dynlplus_b200 import amg, batched, cc, graphs, kernels, solvers, stream
from dynlplus_b200.backend import CSR

pytestmark = pytest.mark.gpu


def labelled_graph(n=3000, K=3, seed=1, weights="lognormal"):
    ds = graphs.planted_partition(n, K, 12, 4, weights=weights, seed=seed)
    return ds, torch.as_tensor(graphs.label_mask(n, 0.05, seed=seed)).cuda()


def same_system(a, b):
    assert a.n_u == b.n_u > 0 and torch.equal(a.U, b.U)
    for x, y in ((a.W.indptr, b.W.indptr), (a.W.indices, b.W.indices), (a.W.data, b.W.data)):
        assert torch.equal(x, y)
    for name in ("s", "diag", "B", "rhs", "rhs_h"):
        assert torch.equal(getattr(a, name), getattr(b, name))
    assert (a.n_active, a.n_ungrounded) == (b.n_active, b.n_ungrounded)


@pytest.mark.parametrize("layout", ["columns", "expanded", "other types"])
def test_build_system_takes_masks_of_any_layout(layout):
    """Masks that are columns of one matrix, expanded or of another type give the system of their plain copies."""
    ds, lab = labelled_graph()
    on = torch.ones_like(lab)
    want = stream.build_system(ds, on, lab)
    if layout == "columns":
        M = torch.stack([on, lab], 1)
        a, b = M[:, 0], M[:, 1]
    elif layout == "expanded":
        a, b = torch.ones(1, dtype=torch.bool, device="cuda").expand(ds.n), torch.stack([lab, lab], 1)[:, 1]
    else:
        a, b = on.to(torch.int64), torch.stack([lab, lab], 1).to(torch.float32)[:, 0]
    same_system(stream.build_system(ds, a, b), want)


@pytest.mark.parametrize("wdtype", ["float32", "float64"])
@pytest.mark.parametrize("K,eta", [(2, 0.0), (5, 0.3)])
def test_bf16_system_rounds_its_operator_only(K, eta, wdtype):
    """The label weights (B, s, rhs) of a bf16 system come from the weights as they are, in its fp64 twin to
    fp64 rounding; the operator's entries are the rounded ones and the diagonal has their row sums."""
    from oracle import ref_np as O
    n = 1003
    ds = graphs.er_graph(n, 9, K, weights="lognormal", seed=K, dtype=wdtype)
    lab = np.random.default_rng(K).random(n) < 0.2
    on = torch.ones(n, dtype=torch.bool, device="cuda")
    S = stream.build_system(ds, on, torch.as_tensor(lab).cuda(), dtype="bfloat16", eta=eta)
    want = O.build_system(ds.A.to_scipy(), ds.y.cpu().numpy(), K, np.ones(n, bool), lab, eta=eta)
    T = S.astype(torch.float64)
    assert np.array_equal(S.U.cpu().numpy(), want["U"])
    w = torch.as_tensor(want["W"].data).to(torch.bfloat16)
    assert torch.equal(S.W.data.cpu(), w) and np.array_equal(S.W.indices.cpu().numpy(), want["W"].indices)
    rowsum = np.add.reduceat(np.append(w.double().numpy(), 0.0), want["W"].indptr[:-1]) * (np.diff(want["W"].indptr) > 0)
    for name, ref in (("s", want["s"]), ("B", want["B"]), ("rhs", want["rhs"]), ("diag", want["s"] + rowsum)):
        got = getattr(T, name).cpu().numpy()
        np.testing.assert_allclose(got, ref, rtol=1e-13, atol=1e-13)
        low = getattr(S, name)
        assert low.dtype == torch.bfloat16 and torch.equal(low, getattr(T, name).to(torch.bfloat16))


@pytest.mark.parametrize("with_h", [True, False])
def test_batch_takes_each_systems_own_right_hand_side(with_h):
    """Systems whose right-hand side was replaced (their [rhs | diag] copy was not) are solved for the new one:
    the batch holds it, and the scores are those of the scaled system."""
    ds, lab = labelled_graph()
    S = stream.build_system(ds, torch.ones_like(lab), lab, dtype="float64")
    T = dataclasses.replace(S, rhs=2 * S.rhs, _conv={})
    bs = batched.BatchedSystems([S, T, S], with_h=with_h)
    h = [S.diag[:, None]] if with_h else []
    assert torch.equal(bs.rhs, torch.cat([torch.cat([x.rhs, *h], 1) for x in (S, T, S)]))
    for solve in (batched.solve_many, batched.solve_many_mixed):
        (a, b), _ = solve([S, T], target_relres=1e-8)
        for sys, F in ((S, a), (T, b)):
            R = solvers.residual(sys, F.contiguous(), sys.rhs)
            assert float((R.norm(dim=0) / sys.rhs.norm(dim=0)).max()) <= 1.01e-8


def random_csr(n, deg, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    col = torch.randint(0, n, (n * deg,), generator=g, device="cuda").to(torch.int32)
    ip = torch.arange(0, n * deg + 1, deg, device="cuda").to(torch.int32)
    return CSR(torch.rand(n * deg, generator=g, device="cuda"), col, ip, (n, n))


def test_captured_product_keeps_its_scratch():
    """A product whose odd rows go through scratch, captured into a graph: replayed after a larger one has run and
    the memory it left was taken, it gives the product of the values X then holds and writes nothing else."""
    n, C = 60_000, 17
    W, X = random_csr(n, 16, 0), torch.rand((n, C), device="cuda")
    Y = torch.empty_like(X)
    kernels.spmm_axpy(W, X, out=Y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        kernels.spmm_axpy(W, X, out=Y)
    V, U = random_csr(2 * n, 16, 1), torch.rand((2 * n, C), device="cuda")
    kernels.spmm_axpy(V, U)
    taken = [torch.full((1 << 20,), 7.0, device="cuda") for _ in range(16)]
    X.uniform_(0, 1)
    want = kernels.spmm_axpy(W, X)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(Y, want)
    assert all(bool((t == 7.0).all()) for t in taken)


def test_product_without_room_for_its_scratch(monkeypatch):
    """Where the scratch for odd rows cannot be allocated the product gathers them as they are: fp64 product of
    the same values within the roundoff of 16 terms in [0, 1)."""
    n, C = 60_000, 17
    W, X, Y = random_csr(n, 16, 0), torch.rand((n, C), device="cuda"), torch.empty((n, C), device="cuda")
    empty = torch.empty

    def full(*size, **kw):
        if kw.get("dtype") == torch.uint8:
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **kw)
    monkeypatch.setattr(torch, "empty", full)
    kernels.spmm_axpy(W, X, out=Y)
    monkeypatch.undo()
    want = kernels.spmm_axpy(CSR(W.data.double(), W.indices, W.indptr, W.shape), X.double())
    assert float((Y.double() - want).abs().max()) <= 16 * 16 * 2.0 ** -24


@pytest.mark.parametrize("cap", [0, 2.5, 2**31 - 1, 2**31, 2**33 + 5, float("inf")])
def test_frontier_solve_takes_any_cap(cap):
    """The number of rounds of the device loop under caps beyond an int32, infinite and fractional, against the host
    loop's."""
    n = 3000
    ds, lab = labelled_graph(n)
    S = stream.build_system(ds, torch.ones_like(lab), lab)
    a, b = (solvers.DynLP(n, 3, max_iter=cap) for _ in range(2))
    sa, sb = a.solve(S), b.solve(S, record=[])
    assert sa.iters == sb.iters and torch.equal(a.F, b.F) and (sa.iters > 100 or cap < 3)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_build_system_refuses_masks_and_labels_of_another_length(dtype):
    ds, lab = labelled_graph(1000)
    on = torch.ones_like(lab)
    for m in (0, 2, 999, 1001):
        long = torch.ones(m, dtype=torch.bool, device="cuda")
        for a, b in ((long, lab), (on, long), (long, long)):
            with pytest.raises(RuntimeError):
                stream.build_system(ds, a, b, dtype=dtype)
    with pytest.raises(RuntimeError):
        stream.build_system(ds, on[:, None], lab, dtype=dtype)
    short = graphs.Dataset("x", ds.A, ds.y[:999], ds.K, ds.order)
    with pytest.raises(IndexError):
        stream.build_system(short, on, lab, dtype=dtype)
    # one flag for all, and labels beyond the graph's vertices, are taken as before
    want = stream.build_system(ds, on, lab, dtype=dtype)
    more = graphs.Dataset("x", ds.A, torch.cat([ds.y, ds.y[:5]]), ds.K, ds.order)
    same_system(stream.build_system(more, on[:1], lab, dtype=dtype), want)


@pytest.mark.parametrize("m", [3, 2000])
def test_fh_components_checks_its_edges(m):
    """Edge ends, weights and grounding of other lengths and ends outside [0, m) are refused; ends counted from the
    last vertex are taken as indices are."""
    g = torch.Generator(device="cuda").manual_seed(m)
    u = torch.randint(0, m - 1, (4 * m,), generator=g, device="cuda")
    v = (u + 1 + torch.randint(0, m - 1, (4 * m,), generator=g, device="cuda")) % m
    rows, cols = torch.cat([u, v]), torch.cat([v, u])
    d = torch.rand(4 * m, generator=g, device="cuda").repeat(2)
    ground = (torch.arange(m, device="cuda") % 7 == 0).float()
    want, nc = cc.fh_components(m, rows, cols, d, 0.3, ground)
    lab, n2 = cc.fh_components(m, rows - m, torch.where(cols % 2 == 0, cols - m, cols), d, 0.3, ground)
    assert n2 == nc and torch.equal(lab, want)
    for a, b, c, gr in ((rows, cols[:-1], d, ground), (rows, cols, d[:1], ground), (rows, cols, d, ground[:-1]),
                        (rows, cols, torch.cat([d, d]), None), (rows, cols, d, torch.cat([ground, ground]))):
        with pytest.raises(IndexError):
            cc.fh_components(m, a, b, c, 0.3, gr)
    for side in (0, 1):
        for value in (m, -m - 1, 2**31 - 1):
            ends = [rows.clone(), cols.clone()]
            ends[side][-1] = value
            with pytest.raises(IndexError):
                cc.fh_components(m, *ends, d, 0.3, ground)


@pytest.mark.parametrize("end", [2**32 + 1, -2**32 + 1, 2**31, 2**63 - 1])
def test_fh_components_refuses_ends_past_int32(end):
    rows, cols = torch.tensor([[0, 1, 0, 2], [1, 0, 2, 0]], device="cuda")
    cols[0] = end
    with pytest.raises(IndexError):
        cc.fh_components(3, rows, cols, torch.ones(4, device="cuda"), 0.5)


@pytest.mark.parametrize("first", [0.0, -0.0])
def test_fh_components_takes_both_zeros_as_equal(first):
    """Of two lightest edges, one of weight 0 and one of weight -0, the one to the smaller component is taken."""
    rows, cols = torch.tensor([[0, 1, 0, 2], [1, 0, 2, 0]], device="cuda")
    d = torch.tensor([first, first, -first, -first], device="cuda")
    lab, nc = cc.fh_components(3, rows, cols, d, -1.0, torch.tensor([0.0, 1.0, 1.0], device="cuda"))
    assert nc == 2 and lab.tolist() == [0, 0, 1]


LOST_WAIT = r"""
#include "cc.cu"
// The grounding kernel as it is launched, on two blocks, with its barrier's `abort` set beforehand: a block that has to
// wait gives up after its first 1,024 polls, the block that arrives last finds every arrival and passes.
extern "C" int lost_wait(int32_t n, const int32_t *rbeg, const int32_t *rend, const int32_t *col, const float *w,
                         const uint8_t *vmask, const uint8_t *sink, uint8_t *umask, uint8_t *in_t, int32_t *count,
                         int32_t *err, int32_t *info, uint8_t *reached, int32_t *flags, int32_t *parent, GridBar *bar) {
  GridBar b{};
  b.abort = 1;
  cudaMemcpy(bar, &b, sizeof(b), cudaMemcpyHostToDevice);
  void *args[] = {&n,     &rbeg, &rend,  &col, &w,    &vmask,   &sink,  &reached,
                  &flags, &parent, &umask, &in_t, &count, &err, &info, &bar};
  const void *kern = (const void *)k_ground_whole<float>;
  cudaError_t e = cudaLaunchCooperativeKernel(kern, dim3(2), dim3(kGroundThreads), args, 0, nullptr);
  return e != cudaSuccess ? (int)e : (int)cudaDeviceSynchronize();
}
"""


def test_a_wait_lost_in_any_block_is_reported(tmp_path):
    """Block 1 of the grounding gives up at the only barrier of a run, block 0 (it has one long row) passes and
    writes its rows: the run says that a wait was lost, since block 1's rows are missing."""
    import ctypes as ct
    import subprocess
    from dynlplus_b200 import _lib, build
    from dynlplus_b200.backend import ptr
    _lib.lib()
    src, so = tmp_path / "lost_wait.cu", tmp_path / "lost_wait.so"
    src.write_text(LOST_WAIT)
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", "-cudart", "static", str(src), "-o", str(so),
                    build.LIB], check=True)
    n, m = 2048, 200_000
    rend = torch.full((n,), m, dtype=torch.int32, device="cuda")
    rbeg = rend.clone()
    rbeg[0] = 0  # row 0 has all the entries, none of them to a reached vertex
    col = torch.full((m,), 5, dtype=torch.int32, device="cuda")
    i32, u8 = (lambda k: torch.zeros(k, dtype=torch.int32, device="cuda")), (lambda k: torch.zeros(k, dtype=torch.uint8, device="cuda"))
    vmask, sink, umask, in_t, w = u8(n) + 1, u8(n), u8(n) + 1, u8(n), torch.ones(m, device="cuda")
    count, err, info, reached, flags, parent, bar = i32(1), i32(1), i32(4), u8(n), i32(64), i32(n + 1), i32(64)
    torch.cuda.synchronize()
    args = [ct.c_void_p(ptr(t)) for t in (rbeg, rend, col, w, vmask, sink, umask, in_t, count, err, info, reached, flags,
                                          parent, bar)]
    assert ct.CDLL(str(so)).lost_wait(ct.c_int32(n), *args) == 0
    assert int(umask[:1024].sum()) == 0 and int(umask[1024:].sum()) == 1024  # block 0 finished, block 1 did not
    assert int(info[3]) == 1


@pytest.mark.parametrize("call", ["grounding", "frontier", "push"])
def test_a_hub_keeps_the_other_blocks_waiting(call):
    """A vertex of 8 million neighbours, whose row one thread or lane group walks for seconds while every other block
    waits at the barrier: the wait is as long as the row, and the result is the star graph's."""
    n = 8_000_000
    ip = torch.cat([torch.zeros(1, dtype=torch.int32, device="cuda"), torch.arange(n - 1, 2 * n - 1, device="cuda").to(torch.int32)])
    col = torch.cat([torch.arange(1, n, device="cuda"), torch.zeros(n - 1, dtype=torch.int64, device="cuda")]).to(torch.int32)
    A = CSR(torch.ones(2 * n - 2, device="cuda"), col, ip, (n, n))
    hub = torch.zeros(1, dtype=torch.int32, device="cuda")
    diag = torch.full((n,), 2.0, dtype=torch.float64, device="cuda")
    diag[0] = n
    if call == "grounding":  # the hub's last neighbour is the only labelled vertex
        sink = torch.zeros(n, dtype=torch.uint8, device="cuda")
        sink[-1] = 1
        umask, in_t = torch.zeros_like(sink), torch.zeros_like(sink)
        assert cc.ground_reach(A, 1 - sink, sink, umask, in_t)[0] == n - 1
        assert torch.equal(umask, 1 - sink)
    elif call == "frontier":  # the hub moves to (n - 1) / 2 / n, then the leaves to half of it
        X = torch.full((n, 1), 0.5, dtype=torch.float64, device="cuda")
        rounds = kernels.FrontierOps(A, 1).solve(hub, X, torch.zeros_like(X), diag, 1e-9, 2)
        assert rounds == 2 and abs(float(X[0, 0]) - 0.5 * (n - 1) / n) <= 1e-9
        assert float((X[1:] - 0.25).abs().max()) <= 1e-6
    else:  # the hub's residual n becomes a score of 1 and a residual of 1 at every leaf
        Z, R = torch.zeros((n, 1), dtype=torch.float64, device="cuda"), torch.zeros((n, 1), dtype=torch.float64, device="cuda")
        R[0] = float(n)
        rounds, ok, edges = kernels.FusedPush(A, 1).run(Z, R, diag, [0.9], hub, 5)
        assert (rounds, ok, edges) == (1, True, n - 1) and float(Z[0, 0]) == 1.0
        assert bool((R[1:] == 1.0).all()) and float(R[0, 0]) == 0.0


@pytest.mark.parametrize("n,K,weights", [(10_000, 8, "unit"), (60_000, 8, "unit"), (20_000, 8, "lognormal"), (30_000, 12, "lognormal"),
                                         (50_000, 5, "lognormal")])
def test_violation_stops_near_the_fp32_floor(n, K, weights):
    """fp32 solves that stop by the violation rule alone and recheck themselves, down to 6e-8: the device-side loop
    takes the host loop's iterations and its iterate has the same violation (a failed recheck does not cost it)."""
    ds = graphs.planted_partition(n, K, 12, 4, weights=weights, seed=3)
    lab = torch.as_tensor(graphs.label_mask(n, 0.01, seed=3)).cuda()
    S = stream.build_system(ds, torch.ones_like(lab), lab)
    S64 = S.astype(torch.float64)
    for eps in (1e-5, 1.2e-7, 6e-8):
        out = []
        for graph in (True, False):
            Z, st = solvers.padded_empty(S.n_u, K, torch.float32, "cuda", fill=0.0), solvers.Stats()
            solvers.pcg(S, Z, S.rhs, [eps] * K, solvers.jacobi_M(S), 3000, st, use_graph=graph)
            R = solvers.residual(S64, Z.double().contiguous(), S64.rhs)
            out.append((st.iters, float(solvers.rho_cols(S64, R).max()) / eps))
        assert out[0] == out[1] and out[0][1] <= 2.0


@pytest.mark.parametrize("rule", ["relres", "violation"])
@pytest.mark.parametrize("n,K", [(3000, 2), (3000, 3), (20_000, 4), (3000, 16)])
def test_solves_beyond_their_precision_keep_the_launched_loop(n, K, rule):
    """A solve that rechecks its stops and is asked for less than fp32 resolves ends where the launched kernels end, bit
    for bit: the sums of the one launch drift further before its patience ends."""
    ds = graphs.er_graph(n, 10, K, seed=n + K)
    S = stream.build_system(ds, torch.ones(n, dtype=torch.bool, device="cuda"),
                            torch.as_tensor(graphs.label_mask(n, 0.02, seed=n)).cuda(), dtype="float32")
    eps, target = ([1e-7] * S.C, None) if rule == "violation" else (None, 1e-6)
    out = []
    for use_graph in (None, False):
        Z, st = solvers.padded_empty(S.n_u, S.C, torch.float32, "cuda", fill=0.5), solvers.Stats()
        solvers.pcg(S, Z, S.rhs.contiguous(), eps, solvers.jacobi_M(S), 100_000, st, target_relres=target,
                    use_graph=use_graph)
        out.append((st.iters, Z.clone()))
    assert out[0][0] == out[1][0] and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("K,dtype", [(3, "float32"), (8, "float64")])
def test_batched_alpha_is_folded_once_for_many_tiles(K, dtype):
    """Instances of 1,024 and 1,025 tiles (where the alphas change from a fold in every tile's block to one of their
    own): each beside a small instance is bit for bit what it is alone, and from 1,025 tiles on an iteration has one
    more launch, so that no block but one reads all tiles' sums."""
    from dynlplus_b200 import _lib
    dt = getattr(torch, dtype)

    def system(n):  # n rows, all grounded: degree 24 leaves no vertex alone
        ds = graphs.er_graph(n + 1, 24, K, seed=n)
        return stream.build_system(ds, torch.ones(n + 1, dtype=torch.bool, device="cuda"),
                                   torch.arange(n + 1, device="cuda") == n, dtype="float64", eta=0.5)
    small, launches = system(500), []
    for n in (1024, 1025):
        S = system(n)
        alone = batched.BatchedSystems([S], tile_rows=1, dtype=dt)
        both = batched.BatchedSystems([small, S], tile_rows=1, dtype=dt)
        assert alone.ntiles == n
        before = _lib.lib().dlp_launch_count()
        Z, it, status, _ = alone.solve(target_relres=1e-5, check_every=64)  # one chunk of 64 iterations, then a recheck
        launches.append(_lib.lib().dlp_launch_count() - before)
        Z2, it2, status2, _ = both.solve(target_relres=1e-5, check_every=64)
        assert status[0] == 5 and (status2 == 5).all() and it[0] == it2[1] < 64
        assert torch.equal(Z2[both.offsets[1]:], Z)
    assert launches[1] - launches[0] == 64


@pytest.mark.parametrize("n", [300, 1928, 1929, 2100])
def test_dense_inverse_is_queued_and_captured(n):
    """The in-place inverse in one launch (up to 1,928 rows here) and with two launches a pivot, as it runs and
    replayed from a captured graph, against numpy: n unit roundoffs times a condition number of at most 41."""
    from dynlplus_b200 import _lib
    from dynlplus_b200.backend import ptr
    from dynlplus_b200.backend import stream as cur
    rng = np.random.default_rng(n)
    A = rng.uniform(-1, 0, (n, n))
    A = (A + A.T) / 2
    np.fill_diagonal(A, 0)
    A[np.arange(n), np.arange(n)] = np.abs(A).sum(1) * 1.05 + 0.01
    want = np.linalg.inv(A)
    tol = n * 2.3e-16 * 41 * np.abs(want).max()
    A = torch.as_tensor(A).cuda()
    D = A.clone()
    ws = torch.empty(_lib.lib().dlp_dense_spd_inverse_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    _lib.call("dlp_dense_spd_inverse", n, ptr(D), ptr(ws), ws.numel(), cur())
    assert np.abs(D.cpu().numpy() - want).max() <= tol
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _lib.call("dlp_dense_spd_inverse", n, ptr(D), ptr(ws), ws.numel(), cur())
    for _ in range(2):
        D.copy_(A)
        g.replay()
        assert np.abs(D.cpu().numpy() - want).max() <= tol


@pytest.mark.parametrize("shape", ["path", "reversed path", "two paths", "grid", "star", "binary tree"])
@pytest.mark.parametrize("shuffled", [False, True])
def test_components_of_long_and_narrow_graphs(shape, shuffled):
    """Edge lists whose components take more rounds than are run (the unions join the rest) and those of a few, with
    vertices in order and in random order, against SciPy; tails of isolated vertices."""
    import scipy.sparse as ssp
    from scipy.sparse.csgraph import connected_components
    n, k = 700_000, np.arange(600_000)
    if shape == "path":
        u, v = k[:-1], k[1:]
    elif shape == "reversed path":
        u, v = k[::-1][:-1], k[::-1][1:]
    elif shape == "two paths":
        u, v = k[:-2], k[2:]
    elif shape == "grid":
        s = 770
        g = np.arange(s * s)
        u, v = np.r_[g[g % s < s - 1], g[: s * (s - 1)]], np.r_[g[g % s < s - 1] + 1, g[: s * (s - 1)] + s]
    elif shape == "star":
        u, v = np.full(k.size - 1, k.size - 1), k[:-1]
    else:
        u, v = k[1:], (k[1:] - 1) // 2
    rng = np.random.default_rng(0)
    if shuffled:
        p = rng.permutation(n)
        u, v = p[u], p[v]
    _, want = connected_components(ssp.coo_matrix((np.ones(len(u)), (u, v)), (n, n)), directed=False)
    first = np.full(want.max() + 1, n)
    np.minimum.at(first, want, np.arange(n))
    want = np.argsort(np.argsort(first))[want]
    lab, nc = cc.connected_components(n, torch.as_tensor(u.astype(np.int32)).cuda(), torch.as_tensor(v.astype(np.int32)).cuda())
    assert nc == want.max() + 1 and np.array_equal(lab.cpu().numpy(), want)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float64"])
@pytest.mark.parametrize("deg", [3, 7, 9, 47, 49])
def test_spmm_layouts_by_degree(deg, dtype):
    """Products on both sides of the degrees where the lane layout changes (8 and 48), at the widths that change it,
    for rows on a vector pitch, packed rows and an offset view, with the library's entry slots and a given number,
    against the same product in fp64: unit roundoff of the accumulation times the row's length and weight sum."""
    n, dt = 3001, getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(deg)
    W = random_csr(n, deg, deg)
    W = CSR(W.data.to(dt), W.indices, W.indptr, W.shape)
    W64 = CSR(W.data.double(), W.indices, W.indptr, W.shape)
    a = torch.rand(n, generator=g, device="cuda").to(torch.float32 if dtype == "bfloat16" else dt)
    tol = (deg + 2) ** 2 * (2.0 ** -53 if dtype == "float64" else 2.0 ** -24)
    for C in (3, 4, 6, 16, 17, 32, 34, 48, 63, 64):
        base = torch.rand((n, C + 8), generator=g, device="cuda").to(dt)
        padded = solvers.padded_empty(n, C, dt, "cuda", 0.0)
        padded.copy_(base[:, :C])
        for X in (padded, base[:, :C].contiguous(), base[:, 1:C + 1]):
            want = kernels.spmm_axpy(W64, X.double(), a=a.double(), b=-1.0, group=1)
            for group in ("auto", 1, 4):
                Y = kernels.spmm_axpy(W, X, a=a, b=-1.0, group=group)
                assert float((Y.double() - want).abs().max()) <= tol


@pytest.mark.parametrize("count", [199_999, 200_000])
def test_push_rounds_of_many_candidates_are_launched(count):
    """On both sides of the number of candidates from which rounds are launched: the launches say which form ran, and
    both forms' rounds, edge visits and results equal those of the rounds launched on request."""
    from dynlplus_b200 import _lib
    n, C = 210_000, 2
    ds = graphs.er_graph(n, 6, 4, seed=2)
    lab = torch.as_tensor(graphs.label_mask(n, 0.02, seed=2)).cuda()
    S = stream.build_system(ds, torch.ones_like(lab), lab, dtype="float64")
    cand = torch.arange(count, dtype=torch.int32, device="cuda")
    g = torch.Generator().manual_seed(0)
    base = torch.rand((S.n_u, C), generator=g, dtype=torch.float64).cuda()
    out = []
    for whole in (True, False):
        Z, R = torch.zeros_like(base), base.clone()
        before = _lib.lib().dlp_launch_count()
        rounds, ok, edges = kernels.FusedPush(S.W, C).run(Z, R, S.diag, [5e-2] * C, cand, 12, use_graph=whole)
        out.append((_lib.lib().dlp_launch_count() - before, rounds, edges, Z, R))
    (la, ra, ea, za, xa), (lb, rb, eb, zb, xb) = out
    assert (ra, ea) == (rb, eb) and ra >= 2
    assert (la == 1) == (count < 200_000) and (la == lb) == (count >= 200_000)
    # every value is a sum of at most 64 rounded terms a round, each no larger than the largest score times its weight
    lim = 64 * ra * 2.0 ** -53 * float(S.diag.max()) * float(za.abs().max())
    assert float((za - zb).abs().max()) <= lim and float((xa - xb).abs().max()) <= lim


@pytest.mark.parametrize("shape,n,sinks", [("path", 3000, 1), ("path", 200_000, 3), ("grid", 40_000, 1), ("grid", 250_000, 2),
                                           ("shuffled grid", 40_000, 1), ("shuffled path", 30_000, 2)])
def test_grounding_that_sweeps_do_not_settle(shape, n, sinks):
    """Long graphs, in order and shuffled, with inert entries that cut parts off and vertices outside the mask: the
    grounded set, its changes and counts against SciPy's components, and the union-find did finish it."""
    import scipy.sparse as ssp
    from scipy.sparse.csgraph import connected_components
    rng = np.random.default_rng(n)
    k = np.arange(n)
    if "path" in shape:
        u, v = k[:-1], k[1:]
    else:
        s = int(round(n ** 0.5))
        u = np.r_[k[k % s < s - 1], k[: s * (s - 1)]]
        v = np.r_[k[k % s < s - 1] + 1, k[: s * (s - 1)] + s]
    ends = np.sort(rng.choice(n, sinks, replace=False))
    cut = rng.random(len(u)) < (0.3 / n ** 0.5 if "path" in shape else 0.05)
    if shape.startswith("shuffled"):
        p = rng.permutation(n)
        u, v, ends = p[u], p[v], p[ends]
    A = ssp.coo_matrix((np.where(cut, 2.0, 1.0).astype(np.float32), (u, v)), (n, n)).tocsr()
    A = (A + A.T).tocsr()
    W = CSR.from_scipy(A)
    W.data[W.data == 2.0] = 0.0  # stored, inert
    sink = np.zeros(n, np.uint8)
    sink[ends] = 1
    vmask = 1 - sink
    vmask[rng.integers(0, n, 3)] = 0
    live = ssp.coo_matrix((np.ones((~cut).sum()), (u[~cut], v[~cut])), (n, n)).tocoo()
    r, c = np.r_[live.row, live.col], np.r_[live.col, live.row]
    keep = (vmask[r] > 0) & ((vmask[c] > 0) | (sink[c] > 0))
    _, lab = connected_components(ssp.coo_matrix((np.ones(keep.sum()), (r[keep], np.where(vmask[c[keep]] > 0, c[keep], n))),
                                                 (n + 1, n + 1)), directed=False)
    want = (vmask > 0) & (lab[:n] == lab[n])
    old = rng.random(n) < 0.5
    T = lambda x: torch.as_tensor(x.astype(np.uint8)).cuda()  # noqa: E731
    umask, in_t = T(old), T(np.zeros(n))
    changes, sweeps = cc.ground_reach(W, T(vmask), T(sink), umask, in_t, w=W.data)
    assert sweeps == -32 and 0 < want.sum() < n - sinks
    assert np.array_equal(umask.cpu().numpy() != 0, want)
    assert changes == (want != old).sum() and np.array_equal(in_t.cpu().numpy() != 0, want != old)


@pytest.mark.parametrize("K", [1, 4, 8, 11])
def test_batched_fp32_rows_are_summed_in_four_slots(K):
    """The fp32 batched solve adds a row's products in four chains (an accuracy of the scores, whatever the degrees of
    the batch): bit for bit what four entry slots on request give, at degrees from 6 to 60."""
    for n, deg in ((3000, 6), (2000, 16), (1000, 60)):
        ds = graphs.er_graph(n, deg, max(K, 2), seed=n)
        S = stream.build_system(ds, torch.ones(n, dtype=torch.bool, device="cuda"),
                                torch.as_tensor(graphs.label_mask(n, 0.05, seed=n)).cuda(), dtype="float32")
        if K == 1:
            assert S.C == 1
        bs = batched.BatchedSystems([S], dtype=torch.float32)
        a = bs.solve(target_relres=1e-5)
        b = bs.solve(target_relres=1e-5, group=4)
        assert a[1][0] == b[1][0] and torch.equal(a[0], b[0])


def test_coarse_operator_of_converted_inputs():
    """Weights and aggregates that are converted on the way give the coarse operator of their fp32 and int32 copies."""
    n, nc = 200_000, 50
    W = random_csr(n, 1, 3)  # as many entries as rows: the copies are of one size
    agg = torch.randint(0, nc, (n,), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    want, _ = amg.coarsen(W, None, agg.to(torch.int32), nc)
    wide = torch.stack([agg, agg], 1)[:, 0]  # int64, strided
    got, _ = amg.coarsen(CSR(W.data.double(), W.indices, W.indptr, W.shape), None, wide, nc)
    assert all(torch.equal(a, b) for a, b in ((got.indptr, want.indptr), (got.indices, want.indices), (got.data, want.data)))


def test_rows_are_taken_by_ids_on_the_host():
    X, idx = torch.randn(100, 5, device="cuda", dtype=torch.float64), torch.tensor([3, 99, 0])
    assert torch.equal(kernels.rows_take(X, idx, torch.float32), X[idx].float())


@pytest.mark.parametrize("C", [1, 5])
def test_rows_are_taken_by_negative_ids(C):
    X = torch.randn(100, C, device="cuda", dtype=torch.float64)
    idx = torch.tensor([-1, 0, -100, 99, -37], device="cuda")
    assert torch.equal(kernels.rows_take(X, idx, torch.float32), X[idx].float())
    assert torch.isnan(kernels.rows_take(X, torch.tensor([100, -101], device="cuda"), torch.float32)).all()
