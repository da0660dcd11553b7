"""The solvers' fast paths against the general ones, at the sizes where they can go wrong."""
import numpy as np
import pytest
import torch

from dynlplus_b200 import graphs, kernels, solvers, stream

pytestmark = pytest.mark.gpu


def grounded(n, K, seed=0, weights="unit", dtype="float32", deg=(12, 4)):
    ds = graphs.planted_partition(n, K, *deg, weights=weights, seed=seed)
    lab = graphs.label_mask(n, 0.02, seed=seed)
    return ds, lab, stream.build_system(ds, torch.ones(n, dtype=torch.bool, device="cuda"), lab, dtype=dtype)


@pytest.mark.parametrize("method,lowp,target", [("pcg", False, 1e-6), ("pcg", True, 1e-6), ("amg", False, 1e-8),
                                                ("amg", True, 1e-8)])
def test_first_solve_asks_for_what_its_precision_resolves(method, lowp, target):
    """The relative residual is met by the fp64 refinement in a few dozen iterations in all; a solve
    asked for less than its rounding leaves would run on until its patience (400) ended."""
    n, K = 20_000, 4
    ds, lab, S = grounded(n, K, seed=3, weights="lognormal")
    solver = solvers.DynLPPlus(n, K, "float32", method=method, tol=1e-3, target_relres=target, lowp=lowp)
    st = solver.solve(S)
    S64 = S.astype(torch.float64)
    F = solver.scores(S)
    R = solvers.residual(S64, F.contiguous(), S64.rhs.contiguous())
    rel = float((R.norm(dim=0) / S64.rhs.norm(dim=0)).max())
    assert rel <= target and st.cert <= 1e-3
    assert st.iters < 150


@pytest.mark.parametrize("n,K,dtype,deg,max_iter", [(40, 2, "float32", 6, 10**7), (257, 2, "float32", 6, 10**7),
                                                    (5000, 3, "float32", 10, 10**7), (5000, 9, "float64", 10, 10**7),
                                                    (3001, 33, "float32", 24, 10**7), (20_000, 4, "float32", 10, 7),
                                                    (20_000, 2, "float32", 10, 8), (300_001, 2, "float32", 6, 12),
                                                    (299_999, 2, "float32", 6, 12)])
def test_frontier_rounds_on_the_device_equal_the_host_loop(n, K, dtype, deg, max_iter):
    """DynLP with its rounds in one launch against the same rounds launched one by one: the same
    per-row arithmetic on the same frontiers, so scores, rounds and edge visits are equal."""
    ds = graphs.er_graph(n, deg, K, weights="lognormal", seed=n)
    lab = graphs.label_mask(n, max(0.02, 1.0 / n), seed=1)
    S = stream.build_system(ds, torch.ones(n, dtype=torch.bool, device="cuda"), lab, dtype=dtype)
    a, b = (solvers.DynLP(n, K, dtype, delta=1e-4, max_iter=max_iter) for _ in range(2))
    rounds = []
    sa, sb = a.solve(S), b.solve(S, record=rounds)
    assert torch.equal(a.F, b.F)
    assert sa.iters == sb.iters == len(rounds) and sa.edges == sb.edges
    assert sa.iters == min(sa.iters, max_iter)


def pcg_case(n, C, dtype, deg=8, seed=0):
    """A grounded system A = diag - W of n rows (some without entries) and right-hand sides."""
    rng = np.random.default_rng(seed)
    m = int(n * deg / 2)
    import scipy.sparse as ssp
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    W = ssp.coo_matrix((rng.uniform(0.2, 1.5, m), (u, v)), (n, n)).tocsr()
    W = W + W.T
    W.setdiag(0)
    W.eliminate_zeros()
    W = W.astype(np.float32)
    diag = np.asarray(W.sum(1)).ravel().astype(np.float64) + rng.uniform(0.05, 0.5, n)
    rhs = rng.uniform(0, 1, (n, C))
    dt = getattr(torch, dtype)
    from dynlplus_b200.backend import CSR
    Wd = CSR.from_scipy(W)
    if not Wd.indices.numel():  # the kernels want valid pointers
        Wd = CSR(torch.zeros(1, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), Wd.indptr, Wd.shape)

    class Sys:
        pass
    S = Sys()
    S.W, S.nnz = Wd, int(W.nnz)
    S.diag = torch.as_tensor(diag).to(dt).cuda()
    return S, W, S.diag.double().cpu().numpy(), torch.as_tensor(rhs).to(dt).cuda()


# block boundaries of the rows (8 per block, then 148 blocks), one and several vectors per row, both vector
# widths, the size the launch path starts at (100,000 rows) and the next one
@pytest.mark.parametrize("n,C,dtype", [(1, 1, "float32"), (7, 4, "float32"), (9, 5, "float64"), (8 * 148, 8, "float32"),
                                       (8 * 148 + 1, 9, "float32"), (5000, 3, "float64"), (5001, 17, "float32"),
                                       (3000, 33, "float32"), (2999, 64, "float32"), (4001, 64, "float64"),
                                       (100_000, 1, "float32"), (100_001, 1, "float32")])
def test_whole_solve_in_one_launch_equals_the_kernel_loop(n, C, dtype):
    """The one-launch PCG against the same iteration launched kernel by kernel: iteration counts within one
    and both at the target (a rounding can move the stop by an iteration), the iterates together, from
    zero and from a given start, with the recheck and without."""
    import scipy.sparse as ssp
    S, W, diag, rhs = pcg_case(n, C, dtype, seed=n + C)
    f32 = dtype == "float32"
    target = 1e-4 if f32 else 1e-11
    A = ssp.diags(diag) - W.astype(np.float64)
    b = rhs.double().cpu().numpy()
    for zero, confirm in ((True, True), (False, True), (True, False)):
        out = []
        for graph in (True, False):
            Z = solvers.padded_empty(n, C, rhs.dtype, "cuda", fill=0.25)
            st = solvers.Stats()
            solvers.TWO_KERNEL = graph
            try:
                solvers.pcg(S, Z, rhs, None, solvers.jacobi_M(S), 3000, st, target_relres=target, use_graph=graph,
                            zero_start=zero, confirm=confirm)
            finally:
                solvers.TWO_KERNEL = True
            out.append((Z.double().cpu().numpy(), st.iters))
        assert abs(out[0][1] - out[1][1]) <= 1
        for Z, _ in out:
            assert (np.linalg.norm(b - A @ Z, axis=0) / np.linalg.norm(b, axis=0)).max() <= 1.2 * target
        # two iterates at relative residual t differ by at most 2 t cond(A); diagonal dominance by at
        # least 0.05 bounds the inverse
        assert np.abs(out[0][0] - out[1][0]).max() <= 2.4 * target * np.linalg.norm(b, axis=0).max() / 0.05


def test_whole_solve_stop_rules():
    """Iteration cap, patience, an unreachable target and a non-finite right-hand side, as in the loop."""
    S, W, diag, rhs = pcg_case(4000, 5, "float32", seed=2)
    for graph in (True, False):
        st, Z = solvers.Stats(), solvers.padded_empty(4000, 5, torch.float32, "cuda")
        solvers.pcg(S, Z, rhs, None, solvers.jacobi_M(S), 7, st, target_relres=1e-12, use_graph=graph, zero_start=True)
        assert st.iters == 7
        st = solvers.Stats()
        solvers.pcg(S, Z, rhs, None, solvers.jacobi_M(S), 3000, st, target_relres=1e-30, patience=20, use_graph=graph,
                    zero_start=True)
        assert st.iters < 200
        bad = rhs.clone()
        bad[17, 3] = float("nan")
        with pytest.raises(FloatingPointError):
            solvers.pcg(S, Z, bad, None, solvers.jacobi_M(S), 50, solvers.Stats(), target_relres=1e-5, use_graph=graph,
                        zero_start=True)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float64"])
@pytest.mark.parametrize("C", [3, 7, 8, 9, 16, 17, 32, 33, 64])
def test_spmm_layouts_and_padded_copies(C, dtype):
    """The SpMM over rows on a vector pitch, on their own odd pitch and on an offset view, at a size where
    odd rows are copied to a vector pitch, against an fp64 product. Tolerance: the working precision's unit
    roundoff times the row's length and weight sum (fp32 accumulation for bf16)."""
    from dynlplus_b200 import kernels
    from dynlplus_b200.backend import CSR
    n, dt = max(200_000, int(13e6 / C / 8)), getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(C)
    deg = torch.randint(0, 16, (n,), generator=g, device="cuda")
    ip = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ip[1:] = torch.cumsum(deg, 0)
    m = int(ip[-1])
    col = torch.randint(0, n, (m,), generator=g, device="cuda")
    w = torch.rand(m, generator=g, device="cuda").to(dt)
    W = CSR(w, col.to(torch.int32), ip.to(torch.int32), (n, n))
    base = torch.rand((n, C + 8), generator=g, device="cuda").to(dt)
    a = torch.rand(n, generator=g, device="cuda").to(torch.float32 if dtype == "bfloat16" else dt)
    A = torch.sparse_csr_tensor(ip, col, w.double(), (n, n))
    tol = 16 * 16 * (2.0 ** -53 if dtype == "float64" else 2.0 ** -24)
    pad = (C * base.element_size() + 15) // 16 * 16 // base.element_size()
    for X in (base[:, :C].contiguous(), base[:, 1:C + 1], torch.nn.functional.pad(base[:, :C], (0, pad - C))[:, :C]):
        Y = kernels.spmm_axpy(W, X, a=a, b=-1.0)
        want = a.double()[:, None] * X.double() - A @ X.double()
        assert float((Y.double() - want).abs().max()) <= tol


@pytest.mark.parametrize("K", [16, 32])
def test_wide_class_sum_corrections(K):
    """Corrections with the last class derived, at the widths where they are on by default: the target is
    met on the fp64 residual of every column and the scores of solved rows sum to one."""
    n = 5000
    ds = graphs.planted_partition(n, K, 12, 4, weights="lognormal", seed=K)
    lab = graphs.label_mask(n, 0.05, seed=K)
    es = stream.EdgeStream(ds, lab)
    solver = solvers.IncrementalLP(n, K, "float32", tol=1e-3, method="pcg", target_relres=1e-6)
    assert solver.class_sum
    solver.solve(es.system)
    up = graphs.EdgeUpdates(ds.A, seed=1, weights="lognormal")
    for _ in range(3):
        S = es.apply_edges(**up.next(200))
        st = solver.solve(S)
        S64 = S.astype(torch.float64)
        R = solvers.residual(S64, solver.Z[:, :K].contiguous(), S64.rhs.contiguous())
        assert st.relres <= 1e-6 and float((R.norm(dim=0) / S64.rhs.norm(dim=0)).max()) <= 1.01e-6
        assert float((solver.Z[:, :K][S.solved].sum(1) - 1).abs().max()) <= 1e-9


@pytest.mark.parametrize("n", [1, 2, 147, 149, 500, 1500, 1900])
def test_dense_inverse_in_one_launch(n):
    """The in-place inverse of a diagonally dominant symmetric matrix (the sizes around one row per block,
    and past what shared memory holds) against numpy; tolerance: n unit roundoffs times the condition
    number, at most 41 by the dominance margin."""
    from dynlplus_b200 import _lib
    from dynlplus_b200.backend import ptr, workspace
    from dynlplus_b200.backend import stream as cur
    rng = np.random.default_rng(n)
    A = rng.uniform(-1, 0, (n, n))
    A = (A + A.T) / 2
    np.fill_diagonal(A, 0)
    A[np.arange(n), np.arange(n)] = np.abs(A).sum(1) * 1.05 + 0.01
    D = torch.as_tensor(A).cuda()
    ws = workspace("amg_inverse").get(_lib.lib().dlp_dense_spd_inverse_workspace_bytes(n))
    _lib.call("dlp_dense_spd_inverse", n, ptr(D), ptr(ws), ws.numel(), cur())
    want = np.linalg.inv(A)
    assert np.abs(D.cpu().numpy() - want).max() <= n * 2.3e-16 * 41 * np.abs(want).max()


@pytest.mark.parametrize("sizes", [[1, 31, 32, 33], [2, 512, 513, 40], [700, 1, 0, 5]])
def test_aggregate_members_of_every_length(sizes):
    """Members of each aggregate in ascending order, at the lengths the three sorts take."""
    from dynlplus_b200 import amg
    agg = np.repeat(np.arange(len(sizes)), sizes)
    agg = agg[np.random.default_rng(0).permutation(agg.size)]
    off, mem = amg.members(torch.as_tensor(agg.astype(np.int32)).cuda(), len(sizes))
    off, mem = off.cpu().numpy(), mem.cpu().numpy()
    for a in range(len(sizes)):
        assert np.array_equal(mem[off[a]:off[a + 1]], np.flatnonzero(agg == a))


@pytest.mark.parametrize("C,dtype", [(1, "float32"), (17, "float32"), (64, "float64"), (70, "float32")])
def test_restriction_and_coarse_entries_of_long_aggregates(C, dtype):
    """Sums over aggregates of 1, 64, 65 and 3,000 members, and coarse entries from runs of as many fine
    ones, against numpy; tolerance: the run's length in unit roundoffs of the working precision."""
    from dynlplus_b200 import _lib, amg
    from dynlplus_b200.backend import CSR, code, ptr
    from dynlplus_b200.backend import stream as cur
    import scipy.sparse as ssp
    sizes = [1, 64, 65, 3000, 300]
    n, nc = sum(sizes), len(sizes)
    rng = np.random.default_rng(C)
    agg = np.repeat(np.arange(nc), sizes)[rng.permutation(n)].astype(np.int32)
    off, mem = amg.members(torch.as_tensor(agg).cuda(), nc)
    R = rng.uniform(0, 1, (n, C))
    Rd = torch.as_tensor(R).to(getattr(torch, dtype)).cuda()
    out = torch.empty((nc, C), dtype=Rd.dtype, device="cuda")
    _lib.call("dlp_amg_restrict", nc, C, ptr(off), ptr(mem), ptr(Rd), C, ptr(out), C, code(Rd), cur())
    Rr = Rd.double().cpu().numpy()
    want = np.stack([Rr[agg == a].sum(0) for a in range(nc)])
    eps = 2.0 ** -24 if dtype == "float32" else 2.0 ** -53
    assert (np.abs(out.double().cpu().numpy() - want) <= 3000 * eps * want).all()
    m = 60_000
    W = ssp.coo_matrix((rng.uniform(0.5, 1.5, m).astype(np.float32), (rng.integers(0, n, m), rng.integers(0, n, m))),
                       (n, n)).tocsr()
    Wc, _ = amg.coarsen(CSR.from_scipy(W), None, torch.as_tensor(agg).cuda(), nc)
    P = ssp.coo_matrix((np.ones(n), (np.arange(n), agg)), (n, nc)).tocsr()
    D = np.asarray((P.T @ W.astype(np.float64) @ P).todense())
    np.fill_diagonal(D, 0)
    got = np.asarray(Wc.to_scipy().astype(np.float64).todense())
    assert np.abs(got - D).max() <= 2.0 ** -23 * D.max()


@pytest.mark.parametrize("kind,n", [("random", 1), ("random", 1023), ("random", 1025), ("random", 60_000), ("path", 5000),
                                    ("path", 20)])
def test_grounding_in_one_launch(kind, n):
    """The grounded set, its changes and counts against SciPy's components: random graphs (sweeps settle),
    and a path longer than 32 sweeps may cover (the union-find in the same launch)."""
    import scipy.sparse as ssp
    from scipy.sparse.csgraph import connected_components
    from dynlplus_b200 import _lib, cc
    from dynlplus_b200.backend import CSR, code, ptr, workspace
    from dynlplus_b200.backend import stream as cur
    rng = np.random.default_rng(n)
    if kind == "path":
        order = rng.permutation(n)
        u, v = order[:-1], order[1:]
    else:
        m = int(0.9 * n)
        u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    A = ssp.coo_matrix((np.ones(len(u), np.float32), (u, v)), (n, n)).tocsr()
    A = ((A + A.T) > 0).astype(np.float32).tocsr()
    A.setdiag(0)
    A.eliminate_zeros()
    dead = rng.random(A.nnz) < (0.0 if kind == "path" else 0.1)  # dead entries, both directions
    C = A.tocoo()
    key = np.minimum(C.row, C.col).astype(np.int64) * n + np.maximum(C.row, C.col)
    dead = np.isin(key, key[dead])
    sink = np.zeros(n, np.uint8)
    sink[(order[:1] if kind == "path" else rng.integers(0, n, max(1, n // 50)))] = 1
    vmask = (1 - sink).astype(np.uint8)
    if n > 100:
        vmask[rng.integers(0, n, n // 20)] = 0  # neither masked nor sink
    Wd = CSR.from_scipy(A)
    if not A.nnz:
        Wd = CSR(torch.zeros(1, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), Wd.indptr, Wd.shape)
    else:
        Wd.data[torch.as_tensor(dead).cuda()] = 0
    old = (rng.random(n) < 0.5).astype(np.uint8)
    T = lambda x: torch.as_tensor(x.copy()).cuda()  # noqa: E731
    um, it = T(old), torch.zeros(n, dtype=torch.uint8, device="cuda")
    ce, info = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.full((4,), 7, dtype=torch.int32, device="cuda")
    ws = workspace("ground_reach").get(_lib.lib().dlp_ground_reach_workspace_bytes(n))
    vm, sk = T(vmask), T(sink)
    _lib.call("dlp_ground_reach_async", n, ptr(Wd.rbeg), ptr(Wd.rend), ptr(Wd.indices), ptr(Wd.data), code(Wd.data),
              ptr(vm), ptr(sk), ptr(um), ptr(it), ptr(ce[:1]), ptr(ce[1:]), ptr(info), ptr(ws), ws.numel(), cur())
    live = A.tocoo()
    keep = ~dead & (vmask[live.row] > 0) & ((vmask[live.col] > 0) | (sink[live.col] > 0))
    r, c = live.row[keep], np.where(vmask[live.col[keep]] > 0, live.col[keep], n)
    _, lab = connected_components(ssp.coo_matrix((np.ones(len(r)), (r, c)), (n + 1, n + 1)), directed=False)
    want = ((vmask > 0) & (lab[:n] == lab[n])).astype(np.uint8)
    assert np.array_equal(um.cpu().numpy(), want)
    assert np.array_equal(it.cpu().numpy(), (want != old).astype(np.uint8))
    active, lost, sweeps, bad = info.tolist()
    assert (active, lost, bad) == (int(vmask.sum() + sink.sum()), int((vmask > want).sum()), 0)
    assert ce.tolist() == [int((want != old).sum()), 0] and 1 <= abs(sweeps) <= 32


@pytest.mark.parametrize("m,deg,grounds,ties", [(1, 0, True, False), (2, 2, False, False), (513, 4, True, False),
                                                (2000, 3, True, True), (2000, 3, False, True), (75_777, 6, True, False)])
def test_fh_components_on_the_device(m, deg, grounds, ties):
    """The merging rounds in one launch against the oracle's, label for label: random graphs, tied
    weights, with and without grounding, from one vertex to more than one block's worth per SM."""
    from dynlplus_b200 import cc
    from oracle import ref_np as O
    rng = np.random.default_rng(m + deg)
    e = m * deg // 2
    u, v = rng.integers(0, m, e), rng.integers(0, m, e)
    d = rng.integers(1, 5, e).astype(np.float32) if ties else rng.uniform(0.05, 2, e).astype(np.float32)
    keep = u != v
    u, v, d = u[keep], v[keep], d[keep]
    rows, cols, dd = np.r_[u, v], np.r_[v, u], np.r_[d, d]
    g = (rng.random(m) < 0.02).astype(np.float32) if grounds else None
    k = 1.5
    want, nc = O.fh_components(m, rows, cols, dd, np.float32(k), g)
    T = lambda x: torch.as_tensor(x).cuda()  # noqa: E731
    lab, n2 = cc.fh_components(m, T(rows), T(cols), T(dd), k, T(g) if g is not None else None)
    assert n2 == nc and np.array_equal(lab.cpu().numpy(), want)


@pytest.mark.parametrize("n,m", [(500_000, 500_000), (900_001, 500_001), (1000, 600_000), (1_100_000, 499_999)])
def test_components_of_long_edge_lists(n, m):
    """Component labels around the line where the rounds start, a dense graph and one past the giant
    component, against SciPy; an endpoint outside the range is refused in the rounds too."""
    import scipy.sparse as ssp
    from scipy.sparse.csgraph import connected_components
    from dynlplus_b200 import cc
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    _, want = connected_components(ssp.coo_matrix((np.ones(m), (u, v)), (n, n)), directed=False)
    first = np.full(want.max() + 1, n)
    np.minimum.at(first, want, np.arange(n))
    want = np.argsort(np.argsort(first))[want]  # ranks by smallest vertex
    T = lambda x: torch.as_tensor(x.astype(np.int32)).cuda()  # noqa: E731
    lab, nc = cc.connected_components(n, T(u), T(v))
    assert nc == want.max() + 1 and np.array_equal(lab.cpu().numpy(), want)
    u[m // 2] = n
    with pytest.raises(ValueError):
        cc.connected_components(n, T(u), T(v))


@pytest.mark.parametrize("n,K,dtype,wdtype,eta", [(6, 2, "float32", "float32", 0.0), (33, 3, "float64", "float64", 0.1),
                                                  (257, 9, "float32", "float64", 0.0), (5000, 2, "float64", "float32", 0.3),
                                                  (4999, 17, "float32", "float32", 0.0)])
def test_built_system_equals_the_oracle(n, K, dtype, wdtype, eta):
    """The system of a graph with inactive vertices and isolated ones: sets, columns and weights equal the
    oracle's, sums to 1e-12 (1e-6 in fp32), in both precisions it carries."""
    from oracle import ref_np as O
    rng = np.random.default_rng(n)
    ds = graphs.er_graph(n, 5, K, weights="lognormal", seed=n, dtype=wdtype)
    y = ds.y.cpu().numpy()
    active, lab = rng.random(n) < 0.9, rng.random(n) < 0.15
    lab[:2] = active[:2] = True
    want = O.build_system(ds.A.to_scipy(), y, K, active, lab, eta=eta)
    S = stream.build_system(ds, torch.as_tensor(active).cuda(), torch.as_tensor(lab).cuda(), dtype=dtype, eta=eta)
    assert np.array_equal(S.U.cpu().numpy(), want["U"]) and S.n_ungrounded == want["n_ungrounded"]
    assert S.n_active == int(active.sum()) and S.U.dtype == torch.int64
    for T in (S, S.astype(torch.float64)):
        W, Ww = T.W.to_scipy(), want["W"]
        assert np.array_equal(W.indptr, Ww.indptr) and np.array_equal(W.indices, Ww.indices)
        assert np.array_equal(W.data.astype(np.float64), Ww.data.astype(W.data.dtype).astype(np.float64))
        tol = 1e-12 if T.diag.dtype == torch.float64 and (wdtype == "float32" or dtype == "float64") else 1e-6
        for name in ("s", "diag", "B", "rhs"):
            np.testing.assert_allclose(getattr(T, name).double().cpu().numpy(), want[name], rtol=tol, atol=tol)
        h = torch.cat([T.rhs, T.diag[:, None]], 1)
        assert torch.equal(T.rhs_h, h) and T.rhs.is_contiguous()
    bad = ds.y.clone()
    bad[0] = K
    with pytest.raises(IndexError):
        stream.build_system(graphs.Dataset("x", ds.A, bad, K, ds.order), torch.as_tensor(active).cuda(),
                            torch.as_tensor(lab).cuda(), dtype=dtype)


@pytest.mark.parametrize("K,dtype", [(2, "float64"), (4, "float64"), (8, "float64"), (4, "float32"), (8, "float32"),
                                     (16, "float64")])
def test_uneven_batch_equals_each_system_alone(K, dtype):
    """Systems of very different sizes in one batch: bit for bit the scores, iterations and status each has
    alone, the target met on the fp64 residual (or the precision's floor), from zero and from a start."""
    from dynlplus_b200 import batched
    dt = getattr(torch, dtype)
    systems = [grounded(n, K, seed=n, deg=(6, 4))[2] for n in (60, 127, 130, 1000, 5000, 20_000)]
    target = 1e-8 if dt == torch.float64 else 1e-4
    for start in (False, True):
        bs = batched.BatchedSystems(systems, dtype=dt)
        Z0 = torch.full((bs.N, bs.Ch), 0.3, dtype=dt, device="cuda") if start else None
        Z, it, status, rel = bs.solve(target_relres=target, Z0=Z0)
        assert (status == 5).all() and (rel <= target).all()
        for k, s in enumerate(systems):
            one = batched.BatchedSystems([s], dtype=dt)
            a, b = bs.offsets[k], bs.offsets[k + 1]
            Z1, it1, st1, rel1 = one.solve(target_relres=target, Z0=Z0[a:b] if start else None)
            assert torch.equal(Z[a:b], Z1) and it[k] == it1[0] and rel[k] == rel1[0]
            S64 = s.astype(torch.float64)
            R = solvers.residual(S64, Z[a:b, : s.C].double().contiguous(), S64.rhs.contiguous())
            bn = S64.rhs.norm(dim=0)  # a zero right-hand side (a class without a label) counts as one, as in the solver
            assert bool((R.norm(dim=0) <= 1.01 * target * torch.where(bn > 0, bn, torch.ones_like(bn))).all())


@pytest.mark.parametrize("dt", ["float32", "float64"])
@pytest.mark.parametrize("C", [1, 4, 5, 8, 9, 16, 17, 32, 33])
def test_push_in_one_launch_equals_the_launched_rounds(C, dt):
    """One cooperative launch against the rounds launched by the host. fp64: the same frontiers (rounds and
    edge visits), Z and R equal up to the order of the atomic sums. Both types: R stays the residual of Z, no
    row violates at the end, and columns beyond C keep their values."""
    n, tdt = 3001, getattr(torch, dt)
    ds = graphs.er_graph(n, 11, 4, seed=C)
    es = stream.EdgeStream(ds, graphs.label_mask(n, 0.05, seed=C), dtype="float32")
    S = es.system.astype(torch.float64)
    W, diag = es.G, S.diag.to(tdt)
    g = torch.Generator().manual_seed(C)
    base = (torch.rand((n, C), generator=g, dtype=torch.float64).to("cuda") * S.solved[:, None]).to(tdt)
    eps = [1e-2] * C
    cand = torch.nonzero(S.solved).flatten().to(torch.int32)
    out = []
    for whole in (True, False):
        Z, R = torch.zeros((n, C + 3), dtype=tdt, device="cuda"), torch.full((n, C + 3), 7.0, dtype=tdt, device="cuda")
        R[:, :C] = base
        rounds, ok, edges = kernels.FusedPush(W, C).run(Z[:, :C], R[:, :C], diag, eps, cand, 10_000, use_graph=whole)
        assert ok and float((R[:, C:] - 7.0).abs().max()) == 0.0 and float(Z[:, C:].abs().max()) == 0.0
        z, x = Z[:, :C].double().contiguous(), R[:, :C].double()
        assert bool((x.abs() <= eps[0] * diag.double()[:, None] * (1 + 1e-6)).all())
        # a value of R takes at most one rounded add per round and entry of its row (degree < 64), each of a
        # residual no larger than diag * max Z; Z one per round
        u = 2.0 ** (-24 if dt == "float32" else -53)
        lim = u * 66 * rounds * float(diag.max()) * max(float(z.abs().max()), 1.0)
        true = base.double() - kernels.spmm_axpy(W, z, a=S.diag, b=-1.0)
        assert float((true - x).abs().max()) <= lim
        out.append((rounds, edges, z, x, lim))
    (r0, e0, z0, x0, lim), (r1, e1, z1, x1, _) = out
    if dt == "float64":
        assert (r0, e0) == (r1, e1)
        assert float((x0 - x1).abs().max()) <= 2 * lim and float((z0 - z1).abs().max()) <= 2 * lim


@pytest.mark.parametrize("n", [35, 257, 5001])
@pytest.mark.parametrize("C", [15, 16, 20, 32, 36])
def test_pcg_sweeps_four_columns_a_thread(C, n):
    """The wide-row sweeps (C of at least 16, a multiple of four, aligned rows) against the scalar ones (a Z on
    an odd pitch keeps the direction sweep scalar; C = 15 both): the true residual meets the target from a
    warm and a zero start, and columns beyond C keep their values."""
    ds = graphs.er_graph(n, 8, 4, seed=n)
    lab = torch.as_tensor(graphs.label_mask(n, 0.2, seed=n)).cuda()
    S = stream.build_system(ds, torch.ones(n, dtype=torch.bool, device="cuda"), lab, eta=1e-3, dtype="float32")
    m = S.n_u
    g = torch.Generator().manual_seed(C * n)
    rhs = torch.rand((m, C), generator=g).cuda()
    rn = rhs.double().norm(dim=0)
    target = 1e-4  # far above the fp32 floor of these systems
    for odd in (False, True):
        for zero in (False, True):
            Z = solvers.padded_empty(m, C, torch.float32, "cuda", fill=0.5) if not odd else \
                torch.full((m, C + 5 - C % 2), 0.5, device="cuda")[:, :C]
            st = solvers.Stats()
            solvers.pcg(S, Z, rhs, None, solvers.jacobi_M(S), 3000, st, target_relres=target, use_graph=False,
                        zero_start=zero)
            R = rhs.double() - kernels.spmm_axpy(S.W, Z.double().contiguous(), a=S.diag.double(), b=-1.0)
            assert float((R.norm(dim=0) / rn).max()) <= 1.05 * target and 1 < st.iters < 3000
            if odd:
                assert float((Z.as_strided((m, 1), (Z.stride(0), 1), Z.storage_offset() + C) - 0.5).abs().max()) == 0.0


@pytest.mark.parametrize("src,dst", [("float32", "float32"), ("float32", "float64"), ("float64", "float32"),
                                     ("float64", "float64")])
@pytest.mark.parametrize("n,C", [(0, 3), (1, 1), (257, 5), (4099, 33)])
def test_rows_take_equals_indexing(n, C, src, dst):
    """Rows by id against tensor indexing, every value the same: from and into rows on a pitch of their own,
    other id types and layouts on the general path, and an id outside the source gives NaN."""
    g = torch.Generator().manual_seed(n + C)
    X = torch.randn((5000, C + 2), generator=g, dtype=torch.float64).to("cuda").to(getattr(torch, src))[:, :C]
    idx = torch.randint(0, 5000, (n,), generator=g).cuda()
    want = X[idx].to(getattr(torch, dst))
    out = torch.full((n, C + 3), 3.0, dtype=want.dtype, device="cuda")
    kernels.rows_take(X, idx, want.dtype, out=out[:, :C])
    assert torch.equal(out[:, :C], want) and bool((out[:, C:] == 3.0).all())
    assert torch.equal(kernels.rows_take(X, idx, want.dtype), want)
    assert torch.equal(kernels.rows_take(X, idx.to(torch.int32), want.dtype), want)
    assert torch.equal(kernels.rows_take(X.t().contiguous().t(), idx, want.dtype), want)
    if n > 1:
        bad = idx.clone()
        bad[1] = 5000
        assert bool(kernels.rows_take(X, bad, want.dtype)[1].isnan().all())


@pytest.mark.parametrize("n,K", [(10_000, 8), (20_000, 8), (10_000, 10)])
def test_plain_fp32_solve_to_its_floor_in_the_device_loop(n, K):
    """fp32 solves to 1e-6 with their own rechecks, at the floor of fp32: the device-side loop takes the host
    loop's iterations (a failed recheck may not cost it the iterate)."""
    ds = graphs.sbm(n, K=K, deg=16.0, seed=3)
    lab = torch.as_tensor(graphs.label_mask(n, 0.01, seed=3)).cuda()
    S = stream.build_system(ds, torch.ones(n, dtype=torch.bool, device="cuda"), lab, dtype="float32")
    its = []
    for graph in (True, False):
        Z, st = solvers.padded_empty(S.n_u, K, torch.float32, "cuda", fill=0.0), solvers.Stats()
        solvers.pcg(S, Z, S.rhs, None, solvers.jacobi_M(S), 10_000, st, target_relres=1e-6, use_graph=graph)
        its.append(st.iters)
    assert its[0] == its[1]
