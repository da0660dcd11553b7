"""Performance cases of the framework's main paths, through its public entry points.

Every case is a call that a program using this library makes: one edge batch on a resident graph
(`EdgeStream.apply_edges` + `IncrementalLP.solve` + `relabel`), a static solve of a new graph, the
fp64 reference solve, the AMG-preconditioned solve, batches of independent solves, one application of
a system's operator, component labels of an edge list, and a vertex-arrival stream. Graphs are the
benchmark's families (planted partition and Erdos-Renyi, unit or lognormal(0, 0.5) weights), made on
the GPU from the seed.
"""
import math

import numpy as np
import torch

from dynlplus_b200 import batched, cc, graphs, kernels, solvers, stream
from dynlplus_b200.backend import CSR

DEV = "cuda"
F64 = torch.float64


# -- the cases --------------------------------------------------------------------------------------
def _update(name, n, K, deg_in, deg_cross, weights, batch, target, labelled, components=False):
    return {"name": name, "kind": "update", "n": n, "K": K, "deg_in": deg_in, "deg_cross": deg_cross,
            "weights": weights, "batch": batch, "target": target, "labelled": labelled, "components": components}


def listed():
    return [
        # a handful of edges on a small resident graph: the latency of one update (launches, host reads)
        _update("update-3k", 3000, 4, 12.0, 4.0, "unit", 16, 1e-6, 0.01),
        # the default solver (certified to 1e-3, no residual target) on a weighted binary graph: a small
        # batch that the residual push repairs locally
        _update("update-60k-push", 60_017, 2, 12.0, 4.0, "lognormal", 200, 0.0, 0.01),
        # the headline stream: Erdos-Renyi, 8 classes, 10,000 updates, component ids after the batch
        _update("update-1m", 1_000_000, 8, 0.0, 10.0, "unit", 10_000, 1e-6, 0.005, True),
        # the serving stream's class count on weighted blocks: wide score rows
        _update("update-250k-k32", 250_000, 32, 12.0, 4.0, "lognormal", 3000, 1e-6, 0.01),
        # the static solve: build the grounded system of a graph and solve it to 1e-6
        {"name": "static-100k", "kind": "static", "n": 100_000, "K": 4, "deg_in": 12.0, "deg_cross": 4.0,
         "weights": "unit", "target": 1e-6},
        # the high-accuracy fp64 solution that a benchmark run compares its scores with
        {"name": "reference-40k", "kind": "reference", "n": 40_009, "K": 5, "deg_in": 12.0, "deg_cross": 4.0,
         "weights": "lognormal"},
        # aggregation AMG, setup and solve to 1e-8, with bf16 sweeps and fp64 refinement
        {"name": "amg-120k", "kind": "amg", "n": 120_000, "K": 16, "deg_in": 24.0, "deg_cross": 8.0,
         "weights": "lognormal", "lowp": True},
        # fresh solves that a server takes together: systems built and solved in mixed precision
        {"name": "fresh-24", "kind": "fresh", "count": 24, "n_min": 2000, "n_max": 60_000, "mixed": True},
        # many uneven systems in one batched fp64 solve
        {"name": "batched-48", "kind": "batched", "count": 48, "n_min": 2000, "n_max": 40_000, "mixed": False},
        # one application of the operator diag X - W X at a width between the padded ones
        {"name": "apply-500k-c17", "kind": "apply", "n": 500_000, "C": 17, "deg": 16.0, "dtype": "float32"},
        # component labels of an edge list (many components of every size)
        {"name": "components-2m", "kind": "components", "n": 2_000_000, "deg": 1.5},
        # the reference benchmark's own form: vertices arrive in batches, frontier Jacobi on each
        {"name": "arrivals-20k", "kind": "arrivals", "n": 20_000, "K": 2, "deg": 10.0, "batches": 4,
         "solver": "dynlp", "resident": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update", "update", "update", "static", "reference", "amg", "fresh", "batched", "apply",
                       "apply", "components", "arrivals"])
    weights = rng.choice(["unit", "lognormal"])
    if kind == "update":
        K = rng.choice([2, 3, 4, 5, 8, 8, 12, 16, 32])
        n = _log(rng, 2000, min(1_000_000, 8_000_000 // K))
        deg = rng.uniform(8.0, 10.0 if n > 400_000 else 20.0)
        share = rng.choice([0.0, 0.5, 0.75])
        return {"kind": kind, "n": n, "K": K, "deg_in": round(deg * share, 2), "deg_cross": round(deg * (1 - share), 2),
                "weights": weights, "batch": _log(rng, 10, max(20, n // 100)), "target": rng.choice([1e-6, 1e-6, 0.0]),
                "labelled": rng.choice([0.005, 0.01, 0.02]) if n > 10_000 else 0.02,
                "components": rng.random() < 0.5}
    if kind in ("static", "reference", "amg"):
        n = _log(rng, 2000, {"static": 100_000, "reference": 40_000, "amg": 120_000}[kind])
        K = rng.choice([2, 3, 4]) if kind == "static" else rng.choice([2, 3, 5]) if kind == "reference" else \
            rng.choice([2, 4, 8, 16])
        c = {"kind": kind, "n": n, "K": K, "deg_in": 12.0, "deg_cross": 4.0, "weights": weights}
        if kind == "static":
            c["target"] = 1e-6
        if kind == "amg":
            c["lowp"] = rng.random() < 0.5
        return c
    if kind in ("fresh", "batched"):
        return {"kind": kind, "count": rng.randint(3, 24 if kind == "fresh" else 48), "n_min": 2000,
                "n_max": _log(rng, 4000, 60_000 if kind == "fresh" else 40_000), "mixed": kind == "fresh"}
    if kind == "apply":
        C = rng.choice([1, 2, 3, 4, 5, 6, 8, 9, 12, 16, 17, 24, 33, 48])
        return {"kind": kind, "n": _log(rng, 1000, 8_500_000 // max(C, 17)), "C": C, "deg": round(rng.uniform(6, 16), 1),
                "dtype": rng.choice(["float32", "float32", "float64", "bfloat16"])}
    if kind == "components":
        return {"kind": kind, "n": _log(rng, 1000, 2_000_000), "deg": round(rng.uniform(0.8, 1.5), 2)}
    return {"kind": kind, "n": _log(rng, 2000, 20_000), "K": rng.choice([2, 3, 4]), "deg": round(rng.uniform(6, 10), 1),
            "batches": rng.randint(2, 4), "solver": rng.choice(["dynlp", "dynlp-fh", "dynlp+auto", "dynlp+inc"]),
            "resident": True}


# -- inputs, made from the seed alone ---------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + 17)


def _uniform(g, m, n):
    return torch.randint(0, n, (m,), generator=g, device=DEV)


def _csr_of(key, w, n):
    """Symmetric CSR (int32 indptr, int32 columns, weights) of the sorted unique keys u * n + v, u < v."""
    u, v = key // n, key % n
    full = torch.cat([u * n + v, v * n + u])
    order = torch.argsort(full)
    full = full[order]
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.bincount(full // n, minlength=n), 0)
    return indptr.to(torch.int32), (full % n).to(torch.int32), torch.cat([w, w])[order].contiguous()


def _edge_weights(g, m, weights):
    if weights == "unit":
        return torch.ones(m, device=DEV)
    return torch.exp(0.5 * torch.randn(m, generator=g, device=DEV))


def _graph(g, n, K, deg_in, deg_cross, weights, connected=False):
    """Unordered edges (sorted keys) with weights, and labels: K equal blocks, n deg_in / 2 pairs within
    the blocks and n deg_cross / 2 uniform ones; without in-block pairs (Erdos-Renyi) uniform labels.
    connected: n - 1 of the uniform pairs attach each vertex to a uniform earlier one instead, so that
    every unlabelled vertex is grounded."""
    bs = max(n // K, 1)
    parts = []
    if deg_in > 0:
        y = torch.clamp(torch.arange(n, device=DEV) // bs, max=K - 1)
        u = _uniform(g, int(n * deg_in / 2), n)
        lo = y[u] * bs
        hi = torch.where(y[u] == K - 1, n, lo + bs)
        v = lo + (torch.rand(u.numel(), generator=g, device=DEV, dtype=F64) * (hi - lo)).long()
        parts.append((u, v))
    else:
        y = _uniform(g, n, K)
    if connected:
        later = torch.arange(1, n, device=DEV)
        parts.append((later, (torch.rand(n - 1, generator=g, device=DEV, dtype=F64) * later).long()))
        deg_cross = max(deg_cross - 2.0, 0.0)
    parts.append((_uniform(g, int(n * deg_cross / 2), n), _uniform(g, int(n * deg_cross / 2), n)))
    u, v = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    a, b = torch.minimum(u, v), torch.maximum(u, v)
    key = torch.unique((a * n + b)[a != b])
    return key, _edge_weights(g, key.numel(), weights), y.to(torch.int32)


def _labelled(g, n, K, y, share):
    """Uniform labelled vertices, the same number of every class: max(1, round(share n / K))."""
    m = max(1, int(round(share * n / K)))
    perm = torch.randperm(n, generator=g, device=DEV)
    by_class = perm[torch.argsort(y[perm], stable=True)]
    size = torch.bincount(y.long(), minlength=K)
    beg = torch.cumsum(size, 0) - size
    lab = torch.zeros(n, dtype=torch.bool, device=DEV)
    lab[by_class[(beg[:, None] + torch.arange(m, device=DEV)[None, :]).flatten()]] = True
    return lab


def _dataset(name, csr, y, K):
    indptr, col, w = csr
    n = y.numel()
    return graphs.Dataset(name, CSR(w, col, indptr, (n, n)), y, K, torch.arange(n, device=DEV))


def _make_graph(case, seed):
    g = _gen(seed)
    key, w, y = _graph(g, case["n"], case["K"], case["deg_in"], case["deg_cross"], case["weights"],
                       connected=case["kind"] != "update")
    lab = _labelled(g, case["n"], case["K"], y, case.get("labelled", 0.01))
    return g, key, w, y, lab


def _batch(g, case, key):
    """Half of the batch inserts uniform non-edges, half deletes uniform edges: (new keys, their
    weights, positions of the deleted keys)."""
    n, ni = case["n"], case["batch"] // 2
    u, v = _uniform(g, 4 * ni + 64, n), _uniform(g, 4 * ni + 64, n)
    a, b = torch.minimum(u, v), torch.maximum(u, v)
    cand = torch.unique((a * n + b)[a != b])
    pos = torch.clamp(torch.searchsorted(key, cand), max=key.numel() - 1)
    cand = cand[key[pos] != cand]
    new = cand[torch.randperm(cand.numel(), generator=g, device=DEV)[:ni]]
    gone = torch.randperm(key.numel(), generator=g, device=DEV)[: case["batch"] - ni]
    return new, _edge_weights(g, new.numel(), case["weights"]), gone


def _many(case, seed):
    """The graphs of one batch of independent solves: sizes log-uniform, 2, 4 or 8 blocks, mean degree
    8 to 24, unit weights, 1% labelled; the sizes are the case's, the edges the seed's."""
    rs = np.random.RandomState(case["count"] * 7919 + case["n_max"])
    for i in range(case["count"]):
        n = int(round(math.exp(rs.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        K, deg = int(rs.choice([2, 4, 8])), float(rs.uniform(8, 24))
        g = _gen(seed * 4099 + i)
        key, w, y = _graph(g, n, K, 0.75 * deg, 0.25 * deg, "unit", connected=True)
        yield n, K, key, w, y, _labelled(g, n, K, y, 0.01)


def _host(x):
    """An array of an edge batch as it arrives: in pinned host memory."""
    return x.cpu().pin_memory()


def _apply_inputs(case, seed):
    g = _gen(seed)
    n, dt = case["n"], getattr(torch, case["dtype"])
    key, w, _ = _graph(g, n, 2, 0.0, case["deg"], "lognormal")
    X = torch.rand((n, case["C"]), generator=g, device=DEV).to(dt)
    csr = _csr_of(key, w.to(dt), n)
    diag = torch.zeros(n, dtype=F64, device=DEV).index_add_(
        0, torch.repeat_interleave(torch.arange(n, device=DEV), torch.diff(csr[0].long())), csr[2].double())
    return csr, X, (diag + 0.25).to(torch.float32 if dt == torch.bfloat16 else dt)


def _edge_list(case, seed):
    g = _gen(seed)
    n, m = case["n"], int(case["n"] * case["deg"] / 2)
    return n, _uniform(g, m, n).to(torch.int32), _uniform(g, m, n).to(torch.int32)


# -- the calls --------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "update":
        n, K = case["n"], case["K"]
        g, key, w, y, lab = _make_graph(case, seed)
        new, nw, gone = _batch(g, case, key)
        es = stream.EdgeStream(_dataset("update", _csr_of(key, w, n), y, K), lab, components=case["components"])
        if case["target"]:
            solver = solvers.IncrementalLP(n, K, "float32", tol=1e-3, method="pcg", target_relres=case["target"])
        else:
            solver = solvers.IncrementalLP(n, K)
        solver.solve(es.system)
        iu, iv, iw = _host((new // n).to(torch.int32)), _host((new % n).to(torch.int32)), _host(nw)
        du, dv = _host((key[gone] // n).to(torch.int32)), _host((key[gone] % n).to(torch.int32))
        dw = _host(w[gone])
        # the batch and the one that takes it back: every pass updates the resident graph, in turn
        turns = [dict(ins_u=iu, ins_v=iv, ins_w=iw, del_u=du, del_v=dv),
                 dict(ins_u=du, ins_v=dv, ins_w=dw, del_u=iu, del_v=iv)]
        return {"kind": kind, "stream": es, "solver": solver, "turns": turns, "components": case["components"]}
    if kind in ("static", "reference", "amg"):
        n, K = case["n"], case["K"]
        _, key, w, y, lab = _make_graph(case, seed)
        ds = _dataset(kind, _csr_of(key, w, n), y, K)
        s = {"kind": kind, "ds": ds, "lab": lab, "all": torch.ones(n, dtype=torch.bool, device=DEV), "case": case}
        if kind != "static":
            s["system"] = stream.build_system(ds, s["all"], lab, dtype="float64" if kind == "reference" else "float32")
        return s
    if kind in ("fresh", "batched"):
        todo = []
        for n, K, key, w, y, lab in _many(case, seed):
            ds = _dataset("one", _csr_of(key, w, n), y, K)
            active = torch.ones(n, dtype=torch.bool, device=DEV)
            todo.append((ds, active, lab) if kind == "fresh" else stream.build_system(ds, active, lab, dtype="float32"))
        return {"kind": kind, "todo": todo}
    if kind == "apply":
        (indptr, col, w), X, diag = _apply_inputs(case, seed)
        n = case["n"]
        return {"kind": kind, "W": CSR(w, col, indptr, (n, n)), "X": X, "diag": diag}
    if kind == "components":
        return {"kind": kind, "edges": _edge_list(case, seed)}
    g = _gen(seed)
    n, K = case["n"], case["K"]
    key, w, y = _graph(g, n, K, 0.85 * case["deg"], 0.15 * case["deg"], "lognormal")
    ds = _dataset("arrivals", _csr_of(key, w, n), y, K)
    ds.order = torch.randperm(n, generator=g, device=DEV)
    make = stream.IncrementalStream if case["resident"] else stream.Stream
    return {"kind": kind, "stream": make(ds, init_frac=0.5, n_batches=case["batches"], seed=int(seed) % 65536), "case": case}


def run(s):
    kind = s["kind"]
    if kind == "update":
        es, solver = s["stream"], s["solver"]
        b = s["turns"][0]
        s["turns"].reverse()
        S = es.apply_edges(**b)
        solver.solve(S)
        solver.relabel(S)
        out = {"scores": solver.F.float()}  # scores are handed on in fp32
        if s["components"]:
            out["components"], out["n_components"] = es.components()
        return out
    if kind == "static":
        ds, c = s["ds"], s["case"]
        S = stream.build_system(ds, s["all"], s["lab"], dtype="float32")
        solver = solvers.DynLPPlus(ds.n, ds.K, "float32", method="pcg", tol=1e-3, target_relres=c["target"])
        solver.solve(S)
        return solver.scores(S).float()
    if kind == "reference":
        F, hmax, _ = solvers.Reference(s["ds"].n, s["ds"].K).solve(s["system"])
        return F
    if kind == "amg":
        solver = solvers.DynLPPlus(s["ds"].n, s["ds"].K, "float32", method="amg", tol=1e-3, target_relres=1e-8,
                                   lowp=s["case"]["lowp"])
        solver.solve(s["system"])
        return solver.scores(s["system"]).float()
    if kind == "fresh":
        systems = [stream.build_system(ds, active, lab, dtype="float32") for ds, active, lab in s["todo"]]
        return [F.float() for F in batched.solve_many_mixed(systems, target_relres=1e-6)[0]]
    if kind == "batched":
        return batched.solve_many(s["todo"], target_relres=1e-6)[0]
    if kind == "apply":
        return kernels.spmm_axpy(s["W"], s["X"], a=s["diag"], b=-1.0)
    if kind == "components":
        return cc.connected_components(*s["edges"])
    c = s["case"]
    solver = solvers.make(c["solver"], c["n"], c["K"], dtype="float32", delta=1e-4, tol=1e-3, group="auto")
    out = []
    for S in s["stream"].batches():
        solver.solve(S)
        out.append(solver.F.float())
    return out


# -- what a pass cannot do without ------------------------------------------------------------------
def work(case):
    """Each input read once and each output written once: the graph (4-byte columns and weights of both
    directions of every edge), the scores before and after, the labels. Flops: one multiply-add per
    stored entry and column for one application of the operator (the number of applications that an
    iterative solve needs is not counted)."""
    kind = case["kind"]
    if kind in ("fresh", "batched"):
        rs = np.random.RandomState(case["count"] * 7919 + case["n_max"])
        b = f = 0.0
        for _ in range(case["count"]):
            n = int(round(math.exp(rs.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
            K, deg = int(rs.choice([2, 4, 8])), float(rs.uniform(8, 24))
            C = 1 if K == 2 else K
            b += n * (deg * 8 + 4 + 8 * C + 8)
            f += 2 * n * deg * C
        return {"bytes": b, "flops": f}
    n = case["n"]
    if kind == "components":
        return {"bytes": 8 * (n * case["deg"] / 2) + 4 * n, "flops": 0}
    if kind == "apply":
        e = {"float32": 4, "float64": 8, "bfloat16": 2}[case["dtype"]]
        o = {"float32": 4, "float64": 8, "bfloat16": 4}[case["dtype"]]
        return {"bytes": n * (case["deg"] * (4 + e) + 4 + case["C"] * (e + o) + o),
                "flops": 2 * n * case["deg"] * case["C"]}
    C = 1 if case["K"] == 2 else case["K"]
    deg = case["deg"] if kind == "arrivals" else case["deg_in"] + case["deg_cross"]
    passes = case["batches"] + 1 if kind == "arrivals" else 1
    return {"bytes": passes * n * (deg * 8 + 4 + 2 * 8 * C + 4), "flops": passes * 2 * n * deg * C}


# -- the same results in 64 bits, from plain torch --------------------------------------------------
def _matvec(indptr, col, w, n):
    A = torch.sparse_csr_tensor(indptr.long(), col.long(), w.double(), (n, n), check_invariants=False)
    return lambda X: A @ X


def _harmonic(indptr, col, w, y, lab, K):
    """The harmonic scores of every unlabelled vertex whose component holds a label (0 elsewhere) by
    fp64 conjugate gradients, and the mask of those vertices."""
    n = y.numel()
    A = _matvec(indptr, col, w, n)
    reach = lab.clone()
    while True:
        more = (A(reach.double()[:, None])[:, 0] > 0) | reach
        if bool((more == reach).all()):
            break
        reach = more
    U = reach & ~lab
    onehot = torch.zeros((n, K), dtype=F64, device=DEV)
    onehot[lab, y[lab].long()] = 1.0
    u = U.double()[:, None]
    rhs = A(onehot) * u
    rhs = rhs[:, 1:2] if K == 2 else rhs
    diag = torch.where(U, A(torch.ones((n, 1), dtype=F64, device=DEV))[:, 0], torch.ones(n, dtype=F64, device=DEV))[:, None]
    X = torch.zeros_like(rhs)
    R = rhs.clone()
    Y = R / diag
    P = Y.clone()
    rz = (R * Y).sum(0)
    stop = 1e-13 * torch.clamp(rhs.norm(dim=0), min=1e-300)
    for _ in range(5000):
        AP = (diag * P - A(P)) * u
        pap = (P * AP).sum(0)
        a = torch.where(pap > 0, rz / torch.where(pap > 0, pap, torch.ones_like(pap)), torch.zeros_like(pap))
        X += a * P
        R -= a * AP
        if bool((R.norm(dim=0) <= stop).all()):
            break
        Y = R / diag
        rz2 = (R * Y).sum(0)
        P = Y + torch.where(rz > 0, rz2 / torch.where(rz > 0, rz, torch.ones_like(rz)), torch.zeros_like(rz)) * P
        rz = rz2
    return X * u, U


def exact(case, seed):
    kind = case["kind"]
    if kind in ("components", "arrivals"):
        return None  # whole numbers; frontier sweeps that stop at a threshold of their own
    if kind == "apply":
        (indptr, col, w), X, diag = _apply_inputs(case, seed)
        X = X.double()
        return diag.double()[:, None] * X - _matvec(indptr, col, w, case["n"])(X)
    if kind in ("fresh", "batched"):
        out = []
        for n, K, key, w, y, lab in _many(case, seed):
            F, U = _harmonic(*_csr_of(key, w, n), y, lab, K)
            out.append(F[U])
        return out
    g, key, w, y, lab = _make_graph(case, seed)
    n, K = case["n"], case["K"]
    if kind == "update":
        new, nw, gone = _batch(g, case, key)
        keep = torch.ones(key.numel(), dtype=torch.bool, device=DEV)
        keep[gone] = False
        key, order = torch.sort(torch.cat([key[keep], new]))
        w = torch.cat([w[keep], nw])[order]
        F, _ = _harmonic(*_csr_of(key, w, n), y, lab, K)
        return {"scores": F, "components": None, "n_components": None} if case["components"] else {"scores": F}
    F, U = _harmonic(*_csr_of(key, w, n), y, lab, K)
    return F[U]
