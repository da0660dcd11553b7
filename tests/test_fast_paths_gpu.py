"""The solvers' fast paths against the general ones, at the sizes where they can go wrong."""
import numpy as np
import pytest
import torch

from dynlplus_b200 import graphs, solvers, stream

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
                                                    (3001, 33, "float32", 24, 10**7), (20_000, 4, "float32", 10, 7)])
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
