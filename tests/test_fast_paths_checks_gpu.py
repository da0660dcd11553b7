"""What the fast paths take besides plain calls: layouts, types, limits and inputs that are refused."""
import numpy as np
import pytest
import torch

from dynlplus_b200 import graphs, stream

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
