"""The grounded system's own bookkeeping (host logic, on CPU tensors)."""
import dataclasses

import torch

from dynlplus_b200.backend import CSR
from dynlplus_b200.stream import System


def test_solved_rows_are_those_of_the_systems_mask():
    """The stream's count stands for its own mask; a system with another one counts it."""
    n = 6
    W = CSR(torch.ones(1), torch.zeros(1, dtype=torch.int32), torch.tensor([0, 1, 1, 1, 1, 1, 1], dtype=torch.int32), (n, n))
    z = torch.zeros(n)
    no = torch.zeros(n, dtype=torch.bool)
    mask = torch.tensor([1, 1, 0, 1, 0, 0], dtype=torch.bool)
    S = System(t=0, U=torch.arange(n), W=W, s=z, diag=z + 1, B=torch.zeros(n, 2), rhs=torch.zeros(n, 1),
               prior=torch.zeros(1), is_new=no, seed=no, comps={}, K=2, C=1, eta=0.0, n_inserted=0, n_deleted=0, n_active=n,
               solved=mask)
    assert S.n_solved == 3
    S.solved_count = 3
    assert S.n_solved == 3 and S.astype("float64").n_solved == 3 and S.astype("float64").solved_count == 3
    T = dataclasses.replace(S, solved=torch.ones(n, dtype=torch.bool))
    assert T.n_solved == n
    assert dataclasses.replace(S, solved=None).n_solved == n
