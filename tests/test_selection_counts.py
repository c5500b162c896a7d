"""Budget arithmetic of the variable-length selection modes on the host, and what its one-launch form refuses."""

import pytest
import torch

from mcsparse_b200.kernels.flash_mcsa.token_sparse import selection_budgets, selection_counts
from oracle.select import selection_counts_ref


@pytest.mark.parametrize("L,n_sink,hi", [(100, 0, 100), (100, 5, 100), (4096, 4, 4096), (32760, 4, 40000), (640, 64, 3)])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_selection_counts_match_oracle(L, n_sink, hi, dtype):
    base = torch.randint(0, hi + 1, (2, 50), generator=torch.Generator().manual_seed(L)).to(dtype)
    assert torch.equal(selection_counts(L, n_sink, 128, base), selection_counts_ref(L, n_sink, 128, base).clamp(max=L))


def test_selection_budgets_refuse_what_they_cannot_read():
    with pytest.raises(RuntimeError):
        selection_budgets(1000, 4, 128, torch.ones(3, dtype=torch.int32))          # not on the GPU
    with pytest.raises(TypeError):
        selection_budgets(1000, 4, 128, torch.ones(3))                             # not counts
