"""failed = min(failed, min(info)) for values of either sign."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 1025, 400_003])
@pytest.mark.parametrize("start,low,want", [(5, 3, 3), (5, 9, 5), (0, 7, 0), (-1, 0, -1), (2, -4, -4), (-4, -2, -4)])
def test_minimum_of_both(n, start, low, want):
    from lakde_b200 import kernels as K

    info = torch.full((n,), 2**31 - 1, dtype=torch.int32, device="cuda")
    info[n // 2] = low
    failed = torch.full((), start, dtype=torch.int32, device="cuda")
    K.fold_info(info, failed)
    assert int(failed) == want
