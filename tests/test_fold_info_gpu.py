"""The fit's worst factorisation status: one launch over all kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 256, 1024, 1025, 296 * 1024 + 1, 400_003])
def test_worst_status(n):
    from lakde_b200 import kernels as K

    info = torch.zeros(n, dtype=torch.int32, device="cuda")
    failed = torch.zeros((), dtype=torch.int32, device="cuda")
    K.fold_info(info, failed)
    assert int(failed) == 0
    if n:
        info[n - 1] = -1
        K.fold_info(info, failed)
        assert int(failed) == -1
        info[n - 1], info[n // 2] = 0, -2
        K.fold_info(info, failed)
        assert int(failed) == -2
        info.zero_()
        K.fold_info(info, failed)  # a failure stays
        assert int(failed) == -2
