"""The fused D <= 8 pass either side of each bound of its packing rule, by
dimension and type (the lanes a row follow the number of points, five more than
rows here; the rows a warp the number of rows)."""

import pytest
import torch

from tests.test_vi_rows_forms_gpu import test_row_packings as compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,D,dtype", [
    (2995, 3, torch.float32), (7995, 7, torch.float32), (7996, 8, torch.float64),
    (17995, 5, torch.float32), (17996, 5, torch.float32), (17995, 8, torch.float32), (17996, 8, torch.float32),
    (17996, 4, torch.float32), (23995, 4, torch.float32), (23995, 8, torch.float64), (23996, 2, torch.float64),
    (40000, 6, torch.float32), (40001, 6, torch.float32), (50000, 4, torch.float32), (50001, 3, torch.float32),
    (56000, 5, torch.float64), (56001, 8, torch.float64), (72001, 4, torch.float64),
])
def test_either_side_of_a_bound(N, D, dtype):
    compare(N, D, dtype)
