"""weighted_gram with infinite and NaN weights: as the sum of w_n times the
finished products, element by element."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", [1, 5, 8, 9, 24, 33, 64])
@pytest.mark.parametrize("N,at", [(1, 0), (3, 1), (5, 4), (700, 0), (700, 699), (5000, 2500)])
@pytest.mark.parametrize("weight", [float("inf"), float("-inf"), float("nan")])
def test_one_weight_that_is_not_finite(dtype, D, N, at, weight):
    from lakde_b200 import kernels as K

    g = torch.Generator(device="cuda").manual_seed(N + D)
    W = torch.randn(N, D, D, generator=g, device="cuda", dtype=torch.float64).to(dtype).triu()
    w = torch.rand(N, generator=g, device="cuda", dtype=torch.float64).to(dtype)
    w[at] = weight
    got = K.weighted_gram(W, w)
    one = (W[at].double() @ W[at].double().T) * weight
    assert torch.equal(torch.isnan(got), torch.isnan(one))
    assert torch.equal(torch.isposinf(got), torch.isposinf(one))
    assert torch.equal(torch.isneginf(got), torch.isneginf(one))
