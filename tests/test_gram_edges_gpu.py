"""The weighted Gram sum at every padded dimension and at kernel counts around
the grid's warps, against float64.  Each element is a sum of at most N D
products, so it is within N D rounding errors of 2^-53 of the sum of their
magnitudes."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", [1, 2, 8, 9, 16, 23, 24, 25, 32, 41, 48, 49, 64])
def test_weighted_gram_edges(D, dtype):
    from lakde_b200 import kernels as K

    for N in (1, 3, 5, 1775, 1777, 2400):
        g = torch.Generator(device="cuda").manual_seed(100 * D + N)
        W = torch.randn(N, D, D, generator=g, device="cuda", dtype=torch.float64).triu().to(dtype)
        w = torch.rand(N, generator=g, device="cuda", dtype=torch.float64).to(dtype)
        Wd = W.double()
        ref = ((w.double()[:, None, None] * Wd) @ Wd.mT).sum(0)
        mag = ((w.double()[:, None, None] * Wd.abs()) @ Wd.abs().mT).sum(0)
        err = (K.weighted_gram(W, w) - ref).abs()
        assert (err <= 2 * (N * D + 4) * 2.0**-53 * mag).all(), N
