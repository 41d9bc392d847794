"""chol_quad_form and the predictive density where a CTA's chunk of kernels is
shorter than a stage, fills one, or fills two and a part (only what is staged is
cleared): against float64 torch, with garbage left in the SMs' shared memory by
a launch on NaN inputs before."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _inputs(N, M, D, dtype, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    W = torch.randn(N, D, D, generator=g, device=DEV, dtype=torch.float64).triu(1) / D**0.5
    W = W + torch.diag_embed(0.5 + torch.rand(N, D, generator=g, device=DEV, dtype=torch.float64))
    X = torch.randn(N, D, generator=g, device=DEV, dtype=torch.float64)
    Y = torch.randn(M, D, generator=g, device=DEV, dtype=torch.float64)
    return W.to(dtype), X.to(dtype), Y.to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", [1, 3, 8, 13, 16, 21, 32, 40, 63])
@pytest.mark.parametrize("N,M", [(1, 1), (1, 5000), (9, 700), (64, 2000), (70, 60_000), (700, 1000), (1000, 1)])
def test_quad_form(dtype, D, N, M):
    from lakde_b200 import kernels as K

    W, X, Y = _inputs(N, M, D, dtype, N + M + D)
    bad = torch.full((64, D, D), float("nan"), dtype=dtype, device=DEV)
    K.chol_quad_form(bad, torch.full((64, D), float("nan"), dtype=dtype, device=DEV), Y[:1].expand(4096, D).contiguous())
    got = K.chol_quad_form(W, X, Y).double()
    W64, X64, Y64 = W.double(), X.double(), Y.double()
    u = torch.finfo(dtype).eps
    for n0 in range(0, N, 16):
        d = Y64[None] - X64[n0 : n0 + 16, None]
        y = d @ W64[n0 : n0 + 16]
        # y_i = sum of D products: (D + 2) u times the sum of their magnitudes; then squared and summed
        mag = (Y64.abs()[None] + X64.abs()[n0 : n0 + 16, None]) @ W64[n0 : n0 + 16].abs()
        want = y.square().sum(2)
        tol = (D + 3) * u * (2 * y.abs() * mag + (D + 3) * u * mag.square()).sum(2) + D * u * want
        assert ((got[n0 : n0 + 16] - want).abs() <= tol).all()
