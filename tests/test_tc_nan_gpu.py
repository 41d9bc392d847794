"""NaN inputs of the tensor-core kernels: what a failed factor or a NaN point
makes of a density, a log rho or a scatter matrix stays visible."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _mixture(N, Nq, D, seed=0):
    g = torch.Generator().manual_seed(seed)
    X = torch.randn(N, D, generator=g)
    Y = torch.randn(Nq, D, generator=g)
    W = torch.randn(N, D, D, generator=g).triu(1) / D**0.5 + torch.diag_embed(0.5 + torch.rand(N, D, generator=g))
    nu = D + 1 + torch.rand(N, generator=g)
    lc = torch.randn(N, generator=g)
    return [v.to(DEV) for v in (X, W, nu, lc, Y)]


@pytest.mark.parametrize("D", [13, 21, 43, 63])
@pytest.mark.parametrize("N,Nq", [(1, 5), (3, 300), (100, 100), (5000, 300)])
@pytest.mark.parametrize("part", ["factor", "coefficient"])
def test_density_keeps_the_nan_of_one_failed_kernel(D, N, Nq, part):
    """One kernel with a NaN factor or coefficient, below and above the number
    of CTAs: NaN for every query wherever lakde_log_pred_density says so."""
    from lakde_b200 import kernels as K

    X, W, nu, lc, Y = _mixture(N, Nq, D)
    at = N // 2
    if part == "factor":
        W[at] = float("nan")
    else:
        lc[at] = float("nan")
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    plain = K.log_pred_density(X, W, nu, lc, Y)
    mixed = K.log_pred_density_tc(X, K.pack_w_cores(W), nu, lc, Y, err)
    assert int(err) == 0
    if N > 1:
        assert torch.isnan(plain).all()
    assert torch.equal(torch.isnan(mixed), torch.isnan(plain))
    assert torch.equal(torch.isneginf(mixed), torch.isneginf(plain))
