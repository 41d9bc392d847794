"""lakde_posterior_factor either side of the number of matrices up to which its
registers are left free (17 to 32 dimensions and below): the same bits, and the
factor of each matrix against float64 torch."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", [9, 16, 17, 24, 32])
def test_either_side_gives_the_same_bits(dtype, D):
    from lakde_b200 import kernels as K

    g = torch.Generator(device="cuda").manual_seed(D)
    N = 1185
    A = torch.randn(N, D, D + 4, generator=g, device="cuda", dtype=torch.float64)
    S = (A @ A.mT / D + 0.1 * torch.eye(D, device="cuda", dtype=torch.float64)).to(dtype)
    P = S.flip(0).contiguous()
    T = torch.linalg.cholesky(P.double()).to(dtype).contiguous()
    nu_0 = torch.full((1,), float(D), dtype=dtype, device="cuda")
    a = torch.full((N,), 2.0, dtype=dtype, device="cuda")
    b = 1 + torch.rand(N, generator=g, device="cuda", dtype=torch.float64).to(dtype)

    def run(n):
        jit = torch.zeros(n, dtype=dtype, device="cuda")
        W, ld, info, L, tr = K.posterior_factor(S[:n].contiguous(), jit, torch.finfo(dtype).eps,
                                                P=P[:n].contiguous(), nu_0=nu_0, a=a[:n].contiguous(),
                                                b=b[:n].contiguous(), T=T[:n].contiguous(), want_L=True, T_lower=True)
        assert int(info.abs().max()) == 0 and float(jit.abs().max()) == 0
        return W, ld, L, tr

    whole = run(N)
    for n in (1184, 1, 777):
        for x, y in zip(run(n), whole):
            torch.testing.assert_close(x, y[:n], rtol=0, atol=0)
    # A_n = S + nu_0 a / b P in the data type (three roundings), W_triu = L^-T
    scale = (nu_0.double() * a.double() / b.double())[:, None, None]
    A64 = S.double() + scale * P.double()
    W64 = whole[0].double()
    u = torch.finfo(dtype).eps
    cond = torch.linalg.cond(A64).max()
    err = (W64.mT @ A64 @ W64 - torch.eye(D, device="cuda", dtype=torch.float64)).abs().max()
    assert float(err) <= 8 * D * u * float(cond)
