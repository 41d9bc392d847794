"""The kernels x points sweep behind chol_quad_form, the predictive density and
its backward, at the edges of its tiles: one point, one kernel, a point more
and fewer than a CTA's tile, a kernel more than a staged group, every padded
dimension, and factors or points with infinities.

Tolerances: y_i is a sum of at most D products of a rounded difference, Q a sum
of D squares, so |Q - exact| <= 2 (D + 3) u sum_i (sum_j |U_ji| |d_j|)^2 to first
order, u the unit roundoff."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS = [1, 2, 3, 4, 8, 11, 16, 24, 25, 32, 33, 48, 63, 64]
ROUND = {torch.float32: 2.0**-24, torch.float64: 2.0**-53}


@pytest.fixture(scope="module")
def K():
    from lakde_b200 import kernels

    return kernels


def inputs(N, M, D, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    W = rn(N, D, D).triu(1) / math.sqrt(D) + torch.diag_embed(0.5 + rn(N, D).abs())
    return W.to(dtype), rn(N, D).to(dtype), rn(M, D).to(dtype)


def quad_ref(W, Xn, Xm):
    """Q and its first-order error scale in float64."""
    d = Xm.double()[None] - Xn.double()[:, None]
    Wd = W.double()
    return (d @ Wd).square().sum(2), (d.abs() @ Wd.abs()).square().sum(2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", DIMS)
def test_quad_edges(K, D, dtype):
    for N, M in [(1, 1), (3, 127), (33, 129), (9, 255), (17, 513), (70, 257)]:
        W, Xn, Xm = inputs(N, M, D, dtype, 100 * D + N)
        ref, scale = quad_ref(W, Xn, Xm)
        err = (K.chol_quad_form(W, Xn, Xm).double() - ref).abs()
        assert (err <= 2 * (D + 3) * ROUND[dtype] * scale).all(), (N, M)


@pytest.mark.parametrize("D", [2, 8, 24, 48, 64])
def test_quad_infinities(K, D):
    """An infinite coordinate gives an infinite (never a NaN) quad form where
    no 0 * inf belongs to the sum, a NaN one a NaN.  At the kernels' padded
    dimensions only: below them the zero columns of the padding always took
    part (0 * inf)."""
    W, Xn, Xm = inputs(5, 40, D, torch.float32, D)
    W = W.abs().triu() + 0.1 * torch.ones_like(W).triu()
    Xm[3, D - 1] = math.inf
    Xm[5, 0] = -math.inf
    Xm[7, D // 2] = math.nan
    q = K.chol_quad_form(W, Xn, Xm)
    assert torch.isinf(q[:, [3, 5]]).all() and torch.isnan(q[:, 7]).all()
    rest = [m for m in range(40) if m not in (3, 5, 7)]
    ref, scale = quad_ref(W, Xn, Xm[rest])
    assert ((q[:, rest].double() - ref).abs() <= 2 * (D + 3) * 2.0**-24 * scale).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", DIMS)
def test_density_edges(K, D, dtype):
    """log p against float64; the tolerance is the spread of the terms' own
    error: h dQ / (1 + Q) (h = (nu + 1) / 2), the rounding of the terms, and the
    hardware log / exp of the float32 path (2e-4, as the other density tests)."""
    for N, M in [(1, 1), (7, 130), (33, 513), (300, 257)]:
        W, X, Y = inputs(N, M, D, dtype, 100 * D + N)
        g = torch.Generator(device="cuda").manual_seed(N)
        nu = (D + 1 + 4 * torch.rand(N, generator=g, device="cuda", dtype=torch.float64)).to(dtype)
        lc = torch.randn(N, generator=g, device="cuda", dtype=torch.float64).to(dtype)
        out = K.log_pred_density(X, W, nu, lc, Y).double()
        q, scale = quad_ref(W, X, Y)
        h = (nu.double()[:, None] + 1) / 2
        lp = lc.double()[:, None] - h * torch.log1p(q)
        ref = torch.logsumexp(lp, 0) - math.log(N)
        u = ROUND[dtype]
        tol = (h * 2 * (D + 3) * u * scale / (1 + q)).amax(0) + 64 * u * lp.abs().amax(0)
        tol = tol + (2e-4 if dtype == torch.float32 else 1e-13)
        assert ((out - ref).abs() <= tol).all(), (N, M)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", [1, 2, 8, 13, 24, 32, 33, 64])
def test_backward_edges(D, dtype):
    """Score and factor gradients against float64 autograd of the same formula.
    Errors are relative to the sum of the absolute terms of each output."""
    from lakde_b200.grad import log_pred_density

    for N, M in [(1, 1), (9, 129), (70, 257)]:
        W, X, Y = inputs(N, M, D, dtype, 100 * D + N)
        L = W.mT.contiguous()
        nu = torch.full((N,), D + 2.0, device="cuda", dtype=dtype)
        a, b = Y.clone().requires_grad_(), L.clone().requires_grad_()
        log_pred_density(X, b, nu, a).sum().backward()
        Yd, Ld = Y.double().requires_grad_(), L.double().requires_grad_()
        z = torch.linalg.solve_triangular(Ld, (Yd[None] - X.double()[:, None]).mT, upper=False)
        logdet = -2 * torch.diagonal(Ld, dim1=1, dim2=2).log().sum(1)
        h = (nu.double() + 1) / 2
        lp = (0.5 * logdet)[:, None] - h[:, None] * torch.log1p(z.square().sum(1))
        torch.logsumexp(lp, 0).sum().backward()
        # condition of the factors times the sums' length times the roundoff
        tol = 200 * (D + math.sqrt(M * N)) * ROUND[dtype]
        for got, ref in ((a.grad, Yd.grad), (b.grad, Ld.grad.tril())):
            cond = torch.linalg.cond(Ld.detach()).max().item()
            assert (got.double() - ref).norm() <= tol * max(cond, 1.0) * ref.norm() + tol, (N, M)
