"""Backward of the predictive density element by element: cw, sw, S_c and the
score of lakde_log_pred_density_bwd against float64, at the edges of query
tiles, kernel groups and chunks, with bounds from the absolute terms of each
output, so that a query, a kernel or a column left out shows."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", [1, 2, 5, 8, 13, 24, 33, 48, 64])
@pytest.mark.parametrize("N,M", [(1, 1), (5, 129), (70, 257), (130, 63), (601, 64), (40, 1030)])
def test_elements(dtype, D, N, M):
    from lakde_b200 import kernels as K

    g = torch.Generator(device=DEV).manual_seed(97 * N + M + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    W = rnd(N, D, D).triu(1) / (2 * D) + torch.diag_embed(0.5 + torch.rand(N, D, generator=g, device=DEV,
                                                                          dtype=torch.float64))
    X, Y = rnd(N, D).to(dtype), rnd(M, D).to(dtype)
    W = W.to(dtype)
    nu = (D + 1 + torch.rand(N, generator=g, device=DEV, dtype=torch.float64)).to(dtype)
    lc = rnd(N).to(dtype)
    gout = rnd(M).to(dtype)
    out = K.log_pred_density(X, W, nu, lc, Y)
    gY, sw, S = K.log_pred_density_bwd(X, W, nu, lc, Y, out, gout)

    # float64 from the same rounded inputs, the softmax weights from the same `out`
    X6, Y6, W6, nu6, lc6, g6 = (v.double() for v in (X, Y, W, nu, lc, gout))
    u = torch.finfo(dtype).eps
    d = Y6[None] - X6[:, None]  # N, M, D
    z = d @ W6
    zm = (Y6.abs()[None] + X6.abs()[:, None]) @ W6.abs()  # the magnitudes behind z
    dm = Y6.abs()[None] + X6.abs()[:, None]
    Q = z.square().sum(2)
    dQ = (D + 4) * u * (2 * z.abs() * zm).sum(2) + D * u * Q + ((D + 4) * u) ** 2 * zm.square().sum(2)
    h = (nu6 + 1)[:, None] / 2
    lp = lc6[:, None] - h * torch.log1p(Q)
    w = torch.exp(lp - (out.double() + math.log(N))[None])
    # of w: h dQ / (1 + Q) through the log, the rounding of lp, of `out` + log N and of exp and log
    lw = h * (dQ / (1 + Q) + 4 * u * torch.log1p(Q)) + 6 * u * (lp.abs() + lc6.abs()[:, None] + out.double().abs()[None] +
                                                               math.log(N)) + 6 * u
    assert lw.max() < 0.05  # the bound below is of first order
    rel = 1.1 * lw + dQ / (1 + Q) + 8 * u
    c = g6[None] * w / (1 + Q)
    ca = c.abs()

    sw_want, sw_tol = (g6[None] * w).sum(1), ((1.1 * lw + (M + 8) * u) * (g6[None] * w).abs()).sum(1)
    assert ((sw.double() - sw_want).abs() <= sw_tol).all()

    S_want = torch.einsum("nm,nmi,nmj->nij", c, d, d)
    S_tol = torch.einsum("nm,nmi,nmj->nij", ca * (rel + (M + 8) * u), dm, dm)
    assert ((S.double() - S_want).abs() <= S_tol).all()
    assert torch.equal(S, S.mT)

    Uz = torch.einsum("nij,nmj->nmi", W6, z)
    Uzm = torch.einsum("nij,nmj->nmi", W6.abs(), zm)
    f = -2 * h * c
    want = (f[..., None] * Uz).sum(0)
    tol = (f.abs()[..., None] * (rel[..., None] * Uz.abs() + (2 * D + N + 12) * u * Uzm)).sum(0)
    assert ((gY.double() - want).abs() <= tol).all()
