"""The fused D <= 8 pass packs 2 to 32 rows a warp by the number of rows; row
counts at the edges of each packing, ragged rows, against the unfused kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 7, 3000, 3001, 8000, 8001, 24000, 24001, 72000, 72001])
@pytest.mark.parametrize("D,dtype", [(2, torch.float32), (5, torch.float64), (8, torch.float32)])
def test_row_packings(N, D, dtype):
    from lakde_b200 import kernels as K

    g = torch.Generator().manual_seed(N + D)
    npts, lo = N + 5, 3  # rows are points 3 .. N + 2
    X = torch.randn(npts, D, generator=g, dtype=torch.float64)
    counts = torch.randint(0, 40, (N,), generator=g)
    counts[0] = 37  # a group of lanes and a batch left ragged
    rowptr = torch.cat((torch.zeros(1, dtype=torch.int64), counts.cumsum(0)))
    nnz = int(rowptr[-1])
    col = torch.randint(npts, (nnz,), generator=g, dtype=torch.int32)
    r = torch.rand(nnz, generator=g, dtype=torch.float64)
    A = torch.randn(N, D, D, generator=g, dtype=torch.float64)
    P = 0.2 * (A @ A.mT) + torch.eye(D, dtype=torch.float64)
    T = torch.linalg.cholesky(P).contiguous()  # row-major: its rows are read as they are
    a, b = 2 + 2 * torch.rand(N, generator=g), 1 + 2 * torch.rand(N, generator=g)
    X, r, P, T, a, b = (t.to(dtype).cuda() for t in (X, r, P, T, a, b))
    rowptr, col = rowptr.cuda(), col.cuda()
    nu0, b0, eps = D + 0.5, 1e-6, torch.finfo(dtype).eps

    def unfused(*ts):  # in float64
        X, r, P, T, a, b = (t.double() for t in ts)
        S, nu = K.mstep(rowptr, col, r, X, nu0, kernel_offset=lo)
        jit = torch.zeros(N, dtype=torch.float64).cuda()
        W, logdet, info, _, trace = K.posterior_factor(
            S, jit, eps, P=P, nu_0=torch.tensor(nu0).cuda(), a=a, b=b, T=T)
        lr = K.estep_logrho(rowptr, col, X, W, nu, logdet, kernel_offset=lo)
        return nu, logdet, nu * trace, b0 + nu0 * nu * trace / 2, lr

    ref = unfused(X, r, P, T, a, b)
    order = torch.argsort(counts, descending=True, stable=True).to(torch.int32).cuda()
    nu, ld, mm, jit = (torch.full((N,), float("nan"), dtype=dtype).cuda() for _ in range(4))
    jit.zero_()
    info = torch.full((N,), 7, dtype=torch.int32).cuda()
    lr = torch.full((nnz,), float("nan"), dtype=dtype).cuda()
    K.vi_rows(rowptr, col, r, X, nu0, a, b, b0, jit, eps, nu, ld, info, lr, P=P, T=T, order=order, mm=mm,
              kernel_offset=lo)
    assert (info == 0).all() and (jit == 0).all()
    # S is summed and the factor rounded in the type of the data: at most 40
    # terms, condition below 1e3 (P >= I, eigenvalues of S + P below 1e3)
    tol = 1e-4 if dtype == torch.float32 else 1e-11
    for name, got, want in zip(("nu", "logdet", "mm", "b"), (nu, ld, mm, b), ref):
        torch.testing.assert_close(got.double(), want, rtol=tol, atol=tol * D, msg=lambda m: f"{name}: {m}")
    own = torch.isinf(ref[4])
    assert torch.equal(own, torch.isinf(lr.double()))
    scale = float(ref[4][~own].abs().max()) if (~own).any() else 1.0
    torch.testing.assert_close(lr.double()[~own], ref[4][~own], rtol=tol, atol=tol * scale)
