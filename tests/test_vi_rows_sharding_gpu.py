"""A shard of lakde_vi_rows gives the rows of the full launch bit for bit, also
where the shard alone would take another launch form than the full set."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("D", [2, 3, 5, 8])
@pytest.mark.parametrize("N,cuts", [
    (3200, (0, 1500, 3200)),
    (9000, (0, 2900, 7000, 9000)),
    (26000, (0, 100, 7900, 26000)),
    (80000, (0, 2000, 26000, 80000)),
])
def test_shards_are_the_rows_of_the_full_launch(dtype, D, N, cuts):
    from lakde_b200 import kernels as K

    g = torch.Generator().manual_seed(N + D)
    lengths = (20 * torch.exp(0.5 * torch.randn(N, generator=g))).round().long().clamp(0, 200)
    rowptr = torch.cat((torch.zeros(1, dtype=torch.int64), lengths.cumsum(0)))
    nnz = int(rowptr[-1])
    X = torch.randn(N, D, generator=g, dtype=torch.float64).to(dtype).to(DEV)
    col = torch.randint(N, (nnz,), generator=g).to(torch.int32).to(DEV)
    r = torch.rand(nnz, generator=g, dtype=torch.float64).to(dtype).to(DEV)
    A = torch.randn(N, D, D + 3, generator=g, dtype=torch.float64)
    P64 = A @ A.mT / (D + 3) + 0.1 * torch.eye(D, dtype=torch.float64)
    P = P64.to(dtype).contiguous().to(DEV)
    T = torch.linalg.cholesky(P64).to(dtype).contiguous().to(DEV)
    a = torch.full((N,), 1.0 + D / 2, dtype=dtype, device=DEV)
    b0 = (0.5 + 1.5 * torch.rand(N, generator=g, dtype=torch.float64)).to(dtype).to(DEV)

    def run(lo, hi):
        p0, p1 = int(rowptr[lo]), int(rowptr[hi])
        n = hi - lo
        z = lambda: torch.zeros(n, dtype=dtype, device=DEV)  # noqa: E731
        out = dict(b=b0[lo:hi].clone(), jitter=z(), nu=z(), logdet=z(), mm=z(),
                   info=torch.zeros(n, dtype=torch.int32, device=DEV),
                   logrho=torch.zeros(p1 - p0, dtype=dtype, device=DEV))
        rp = (rowptr[lo : hi + 1] - p0).to(DEV)
        order = torch.argsort(rp[1:] - rp[:-1], descending=True, stable=True).to(torch.int32)
        K.vi_rows(rp, col[p0:p1].contiguous(), r[p0:p1].contiguous(), X, float(D), a[lo:hi].contiguous(), out["b"],
                  1e-6, out["jitter"], torch.finfo(dtype).eps, out["nu"], out["logdet"], out["info"], out["logrho"],
                  P=P[lo:hi].contiguous(), T=T[lo:hi].contiguous(), order=order, mm=out["mm"], kernel_offset=lo)
        return out

    full = run(0, N)
    for lo, hi in zip(cuts, cuts[1:]):
        part = run(lo, hi)
        for key in ("b", "jitter", "nu", "logdet", "info", "mm"):
            torch.testing.assert_close(part[key], full[key][lo:hi], rtol=0, atol=0, msg=f"{key} of rows {lo}..{hi}")
        p0, p1 = int(rowptr[lo]), int(rowptr[hi])
        torch.testing.assert_close(part["logrho"], full["logrho"][p0:p1], rtol=0, atol=0)
