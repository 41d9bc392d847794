"""lakde_vi_rows on point rows at every alignment its element type allows: the
wide loads are taken only where the rows are 32-byte aligned, and the results
are those of an aligned copy bit for bit (D = 8 and, in float64, 4 have rows of
32 and 64 bytes; D = 5 is padded to 8 and read element-wise)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _at_offset(X, elements):
    """A contiguous copy of X that starts `elements` elements past a 256-byte aligned address."""
    buf = torch.empty(X.numel() + elements, dtype=X.dtype, device=X.device)
    out = buf[elements:].view_as(X)
    out.copy_(X)
    assert buf.data_ptr() % 256 == 0
    return out


def _run(X, P, T, rowptr, col, r, order):
    from lakde_b200 import kernels as K

    N, D = X.shape
    z = lambda: torch.zeros(N, dtype=X.dtype, device=DEV)  # noqa: E731
    out = dict(b=torch.ones_like(z()), jitter=z(), nu=z(), logdet=z(), mm=z(),
               info=torch.zeros(N, dtype=torch.int32, device=DEV),
               logrho=torch.zeros(col.numel(), dtype=X.dtype, device=DEV))
    K.vi_rows(rowptr, col, r, X, float(D), torch.full_like(z(), 1.0 + D / 2), out["b"], 1e-6, out["jitter"],
              torch.finfo(X.dtype).eps, out["nu"], out["logdet"], out["info"], out["logrho"], P=P, T=T, order=order,
              mm=out["mm"])
    return out


@pytest.mark.parametrize("form", ["two_lanes_per_row", "thread_per_row"])
@pytest.mark.parametrize("dtype,D", [(torch.float32, 8), (torch.float64, 8), (torch.float64, 4), (torch.float32, 4),
                                     (torch.float32, 5), (torch.float64, 5)])
@pytest.mark.parametrize("N", [130, 3500, 9000, 25000, 73000])
def test_vi_rows_at_every_alignment(form, dtype, D, N):
    from lakde_b200 import tuning

    g = torch.Generator().manual_seed(N + D)
    k = 12
    X = torch.randn(N, D, generator=g, dtype=torch.float64).to(dtype).to(DEV)
    col = torch.randint(N, (N * k,), generator=g).to(torch.int32).to(DEV)
    r = torch.rand(N * k, generator=g, dtype=torch.float64).to(dtype).to(DEV)
    rowptr = torch.arange(0, N * k + 1, k, device=DEV)
    order = torch.randperm(N, generator=g).to(torch.int32).to(DEV)
    A = torch.randn(N, D, D + 3, generator=g, dtype=torch.float64).to(DEV)
    P64 = A @ A.mT / (D + 3) + 0.1 * torch.eye(D, dtype=torch.float64, device=DEV)
    P, T = P64.to(dtype).contiguous(), torch.linalg.cholesky(P64).to(dtype).contiguous()
    before = tuning.get_choice("vi_rows", D)
    try:
        tuning.set_choice("vi_rows", D, form)
        want = _run(X, P, T, rowptr, col, r, order)
        assert int(want["info"].min()) == 0
        es = X.element_size()
        for offset in (4, 8, 16, 32):
            if offset < es:
                continue
            got = _run(_at_offset(X, offset // es), _at_offset(P, offset // es), _at_offset(T, offset // es), rowptr,
                       col, r, order)
            for key in want:
                torch.testing.assert_close(got[key], want[key], rtol=0, atol=0, msg=f"{key} at offset {offset}")
    finally:
        tuning.set_choice("vi_rows", D, before)
