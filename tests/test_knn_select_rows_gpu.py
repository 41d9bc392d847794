"""lakde_knn_select on either side of the rule that gives a row a warp or a
block: the neighbours and distances of an exact float64 ranking."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("include_self", [False, True])
@pytest.mark.parametrize("nb,N,k", [
    (1, 32769, 5), (255, 40_000, 20), (256, 40_000, 20), (256, 131_073, 20), (1184, 131_073, 5), (1185, 131_073, 5),
    (7, 32768, 152), (599, 3000, 153), (600, 3000, 153), (600, 3000, 492), (599, 700, 492), (1185, 1300, 493),
])
def test_either_form(nb, N, k, include_self):
    from lakde_b200 import kernels as K

    g = torch.Generator(device="cuda").manual_seed(nb + N + k)
    X = torch.randn(N, 3, generator=g, device="cuda", dtype=torch.float64)
    X[N // 2] = X[N // 3]  # equal distances: by index
    row0 = (N - nb) // 2
    rows = torch.arange(nb, device="cuda")
    e = torch.zeros(nb, N, device="cuda", dtype=torch.float64)
    for d in range(3):  # in the kernel's order, so that equal stays equal
        df = X[None, :, d] - X[row0 : row0 + nb, None, d]
        e = torch.addcmul(e, df, df)
    idx = torch.empty(nb, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(nb, k, dtype=torch.float64, device="cuda")
    K.knn_select(e, X, row0, k, include_self=include_self, out_idx=idx, out_dist=dist)
    if not include_self:
        e[rows, row0 + rows] = torch.inf
    want, at = e.sort(dim=1, stable=True)
    assert torch.equal(idx.long(), at[:, :k])
    torch.testing.assert_close(dist, want[:, :k].sqrt(), rtol=1e-14, atol=0)
