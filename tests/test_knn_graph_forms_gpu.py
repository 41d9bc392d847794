"""compute_knn_graph on either side of the size from which the norms join the
distance GEMM as a dimension, in whole and in cut blocks."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 1025, 8192, 8193, 9001])
@pytest.mark.parametrize("D,offset", [(2, 0.0), (21, 50.0)])
@pytest.mark.parametrize("bsize", [1000, 1024])
def test_exact_on_either_side(N, D, offset, bsize):
    from lakde_b200.utils import compute_knn_graph

    g = torch.Generator(device="cuda").manual_seed(N + D)
    X = torch.randn(N, D, generator=g, device="cuda") + offset
    k = min(20, N - 1)
    dist, idx = compute_knn_graph(X, k, bsize=bsize, return_dists=True, dtype=torch.int64)
    Xd = X.double()
    for i in range(0, N, 2048):
        e = torch.zeros(min(2048, N - i), N, device="cuda", dtype=torch.float64)
        for d in range(D):
            df = Xd[None, :, d] - Xd[i : i + 2048, None, d]
            e = torch.addcmul(e, df, df)
        rows = torch.arange(len(e), device="cuda")
        e[rows, i + rows] = torch.inf
        want, at = e.sort(dim=1, stable=True)
        assert torch.equal(idx[i : i + 2048], at[:, :k])
        torch.testing.assert_close(dist[i : i + 2048].double(), want[:, :k].sqrt(), rtol=1e-7, atol=0)
