"""Points with a coordinate that is not finite have no neighbours (-1) and are
nobody's, in both forms of the distance GEMM and of the selection."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("N,D,k", [(60, 2, 5), (700, 3, 300), (1500, 1, 30), (9000, 5, 40), (9000, 5, 600)])
def test_rows_and_columns(N, D, k, bad):
    from lakde_b200.utils import compute_knn_graph

    g = torch.Generator(device="cuda").manual_seed(N)
    X = torch.randn(N, D, generator=g, device="cuda")
    rows = torch.tensor([0, 17, N - 1], device="cuda")
    X[rows, 0] = bad
    dist, idx = compute_knn_graph(X, k, return_dists=True)
    good = torch.ones(N, dtype=torch.bool, device="cuda")
    good[rows] = False
    assert (idx[rows] == -1).all() and torch.isinf(dist[rows]).all()
    # the others: the graph of the finite points alone
    d2, i2 = compute_knn_graph(X[good].contiguous(), k, return_dists=True)
    at = good.nonzero().squeeze(1)
    assert torch.equal(idx[good].long(), at[i2.long()])
    assert torch.equal(dist[good], d2)
