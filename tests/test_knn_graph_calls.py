"""Calls of compute_knn_graph that do not depend on a GPU's arithmetic, with
the selection kernel replaced by a sort on the CPU."""

import pytest
import torch

from lakde_b200 import utils


@pytest.fixture
def blocks(monkeypatch):
    """The (rows, columns) of every distance block handed to the selection."""
    seen = []

    def select(dist, X, row0, k, include_self=False, out_idx=None, out_dist=None):
        assert not dist.requires_grad
        nb, N = dist.shape
        seen.append((nb, N))
        e = (X[row0 : row0 + nb, None] - X[None]).square().sum(2)
        # the block orders the points as the distances do
        assert torch.equal(dist.argsort(dim=1, stable=True), e.argsort(dim=1, stable=True))
        if not include_self:
            e[torch.arange(nb), torch.arange(nb) + row0] = torch.inf
        d, i = e.sort(dim=1, stable=True)
        out_idx.copy_(i[:, :k])
        if out_dist is not None:
            out_dist.copy_(d[:, :k].sqrt())
        return out_idx

    monkeypatch.setattr(utils.kernels, "knn_select", select)
    return seen


def _points(N, D, seed=0):
    return torch.randn(N, D, generator=torch.Generator().manual_seed(seed), dtype=torch.float64)


def _exact(X, k):
    e = (X[:, None] - X[None]).square().sum(2)
    e.fill_diagonal_(torch.inf)
    d, i = e.sort(dim=1, stable=True)
    return d[:, :k].sqrt(), i[:, :k]


def test_no_points(blocks):
    I = utils.compute_knn_graph(torch.empty(0, 5), 3)
    assert I.shape == (0, 3) and I.dtype == torch.int32
    d, I = utils.compute_knn_graph(torch.empty(0, 5), 3, return_dists=True)
    assert d.shape == I.shape == (0, 3)
    assert blocks == []


def test_points_that_require_grad(blocks):
    X = _points(60, 4).requires_grad_()
    d, I = utils.compute_knn_graph(X, 7, return_dists=True)
    ed, ei = _exact(X.detach(), 7)
    assert torch.equal(I.long(), ei)
    torch.testing.assert_close(d, ed)
    assert not d.requires_grad


@pytest.mark.parametrize("bsize,sizes", [(16, [16, 16, 16, 2]), (50, [50]), (77, [50]), (1024, [50])])
def test_a_small_block_size_bounds_the_block(blocks, bsize, sizes):
    """Below the default, bsize is the number of rows of distances held at once."""
    X = _points(50, 3)
    assert torch.equal(utils.compute_knn_graph(X, 5, bsize=bsize).long(), _exact(X, 5)[1])
    assert blocks == [(nb, 50) for nb in sizes]


def test_the_default_block_grows_to_two_gigabytes(blocks, monkeypatch):
    X = _points(1500, 2)
    utils.compute_knn_graph(X, 5)
    utils.compute_knn_graph(X, 5, bsize=1400)
    utils.compute_knn_graph(X, 5, bsize=1023)
    assert blocks == [(1500, 1500), (1500, 1500), (1023, 1500), (477, 1500)]


@pytest.mark.parametrize("bsize", [0, -1])
def test_block_size_must_be_positive(blocks, bsize):
    with pytest.raises(ValueError):
        utils.compute_knn_graph(_points(20, 2), 3, bsize=bsize)
