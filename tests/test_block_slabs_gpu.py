"""The block schedule's dense E-step over slabs of points: any slab width gives
the entries of one slab over all points, in the same order."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,block,entries", [
    (300, 64, 1),            # a slab per block of points, ragged last block (44 rows)
    (300, 64, 64 * 64 * 2),  # two blocks a slab, the last slab of one ragged block
    (256, 64, 64 * 64 * 3),  # slabs of three blocks, whole last slab of one
    (50, 64, 1),             # one kernel block, fewer points than a block
])
@pytest.mark.parametrize("threshold", [0, 1e-3])
def test_slab_width(monkeypatch, n, block, entries, threshold):
    from lakde_b200 import LocalKNearestKDE
    from lakde_b200 import local_adaptive_kde as la

    g = torch.Generator().manual_seed(n)
    X = torch.randn(n, 3, generator=g, dtype=torch.float64).cuda()
    model = LocalKNearestKDE(k_or_knn_graph=12, block_size=block)
    model.fit(X, iterations=1, sparsity_threshold=threshold)
    for bi in range(model.num_blocks(n)):
        sigma_0, _ = model.calc_prior_cov(X, bi)
        S, nu = model.calc_posterior_contribs(X, bi)
        W = model.calc_posterior(bi, sigma_0, S)
        out = []
        for e in (la.DENSE_ENTRIES, entries):
            monkeypatch.setattr(la, "DENSE_ENTRIES", e)
            out.append(model.partial_expectation_step(X, bi, W, nu, sparsity_threshold=threshold))
        monkeypatch.undo()
        (i0, v0, c0), (i1, v1, c1) = out
        assert torch.equal(i0, i1)
        # a column's log-sum over at most 64 kernels in float64: 64 eps, and
        # as much again through the exponential at |log rho| < 1e3
        torch.testing.assert_close(c1, c0, rtol=1e-12, atol=1e-12)
        torch.testing.assert_close(v1, v0, rtol=1e-10, atol=0)
