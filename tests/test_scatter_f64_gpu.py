"""Scatter covariance in float64 above 16 dimensions: a warp per row, four pairs
a step, 32 pairs an index load.  Row lengths around those edges, dimensions at
the edges of the 8-wide tiles, both index types."""

import numpy as np
import pytest
import torch

import oracle.lakde_oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 3, 4, 5, 31, 32, 33, 36, 64, 65, 130, 0, 2]


@pytest.mark.parametrize("D", [17, 24, 25, 32, 33, 41, 48, 49, 63, 64])
@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
def test_row_lengths(D, idx):
    from lakde_b200 import kernels as K

    rng = np.random.default_rng(D)
    N, M = len(LENGTHS), 97
    rowptr = np.concatenate(([0], np.cumsum(LENGTHS)))
    col = rng.integers(0, M, rowptr[-1])
    val = rng.uniform(0, 1, rowptr[-1])
    Xn, Xm = rng.standard_normal((N, D)), rng.standard_normal((M, D))
    ref = O.calc_W_inv(rowptr, col, val, Xn, Xm)
    t = lambda a, **k: torch.as_tensor(a, **k).cuda()
    S = K.calc_W_inv(t(rowptr, dtype=idx), t(col, dtype=idx), t(val), t(Xn), t(Xm)).cpu().numpy()
    # each entry is a sum of at most 130 products of centred differences (three
    # roundings a term): 133 half-eps of the sum of their sizes
    sizes = np.zeros_like(S)
    for n in range(N):
        sl = slice(rowptr[n], rowptr[n + 1])
        dl = np.abs(Xm[col[sl]] - Xn[n])
        sizes[n] = np.einsum("k,ki,kj->ij", val[sl], dl, dl)
    assert np.all(np.abs(S - ref) <= 2 * 133 * np.finfo(np.float64).eps * sizes)
    assert np.array_equal(S, S.transpose(0, 2, 1))

    # the row sums, and a row with an index out of range
    X = t(np.concatenate((Xn, Xm)))
    _, nu = K.mstep(t(rowptr, dtype=idx), t(col, dtype=idx), t(val), X, 3.5)
    nu_ref = 3.5 + np.array([val[a:b].sum() for a, b in zip(rowptr[:-1], rowptr[1:])])
    np.testing.assert_allclose(nu.cpu().numpy(), nu_ref, rtol=133 * np.finfo(np.float64).eps)
    col[rowptr[6] + 31] = M
    S = K.calc_W_inv(t(rowptr, dtype=idx), t(col, dtype=idx), t(val), t(Xn), t(Xm)).cpu().numpy()
    assert np.isnan(S[6]).all() and np.isfinite(np.delete(S, 6, 0)).all()


@pytest.mark.parametrize("D", [17, 63])
def test_infinities(D):
    """An infinite coordinate reaches its own row and column of its row's sum only."""
    from lakde_b200 import kernels as K

    g = torch.Generator().manual_seed(D)
    X = torch.randn(40, D, generator=g, dtype=torch.float64).cuda()
    X[7, D - 1] = float("inf")
    rowptr = torch.tensor([0, 6, 12]).cuda()
    col = torch.tensor([1, 2, 3, 4, 5, 7, 8, 9, 10, 11, 12, 13]).cuda()
    S = K.calc_W_inv(rowptr, col, torch.ones(12, dtype=torch.float64).cuda(), X[:2].contiguous(), X).cpu()
    assert S[0, : D - 1, : D - 1].isfinite().all() and S[1].isfinite().all()
    assert S[0, D - 1, D - 1] == float("inf") and S[0, D - 1, : D - 1].isinf().all()
