"""Selection of the nearest neighbours from a distance block at the edges of
the per-row kernels: row lengths around the warps' 256-value steps and quarters,
candidate counts around the buffer rules, the point itself in and out, adversarial
orders, equal distances, NaN and infinities.  The result is exact, so it is
compared exactly."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(dist, X, row0, k, include_self):
    """kc = k + 8 smallest by (value, index), then k by (exact distance, index)."""
    out = []
    for r in range(dist.size(0)):
        d = dist[r].clone()
        d[torch.isnan(d)] = float("inf")
        if not include_self:
            d[row0 + r] = float("inf")
        avail = d.numel() if include_self else d.numel() - 1
        cand = torch.sort(d, stable=True).indices[: min(k + 8, avail)].sort().values
        cand = cand[torch.isfinite(d[cand])]
        e = torch.zeros(len(cand), dtype=torch.float64, device=d.device)
        for i in range(X.size(1)):  # the kernel's order of additions
            e = torch.addcmul(e, X[cand, i] - X[row0 + r, i], X[cand, i] - X[row0 + r, i])
        e, at = torch.sort(e, stable=True)
        idx = cand[at][:k]
        out.append(torch.cat((idx, idx.new_full((k - len(idx),), -1))))
    return torch.stack(out)


@pytest.mark.parametrize("N", [2, 9, 255, 256, 257, 1023, 1025, 2049, 5000])
@pytest.mark.parametrize("k", [1, 24, 25, 152, 153, 492, 493])
def test_selection_edges(N, k):
    from lakde_b200 import kernels as K

    g = torch.Generator(device="cuda").manual_seed(N + k)
    X = torch.randint(-40, 40, (N, 3), generator=g, device="cuda").double()  # exact sums, many ties
    d = (X[:, None] - X[None]).square().sum(2) if N <= 1100 else (
        X.square().sum(1)[None] + X.square().sum(1)[:, None] - 2 * X @ X.T)
    for include_self in (False, True):
        if k > (N if include_self else N - 1):
            continue
        nb = min(N, 5)
        row0 = N - nb
        block = d[row0:].contiguous()
        got = K.knn_select(block, X, row0, k, include_self=include_self)
        assert torch.equal(got, reference(block, X, row0, k, include_self))


@pytest.mark.parametrize("k", [16, 200])
def test_adversarial_orders(k):
    """Descending values cut the buffers at every step; NaN and inf are never
    chosen; fewer finite values than k leave -1."""
    from lakde_b200 import kernels as K

    N = 3001
    X = torch.arange(N, 0, -1, dtype=torch.float64, device="cuda")[:, None].contiguous()
    rows = [(X[:, 0] - X[-1, 0]).square(), (X[:, 0] - X[-2, 0]).square(), (X[:, 0] - X[-3, 0]).square()]
    block = torch.stack(rows[::-1]).contiguous()
    block[1, ::3] = float("nan")
    block[2, 100:] = float("inf")
    got = K.knn_select(block, X, N - 3, k)
    assert torch.equal(got, reference(block, X, N - 3, k, False))
