"""The block schedule's rebalance holds no copy of the stored columns."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("index_dtype", [torch.int32, torch.int64, torch.int16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_rebalance_result_and_peak(dtype, index_dtype):
    from lakde_b200 import LocalKNearestKDE

    N, blocks = 4000, 8
    rows = N // blocks
    g = torch.Generator(device="cuda").manual_seed(0)
    X = torch.randn(N, 2, generator=g, device="cuda", dtype=dtype)
    model = LocalKNearestKDE(k_or_knn_graph=12, block_size=rows)
    dense = torch.rand(N, N, generator=g, device="cuda", dtype=dtype) + 0.1
    i, j = torch.meshgrid(torch.arange(rows, device="cuda"), torch.arange(N, device="cuda"), indexing="ij")
    ind = torch.stack((i.reshape(-1), j.reshape(-1))).to(index_dtype)
    del i, j
    model.rnm_blocks = [(ind, dense[b * rows : (b + 1) * rows].reshape(-1).clone()) for b in range(blocks)]
    old = torch.randn(N, generator=g, device="cuda", dtype=dtype)
    new = old + 0.3 * torch.randn(N, generator=g, device="cuda", dtype=dtype)
    model.rnm_log_consts = old
    scaled = dense.double() * torch.exp(old - new).double()[None]
    scaled[2 * rows : 3 * rows] = dense[2 * rows : 3 * rows].double()
    want = scaled / scaled.sum(0)
    del dense, scaled
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    c = model.rebalance_responsibilities_(X, 2, new.clone())
    peak = torch.cuda.max_memory_allocated() - held
    # one block's gathered coefficients (and its columns, when their type is
    # converted), never all blocks' columns
    block = rows * N
    assert peak <= 1.1 * block * (X.element_size() + (8 if index_dtype == torch.int16 else 0)) + 2**20
    got = torch.cat([v for _, v in model.rnm_blocks]).reshape(N, N)
    # sums of 4,000 positive terms in any order: 4,000 eps, and a few for the factors
    tol = 4100 * torch.finfo(dtype).eps
    torch.testing.assert_close(got.double(), want, rtol=tol, atol=0)
    torch.testing.assert_close(c.isfinite().all(), torch.tensor(True, device="cuda"))
