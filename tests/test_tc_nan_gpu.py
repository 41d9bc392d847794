"""NaN inputs of the tensor-core kernels: what a failed factor or a NaN point
makes of a density, a log rho or a scatter matrix stays visible."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _mixture(N, Nq, D, seed=0):
    g = torch.Generator().manual_seed(seed)
    X = torch.randn(N, D, generator=g)
    Y = torch.randn(Nq, D, generator=g)
    W = torch.randn(N, D, D, generator=g).triu(1) / D**0.5 + torch.diag_embed(0.5 + torch.rand(N, D, generator=g))
    nu = D + 1 + torch.rand(N, generator=g)
    lc = torch.randn(N, generator=g)
    return [v.to(DEV) for v in (X, W, nu, lc, Y)]


@pytest.mark.parametrize("D", [13, 21, 43, 63])
@pytest.mark.parametrize("N,Nq", [(1, 5), (3, 300), (100, 100), (5000, 300)])
@pytest.mark.parametrize("part", ["factor", "coefficient"])
def test_density_keeps_the_nan_of_one_failed_kernel(D, N, Nq, part):
    """One kernel with a NaN factor or coefficient, below and above the number
    of CTAs: NaN for every query wherever lakde_log_pred_density says so."""
    from lakde_b200 import kernels as K

    X, W, nu, lc, Y = _mixture(N, Nq, D)
    at = N // 2
    if part == "factor":
        W[at] = float("nan")
    else:
        lc[at] = float("nan")
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    plain = K.log_pred_density(X, W, nu, lc, Y)
    mixed = K.log_pred_density_tc(X, K.pack_w_cores(W), nu, lc, Y, err)
    assert int(err) == 0
    if N > 1:
        assert torch.isnan(plain).all()
    assert torch.equal(torch.isnan(mixed), torch.isnan(plain))
    assert torch.equal(torch.isneginf(mixed), torch.isneginf(plain))


def _pairs(N, k, seed):
    """k pairs a row, the row's own point among them."""
    g = torch.Generator().manual_seed(seed)
    col = torch.stack([torch.randperm(N, generator=g)[:k] for _ in range(N)])
    col[:, 0] = torch.arange(N)
    rowptr = torch.arange(0, N * k + 1, k)
    r = torch.rand(N * k, generator=g) + 0.1
    return rowptr.to(DEV), col.reshape(-1).to(torch.int32).to(DEV), r.to(DEV)


@pytest.mark.parametrize("D", [9, 16, 21, 43, 63])
def test_nan_point_reaches_log_rho_and_scatter(D):
    """One NaN coordinate of one point: the log rho and the entries of S_n that
    it takes part in are NaN exactly where the plain kernels say so."""
    from lakde_b200 import kernels as K

    N, k = 150, 20
    X, W, nu, _, _ = _mixture(N, 1, D, seed=D)
    X[7, D // 2] = float("nan")
    rowptr, col, r = _pairs(N, k, D)
    ld = torch.zeros(N, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    S, _ = K.mstep(rowptr, col, r, X, D + 1.0)
    St, _ = K.mstep_tc(rowptr, col, r, X, D + 1.0, err)
    lr = K.estep_logrho(rowptr, col, X, W, nu, ld)
    lrt = K.estep_tc(rowptr, col, X, K.pack_w_cores(W), nu, ld, err)
    assert int(err) == 0
    assert torch.isnan(S).any() and torch.isnan(lr).any()
    assert torch.equal(torch.isnan(St), torch.isnan(S))
    assert torch.equal(torch.isnan(lrt), torch.isnan(lr))


@pytest.mark.parametrize("D", [9, 21, 43, 63])
def test_nan_query_gives_no_finite_density(D):
    from lakde_b200 import kernels as K

    X, W, nu, lc, Y = _mixture(400, 300, D, seed=D)
    Y[3, D - 1] = Y[299, 0] = float("nan")
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    plain = K.log_pred_density(X, W, nu, lc, Y)
    mixed = K.log_pred_density_tc(X, K.pack_w_cores(W), nu, lc, Y, err)
    assert int(err) == 0
    assert not torch.isfinite(mixed[[3, 299]]).any()
    assert torch.equal(torch.isfinite(mixed), torch.isfinite(plain))


@pytest.mark.parametrize("D", [9, 24, 48, 63])
def test_w_cores_of_a_nan_factor_are_nan(D):
    """The canonical NaN of device arithmetic (all mantissa bits set) and the
    negative one, whose rounding would carry to a zero."""
    from lakde_b200 import kernels as K

    _, W, _, _, _ = _mixture(4, 1, D)
    W[1] = torch.full((D, D), 0x7FFFFFFF, dtype=torch.int32, device=DEV).view(torch.float32)
    W[2] = torch.full((D, D), -1, dtype=torch.int32, device=DEV).view(torch.float32)
    cores = K.pack_w_cores(W)
    n = torch.isnan(cores).sum(1).tolist()
    assert n == [0, D * (D + 1), D * (D + 1), 0]  # hi and lo of each lower element


@pytest.mark.parametrize("D", [10, 21, 43, 63])
def test_nan_centre_gives_nan_density(D):
    """A NaN coordinate of one kernel centre, in the first, an odd and the last
    dimension (a chunk of four cut by D)."""
    from lakde_b200 import kernels as K

    for at in (0, 5, D - 1):
        X, W, nu, lc, Y = _mixture(300, 200, D, seed=D + at)
        X[17, at] = float("nan")
        err = torch.zeros(1, dtype=torch.int32, device=DEV)
        assert torch.isnan(K.log_pred_density(X, W, nu, lc, Y)).all()
        assert torch.isnan(K.log_pred_density_tc(X, K.pack_w_cores(W), nu, lc, Y, err)).all()
        assert int(err) == 0


@pytest.mark.parametrize("D", [9, 21, 43, 63])
def test_padding_columns_may_hold_nan(D):
    """Columns past D of 16-byte aligned rows are never used: NaN there changes no bit."""
    from lakde_b200 import kernels as K

    N, k = 150, 20
    X, W, nu, lc, Y = _mixture(N, 130, D, seed=D)
    rowptr, col, r = _pairs(N, k, D)
    ld = torch.zeros(N, device=DEV)
    Wc = K.pack_w_cores(W)
    outs = []
    for fill in (0.0, float("nan")):
        Xp = torch.full((N, (D + 3) // 4 * 4), fill, device=DEV)[:, :D]
        Yp = torch.full((130, (D + 3) // 4 * 4), fill, device=DEV)[:, :D]
        Xp.copy_(X)
        Yp.copy_(Y)
        err = torch.zeros(1, dtype=torch.int32, device=DEV)
        S, nuo = K.mstep_tc(rowptr, col, r, Xp, D + 1.0, err)
        outs.append((S, nuo, K.estep_tc(rowptr, col, Xp, Wc, nu, ld, err),
                     K.log_pred_density_tc(Xp, Wc, nu, lc, Yp, err)))
        assert int(err) == 0
    for a, b in zip(*outs):
        assert torch.isfinite(a[~torch.isneginf(a)]).all()
        torch.testing.assert_close(a, b, rtol=0, atol=0)
