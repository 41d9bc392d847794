"""Performance cases of the framework: what a user has it do, through its
public entry points, with inputs made from a seed alone.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` builds what a program has in hand before the call, ``run`` makes
one pass, ``work`` counts what a pass cannot do without, and ``exact`` gives
the outputs in 64 bits from plain torch.

Kinds:

* ``fit``     fused VI iterations of LocalKNearestKDE (the framework's main path)
* ``hier``    the same of LocalHierarchicalKDE on uneven neighbourhoods
* ``block``   the default block schedule of LocalKNearestKDE
* ``predict`` log_pred_density of a fitted model on held-out queries
* ``score``   differentiable log density, forward and backward
* ``quad``    the drop-in op chol_quad_form
* ``scatter`` the drop-in op calc_W_inv
* ``knn``     the kNN graph every fit starts from

The models are built with ``autotune=False``: the launch forms the tuner picks
from are equivalent, and a choice made by timing would differ from run to run.
"""

import math

import torch

DEVICE = "cuda"
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # the smallest fit: 2-d toy data, ten iterations; latency of the replayed launches
        {"name": "fit_circle2d", "kind": "fit", "n": 2000, "d": 2, "k": 20, "iterations": 10, "dtype": "f32"},
        # tabular data of dimension 8 at the size of a real set
        {"name": "fit_gas8", "kind": "fit", "n": 200_000, "d": 8, "k": 50, "iterations": 2, "dtype": "f32"},
        # dimension 21 (odd, padded to 24 / 32 inside), an ordinary fit
        {"name": "fit_spec21", "kind": "fit", "n": 60_000, "d": 21, "k": 64, "iterations": 2, "dtype": "f32"},
        # the headline workload's dimension and K at a tenth of its rows, odd row count
        {"name": "fit_bsds63", "kind": "fit", "n": 100_003, "d": 63, "k": 100, "iterations": 1, "dtype": "f32"},
        # hierarchical model, lognormal neighbourhoods of a handful to thousands of pairs
        {"name": "hier_embed43", "kind": "hier", "n": 20_000, "d": 43, "k": 64, "cap": 2048, "iterations": 1,
         "dtype": "f32"},
        # the constructor's default schedule (block coordinate ascent) on the toy set
        {"name": "block_circle2d", "kind": "block", "n": 2000, "d": 2, "k": 20, "iterations": 1, "dtype": "f32"},
        # held-out density, tabular data of dimension 8
        {"name": "predict_gas8", "kind": "predict", "n": 100_000, "d": 8, "k": 50, "nq": 20_000, "dtype": "f32"},
        # held-out density in dimension 63
        {"name": "predict_bsds63", "kind": "predict", "n": 30_000, "d": 63, "k": 100, "nq": 5000, "dtype": "f32"},
        # gradients of the density for queries and factors (score, factor gradients)
        {"name": "score_spec21", "kind": "score", "n": 20_000, "d": 21, "nq": 4096, "dtype": "f32"},
        # a block of kernels against all points of a set, the reference's own op
        {"name": "quad_d63", "kind": "quad", "n": 512, "d": 63, "m": 20_011, "dtype": "f32"},
        # scatter covariances in float64, the data type of the parity runs
        {"name": "scatter_d43_f64", "kind": "scatter", "n": 20_000, "d": 43, "k": 64, "dtype": "f64"},
        # the exact neighbour graph with distances
        {"name": "knn_d21", "kind": "knn", "n": 50_000, "d": 21, "k": 64, "dtype": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _k_for(rng, d):
    """Neighbour counts as they are used: enough for a full-rank local covariance."""
    lo = max(16, 2 * d)
    return min(128, rng.randint(lo, 2 * lo))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "hier", "predict", "predict", "score", "quad", "scatter", "knn", "block"])
    d = rng.choice([2, 3, 5, 8, 13, 16, 21, 24, 32, 36, 43, 48, 57, 63, 64])
    dtype = rng.choice(["f32", "f32", "f32", "f64"])
    k = _k_for(rng, d)
    if kind == "fit":
        n = min(_log_int(rng, 1000, 100_000), int(1.2e9 / (k * max(d, 8) ** 2) * (1 if dtype == "f32" else 0.2)) + 900)
        return {"kind": kind, "n": n, "d": d, "k": k, "iterations": rng.randint(1, 3), "dtype": dtype}
    if kind == "hier":
        d = min(d, 43)
        return {"kind": kind, "n": _log_int(rng, 1500, 20_000), "d": d, "k": _k_for(rng, d),
                "cap": rng.choice([256, 1024]), "iterations": rng.randint(1, 2), "dtype": "f32"}
    if kind == "block":
        d = min(d, 21)
        return {"kind": kind, "n": _log_int(rng, 600, 3000), "d": d, "k": _k_for(rng, d), "iterations": 1,
                "dtype": dtype}
    if kind == "predict":
        n, nq = _log_int(rng, 1000, 60_000), _log_int(rng, 1, 8000)
        scale = 1 if dtype == "f32" else 0.05
        while n * nq * d * d > 4e11 * scale and nq > 1:
            nq //= 2
        return {"kind": kind, "n": n, "d": d, "k": k, "nq": max(nq, 1), "dtype": dtype}
    if kind == "score":
        d = min(d, 32)
        n, nq = _log_int(rng, 500, 20_000), _log_int(rng, 50, 4096)
        if dtype == "f64":
            nq = max(1, nq // 8)
        return {"kind": kind, "n": n, "d": d, "nq": nq, "dtype": dtype}
    if kind == "quad":
        return {"kind": kind, "n": _log_int(rng, 1, 1024), "d": d, "m": _log_int(rng, 1, 20_000), "dtype": dtype}
    if kind == "scatter":
        return {"kind": kind, "n": _log_int(rng, 500, 20_000), "d": d, "k": k, "dtype": dtype}
    return {"kind": kind, "n": _log_int(rng, 1000, 40_000), "d": d, "k": k, "dtype": "f32"}


# ------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _factor(g, d, lo):
    """Random covariance factor: eigenvalues 1 / k for d >= 32, else log-uniform in [lo, 1]."""
    q, r = torch.linalg.qr(torch.randn(d, d, generator=g, device=DEVICE, dtype=torch.float64))
    q = q * torch.sign(torch.diagonal(r))
    if d >= 32:
        eig = torch.arange(1, d + 1, device=DEVICE, dtype=torch.float64) ** -1.0
    else:
        eig = torch.exp(torch.rand(d, generator=g, device=DEVICE, dtype=torch.float64) * -math.log(lo) + math.log(lo))
    return q * eig.sqrt()


def _mixture(g, n, d, comps):
    x = torch.empty(n, d, device=DEVICE, dtype=torch.float64)
    lab = torch.randint(len(comps), (n,), generator=g, device=DEVICE)
    z = torch.randn(n, d, generator=g, device=DEVICE, dtype=torch.float64)
    for c, (mean, fac) in enumerate(comps):
        own = (lab == c).nonzero().squeeze(1)
        x[own] = mean + z[own] @ fac.T
    return x


def _data(seed, n, d, nq, dtype, embedded=False):
    """Training points [n, d] and queries [nq, d] of one mixture: a circle of
    Gaussians at d = 2, full-covariance mixtures above (a heavy-tailed
    component up to d = 8, 1,000 near-duplicate points in large sets of
    d >= 32), or a 10-dimensional mixture embedded in d dimensions with noise."""
    g = _generator(seed)
    total = n + nq
    if d == 2:
        ang = torch.randint(8, (total,), generator=g, device=DEVICE).double() * (2 * math.pi / 8)
        x = torch.stack((2 * ang.cos(), 2 * ang.sin()), 1)
        x = x + 0.2 * torch.randn(total, 2, generator=g, device=DEVICE, dtype=torch.float64)
    elif embedded:
        lat = min(10, d)
        comps = [(2 * torch.randn(lat, generator=g, device=DEVICE, dtype=torch.float64), _factor(g, lat, 1e-2))
                 for _ in range(6)]
        q, _ = torch.linalg.qr(torch.randn(d, d, generator=g, device=DEVICE, dtype=torch.float64))
        x = _mixture(g, total, lat, comps) @ q[:, :lat].T
        x = x + 0.1 * torch.randn(total, d, generator=g, device=DEVICE, dtype=torch.float64)
    else:
        comps = [(2 * torch.randn(d, generator=g, device=DEVICE, dtype=torch.float64), _factor(g, d, 1e-2 if d <= 8 else 0.1))
                 for _ in range(12)]
        x = _mixture(g, total, d, comps)
        if d <= 8:
            tail = (torch.rand(total, generator=g, device=DEVICE) < 0.1).nonzero().squeeze(1)
            z = torch.randn(len(tail), d + 3, generator=g, device=DEVICE, dtype=torch.float64)
            u = z[:, d:].square().sum(1)
            x[tail] = (z[:, :d] @ _factor(g, d, 1e-2).T) / (u / 3).sqrt()[:, None]
        elif d >= 32 and n >= 50_000:
            at = torch.randperm(n, generator=g, device=DEVICE)[:1000]
            x[at] = x[at[0]] + 1e-2 * torch.randn(1000, d, generator=g, device=DEVICE, dtype=torch.float64)
    x = x.to(dtype)
    return x[:n].contiguous(), x[n:].contiguous()


def _knn(X, k):
    """Exact float64 neighbour lists in plain torch (distances, indices)."""
    Xd = X.double()
    sq = (Xd * Xd).sum(1)
    out, dist = [], []
    for i in range(0, len(Xd), 1024):
        d2 = sq[None, :] - 2 * Xd[i : i + 1024] @ Xd.T
        rows = torch.arange(len(d2), device=X.device)
        d2[rows, rows + i] = math.inf
        cand = d2.topk(min(k + 8, len(Xd) - 1), largest=False, sorted=False).indices.sort(1).values
        e = (Xd[cand] - Xd[i : i + 1024, None]).square().sum(2)
        e, at = e.sort(dim=1, stable=True)
        out.append(cand.gather(1, at[:, :k]))
        dist.append(e[:, :k].sqrt())
    return torch.cat(dist), torch.cat(out)


def _counts(seed, n, k, cap):
    """Lognormal neighbourhood sizes (median 64, sigma 1), at least k and at most
    cap: the distribution's quantiles, dealt to the points by the seed."""
    p = (torch.arange(n, device=DEVICE, dtype=torch.float64) + 0.5) / n
    c = torch.exp(math.log(64) + torch.special.ndtri(p))[torch.randperm(n, generator=_generator(seed + 7919), device=DEVICE)]
    return c.round().long().clamp(k, min(cap, n - 1))


def _mixture_model(case, seed):
    """Kernel centres, Cholesky factors of W^-1, degrees of freedom and queries
    of a predictive mixture (scaled local covariances)."""
    dt = DTYPES[case["dtype"]]
    n, d = case["n"], case["d"]
    X, Y = _data(seed, n, d, case["nq"], dt)
    g = _generator(seed + 1)
    nu = d + 1 + 4 * torch.rand(n, generator=g, device=DEVICE, dtype=torch.float64)
    q = torch.randn(n, d, d, generator=g, device=DEVICE, dtype=torch.float64).tril(-1) * (0.3 / math.sqrt(d))
    diag = torch.exp(0.3 * torch.randn(n, d, generator=g, device=DEVICE, dtype=torch.float64))
    L = (q + torch.diag_embed(diag)) * (0.5 * nu.sqrt())[:, None, None]
    return X, L.to(dt).contiguous(), nu.to(dt), Y


def _csr(case, seed):
    """A ragged CSR pattern: about k pairs a row, some rows empty, a few long."""
    n, k = case["n"], case["k"]
    g = _generator(seed + 2)
    len_ = (k * torch.exp(0.7 * torch.randn(n, generator=g, device=DEVICE))).round().long().clamp(0, 12 * k)
    len_[torch.rand(n, generator=g, device=DEVICE) < 0.02] = 0
    rowptr = torch.cat((len_.new_zeros(1), len_.cumsum(0)))
    nnz = int(rowptr[-1])
    col = torch.randint(n, (nnz,), generator=g, device=DEVICE)
    val = torch.rand(nnz, generator=g, device=DEVICE, dtype=torch.float64)
    return rowptr, col, val.to(DTYPES[case["dtype"]])


def _quad_inputs(case, seed):
    dt = DTYPES[case["dtype"]]
    n, m, d = case["n"], case["m"], case["d"]
    X, Y = _data(seed, n, d, m, dt)
    g = _generator(seed + 3)
    W = torch.randn(n, d, d, generator=g, device=DEVICE, dtype=torch.float64).triu(1) / math.sqrt(d)
    W = W + torch.diag_embed(torch.exp(0.5 * torch.randn(n, d, generator=g, device=DEVICE, dtype=torch.float64)))
    return W.to(dt).contiguous(), X, Y


# ---------------------------------------------------------------- the passes
def prepare(case, seed):
    kind = case["kind"]
    dt = DTYPES[case["dtype"]]
    state = {"kind": kind}
    if kind in ("fit", "block", "predict"):
        from lakde_b200 import LocalKNearestKDE

        X, Y = _data(seed, case["n"], case["d"], case.get("nq", 0), dt)
        model = LocalKNearestKDE(k_or_knn_graph=case["k"], fused=kind != "block", autotune=False)
        # two iterations: buffers allocated, and the fused iteration captured
        model.fit(X, iterations=1 if kind == "block" else 2)
        state.update(model=model, X=X, Y=Y, iterations=case.get("iterations", 0))
    elif kind == "hier":
        from lakde_b200 import LocalHierarchicalKDE, PairPattern
        from lakde_b200.utils import compute_knn_graph

        X, _ = _data(seed, case["n"], case["d"], 0, dt, embedded=True)
        counts = _counts(seed, case["n"], case["k"], case["cap"])
        graph = compute_knn_graph(X, int(counts.max()))
        model = LocalHierarchicalKDE(k_or_knn_graph=graph[:, : case["k"]].contiguous(), fused=True,
                                     candidates=PairPattern.from_knn_counts(graph, counts), autotune=False)
        model.fit(X, iterations=2)
        state.update(model=model, X=X, iterations=case["iterations"])
    elif kind == "score":
        X, L, nu, Y = _mixture_model(case, seed)
        state.update(X=X, L=L.requires_grad_(), nu=nu, Y=Y.requires_grad_())
    elif kind == "quad":
        W, Xn, Xm = _quad_inputs(case, seed)
        state.update(W=W, Xn=Xn, Xm=Xm)
    elif kind == "scatter":
        X, _ = _data(seed, case["n"], case["d"], 0, dt)
        rowptr, col, val = _csr(case, seed)
        state.update(X=X, rowptr=rowptr, col=col, val=val)
    elif kind == "knn":
        X, _ = _data(seed, case["n"], case["d"], 0, dt)
        state.update(X=X, k=case["k"])
    return state


def run(state):
    kind = state["kind"]
    if kind in ("fit", "hier"):
        model, X = state["model"], state["X"]
        model.fit(X, iterations=state["iterations"])
        out = {"r": model.responsibilities[1], "c": model.rnm_log_consts, "nu": model.nu, "b": model.b,
               "logdet_W": model.logdet_W}
        if kind == "hier":
            # the shared factor in the type the model works in
            out["W_shared"] = model.W_shared_triu.to(X.dtype)
        return out
    if kind == "block":
        model, X = state["model"], state["X"]
        model.fit(X, iterations=state["iterations"])
        n, bs = len(X), model.block_size
        r = X.new_zeros(n, n)
        for i, (idx, val) in enumerate(model.rnm_blocks):
            r[idx[0].long() + i * bs, idx[1].long()] = val
        return {"r": r, "c": model.rnm_log_consts, "nu": model.nu, "b": model.b, "logdet_W": model.logdet_W}
    if kind == "predict":
        return state["model"].log_pred_density(state["X"], state["Y"])
    if kind == "score":
        from lakde_b200.grad import log_pred_density

        state["Y"].grad = state["L"].grad = None
        lp = log_pred_density(state["X"], state["L"], state["nu"], state["Y"])
        lp.sum().backward()
        return {"log_density": lp.detach(), "score": state["Y"].grad, "grad_L": state["L"].grad}
    from lakde_b200 import kernels as K

    if kind == "quad":
        return K.chol_quad_form(state["W"], state["Xn"], state["Xm"])
    if kind == "scatter":
        return K.calc_W_inv(state["rowptr"], state["col"], state["val"], state["X"], state["X"])
    from lakde_b200.utils import compute_knn_graph

    dist, idx = compute_knn_graph(state["X"], state["k"], return_dists=True)
    return {"dist": dist, "idx": idx}


def work(case):
    kind, n, d = case["kind"], case["n"], case["d"]
    es = 4 if case["dtype"] == "f32" else 8
    tri = d * (d + 1) / 2
    if kind in ("fit", "hier", "predict"):
        pairs = n * case["k"] if kind != "hier" else n * 106.0  # mean of the lognormal sizes
        # scatter sums, factorisation (Cholesky, inverse, trace product), quad forms
        m_flops, f_flops, e_flops = 2 * pairs * tri, 2.0 * n * d**3 / 2, 2 * pairs * (tri + d)
        m_bytes = 4 * pairs + es * pairs + es * n * d
        state_bytes = es * n * (tri + (tri if kind != "hier" else 0)) + 8 * es * n
        if kind == "predict":
            nq = case["nq"]
            return {"bytes": m_bytes + state_bytes / 2 + es * nq * (d + 1),
                    "flops": m_flops + f_flops + 2.0 * n * nq * (tri + 2 * d)}
        it = case["iterations"]
        gram = 2.0 * n * d * tri / 3 if kind == "hier" else 0.0
        # the responsibilities are read and written, the pattern is read twice
        return {"bytes": it * (m_bytes + (4 + es) * pairs + state_bytes), "flops": it * (m_flops + f_flops + e_flops + gram)}
    if kind == "block":
        it = case["iterations"]
        return {"bytes": it * 3.0 * es * n * n, "flops": it * 2.0 * n * n * (2 * tri + d)}
    if kind == "score":
        nq = case["nq"]
        return {"bytes": es * (2 * n * tri + 2 * nq * d + n * d + nq), "flops": 2.0 * n * nq * (4 * tri + 4 * d)}
    if kind == "quad":
        m = case["m"]
        return {"bytes": es * (n * tri + n * d + m * d + float(n) * m), "flops": 2.0 * n * m * (tri + d)}
    if kind == "scatter":
        pairs = 1.27 * n * case["k"]
        return {"bytes": (8 + es) * pairs + es * (n * d + n * d * d), "flops": 2 * pairs * tri}
    return {"bytes": es * n * d + 8.0 * n * case["k"], "flops": 2.0 * n * n * d}


# ------------------------------------------------- 64-bit results, plain torch
def _lse_parts(c, rsum, lse, first):
    if first:
        return lse
    old = torch.log(rsum) + c
    sub = c + torch.log1p(torch.clamp_min(-torch.exp(old - c), -1))
    return torch.logaddexp(sub, lse)


class _ExactVI:
    """Batch VI on a pair pattern (kernel n, point m) in float64 (the locally
    adaptive model of both priors), all quantities recomputed from the data."""

    def __init__(self, X, kern, point, seed_graph, hier):
        self.X, self.hier = X.double(), hier
        self.N, self.D = X.shape
        N, D = X.shape
        order = torch.argsort(kern * N + point)
        self.kern, self.point = kern[order], point[order]
        keys = self.kern * N + self.point
        k = seed_graph.size(1)
        want = seed_graph.reshape(-1) * N + torch.arange(N, device=X.device).repeat_interleave(k)
        self.r = torch.zeros(len(keys), device=X.device, dtype=torch.float64)
        self.r[torch.searchsorted(keys, want)] = 1.0 / k
        self.nu0 = float(D)
        self.a = 1e-6 + self.nu0 * D / 2
        self.b = torch.full((N,), self.a, device=X.device, dtype=torch.float64)
        self.c = self.rsum = None
        if hier:
            Xc = self.X - self.X.mean(0)
            s0 = torch.linalg.cholesky(Xc.T @ Xc / (N - 1))
            self.nsh0 = D - 1 + 1e-2
            self.nsh = self.nsh0 + N * self.nu0
            inv = torch.linalg.inv(s0).T
            self.lambda0 = inv @ inv.T
            self.Wsh = self.nu0 * s0.T / self.nsh
        else:
            ones = torch.full((N * k,), 1.0 / k, device=X.device, dtype=torch.float64)
            rows = torch.arange(N, device=X.device).repeat_interleave(k)
            self.P = self._scatter(rows, seed_graph.reshape(-1), ones)
            self.T = torch.linalg.cholesky(self.P)

    def _prior(self):
        if self.hier:
            sb = self.nsh * self.Wsh @ self.Wsh.T
            return sb, sb
        return self.P, self.T

    def _scatter(self, kern, point, w):
        S = torch.zeros(self.N, self.D, self.D, device=self.X.device, dtype=torch.float64)
        step = max(1, int(4e8 / self.D**2))
        for i in range(0, len(kern), step):
            kk = kern[i : i + step]
            dl = self.X[point[i : i + step]] - self.X[kk]
            S.index_add_(0, kk, (w[i : i + step, None] * dl)[:, :, None] * dl[:, None, :])
        return S

    def factor(self):
        nu = torch.full((self.N,), self.nu0, device=self.X.device, dtype=torch.float64).index_add_(0, self.kern, self.r)
        A = self._scatter(self.kern, self.point, self.r)
        P, T = self._prior()
        A += (self.nu0 * self.a / self.b)[:, None, None] * P
        L = torch.linalg.cholesky(A)
        eye = torch.eye(self.D, device=self.X.device, dtype=torch.float64)
        Li = torch.linalg.solve_triangular(L, eye.expand_as(L), upper=False)
        logdet = 2 * torch.diagonal(Li, dim1=1, dim2=2).log().sum(1)
        # ||T^T W_triu||_F^2 with W_triu = L^-T
        trace = (Li @ T).square().sum((1, 2)) if not self.hier else (T.T @ Li.mT).square().sum((1, 2))
        return Li, nu, logdet, trace

    def estep(self, Li, nu, logdet, first):
        D, N = self.D, self.N
        i = torch.arange(1, D + 1, device=self.X.device, dtype=torch.float64)
        c0 = 0.5 * (torch.digamma(nu[:, None] / 2 + (1 - i) / 2).sum(1) + D * math.log(2) + logdet)
        lr = torch.empty_like(self.r)
        step = max(1, int(4e8 / D**2))
        for s in range(0, len(lr), step):
            kk = self.kern[s : s + step]
            dl = self.X[self.point[s : s + step]] - self.X[kk]
            q = torch.bmm(Li[kk], dl[:, :, None]).square().sum((1, 2))
            lr[s : s + step] = c0[kk] - nu[kk] / 2 * q
        lr[self.kern == self.point] = -math.inf
        mx = torch.full((N,), -math.inf, device=lr.device, dtype=lr.dtype).scatter_reduce_(0, self.point, lr, "amax")
        lse = mx + torch.zeros_like(mx).index_add_(0, self.point, torch.exp(lr - mx[self.point])).log()
        c = _lse_parts(self.c, self.rsum, lse, first)
        r = torch.exp(lr - c[self.point])
        tot = torch.zeros_like(c).index_add_(0, self.point, r).clamp_min(torch.finfo(torch.float64).eps)
        self.c = c + tot.log()
        self.r = r / tot[self.point]
        self.rsum = torch.zeros_like(c).index_add_(0, self.point, self.r)

    def iterate(self, iterations):
        Li, nu, logdet, _ = self.factor()
        if self.hier:
            self.contrib(Li, nu)
        self.estep(Li, nu, logdet, True)
        for _ in range(iterations):
            Li, nu, logdet, trace = self.factor()
            self.estep(Li, nu, logdet, False)
            self.b = 1e-6 + self.nu0 * nu * trace / 2
            if self.hier:
                prec = self.contrib(Li, nu) * self.nu0 + self.nsh0 * self.lambda0
                self.Wsh = torch.linalg.inv(torch.linalg.cholesky(prec)).T
            self.nu, self.logdet = nu, logdet

    def contrib(self, Li, nu):
        w = nu * self.a / self.b
        return torch.einsum("n,nji,njk->ik", w, Li, Li) if self.D <= 16 else ((w[:, None, None] * Li).mT @ Li).sum(0)

    def outputs(self):
        out = {"r": self.r, "c": self.c, "nu": self.nu, "b": self.b, "logdet_W": self.logdet}
        if self.hier:
            out["W_shared"] = self.Wsh
        return out


def _exact_density(X, Li, nu, logdet, Y):
    """-log N + logsumexp of the Student-t components, kernels in chunks."""
    N, D = X.shape
    a1, a2 = (nu + 1) / 2, (nu + 1 - D) / 2
    lc = torch.lgamma(a1) - torch.lgamma(a2) + 0.5 * logdet - 0.5 * D * math.log(math.pi)
    acc = torch.full((len(Y),), -math.inf, device=X.device, dtype=torch.float64)
    step = max(1, int(3e8 / (len(Y) * D)))
    for s in range(0, N, step):
        z = torch.matmul(Y[None] - X[s : s + step, None], Li[s : s + step].mT)
        lp = lc[s : s + step, None] - a1[s : s + step, None] * torch.log1p(z.square().sum(2))
        acc = torch.logaddexp(acc, torch.logsumexp(lp, 0))
    return acc - math.log(N)


def _exact_score(case, seed):
    X, L, nu, Y = (t.double() for t in _mixture_model(case, seed))
    N, D = X.shape
    eye = torch.eye(D, device=X.device, dtype=torch.float64)
    Li = torch.linalg.solve_triangular(L, eye.expand_as(L), upper=False)
    diag = torch.diagonal(L, dim1=1, dim2=2)
    logdet = -2 * diag.log().sum(1)
    lp_all = _exact_density(X, Li, nu, logdet, Y)
    h = (nu + 1) / 2
    lc = torch.lgamma(h) - torch.lgamma((nu + 1 - D) / 2) + 0.5 * logdet - 0.5 * D * math.log(math.pi)
    gY = torch.zeros_like(Y)
    gL = torch.empty_like(L)
    step = max(1, int(3e8 / (len(Y) * D)))
    for s in range(0, N, step):
        sl = slice(s, s + step)
        z = torch.matmul(Y[None] - X[sl, None], Li[sl].mT)
        q = z.square().sum(2)
        w = torch.exp(lc[sl, None] - h[sl, None] * torch.log1p(q) - lp_all - math.log(N))
        cw = w / (1 + q)
        cz = cw[:, :, None] * z
        gY += torch.einsum("nq,nqd->qd", -2 * h[sl, None].expand_as(cw), torch.matmul(cz, Li[sl]))
        # d/dL = 2 h L^-T (sum_y c z z^T) - (sum_y w) diag(1 / L_ii), lower triangle
        m = torch.matmul(cz.mT, z)
        g = 2 * h[sl, None, None] * torch.matmul(Li[sl].mT, m)
        g.diagonal(dim1=1, dim2=2).sub_(w.sum(1)[:, None] / diag[sl])
        gL[sl] = g.tril()
    return {"log_density": lp_all, "score": gY, "grad_L": gL}


def _exact_block(case, seed, warm):
    """The default block schedule (block size 512) in float64, dense r [n, m]."""
    X, _ = _data(seed, case["n"], case["d"], 0, DTYPES[case["dtype"]])
    _, graph = _knn(X, case["k"])
    N, D = X.shape
    X = X.double()
    dl_all = X[None] - X[:, None]  # [n, m] -> x_m - x_n
    k, bs = case["k"], min(512, N)
    r = torch.zeros(N, N, device=X.device, dtype=torch.float64)
    r[graph.reshape(-1), torch.arange(N, device=X.device).repeat_interleave(k)] = 1.0 / k
    nb = X[graph] - X[:, None]
    P = nb.mT @ nb / k
    T = torch.linalg.cholesky(P)
    nu0 = float(D)
    a = 1e-6 + nu0 * D / 2
    b = torch.full((N,), a, device=X.device, dtype=torch.float64)
    nu, logdet = torch.empty_like(b), torch.empty_like(b)
    i = torch.arange(1, D + 1, device=X.device, dtype=torch.float64)
    eye = torch.eye(D, device=X.device, dtype=torch.float64)
    eps = torch.finfo(torch.float64).eps

    def update(sl):
        S = torch.einsum("nm,nmi,nmj->nij", r[sl], dl_all[sl], dl_all[sl])
        nus = nu0 + r[sl].sum(1)
        L = torch.linalg.cholesky((nu0 * a / b[sl])[:, None, None] * P[sl] + S)
        Li = torch.linalg.solve_triangular(L, eye.expand_as(L), upper=False)
        ld = 2 * torch.diagonal(Li, dim1=1, dim2=2).log().sum(1)
        c0 = 0.5 * (torch.digamma(nus[:, None] / 2 + (1 - i) / 2).sum(1) + D * math.log(2) + ld)
        lr = c0[:, None] - nus[:, None] / 2 * torch.matmul(dl_all[sl], Li.mT).square().sum(2)
        own = torch.arange(sl.start, min(sl.stop, N), device=X.device)
        lr[own - sl.start, own] = -math.inf
        return nus, ld, (Li @ T[sl]).square().sum((1, 2)), lr

    blocks = [slice(s, min(s + bs, N)) for s in range(0, N, bs)]
    lrs = []
    for sl in blocks:
        nu[sl], logdet[sl], _, lr = update(sl)
        lrs.append(lr)
    c = torch.logsumexp(torch.cat(lrs), 0)
    r = torch.exp(torch.cat(lrs) - c)
    tot = r.sum(0).clamp_min(eps)
    c, r = c + tot.log(), r / tot
    for _ in range(warm + case["iterations"]):
        for sl in blocks:
            nus, ld, tr, lr = update(sl)
            old = torch.log(r[sl].sum(0)) + c
            sub = c + torch.log1p(torch.clamp_min(-torch.exp(old - c), -1))
            cn = torch.logaddexp(sub, torch.logsumexp(lr, 0))
            r *= torch.exp(c - cn)
            r[sl] = torch.exp(lr - cn)
            tot = r.sum(0).clamp_min(eps)
            c, r = cn + tot.log(), r / tot
            nu[sl], logdet[sl], b[sl] = nus, ld, 1e-6 + nu0 * nus * tr / 2
    return {"r": r, "c": c, "nu": nu, "b": b, "logdet_W": logdet}


def exact(case, seed):
    kind = case["kind"]
    dt = DTYPES[case["dtype"]]
    if kind in ("fit", "hier", "predict"):
        X, Y = _data(seed, case["n"], case["d"], case.get("nq", 0), dt, embedded=kind == "hier")
        N = len(X)
        if kind == "hier":
            counts = _counts(seed, N, case["k"], case["cap"])
            _, graph = _knn(X, int(counts.max()))
            keep = torch.arange(graph.size(1), device=X.device)[None] < counts[:, None]
            kern, point = graph[keep], torch.arange(N, device=X.device).repeat_interleave(counts)
            graph = graph[:, : case["k"]].contiguous()
        else:
            _, graph = _knn(X, case["k"])
            kern, point = graph.reshape(-1), torch.arange(N, device=X.device).repeat_interleave(case["k"])
        vi = _ExactVI(X, kern, point, graph, kind == "hier")
        vi.iterate(2 + case.get("iterations", 0))
        if kind != "predict":
            return vi.outputs()
        Li, nu, logdet, _ = vi.factor()
        return _exact_density(vi.X, Li, nu, logdet, Y.double())
    if kind == "block":
        return _exact_block(case, seed, 1)
    if kind == "score":
        return _exact_score(case, seed)
    if kind == "quad":
        W, Xn, Xm = (t.double() for t in _quad_inputs(case, seed))
        out = torch.empty(len(Xn), len(Xm), device=Xn.device, dtype=torch.float64)
        step = max(1, int(3e8 / (len(Xm) * case["d"])))
        for s in range(0, len(Xn), step):
            out[s : s + step] = torch.matmul(Xm[None] - Xn[s : s + step, None], W[s : s + step]).square().sum(2)
        return out
    if kind == "scatter":
        X, _ = _data(seed, case["n"], case["d"], 0, dt)
        rowptr, col, val = _csr(case, seed)
        X, val = X.double(), val.double()
        kern = torch.repeat_interleave(torch.arange(case["n"], device=X.device), rowptr.diff())
        out = torch.zeros(case["n"], case["d"], case["d"], device=X.device, dtype=torch.float64)
        step = max(1, int(4e8 / case["d"] ** 2))
        for s in range(0, len(col), step):
            dl = X[col[s : s + step]] - X[kern[s : s + step]]
            out.index_add_(0, kern[s : s + step], (val[s : s + step, None] * dl)[:, :, None] * dl[:, None, :])
        return out
    X, _ = _data(seed, case["n"], case["d"], 0, dt)
    return {"dist": _knn(X, case["k"])[0], "idx": None}
