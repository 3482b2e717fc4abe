"""Performance cases of the Gibbs-sweep library: what a program that factorises a sparse matrix
asks of it, through its public entry points, from the smallest default call to the benchmark
matrix, with the 64-bit results of each call in plain torch.

A case is a dict of plain values.  Its `op` names the call:

  sweep       Sampler.sweep: one Gibbs iteration with the evaluation of the test set (the body of
              the loop of `macau_b200.macau` / `bpmf`), BPMF priors on both sides
  rows        Sampler.sample_latents: the rows of one mode given the other mode
  prior       mg_normal_wishart_noalloc: one Normal-Wishart draw from latents in device memory
  side        Sampler.sweep with side information on the rows (Macau prior, block-CG link solve)
  link        Sampler.update_prior of a Macau prior, and the link matrix it drew
  univariate  Sampler.sweep with side information under the univariate sampler
  batch       Batch.sweeps: twenty iterations of many small problems, then their latents and RMSEs
"""
import ctypes
import math

import numpy as np
import torch

from macau_b200 import _lib

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
BURNIN, ITERATION = 10, 12  # the iteration that a pass runs is the third collected sample
LAMBDA_BETA, TOL = 5.0, 1e-6  # defaults of macau()


def listed():
    return [
        # macau() as it is called without options: 64 bits, K = 10, a small matrix, one iteration
        dict(name="default_small", op="sweep", compute="fp64", K=10, rows=2000, cols=1500,
             nobs=60000, degrees="uniform", alpha=4.0, adaptive=False),
        # the same matrix in mixed precision
        dict(name="mixed_small", op="sweep", compute="mixed", K=10, rows=2000, cols=1500,
             nobs=60000, degrees="uniform", alpha=4.0, adaptive=False),
        # a wide model of a small matrix
        dict(name="fp64_wide_k128", op="sweep", compute="fp64", K=128, rows=2000, cols=1500,
             nobs=60000, degrees="uniform", alpha=4.0, adaptive=False),
        # ratings with learned precision, sizes that no tile divides
        dict(name="fp64_adaptive_k20", op="sweep", compute="fp64", K=20, rows=13801, cols=2701,
             nobs=1900001, degrees="powerlaw", alpha=2.0, adaptive=True),
        # the benchmark matrix (20M ratings, 138,000 x 27,000) in 64 bits and in mixed precision
        dict(name="benchmark_fp64_k32", op="sweep", compute="fp64", K=32, rows=138000,
             cols=27000, nobs=20000000, degrees="powerlaw", alpha=2.0, adaptive=False),
        dict(name="benchmark_mixed_k32", op="sweep", compute="mixed", K=32, rows=138000,
             cols=27000, nobs=20000000, degrees="powerlaw", alpha=2.0, adaptive=False),
        # the rows of a wide mixed-precision model
        dict(name="mixed_rows_k64", op="rows", compute="mixed", K=64, rows=30000, cols=6001,
             nobs=3000000, degrees="powerlaw", alpha=2.0),
        # the hyperparameters alone, of latents that another program holds on the GPU
        dict(name="prior_k64", op="prior", K=64, rows=27000),
        # side information: the compound / feature matrix of the benchmark, default tolerance
        dict(name="side_mixed_k32", op="side", compute="mixed", K=32, rows=20000, cols=500,
             nobs=1000000, nfeat=32768, ones=50, alpha=5.0),
        # its link matrix alone in 64 bits, a smaller feature set of odd size
        dict(name="link_fp64_k16", op="link", compute="fp64", K=16, rows=5003, cols=301,
             nobs=100000, nfeat=4099, ones=30, alpha=5.0),
        # the univariate sampler
        dict(name="univariate_fp64_k32", op="univariate", compute="fp64", K=32, rows=5003,
             cols=501, nobs=250000, nfeat=8193, ones=50, alpha=5.0),
        # many small models at once
        dict(name="batch_64", op="batch", nprob=64, rows=4000, cols=1000, alpha=4.0),
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["sweep", "sweep", "sweep", "sweep", "rows", "rows", "prior", "side", "link",
                     "univariate", "batch"])
    compute = rng.choice(["fp64", "fp64", "mixed"])
    if op == "prior":
        return dict(op=op, K=rng.choice([8, 10, 16, 20, 32, 33, 48, 64]), rows=span(500, 138000))
    if op == "batch":
        return dict(op=op, nprob=span(4, 64), rows=span(300, 4000), cols=span(200, 1000),
                    alpha=rng.choice([1.5, 4.0]))
    if op in ("side", "link", "univariate"):
        rows, cols = span(500, 20000), span(50, 500)
        return dict(op=op, compute=compute if op != "link" else "fp64",
                    K=rng.choice([8, 10, 16, 20, 32]), rows=rows, cols=cols,
                    nobs=min(span(5000, 1000000), rows * cols // 4), nfeat=span(300, 8192),
                    ones=rng.choice([10, 30, 50]), alpha=5.0)
    K = rng.choice([5, 8, 10, 16, 20, 24, 32, 32, 40, 64, 100, 128])
    rows = span(300, 138000)
    cols = span(200, min(rows, 27000))
    most = int(20000000 * 1024 / max(K, 16) ** 2)
    nobs = min(span(5000, 20000000), rows * cols // 6, most)
    return dict(op=op, compute=compute, K=K, rows=rows, cols=cols, nobs=nobs,
                degrees=rng.choice(["uniform", "powerlaw"]), alpha=rng.choice([2.0, 4.0]),
                **({} if op == "rows" else dict(adaptive=rng.random() < 0.25)))


# ---- inputs -------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _degrees(n, total, most, kind, g):
    """Expected entries of n rows: equal, or the power law p(k) ~ 1/k clipped to [5, most]."""
    if kind == "uniform":
        return torch.full((n,), total / n, dtype=torch.float64, device=DEVICE)
    d = 5.0 * 4000.0 ** torch.rand(n, generator=g, dtype=torch.float64, device=DEVICE)
    scale = total / d.sum()
    for _ in range(8):
        x = (d * scale).clamp(5.0, float(most))
        scale = scale * total / x.sum()
    return x


def _positions(rows, cols, nobs, kind, g):
    """nobs (or slightly fewer) distinct cells in random order."""
    cr = torch.cumsum(_degrees(rows, nobs, min(20000, cols), kind, g), 0)
    cc = torch.cumsum(_degrees(cols, nobs, min(20000, rows), kind, g), 0)
    key = torch.empty(0, dtype=torch.int64, device=DEVICE)
    for _ in range(4):
        m = int((nobs - len(key)) * 1.15) + 16
        r = torch.searchsorted(cr, torch.rand(m, generator=g, dtype=torch.float64, device=DEVICE) * cr[-1])
        c = torch.searchsorted(cc, torch.rand(m, generator=g, dtype=torch.float64, device=DEVICE) * cc[-1])
        key = torch.unique(torch.cat([key, r.clamp(max=rows - 1) * cols + c.clamp(max=cols - 1)]))
        if len(key) >= nobs:
            break
    key = key[torch.randperm(len(key), generator=g, device=DEVICE)[:nobs]]
    return key // cols, key % cols


def _normal(shape, sd, g):
    return torch.randn(shape, generator=g, dtype=torch.float64, device=DEVICE) * sd


def _spd(K, g):
    a = _normal((K, K), 1.0, g)
    return 6.0 * (a @ a.T / K + torch.eye(K, dtype=torch.float64, device=DEVICE))


def _matrix(case, seed):
    """Ratings, 10% held out, and the chain's state before the pass: latents and, for BPMF priors,
    hyperparameters of a chain past its burn-in."""
    g = _generator(seed)
    rows, cols, K = case["rows"], case["cols"], case["K"]
    r, c = _positions(rows, cols, case["nobs"], case.get("degrees", "uniform"), g)
    sd = K ** -0.25
    U, V = _normal((rows, K), sd, g), _normal((cols, K), sd, g)
    v = _normal((len(r),), 0.8, g) + 3.5
    for s in range(0, len(r), 1 << 21):
        e = slice(s, s + (1 << 21))
        v[e] += (U[r[e]] * V[c[e]]).sum(1)
    if case.get("degrees") == "powerlaw":  # ratings in half steps
        v = (v * 2.0).round().div(2.0).clamp(0.5, 5.0)
    nt = max(1, len(r) // 10)
    d = dict(r=r[nt:], c=c[nt:], v=v[nt:], tr=r[:nt], tc=c[:nt], tv=v[:nt],
             U=U + _normal(U.shape, 0.1, g), V=V + _normal(V.shape, 0.1, g),
             mu=[_normal((K,), 0.1, g) for _ in range(2)], Lambda=[_spd(K, g) for _ in range(2)])
    if "nfeat" in case:  # binary features, Zipf(1.1)-like popularity, Poisson(ones) per row
        nfeat = case["nfeat"]
        p = torch.arange(1, nfeat + 1, dtype=torch.float64, device=DEVICE) ** -1.1
        cnt = torch.poisson(torch.full((rows,), float(case["ones"]), device=DEVICE), generator=g).long()
        fr = torch.repeat_interleave(torch.arange(rows, device=DEVICE), cnt)
        cp = torch.cumsum(p, 0)
        fc = torch.searchsorted(cp, torch.rand(len(fr), generator=g, dtype=torch.float64, device=DEVICE) * cp[-1])
        key = torch.unique(fr * nfeat + fc.clamp(max=nfeat - 1))
        d["fr"], d["fc"] = key // nfeat, key % nfeat
    return d


def _np(x, dtype):
    return np.ascontiguousarray(x.cpu().numpy().astype(dtype, copy=False))


class _Latents:
    """A mode's latents in the sampler's device memory, which lives as long as this object."""

    def __init__(self, sampler, mode):
        ptr, stride, size = sampler.latents_device(mode)
        self.sampler = sampler
        self.__cuda_array_interface__ = {
            "shape": (sampler.dims[mode], stride), "typestr": "<f%d" % size,
            "data": (ptr, False), "version": 3, "strides": None}


class _Chain:
    """A sampler with its data, and the latents that it writes as torch tensors."""

    def __init__(self, case, seed):
        d = _matrix(case, seed)
        shape = (case["rows"], case["cols"])
        mixed = case["compute"] == "mixed"
        s = _lib.Sampler(case["K"], case["alpha"], seed=seed, compute=int(mixed))
        if case.get("adaptive"):
            s.set_noise_adaptive(1.0, 10.0)
        s.set_relation_data(_np(d["r"], np.int32), _np(d["c"], np.int32), _np(d["v"], np.float64), shape)
        if case["op"] not in ("rows", "link"):
            s.set_relation_data_test(_np(d["tr"], np.int32), _np(d["tc"], np.int32),
                                     _np(d["tv"], np.float64), shape)
        if "nfeat" in case:
            f = (_np(d["fr"], np.int32), _np(d["fc"], np.int32), None, (case["rows"], case["nfeat"]))
            if case["op"] == "univariate":
                s.set_side_univariate(0, *f, LAMBDA_BETA)
            else:
                s.set_side(0, *f, LAMBDA_BETA, TOL)
        s.set_samples(BURNIN, 100)
        s.init()
        s.set_latents(0, _np(d["U"], np.float64))
        s.set_latents(1, _np(d["V"], np.float64))
        for m in range(2):
            if m == 1 or "nfeat" not in case:
                s.set_hyper(m, _np(d["mu"][m], np.float64), _np(d["Lambda"][m], np.float64))
        self.s = s
        # tensors over the sampler's own buffers, each keeping the sampler alive
        self.latents = [torch.as_tensor(_Latents(s, m), device=DEVICE) for m in (0, 1)]


def _problems(case, seed):
    """Small matrices of uneven size, K in {8, 16, 32}, 1 to 5% filled, 10% held out: the sizes are
    the case's, the entries the seed's."""
    sizes, rng = np.random.default_rng(case["nprob"]), np.random.default_rng(seed)
    problems, K = [], []
    for _ in range(case["nprob"]):
        nr = int(sizes.integers(case["rows"] // 20 + 1, case["rows"] + 1))
        nc = int(sizes.integers(case["cols"] // 10 + 1, case["cols"] + 1))
        k = int(sizes.choice([8, 16, 32]))
        n = max(32, int(nr * nc * sizes.uniform(0.01, 0.05)))
        pos = rng.permutation(np.unique(rng.integers(0, nr * nc, n)))
        r, c = (pos // nc).astype(np.int32), (pos % nc).astype(np.int32)
        U, V = (rng.normal(0.0, k ** -0.25, (x, k)).astype(np.float32) for x in (nr, nc))
        v = np.einsum("ij,ij->i", U[r], V[c]).astype(np.float64) + rng.normal(0.0, 0.5, len(r))
        nt = max(1, len(r) // 10)
        problems.append(dict(rows=r[nt:], cols=c[nt:], vals=v[nt:], trows=r[:nt], tcols=c[:nt],
                             tvals=v[:nt], shape=(nr, nc)))
        K.append(k)
    return problems, K


def _prior_inputs(case, seed):
    g = _generator(seed)
    K = case["K"]
    return (_normal((case["rows"], K), 0.5, g) + _normal((K,), 0.2, g),
            torch.zeros(K, dtype=torch.float64, device=DEVICE),
            torch.eye(K, dtype=torch.float64, device=DEVICE))


class _Prior:
    def __init__(self, case, seed):
        self.U, self.mu0, self.T = _prior_inputs(case, seed)
        self.seed = int(seed)
        self.mu, self.Lambda = torch.empty_like(self.mu0), torch.empty_like(self.T)
        self.call = _lib.lib().mg_normal_wishart_noalloc
        self.err = ctypes.create_string_buffer(256)


def prepare(case, seed):
    if case["op"] == "prior":
        return case, _Prior(case, seed)
    if case["op"] == "batch":
        problems, K = _problems(case, seed)
        b = _lib.Batch(problems, K, [seed + i for i in range(len(K))], case["alpha"])
        b.init(burnin=BURNIN)
        return case, b
    return case, _Chain(case, seed)


# ---- one pass -----------------------------------------------------------------------------------

def run(state):
    case, st = state
    op = case["op"]
    if op == "prior":
        n, k = st.U.shape
        code = st.call(st.U.data_ptr(), n, k, k, st.mu0.data_ptr(), 2.0, st.T.data_ptr(), k,
                       st.seed, ITERATION, 0, st.mu.data_ptr(), st.Lambda.data_ptr(), None,
                       st.err, len(st.err))
        if code != 0:
            raise RuntimeError(st.err.value.decode())
        return {"mu": st.mu, "Lambda": st.Lambda}
    if op == "batch":
        st.sweeps(BURNIN, 20, eval=True)
        return {"rmse": st.rmse(), "latents": [np.concatenate(
            [st.latents(p, m).reshape(-1) for p in range(st.P)]).astype(np.float32) for m in (0, 1)]}
    s = st.s
    if op == "rows":
        s.sample_latents(0, ITERATION)
        return {"U": st.latents[0]}
    if op == "link":
        s.update_prior(0, ITERATION)
        return {"beta": s.beta(0).astype(np.float32)}  # solved to 1e-6
    s.sweep(ITERATION, eval=True)
    if case["compute"] == "fp64" and op == "sweep":
        return {"U": st.latents[0], "V": st.latents[1], "rmse": list(s.rmse())}
    return {"U": st.latents[0], "V": st.latents[1]}


# ---- what a pass cannot do without -----------------------------------------------------------------

def work(case):
    K = case["K"] if "K" in case else 20
    if case["op"] == "prior":
        n = case["rows"]
        return {"bytes": 8.0 * n * K, "flops": float(n) * K * (K + 1)}
    sweeps = 1
    if case["op"] == "batch":
        sweeps, P = 20, case["nprob"]
        rows, cols = 0.525 * case["rows"] * P, 0.55 * case["cols"] * P
        nnz, test, mixed = 0.9 * 0.03 * rows * cols / P, 0.1 * 0.03 * rows * cols / P, True
    else:
        rows, cols, mixed = float(case["rows"]), float(case["cols"]), case["compute"] == "mixed"
        nnz, test = 0.9 * case["nobs"], 0.1 * case["nobs"]
    entry, value = (8.0, 4.0) if mixed else (12.0, 8.0)
    finish = K ** 3 / 3.0 + 6.0 * K * K
    # a mode's rows: its entries and the other mode's latents in, its own latents out
    half = [(n, nnz * entry + (n + o) * K * value, nnz * (K * (K + 1) + 2.0 * K) + n * finish)
            for n, o in ((rows, cols), (cols, rows))]
    prior = [(n * K * value, n * K * (K + 1.0)) for n in (rows, cols)]
    link = (0.0, 0.0)
    if "nfeat" in case:
        ones = float(case["ones"]) * rows
        link = (8.0 * ones + 8.0 * K * (rows + 2.0 * case["nfeat"]), 8.0 * ones * K)
    if case["op"] == "rows":
        return {"bytes": half[0][1], "flops": half[0][2]}
    if case["op"] == "link":
        return {"bytes": prior[0][0] + link[0], "flops": prior[0][1] + link[1]}
    evaluation = (32.0 * test, 2.0 * K * test)
    noise = (16.0 * nnz, 2.0 * K * nnz) if case.get("adaptive") else (0.0, 0.0)
    parts = [h[1:] for h in half] + prior + [link, evaluation, noise]
    return {"bytes": sweeps * sum(p[0] for p in parts), "flops": sweeps * sum(p[1] for p in parts)}


# ---- the same in 64 bits, without the library -------------------------------------------------------

_M32 = 0xFFFFFFFF


def _philox(c, k0, k1):
    """Philox-4x32-10 (Salmon et al., SC'11) of four counter words (int64 tensors of 32-bit values)."""
    c0, c1, c2, c3 = c
    for r in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & _M32) ^ c1 ^ ((k0 + r * 0x9E3779B9) & _M32), p1 & _M32,
                          ((p0 >> 32) & _M32) ^ c3 ^ ((k1 + r * 0xBB67AE85) & _M32), p0 & _M32)
    return c0, c1, c2, c3


def _uniforms(seed, purpose, mode, index, block):
    """The two 53-bit uniforms in (0, 1) of each block keyed (seed, iteration, purpose, mode, index)."""
    index, block = torch.broadcast_tensors(index, block)
    one = torch.ones_like(index)
    w = _philox((block, index, one * (purpose << 8 | mode), one * ITERATION), seed & _M32, seed >> 32 & _M32)

    def unit(hi, lo):
        return ((((hi << 32) | lo) >> 11) & ((1 << 53) - 1)).double().add(0.5).mul(2.0 ** -53)
    return unit(w[0], w[1]), unit(w[2], w[3])


def _arange(n):
    return torch.arange(n, dtype=torch.int64, device=DEVICE)


def _normals(seed, purpose, mode, n, K):
    """n x K standard normals by Box-Muller, two to a block."""
    u1, u2 = _uniforms(seed, purpose, mode, _arange(n)[:, None], _arange((K + 1) // 2)[None, :])
    rad, th = torch.sqrt(-2.0 * torch.log(u1)), 6.283185307179586 * u2
    return torch.stack([rad * torch.cos(th), rad * torch.sin(th)], 2).reshape(n, -1)[:, :K]


def _gammas(seed, purpose, mode, shapes):
    """Gamma(shape, 1) by Marsaglia and Tsang (2000), shapes of at least 1."""
    out = []
    for i, shape in enumerate(shapes):
        d = shape - 1.0 / 3.0
        c = 1.0 / math.sqrt(9.0 * d)
        u1, u2 = (x.tolist() for x in _uniforms(seed, purpose, mode, torch.full((128,), i, device=DEVICE), _arange(128)))
        got = d
        for t in range(64):
            x = math.sqrt(-2.0 * math.log(u1[2 * t])) * math.cos(6.283185307179586 * u2[2 * t])
            v = (1.0 + c * x) ** 3
            if v > 0.0 and math.log(u1[2 * t + 1]) < 0.5 * x * x + d - d * v + d * math.log(v):
                got = d * v
                break
        out.append(got)
    return torch.tensor(out, dtype=torch.float64, device=DEVICE)


def _grams(r, c, w, V, n):
    """sum v v^T and sum w v of each of n rows."""
    K = V.shape[1]
    order = torch.argsort(r, stable=True)
    c, w = c[order], w[order]
    length = torch.bincount(r, minlength=n)
    start = torch.cumsum(length, 0) - length
    G, b = V.new_zeros(n, K, K), V.new_zeros(n, K)
    by = torch.argsort(length, descending=True)
    most = (1 << 25) // K
    at, host = 0, length[by].tolist()
    while at < n and host[at] > 0:
        L = host[at]
        rows = by[at:at + max(1, most // L)]
        pos = torch.arange(L, device=V.device)
        ok = pos < length[rows][:, None]
        e = (start[rows][:, None] + pos).clamp(max=len(c) - 1)
        X = V[c[e]] * ok[:, :, None]
        G[rows] = X.transpose(1, 2) @ X
        b[rows] = (X.transpose(1, 2) @ (w[e] * ok)[:, :, None])[:, :, 0]
        at += len(rows)
    return G, b


def _sample(d, V, mode, mu, Lambda, alpha, seed, univariate=None):
    """The rows of a mode given the other mode's latents V."""
    K = V.shape[1]
    r, c = (d["r"], d["c"]) if mode == 0 else (d["c"], d["r"])
    n = len(d["U"] if mode == 0 else d["V"])
    G, b = _grams(r, c, (d["v"] - d["v"].mean()) * alpha, V, n)
    z = _normals(seed, 1, mode, n, K)
    if univariate is not None:  # coordinate by coordinate from the current values
        u, lam = univariate.clone(), torch.diagonal(Lambda)
        for k in range(K):
            q = lam[k] + alpha * G[:, k, k]
            rest = (G[:, k] * u).sum(1) - G[:, k, k] * u[:, k]
            u[:, k] = (lam[k] * mu[k] + b[:, k] - alpha * rest) / q + z[:, k] / torch.sqrt(q)
        return u
    G *= alpha
    G += Lambda
    L = torch.linalg.cholesky(G)
    y = torch.linalg.solve_triangular(L, (b + Lambda @ mu)[:, :, None], upper=False)
    return torch.linalg.solve_triangular(L.transpose(1, 2), y + z[:, :, None], upper=True)[:, :, 0]


def _normal_wishart(U, mode, seed, T, nu):
    """(mu, Lambda) of the Normal-Wishart posterior of the rows of U, prior mean 0 and strength 2."""
    n, K = U.shape
    kappa = 2.0 + n
    m = U.sum(0) / kappa
    X = T + U.T @ U - kappa * torch.outer(m, m)
    L = torch.linalg.cholesky(torch.linalg.inv(X))
    C = torch.zeros_like(X)
    off = _normals(seed, 4, mode, K, K)
    diag = torch.sqrt(2.0 * _gammas(seed, 5, mode, [0.5 * (nu + n - i) for i in range(K)]))
    for i in range(K):
        C[i, i] = diag[i]
        C[i, i + 1:] = off[i, :K - 1 - i]
    B = L @ C.T
    Lambda = B @ B.T
    z = _normals(seed, 6, mode, 1, K)[0]
    mu = m + torch.linalg.solve_triangular((B * math.sqrt(kappa)).T, z[:, None], upper=True)[:, 0]
    return mu, Lambda


def _link(d, case, seed):
    """The link matrix that one update draws: (F^T F + lambda I) beta = right-hand side."""
    K, nfeat, n = case["K"], case["nfeat"], case["rows"]
    eye = torch.eye(K, dtype=torch.float64, device=DEVICE)
    mu, Lambda = _normal_wishart(d["U"], 0, seed, eye, K + nfeat)
    Lt = torch.linalg.cholesky(Lambda).T

    def mvn(purpose, count):
        return torch.linalg.solve_triangular(Lt, _normals(seed, purpose, 0, count, K).T, upper=True).T
    F = torch.zeros(n, nfeat, dtype=torch.float64, device=DEVICE)
    F[d["fr"], d["fc"]] = 1.0
    rhs = F.T @ (d["U"] + mvn(2, n) - mu) + math.sqrt(LAMBDA_BETA) * mvn(3, nfeat)
    A = F.T @ F
    A.diagonal().add_(LAMBDA_BETA)
    return torch.cholesky_solve(rhs, torch.linalg.cholesky(A))


def _padded(U):
    """The library's rows: K values in a row of 8, 16, 32, 64 or 128."""
    K = U.shape[1]
    return torch.nn.functional.pad(U, (0, next(p for p in (8, 16, 32, 64, 128) if p >= K) - K))


def exact(case, seed):
    op = case["op"]
    if op == "batch":  # twenty chained iterations from zero: no 64-bit value of theirs is near
        return None
    if op == "prior":
        U, _, T = _prior_inputs(case, seed)
        mu, Lambda = _normal_wishart(U, 0, seed, T, case["K"])
        return {"mu": mu, "Lambda": Lambda}
    d = _matrix(case, seed)
    if op == "link":
        return {"beta": _link(d, case, seed)}
    K, alpha = case["K"], case["alpha"]
    if case.get("adaptive"):
        alpha = 2.0 / (d["v"] - d["v"].mean()).square().mean().item()
    mu, Lambda = list(d["mu"]), list(d["Lambda"])
    if "nfeat" in case:  # before the first update of a prior with side information
        mu[0] = torch.zeros_like(mu[0])
        Lambda[0] = 10.0 * torch.eye(K, dtype=torch.float64, device=DEVICE)
    U = _sample(d, d["V"], 0, mu[0], Lambda[0], alpha, seed, d["U"] if op == "univariate" else None)
    if op == "rows":
        return {"U": _padded(U)}
    V = _sample(d, U, 1, mu[1], Lambda[1], alpha, seed)
    out = {"U": _padded(U), "V": _padded(V)}
    if case["compute"] == "fp64" and op == "sweep":
        p = (U[d["tr"]] * V[d["tc"]]).sum(1) + d["v"].mean()
        out["rmse"] = [(d["tv"] - p / (ITERATION - BURNIN + 1)).square().mean().sqrt().item(),
                       (d["tv"] - p).square().mean().sqrt().item()]
    return out
