"""Chains with a block-CG link, block-CG solves, batches and wide mixed rows against recorded ones, bit
for bit.

A link solve ends at a tolerance, so one rounding in what reaches it moves the link matrix by 1e-7 to
1e-6, and a batch's mixed chains and mixed rows at K > 32 part after a rounding that falls the other
way: these paths keep one order of summation (macau_b200/csrc/hyper_ordered.cu, sample_wide_mixed.cu).  golden/recorded_chains.json holds digests of
their outputs, recorded on a B200 with the scalar kernels that the matrix-instruction and pipelined
ones replaced; a change of the order, of the matrix instruction's rounding or of its place in a row
shows as another digest, whatever its size.
"""
import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

from macau_b200 import _lib

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).parent / "golden" / "recorded_chains.json"
ROWS, COLS, NFEAT = 1500, 301, 403


def digest(*arrays):
    h = hashlib.sha256()
    for a in arrays:
        h.update(np.ascontiguousarray(a, np.float64).tobytes())
    return h.hexdigest()[:16]


def zipf_pairs(rng, nrow, ncol, mean):
    """Distinct (row, column) pairs, mean a row, columns by Zipf(1.1): the first ones are long."""
    p = np.arange(1, ncol + 1, dtype=np.float64) ** -1.1
    n = rng.poisson(mean, nrow)
    r = np.repeat(np.arange(nrow), n)
    c = np.minimum(np.searchsorted(np.cumsum(p) / p.sum(), rng.random(len(r))), ncol - 1)
    key = np.unique(r * ncol + c)
    return (key // ncol).astype(np.int32), (key % ncol).astype(np.int32)


def chain_start(K, mixed, kind, weighted):
    """A sampler with a block-CG link on mode 0 ("one"), on both ("both"), or on mode 1 with the
    univariate prior on mode 0 ("univariate")."""
    rng = np.random.default_rng(1000 * K + 10 * weighted)
    r, c = zipf_pairs(rng, ROWS, COLS, 14)
    U, V = (rng.normal(scale=0.4, size=(n, K)) for n in (ROWS, COLS))
    y = (U[r] * V[c]).sum(1) + rng.normal(scale=0.5, size=len(r)) + 3.0
    s = _lib.Sampler(K, 2.0, seed=31, compute=int(mixed))
    s.set_relation_data(r, c, y, (ROWS, COLS))

    def side(mode, n, nfeat, mean, dense):
        fr, fc = zipf_pairs(rng, n, nfeat, mean)
        if dense:  # one feature that every row has
            keep = fc != 0
            fr = np.concatenate([fr[keep], np.arange(n, dtype=np.int32)])
            fc = np.concatenate([fc[keep], np.zeros(n, np.int32)])
        w = rng.normal(size=len(fr)) if weighted else None
        if mode == 0 and kind == "univariate":
            s.set_side_univariate(mode, fr, fc, w, (n, nfeat), 5.0)
        else:
            s.set_side(mode, fr, fc, w, (n, nfeat), 5.0, 1e-6)

    side(0, ROWS, NFEAT, 20, kind == "univariate")
    if kind != "one":
        side(1, COLS, 57, 6, False)
    s.set_samples(0, 2)
    s.init()
    s.set_latents(0, U)
    s.set_latents(1, V)
    return s


def chain(K, mixed, kind, weighted, sweeps=2):
    s = chain_start(K, mixed, kind, weighted)
    out = {}
    for it in range(sweeps):
        s.sweep(it, eval=False)
        for m in (0, 1):
            out[f"{it} latents {m}"] = digest(s.latents(m))
            mu, Lam, lb = s.hyper(m)
            out[f"{it} hyper {m}"] = digest(mu, Lam)
            if m == 0 or kind != "one":
                univariate = m == 0 and kind == "univariate"
                out[f"{it} link {m}"] = digest(s.beta(m), s.uhat(m))
                out[f"{it} lambda_beta {m}"] = digest(s.lambda_beta_univariate(m) if univariate else lb)
    s.close()
    return out


def solve(n, mixed, weighted):
    rng = np.random.default_rng(77 + n)
    r, c = zipf_pairs(rng, ROWS, NFEAT, 20)
    w = rng.normal(size=len(r)) if weighted else None
    X, it, _ = _lib.blockcg_raw(r, c, w, (ROWS, NFEAT), rng.normal(size=(n, NFEAT)), 5.0, 1e-6,
                                int(mixed))
    return {"X": digest(X), "iterations": digest(float(it))}


def batch():
    rng = np.random.default_rng(5)
    problems, K = [], [8, 16, 32, 5, 20, 27]
    for k, (n, m) in zip(K, ((700, 150), (321, 99), (1003, 211), (33, 40), (260, 300), (517, 64))):
        r, c = zipf_pairs(rng, n, m, 9)
        y = rng.normal(size=len(r))
        problems.append(dict(rows=r[5:], cols=c[5:], vals=y[5:], trows=r[:5], tcols=c[:5],
                             tvals=y[:5], shape=(n, m)))
    b = _lib.Batch(problems, K, list(range(40, 40 + len(K))), 4.0)
    b.init(1)
    b.sweeps(0, 4)
    out = {f"{p} {m}": digest(b.latents(p, m)) for p in range(len(K)) for m in (0, 1)}
    b.close()
    return out


def wide_rows(K):
    """Mixed rows of every length up to 700, those shorter than K redone in FP64: Lambda = 1e-7 I, so
    that their FP32 pivots are rounding alone."""
    lengths = (0, 1, 3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 129, 255, 256, 257, 700)
    rng = np.random.default_rng(K)
    r = np.repeat(np.arange(len(lengths), dtype=np.int32), lengths)
    c = np.concatenate([rng.permutation(720)[:n] for n in lengths]).astype(np.int32)
    s = _lib.Sampler(K, 1.5, seed=2, compute=_lib.MG_COMPUTE_MIXED)
    s.set_relation_data(r, c, rng.normal(size=len(r)), (len(lengths), 720))
    s.set_samples(0, 1)
    s.init()
    s.set_option("split_threshold", 256)  # rows of 257 and 700 entries in parts
    s.set_latents(1, rng.integers(-4, 5, size=(720, K)) / 4.0)
    s.set_hyper(0, np.zeros(K), 1e-7 * np.eye(K))
    s.sample_latents(0, 4)
    out = {"rows": digest(s.latents(0)), "redone": s.stats()["retries"][0]}
    s.close()
    return out


CHAINS = [(K, mixed, kind, weighted) for K in (1, 7, 8, 16, 31, 32, 33, 40, 64) for mixed in (0, 1)
          for kind in ("one", "both", "univariate") for weighted in (0, 1)]
SOLVES = [(n, mixed, weighted) for n in (1, 8, 9, 16, 17, 32, 33, 64) for mixed in (0, 1)
          for weighted in (0, 1)]


def recorded(key):
    return json.loads(GOLDEN.read_text())[key]


@pytest.mark.parametrize("n,mixed,weighted", SOLVES)
def test_solve(n, mixed, weighted):
    assert solve(n, mixed, weighted) == recorded("solve %d %d %d" % (n, mixed, weighted))


@pytest.mark.parametrize("K,mixed,kind,weighted", CHAINS)
def test_chain(K, mixed, kind, weighted):
    assert chain(K, mixed, kind, weighted) == recorded("chain %d %d %s %d" % (K, mixed, kind, weighted))


@pytest.mark.parametrize("K", [33, 48, 64, 65, 100, 128])
def test_wide_rows(K):
    assert wide_rows(K) == recorded("rows %d" % K)


def test_batch():
    assert batch() == recorded("batch")
