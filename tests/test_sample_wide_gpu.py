"""The row sampler for 32 < K <= 128 (sample_wide.cu) at the edges of its entry steps (4 in FP64,
16 with BF16 gathers), chunks (32), component blocks and panels (8), and its FP64 redo."""
import numpy as np
import pytest

from macau_b200 import _lib
from oracle import oracle as orc
from tests.gpu_helpers import gpu_sampler, random_spd, relerr, train_matrix
from tests.test_gpu_parity import FP64_TOL, MIXED_SAMPLE_TOL

pytestmark = pytest.mark.gpu

LENGTHS = (0, 1, 3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 129, 255, 256, 257, 700)


def problem(K, rng, ncol=720):
    rows = np.repeat(np.arange(len(LENGTHS)), LENGTHS)
    cols = np.concatenate([rng.permutation(ncol)[:n] for n in LENGTHS])
    return dict(rows=rows.astype(np.int32), cols=cols.astype(np.int32),
                vals=rng.normal(size=len(rows)), shape=(len(LENGTHS), ncol))


@pytest.mark.parametrize("K", [33, 40, 41, 63, 64, 65, 100, 127, 128])
@pytest.mark.parametrize("compute", [_lib.MG_COMPUTE_FP64, _lib.MG_COMPUTE_MIXED])
def test_row_lengths_match_oracle(K, compute):
    rng = np.random.default_rng(K)
    w = problem(K, rng)
    V = rng.normal(scale=0.4, size=(w["shape"][1], K))
    mu, Lam = rng.normal(scale=0.2, size=K), random_spd(rng, K, 3.0)
    Y = orc.Csr.from_scipy(train_matrix(w))
    for groups in ((1, 2) if K <= 64 else (0,)):
        s = gpu_sampler(w, K, 1.5, seed=K, compute=compute)
        s.set_option("split_threshold", 256)  # rows of 257 and 700 entries in parts
        s.set_option("cta_groups", groups)
        s.set_latents(1, V)
        s.set_hyper(0, mu, Lam)
        s.sample_latents(0, 5)
        want, _ = orc.sample_latents(K, Y, V, s.mean_value(), 1.5, mu, Lam, seed=K, sweep=5, mode=0)
        assert relerr(s.latents(0), want) < (FP64_TOL if compute == _lib.MG_COMPUTE_FP64
                                             else MIXED_SAMPLE_TOL)
        assert s.stats()["retries"] == [0, 0]
        s.close()


@pytest.mark.parametrize("K", [48, 128])
def test_failed_fp32_factors_are_redone_in_fp64(K):
    # Lambda = 1e-7 I: a row of at most K / 2 entries has K / 2 pivots of pure FP32 rounding, and
    # one of them lies below the floor.  (A row one entry short of K has a single such pivot, which
    # may lie above it.)  The latents are exact in BF16 (multiples of 1/4), so that the FP64 redo
    # has the oracle's Gram but for FP32 accumulation, which is exact here too (sums of multiples
    # of 1/16 below 2^20)
    rng = np.random.default_rng(K)
    w = problem(K, rng)
    V = rng.integers(-4, 5, size=(w["shape"][1], K)) / 4.0
    Lam = 1e-7 * np.eye(K)
    s = gpu_sampler(w, K, 1.5, seed=2, compute=_lib.MG_COMPUTE_MIXED)
    s.set_latents(1, V)
    s.set_hyper(0, np.zeros(K), Lam)
    s.sample_latents(0, 4)
    short = np.array(LENGTHS) <= K // 2
    # an empty row's MM is Lambda itself: well conditioned, no redo
    assert s.stats()["retries"][0] >= short.sum() - 1
    want, _ = orc.sample_latents(K, orc.Csr.from_scipy(train_matrix(w)), V, s.mean_value(), 1.5,
                                 np.zeros(K), Lam, seed=2, sweep=4, mode=0)
    # conditions up to ~1e10 in FP64 (1e-6), stored as FP32; the weights are rounded to FP32
    # before the sums (6e-8 of them, times the condition of the row's own entries)
    assert relerr(s.latents(0)[short], want[short]) < MIXED_SAMPLE_TOL
    s.close()
