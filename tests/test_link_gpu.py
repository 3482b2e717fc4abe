"""The link kernels at the edges of their splits: the SpMM (16 gathers in flight, chunks of 32 indices,
parts of 256 entries, 32 or 64 padded components), FP64 rows of a chain with a block-CG link, and the
univariate sampler's levels (a warp per short feature, the whole block per long one)."""
import numpy as np
import pytest
import scipy.sparse as sp

from macau_b200 import _lib
from oracle import oracle as orc
from tests.gpu_helpers import gpu_sampler, random_spd, relerr, train_matrix
from tests.test_gpu_parity import small_uniform, univariate_pair

pytestmark = pytest.mark.gpu

LENGTHS = (0, 1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65, 127, 255, 256, 257, 272, 511, 513, 640)


def side_of_lengths(rng, nrows, lengths, binary):
    cols = np.repeat(np.arange(len(lengths)), lengths)
    rows = np.concatenate([rng.permutation(nrows)[:n] for n in lengths]).astype(np.int32)
    vals = np.ones(len(rows)) if binary else rng.normal(size=len(rows))
    return sp.csr_matrix((vals, (rows, cols)), shape=(nrows, len(lengths)))


@pytest.mark.parametrize("K", [1, 8, 31, 32, 33, 64])
@pytest.mark.parametrize("binary", [True, False])
def test_spmm_row_lengths(K, binary):
    # Uhat = F beta, rows of F of every length: sums of at most 640 products, so FP64 rounding
    rng = np.random.default_rng(K + 100 * binary)
    lengths = (LENGTHS * 15)[:300]
    F = side_of_lengths(rng, 700, lengths, binary).T.tocoo()
    s = gpu_sampler(small_uniform(seed=1, nrow=300), K, 1.5, 5, init=False)
    s.set_side(0, F.row, F.col, None if binary else F.data, F.shape, 50.0, 1e-6)
    s.init()
    s.set_latents(0, rng.normal(scale=0.5, size=(300, K)))
    s.update_prior(0, 2)
    assert relerr(s.uhat(0), F @ s.beta(0)) < 640 * 2.3e-16
    s.close()


@pytest.mark.parametrize("K", [1, 8, 9, 17, 32])
def test_link_chain_rows_and_hyper_match_oracle(K):
    # FP64 rows of a chain with a block-CG link (k_sample's order of summation) and its hyperprior
    rng = np.random.default_rng(K)
    w = small_uniform(seed=3, nrow=297, ncol=131, nobs=9000)
    F = side_of_lengths(rng, 297, (1, 33, 64, 200, 297), False)
    Fc = F.tocoo()
    s = gpu_sampler(w, K, 1.5, 21, init=False)
    s.set_side(0, Fc.row, Fc.col, Fc.data, F.shape, 4.0, 1e-12)
    s.init()
    U, V = (rng.normal(scale=0.4, size=(n, K)) for n in w["shape"])
    mu, Lam = rng.normal(scale=0.2, size=K), random_spd(rng, K, 3.0)
    s.set_latents(1, V)
    s.set_hyper(1, mu, Lam)
    s.set_latents(0, U)
    s.sample_latents(1, 6)
    want, _ = orc.sample_latents(K, orc.Csr.from_scipy(train_matrix(w).T.tocsr()), U,
                                 s.mean_value(), 1.5, mu, Lam, seed=21, sweep=6, mode=1)
    assert relerr(s.latents(1), want) < 1e-9
    s.close()


@pytest.mark.parametrize("binary", [True, False])
@pytest.mark.parametrize("K", [1, 12, 33])
def test_univariate_levels_of_mixed_lengths(K, binary):
    rng = np.random.default_rng(7 * K + binary)
    w = small_uniform(seed=2, nrow=700, ncol=150, nobs=9000)
    short = tuple(rng.integers(0, 4, size=120))
    F = side_of_lengths(rng, 700, short + LENGTHS + short, binary)
    s, m = univariate_pair(w, K, 55, 0, F)
    for it in (0, 1):
        U = rng.normal(scale=0.5, size=(700, K))
        s.set_latents(0, U)
        m.set("latents", 0, U)
        s.update_prior(0, it)
        assert m.update_prior(0, it) == 0
        assert relerr(s.beta(0), m.beta(0)) < 1e-9
        assert relerr(s.uhat(0), m.uhat(0)) < 1e-9
        assert relerr(s.lambda_beta_univariate(0), m.lambda_beta_one(0)) < 1e-9
    s.close()


@pytest.mark.parametrize("nshort", [31, 32, 33, 513, 1400])
@pytest.mark.parametrize("binary", [True, False])
def test_univariate_wide_levels(nshort, binary):
    # features of 0 to 3 entries: a lane each up to two entries, where a level has 32 of them or more
    rng = np.random.default_rng(nshort + binary)
    w = small_uniform(seed=2, nrow=700, ncol=150, nobs=9000)
    lengths = tuple(rng.permutation([0, 1, 2] * nshort)[:nshort]) + (3, 40, 0, 300, 2)
    s, m = univariate_pair(w, 9, 55, 0, side_of_lengths(rng, 700, lengths, binary))
    for it in (0, 1):
        U = rng.normal(scale=0.5, size=(700, 9))
        s.set_latents(0, U)
        m.set("latents", 0, U)
        s.update_prior(0, it)
        assert m.update_prior(0, it) == 0
        assert relerr(s.beta(0), m.beta(0)) < 1e-9
        assert relerr(s.uhat(0), m.uhat(0)) < 1e-9
        assert relerr(s.lambda_beta_univariate(0), m.lambda_beta_one(0)) < 1e-9
    s.close()


@pytest.mark.parametrize("K", [1, 16, 32, 33, 64])
@pytest.mark.parametrize("binary", [True, False])
def test_spmm_many_short_rows(K, binary):
    # 16,384 tasks and more take 8 gathers at a time: rows of F at the edges of these; a row's sum of n
    # <= 40 products is off by at most n n eps times the largest product
    rng = np.random.default_rng(K + binary)
    lengths = ((0, 1, 2, 3, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 40) * 1134)[:17001]
    F = side_of_lengths(rng, 700, lengths, binary).T.tocoo()
    s = gpu_sampler(small_uniform(seed=1, nrow=17001, ncol=60, nobs=40000), K, 1.5, 5, init=False)
    s.set_side(0, F.row, F.col, None if binary else F.data, F.shape, 50.0, 1e-6)
    s.init()
    s.set_latents(0, rng.normal(scale=0.5, size=(17001, K)))
    s.update_prior(0, 2)
    beta = s.beta(0)
    bound = 40 * 40 * 2.3e-16 * np.abs(F.data).max() * np.abs(beta).max()
    assert np.abs(s.uhat(0) - F @ beta).max() < bound
    s.close()
