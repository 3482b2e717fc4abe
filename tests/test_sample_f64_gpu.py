"""The FP64 warp-per-row sampler (mma.sync.m8n8k4.f64 Grams, K <= 32) at the edges of its entry
steps (4), gather ring (12 ahead) and chunks (32), and of its component blocks (8)."""
import numpy as np
import pytest

from macau_b200 import _lib
from oracle import oracle as orc
from tests.gpu_helpers import gpu_sampler, random_spd, relerr, train_matrix

pytestmark = pytest.mark.gpu

TOL = 1e-9  # FP64 on both sides, sums in another order: rounding times the rows' condition number
LENGTHS = (0, 1, 3, 4, 5, 12, 13, 16, 17, 31, 32, 33, 36, 44, 45, 63, 64, 65, 96, 129, 255, 256, 257, 700)


@pytest.mark.parametrize("K", [1, 7, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("groups", [2, 4])
def test_row_lengths_match_oracle(K, groups):
    rng = np.random.default_rng(100 * K + groups)
    ncol = 720
    rows = np.repeat(np.arange(len(LENGTHS)), LENGTHS)
    cols = np.concatenate([rng.permutation(ncol)[:n] for n in LENGTHS])
    w = dict(rows=rows.astype(np.int32), cols=cols.astype(np.int32),
             vals=rng.normal(size=len(rows)), shape=(len(LENGTHS), ncol))
    s = gpu_sampler(w, K, 1.5, seed=K)
    s.set_option("split_threshold", 256)  # rows of 257 and 700 entries in parts
    s.set_option("cta_groups", groups)
    V = rng.normal(scale=0.4, size=(ncol, K))
    mu, Lam = rng.normal(scale=0.2, size=K), random_spd(rng, K, 3.0)
    s.set_latents(1, V)
    s.set_hyper(0, mu, Lam)
    s.sample_latents(0, 5)
    want, _ = orc.sample_latents(K, orc.Csr.from_scipy(train_matrix(w)), V, s.mean_value(), 1.5,
                                 mu, Lam, seed=K, sweep=5, mode=0)
    assert relerr(s.latents(0), want) < TOL
    s.close()
