"""The hyperprior update (hyper_wide.cu, k_stats32) at the edges of its 8 x 8 tiles, of its four-row
steps, of its row blocks (128 rows each) and of the partials the draw adds itself (16 blocks), FP64
and mixed, one mode and both."""
import numpy as np
import pytest

from macau_b200 import _lib
from oracle import oracle as orc
from tests.gpu_helpers import gpu_sampler, relerr
from tests.test_gpu_parity import FP64_TOL

pytestmark = pytest.mark.gpu


def matrix(rows, cols):
    rng = np.random.default_rng(rows)
    return dict(rows=np.arange(rows, dtype=np.int32), cols=np.zeros(rows, np.int32) + cols // 2,
                vals=rng.normal(size=rows), shape=(rows, cols))


@pytest.mark.parametrize("K", [1, 2, 7, 8, 9, 20, 32, 33, 40, 63, 64, 65, 100, 128])
@pytest.mark.parametrize("rows", [1, 130, 517, 2100])
@pytest.mark.parametrize("compute", [_lib.MG_COMPUTE_FP64, _lib.MG_COMPUTE_MIXED])
def test_draw_matches_oracle(K, rows, compute):
    rng = np.random.default_rng(K + rows)
    s = gpu_sampler(matrix(rows, 7), K, 1.0, seed=99, compute=compute)
    # values that FP32 holds exactly: both computes see the oracle's latents
    U = rng.normal(0.3, 1.0, size=(rows, K)).astype(np.float32).astype(np.float64)
    s.set_latents(0, U)
    s.update_prior(0, 11)
    mu, Lam, _ = s.hyper(0)
    mu_o, Lam_o, st = orc.cond_normal_wishart(U, np.zeros(K), 2.0, np.eye(K), K, seed=99, sweep=11,
                                              mode=0)
    assert st == 0
    assert relerr(Lam, Lam_o) < FP64_TOL and relerr(mu, mu_o) < FP64_TOL
    np.testing.assert_array_equal(Lam, Lam.T)
    s.close()


@pytest.mark.parametrize("K", [10, 40, 128])
def test_both_modes_at_once_match_one_at_a_time(K):
    rng = np.random.default_rng(K)
    w = matrix(300, 170)
    a, b = (gpu_sampler(w, K, 1.0, seed=4) for _ in range(2))
    U, V = (rng.normal(size=(n, K)) for n in w["shape"])
    for s in (a, b):
        s.set_latents(0, U)
        s.set_latents(1, V)
    a.sweep(3, eval=False)  # both samplers, then both priors in one launch per step
    for m in (0, 1):
        b.sample_latents(m, 3)
    for m in (0, 1):
        b.update_prior(m, 3)
        for x, y in zip(a.hyper(m)[:2], b.hyper(m)[:2]):
            np.testing.assert_array_equal(x, y)
    a.close()
    b.close()
