"""Two iterations of a chain with a block-CG link against the oracle, over the widths at which its
kernels change (8, 16, 32, 64 columns of a solve; K <= 32 and above): rows with Uhat, statistics,
draws with beta beta^T, solves and lambda_beta."""
import numpy as np
import pytest
import scipy.sparse as sp

from macau_b200 import _lib, workloads
from oracle import oracle as orc
from tests.gpu_helpers import gpu_sampler, oracle_model, relerr
from tests.test_gpu_parity import FP64_TOL, MIXED_SAMPLE_TOL, gpu_cg_parts

pytestmark = pytest.mark.gpu

ROWS, NFEAT, LAMBDA_BETA = 2000, 3000, 50.0


@pytest.fixture
def oracle_parts():
    yield orc.set_reduce_parts
    orc.set_reduce_parts(1)


def workload(K, binary):
    # features at uniform positions: F^T F + 50 I has its spectrum in 50 .. 90 but for the mean's
    # direction, so that a solve to 1e-12 determines the link matrix to about that
    rng = np.random.default_rng(K)
    w = workloads.bpmf_uniform(nrow=ROWS, ncol=301, nobs=20000, seed=K)
    w["tvals"] = []
    F = sp.random(ROWS, NFEAT, density=0.007, random_state=rng, format="coo")
    w["side"] = (F.row.astype(np.int32), F.col.astype(np.int32),
                 None if binary else rng.normal(size=F.nnz), F.shape)
    return w


def pair(K, binary, compute=_lib.MG_COMPUTE_FP64):
    w = workload(K, binary)
    s = gpu_sampler(w, K, 1.5, 21, compute=compute, lambda_beta=LAMBDA_BETA, tol=1e-12)
    return s, oracle_model(w, K, 1.5, 21, lambda_beta=LAMBDA_BETA, tol=1e-12)


def carry(s, m):
    """The GPU's state into the oracle, lambda_beta put back to its start on both sides."""
    s.set_hyper(0, lambda_beta=LAMBDA_BETA)
    m.set("lambda_beta", 0, [LAMBDA_BETA])
    m.set("beta", 0, s.beta(0))
    m.set("uhat", 0, s.uhat(0))
    for mode in (0, 1):
        mu, Lam, _ = s.hyper(mode)
        m.set("mu", mode, mu)
        m.set("Lambda", mode, Lam)
        m.set("latents", mode, s.latents(mode))


@pytest.mark.parametrize("K", [7, 9, 16, 17, 31, 33, 64])
@pytest.mark.parametrize("binary", [True, False])
def test_fp64_chain_matches_oracle(K, binary, oracle_parts):
    s, m = pair(K, binary)
    oracle_parts(gpu_cg_parts(NFEAT))
    for it in range(2):
        for mode in (0, 1):
            s.sample_latents(mode, it)
            m.sample_mode(mode, it)
            assert relerr(s.latents(mode), m.latents(mode)) < FP64_TOL, (it, mode)
            m.set("latents", mode, s.latents(mode))
        for mode in (0, 1):
            s.update_prior(mode, it)
            assert m.update_prior(mode, it) == 0
            mu, Lam, lb = s.hyper(mode)
            assert relerr(mu, m.mu(mode)) < FP64_TOL, (it, mode)
            assert relerr(Lam, m.Lambda(mode)) < FP64_TOL, (it, mode)
        assert relerr(s.beta(0), m.beta(0)) < FP64_TOL, it
        assert relerr(s.uhat(0), m.uhat(0)) < FP64_TOL, it
        lb = s.hyper(0)[2]
        assert abs(lb - m.lambda_beta(0)[0]) / lb < FP64_TOL
        assert np.abs(s.uhat(0)).max() > 0.0
        carry(s, m)
    s.close()


@pytest.mark.parametrize("K", [16, 33, 64])
def test_mixed_rows_with_uhat_match_oracle(K):
    s, m = pair(K, False, _lib.MG_COMPUTE_MIXED)
    for mode in (0, 1):
        s.sample_latents(mode, 0)
    for mode in (0, 1):
        s.update_prior(mode, 0)
    carry(s, m)
    assert np.abs(s.uhat(0)).max() > 0.0
    s.sample_latents(0, 1)
    m.sample_mode(0, 1)
    assert relerr(s.latents(0), m.latents(0)) < MIXED_SAMPLE_TOL
    s.close()
