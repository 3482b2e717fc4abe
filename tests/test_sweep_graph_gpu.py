"""When a sampler's sweeps are captured as a CUDA graph: with the second sweep, not for a single one."""
import numpy as np
import pytest

from macau_b200 import _lib
from tests.gpu_helpers import gpu_sampler
from tests.test_gpu_parity import small_uniform

pytestmark = pytest.mark.gpu


def state(s):
    return [s.latents(m) for m in (0, 1)] + [x for m in (0, 1) for x in s.hyper(m)[:2]]


@pytest.mark.parametrize("compute", [_lib.MG_COMPUTE_FP64, _lib.MG_COMPUTE_MIXED])
def test_graph_is_built_for_a_second_sweep(compute):
    w = small_uniform(seed=4, nrow=300)
    chains = [gpu_sampler(w, 10, 2.0, 3, compute=compute) for _ in range(4)]
    single, together, timed, eager = chains
    eager.set_option("graph", 0)
    captured = []
    for it in range(4):
        single.sweep(it, eval=False)
        captured.append(single.stats()["graph_captured"])
    assert captured == [False, True, True, True]
    together.sweeps(0, 4, eval=False)
    assert together.stats()["graph_captured"]
    assert timed.time_sweeps(0, 4)[0] > 0.0
    assert timed.stats()["graph_captured"]
    eager.sweeps(0, 4, eval=False)
    assert not eager.stats()["graph_captured"]
    want = state(single)
    for s in chains:
        assert s.stats()["sweeps"] == 4
        for a, b in zip(state(s), want):
            assert np.array_equal(a, b)
        s.close()
