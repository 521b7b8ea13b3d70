"""Marginals of many short buckets: 1 to 32 chunks a bucket, on both sides of
the rule between a thread and a warp per run, bit for bit."""
import numpy as np
import pytest

from oracle import sampler as osamp
from tests.helpers import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("k", [3, 4, 5, 6, 7, 8])
def test_runs_of_a_bucket(k, dtype):
    from mettleq_b200.engine import StateVector
    n = 18
    vec = rand_state(n, k, dtype)
    sv = StateVector(n, dtype=dtype)
    sv.set(vec)
    rng = np.random.default_rng(k)
    p = osamp.amp2(vec)
    for wires in ([int(q) for q in rng.permutation(n)[:k]], list(range(n - k, n)), list(range(k))):
        ref = osamp.marginal_probabilities(p, n, wires)
        assert np.array_equal(sv.probabilities(wires), ref)
        assert np.array_equal(sv.sample_indices(40, wires, seed=2), osamp.sample_indices(ref, 2, 40))
    sv.close()
