"""Shots at the counts where the draw kernel or the way back changes, bit for
bit against the oracle."""
import numpy as np
import pytest

from oracle import sampler as osamp
from tests.helpers import rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n,shots", [(1, 24576), (3, 8193), (4, 30000), (10, 24575), (10, 24576), (11, 8192), (16, 40000),
                                     (21, 24577)])
def test_many_shots_match_the_oracle(n, shots, dtype):
    from mettleq_b200.engine import StateVector
    vec = rand_state(n, 5 * n, dtype)
    rng = np.random.default_rng(n)
    if n > 2:
        vec[rng.random(1 << n) < 0.3] = 0
        vec[-(1 << n) // 5:] = 0
    sv = StateVector(n, dtype=dtype)
    sv.set(vec)
    p = osamp.amp2(vec)
    ref = osamp.sample_indices(p, 17, shots, stream_offset=3)
    assert np.array_equal(sv.sample_indices(shots, seed=17, stream_offset=3), ref)
    if n > 3:
        wires = [n - 1, 0, 2]
        m = osamp.marginal_probabilities(p, n, wires)
        assert np.array_equal(sv.sample_indices(shots, wires, seed=5), osamp.sample_indices(m, 5, shots))
    # the counts on both sides of each change draw the same shots
    few = sv.sample_indices(1000, seed=17, stream_offset=3)
    assert np.array_equal(few, ref[:1000])
    sv.close()


def test_many_shots_of_a_zero_state_are_refused():
    from mettleq_b200.engine import StateVector
    sv = StateVector(8)
    sv.set(np.zeros(256, dtype=np.complex64))
    for shots in (9000, 50000):
        with pytest.raises(ValueError):
            sv.sample_indices(shots, seed=1)
    sv.close()
