"""Measurement kernels at the edges of their work split, against the oracle
(bit for bit: sums, offsets and shots are defined to the last rounding)."""
import numpy as np
import pytest

from oracle import sampler as osamp
from tests.helpers import rand_state

pytestmark = pytest.mark.gpu


def _sv(n, dtype, vec):
    from mettleq_b200.engine import StateVector
    sv = StateVector(n, dtype=dtype)
    sv.set(vec)
    return sv


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n,shots", [(1, 1), (2, 5), (3, 33), (5, 100), (10, 257), (11, 1000), (20, 3), (21, 2000)])
def test_shots_over_block_and_superblock_edges(n, shots, dtype):
    """Blocks of fewer than 8 entries up to 1024, one block up to two
    super-blocks; zeros at the end of the state and inside blocks."""
    vec = rand_state(n, 31 + n, dtype)
    rng = np.random.default_rng(n)
    if n > 2:
        vec[rng.random(1 << n) < 0.3] = 0
        vec[-(1 << n) // 5:] = 0
    sv = _sv(n, dtype, vec)
    ref = osamp.sample_indices(osamp.amp2(vec), 91, shots, stream_offset=2)
    assert np.array_equal(sv.sample_indices(shots, seed=91, stream_offset=2), ref)
    sv.close()


def test_zero_state_is_refused():
    sv = _sv(12, np.complex64, np.zeros(1 << 12, dtype=np.complex64))
    for shots in (0, 7):
        with pytest.raises(ValueError):
            sv.sample_indices(shots, seed=1)
    sv.close()
