"""A call that is refused for want of device memory leaves the next ones alone."""
import numpy as np
import pytest

from tests.helpers import device_memory_left

pytestmark = pytest.mark.gpu


def test_the_call_after_a_refused_one():
    from mettleq_b200 import StatevectorMemoryError
    from mettleq_b200.engine import StateVector
    n = 28
    x = np.array([[0, 1], [1, 0]])
    sv = StateVector(n)
    sv.reset()
    sv.apply_single(x, 1)
    rows = [1 << q for q in range(n)]  # reverses the qubits: needs the second buffer, 2 GB
    with device_memory_left(64 << 20):
        with pytest.raises(StatevectorMemoryError):
            sv.apply_xor_affine(rows, 0)
        sv.apply_single(x, 0)  # in place: needs no memory
        sv.synchronize()
    assert sv.probabilities([0, 1, 2, n - 1]).tolist() == [float(i == 0b1100) for i in range(16)]
    sv.apply_xor_affine(rows, 0)
    assert sv.probabilities([0, n - 3, n - 2, n - 1]).tolist() == [float(i == 0b0011) for i in range(16)]
    sv.close()
