"""A call that is refused for want of device memory leaves the next ones alone."""
import numpy as np
import pytest

from tests.helpers import rand_state

pytestmark = pytest.mark.gpu


def test_the_call_after_a_refused_one():
    import torch
    from mettleq_b200 import StatevectorMemoryError
    from mettleq_b200.engine import StateVector
    n = 24
    vec = rand_state(n, 1, np.complex64)
    sv = StateVector(n)
    sv.set(vec)
    sv.apply_single(np.eye(2), 0)
    rows = [1 << q for q in range(n)]  # reverses the qubits: needs the second buffer, 128 MB
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(StatevectorMemoryError):
        sv.apply_xor_affine(rows, 0)
    sv.apply_single(np.array([[0, 1], [1, 0]]), 0)  # in place: needs no memory
    del fill
    torch.cuda.empty_cache()
    half = 1 << (n - 1)
    assert np.array_equal(sv.get(), np.concatenate([vec[half:], vec[:half]]))
    sv.apply_xor_affine(rows, 0)
    assert np.array_equal(sv.get()[:2], [vec[half], vec[0]])
    sv.close()
