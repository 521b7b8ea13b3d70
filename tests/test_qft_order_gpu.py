"""A QFT on ordered wires takes, amplitude by amplitude, the factors of the
contiguous transform: moving the wires to the top, transforming there and
moving back gives the same bits."""
import numpy as np
import pytest

from tests.helpers import rand_state

pytestmark = pytest.mark.gpu


def _move(n, wires):
    """Rows of the map that takes wire j of the list to qubit j, the others
    below in their order (row q: the index bits of the result whose parity is
    qubit q of the source)."""
    rest = [q for q in range(n) if q not in wires]
    rows = [0] * n
    for to, q in enumerate(list(wires) + rest):
        rows[q] = 1 << (n - 1 - to)
    return rows


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("n,k", [(6, 3), (9, 2), (13, 7), (16, 9), (16, 12), (19, 10), (20, 15), (21, 16)])
def test_same_bits_as_the_contiguous_transform(n, k, inverse, dtype):
    from mettleq_b200.engine import StateVector
    for trial in range(3):
        wires = [int(q) for q in np.random.default_rng([n, k, trial]).permutation(n)[:k]]
        vec = rand_state(n, n + trial, dtype)
        a, b = StateVector(n, dtype=dtype), StateVector(n, dtype=dtype)
        a.set(vec)
        a.apply_qft(wires, inverse)
        rows = _move(n, wires)
        back = [0] * n
        for q, r in enumerate(rows):
            back[n - r.bit_length()] = 1 << (n - 1 - q)
        b.set(vec)
        b.apply_xor_affine(rows, 0)
        b.apply_qft(list(range(k)), inverse)
        b.apply_xor_affine(back, 0)
        x, y = a.get(), b.get()
        a.close()
        b.close()
        # (a sweep's 2^-1/2 for an odd number of stages is one rounding, which
        # another division of the stages has elsewhere or not at all)
        eps = np.finfo(dtype).eps
        scale = np.abs(y).max()
        assert np.max(np.abs(x - y)) <= 4 * eps * scale
        if k % 2 == 0 and k <= 7:
            assert np.array_equal(x, y)
