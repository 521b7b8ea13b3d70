"""QFT on ordered wires of a register (no permutation passes) against the
oracle: one tile and several, stages that fill their register phases and
remainders, targets among the low passengers and above them."""
import numpy as np
import pytest

from oracle import OracleSim
from tests.helpers import rand_state

pytestmark = pytest.mark.gpu

TOL = {np.complex64: 1e-5, np.complex128: 1e-12}


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("n,k", [(2, 2), (4, 3), (6, 6), (9, 5), (11, 10), (12, 12), (13, 4), (16, 9), (18, 18), (20, 13)])
def test_ordered_wires(n, k, inverse, dtype):
    from mettleq_b200.engine import StateVector
    for trial in range(2):
        rng = np.random.default_rng(100 * n + k + trial)
        wires = [int(w) for w in rng.permutation(n)[:k]]
        if trial:
            wires = sorted(wires, reverse=True)
        vec = rand_state(n, n + k, dtype)
        sv = StateVector(n, dtype=dtype)
        sv.set(vec)
        sv.apply_qft(wires, inverse=inverse)
        o = OracleSim(n, np.complex128)
        o.set_state(vec.astype(np.complex128))
        (o.iqft if inverse else o.qft)(wires)
        assert np.max(np.abs(sv.get() - o.state)) <= TOL[dtype]
        sv.close()
