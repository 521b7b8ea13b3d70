"""Lists of controlled gates that share wires: many gates in one sweep, in
order, against the oracle."""
import numpy as np
import pytest

from oracle import OracleSim
from tests.helpers import haar_u2, rand_state

pytestmark = pytest.mark.gpu

TOL = {np.complex64: 1e-5, np.complex128: 1e-12}


def _check(n, gates, dtype):
    from mettleq_b200.engine import StateVector
    vec = rand_state(n, len(gates), dtype)
    sv = StateVector(n, dtype=dtype)
    sv.set(vec)
    sv.apply_controlled(gates)
    o = OracleSim(n, np.complex128)
    o.set_state(vec.astype(np.complex128))
    for c, t, u in gates:
        o.apply_multi_controlled_single(u, c, t)
    assert np.max(np.abs(sv.get() - o.state)) <= TOL[dtype]
    sv.close()


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 11, 12, 13, 17, 20])
def test_chains_in_both_directions(n, dtype):
    rng = np.random.default_rng(n)
    for step in (1, -1):
        wires = list(range(n))[::step]
        _check(n, [([a], b, haar_u2(rng)) for a, b in zip(wires, wires[1:])], dtype)


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [2, 3, 5, 9, 12, 14, 18, 21])
def test_random_lists(n, dtype):
    """Repeated targets, targets that are controls of their neighbours, up to
    three controls, more targets than a tile holds and more gates than a sweep."""
    rng = np.random.default_rng(50 + n)
    gates = []
    for _ in range(45):
        k = int(rng.integers(1, min(n, 4) + 1)) if n > 1 else 1
        w = [int(x) for x in rng.permutation(n)[:max(2, k)]]
        if gates and rng.random() < 0.3:
            w = [x for x in w if x != gates[-1][1]] + [gates[-1][1]]
        gates.append((w[:-1], w[-1], haar_u2(rng)))
    _check(n, gates, dtype)
