"""Diagonal layers by tiles of the index space, at the edges of the split into
low and high bits, against the oracle."""
import numpy as np
import pytest

from oracle import OracleSim
from tests.helpers import oracle_apply_terms, rand_state

pytestmark = pytest.mark.gpu

TOL = {np.complex64: 1e-5, np.complex128: 1e-12}


def _terms(n, rng, bonds):
    """Every term kind: one per qubit and one per bond, and a global phase."""
    out = [(5, 0, -1, [0.7])]
    for q in range(n):
        t = float(rng.uniform(-3, 3))
        out.append([(2, q, -1, [t]), (3, q, -1, [t]), (6, q, -1, [np.cos(t), np.sin(t), np.sin(t), -np.cos(t)])][q % 3])
    for i, (a, b) in enumerate(bonds):
        t = float(rng.uniform(-3, 3))
        d = np.exp(1j * rng.uniform(-3, 3, 4))
        out.append([(0, a, b, [t]), (1, a, b, [t]), (4, a, b, [t]), (7, a, b, list(d.view(np.float64)))][i % 4])
    return out


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [10, 11, 12, 13, 14, 19, 21])
def test_all_pairs_of_a_register(n, dtype):
    """Low pairs, mixed pairs and high pairs, in both wire orders; states below
    one tile, of one tile and of many."""
    from mettleq_b200.engine import StateVector
    rng = np.random.default_rng(n)
    bonds = [(a, b) if (a + b) % 3 else (b, a) for a in range(n) for b in range(a + 1, n)]
    if n > 14:
        bonds = [bonds[i] for i in sorted(rng.permutation(len(bonds))[:3 * n])]
    terms = _terms(n, rng, bonds)
    vec = rand_state(n, n, dtype)
    sv = StateVector(n, dtype=dtype)
    sv.set(vec)
    sv.apply_diag_terms(terms)
    o = OracleSim(n, np.complex128)
    o.set_state(vec.astype(np.complex128))
    oracle_apply_terms(o, terms)
    assert np.max(np.abs(sv.get() - o.state)) <= TOL[dtype]
    sv.close()


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_tables_without_unit_modulus_keep_the_window_path(dtype):
    """A projector's zeros and a scaling factor cannot be factored by division."""
    from mettleq_b200.engine import StateVector
    n = 13
    vec = rand_state(n, 2, dtype)
    sv = StateVector(n, dtype=dtype)
    sv.set(vec)
    sv.apply_diag_terms([(7, 0, n - 1, [1, 0, 0, 0, 0, 0, 1, 0]), (0, 2, 9, [0.4])])
    sv.scale(0.5 - 2j)
    o = OracleSim(n, np.complex128)
    o.set_state(vec.astype(np.complex128))
    oracle_apply_terms(o, [(7, 0, n - 1, [1, 0, 0, 0, 0, 0, 1, 0]), (0, 2, 9, [0.4])])
    assert np.max(np.abs(sv.get() - o.state * (0.5 - 2j))) <= TOL[dtype]
    sv.close()
