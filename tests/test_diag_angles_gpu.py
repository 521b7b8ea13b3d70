"""Diagonals as sums of angles: accuracy, exact signs, and the diagonals that
are one small table."""
import math

import numpy as np
import pytest

from oracle import OracleSim
from tests.helpers import oracle_apply_terms, rand_state

pytestmark = pytest.mark.gpu


def _apply(n, dtype, vec, terms):
    from mettleq_b200.engine import StateVector
    sv = StateVector(n, dtype=dtype)
    sv.set(vec)
    sv.apply_diag_terms(terms)
    out = sv.get()
    sv.close()
    return out


@pytest.mark.parametrize("dtype,tol", [(np.complex64, 5.5e-8), (np.complex128, 3e-16)])
@pytest.mark.parametrize("n", [12, 16, 18])
def test_error_of_a_chain_with_far_bonds(n, dtype, tol):
    """Against 80-bit arithmetic, relative to the norm.  complex64: one rounded
    factor (each part to an ulp) and one product, 4.5e-8 in the mean square;
    complex128: three of each, 2e-16.  Twice as many of each, as products of the
    terms' factors have, would exceed the bounds."""
    rng = np.random.default_rng(n)
    bonds = [(i, i + 1) for i in range(n - 1)] + [(i, n - 1 - i) for i in range(4)]
    terms = [(0, a, b, [float(rng.uniform(0, 3))]) for a, b in bonds]
    terms += [(6, q, -1, [math.cos(t), -math.sin(t), math.cos(t), math.sin(t)]) for q, t in enumerate(rng.uniform(-3, 3, n))]
    terms += [(1, 0, n - 1, [1e6]), (4, 1, n - 2, [-700.0]), (2, 3, -1, [7.5]), (3, 4, -1, [-8.5]), (5, 0, -1, [0.3])]
    vec = rand_state(n, n, dtype)
    got = _apply(n, dtype, vec, terms).astype(np.clongdouble)
    ref = vec.astype(np.clongdouble)
    i = np.arange(1 << n)
    for kind, a, b, p in terms:
        x = (i >> (n - 1 - a)) & 1
        y = (i >> (n - 1 - b)) & 1 if b >= 0 else 0
        t = np.longdouble(p[0])
        if kind == 6:
            ref = ref * np.where(x, np.clongdouble(complex(p[2], p[3])), np.clongdouble(complex(p[0], p[1])))
            continue
        ang = {0: -t * (1 - 2 * (x ^ y)), 1: t * (x & y), 2: t / 2 * (2 * x - 1), 3: t * x, 4: t / 2 * x * (2 * y - 1),
               5: t * np.ones_like(x)}[kind]
        ref = ref * (np.cos(ang) + 1j * np.sin(ang))
    err = np.sqrt(np.sum(np.abs(got - ref) ** 2) / np.sum(np.abs(ref) ** 2))
    assert err < tol


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_quarter_turns_are_exact(dtype):
    """CZ, Z and S on many wires only swap and negate parts."""
    n = 14
    terms = [(1, i, (i + 3) % n, [math.pi]) for i in range(n)] + [(3, q, -1, [math.pi]) for q in range(0, n, 3)]
    terms += [(6, q, -1, [1, 0, 0, 1]) for q in range(1, n, 4)]
    vec = rand_state(n, 3, dtype)
    got = _apply(n, dtype, vec, terms)
    i = np.arange(1 << n)
    quarter = np.zeros(1 << n, dtype=int)
    for kind, a, b, _ in terms:
        x = (i >> (n - 1 - a)) & 1
        quarter += {1: 2 * x * ((i >> (n - 1 - b)) & 1), 3: 2 * x, 6: x}[kind]
    ref = np.choose(quarter % 4, [vec, -vec.imag + 1j * vec.real, -vec, vec.imag - 1j * vec.real]).astype(dtype)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [11, 12, 13, 17, 22, 23, 24])
def test_small_tables_and_tiles_agree_with_the_oracle(n, dtype):
    """On both sides of the rule for one small table: spans of six and seven
    bits, up to four and five scattered bits, a global phase alone."""
    rng = np.random.default_rng(n)
    t = lambda: [float(rng.uniform(-3, 3))]
    sets = [[(2, n // 2, -1, t())], [(0, q, q + 1, t()) for q in range(2, 7)], [(0, q, q + 1, t()) for q in range(2, 8)],
            [(5, 0, -1, t())]]
    if n >= 14:
        sets += [[(0, 0, n - 1, t()), (1, 1, n - 1, t()), (4, n - 2, 0, t())], [(0, 0, n - 1, t()), (0, 1, n - 2, t()), (0, 2, n - 1, t())]]
    if n > 17:
        sets = [sets[i] for i in (1, 4)]
    vec = rand_state(n, n, dtype)
    for terms in sets:
        o = OracleSim(n, np.complex128)
        o.set_state(vec.astype(np.complex128))
        oracle_apply_terms(o, terms)
        assert np.max(np.abs(_apply(n, dtype, vec, terms) - o.state)) <= (1e-6 if dtype == np.complex64 else 1e-14)
