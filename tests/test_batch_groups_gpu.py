"""Groups of larger circuits in a batch: matrices of every form (rotations,
general unitaries, zeros on the diagonal or beside it, not unitary), uneven
depths, widths from one high target bit to more than one high sweep."""
import math

import numpy as np
import pytest

from oracle import OracleSim
from tests.helpers import haar_u2

pytestmark = pytest.mark.gpu


def _mats(kind, d, n, rng):
    m = np.empty((d, n, 4), dtype=np.complex128)
    for l in range(d):
        for q in range(n):
            if kind == "haar":
                u = haar_u2(rng)
            elif kind == "fixed":  # H, X, S, identity, Y-like with a phase
                u = [np.array([[1, 1], [1, -1]]) / math.sqrt(2), np.array([[0, 1], [1, 0]]), np.diag([1, 1j]), np.eye(2),
                     np.exp(0.3j) * np.array([[0, -1j], [1j, 0]])][(l + q) % 5]
            else:  # not unitary
                u = np.eye(2) + 0.2 * (rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))
            m[l, q] = np.asarray(u, dtype=np.complex128).reshape(4)
    return m


def _oracle(n, mats, ladder):
    o = OracleSim(n, np.complex128)
    for layer in mats:
        for q in range(n):
            o.apply_single(layer[q].reshape(2, 2), q)
        if ladder:
            for q in range(n - 1):
                o.apply_controlled_single(np.array([[0, 1], [1, 0]]), q, q + 1)
    return np.abs(o.state) ** 2


@pytest.mark.parametrize("lanes", [1, 3])
def test_groups_match_oracle(lanes):
    """Probabilities to 2e-6 of a unit total (scaled by the total where the
    matrices are not unitary), <Z_0> to 1e-5 of it, also after a second run with
    other matrices through the same graph."""
    from mettleq_b200.batch import CircuitBatch
    ns = [14, 14, 14, 14, 15, 15, 16, 17, 18, 19, 20, 21, 14, 16, 13]
    ds = [0, 1, 4, 2, 3, 3, 2, 3, 2, 2, 2, 2, 3, 2, 2]
    kinds = ["haar", "fixed", "haar", "fixed", "other", "haar", "haar", "fixed", "haar", "other", "haar", "haar", "haar",
             "fixed", "haar"]
    ladder = [True] * 12 + [False] * 3
    b = CircuitBatch(ns, ds, ladder=ladder, lanes=lanes)
    try:
        for it in range(2):
            rng = np.random.default_rng(it)
            kinds = kinds if it == 0 else kinds[::-1]
            mats = [_mats(k, d, n, rng) for k, d, n in zip(kinds, ds, ns)]
            b.run(mats)
            z0 = b.z0()
            for c, n in enumerate(ns):
                ref = _oracle(n, mats[c], ladder[c])
                total = ref.sum()
                assert np.max(np.abs(b.probabilities(c) - ref)) < 2e-6 * total, (it, c, n, kinds[c])
                half = len(ref) // 2
                assert abs(z0[c] - (ref[:half].sum() - ref[half:].sum())) < 1e-5 * total, (it, c, n, kinds[c])
    finally:
        b.close()


@pytest.mark.parametrize("n,count", [(14, 160), (16, 40)])
def test_blocks_go_from_one_circuit_to_the_next(n, count):
    """More tiles than resident blocks: a block's next tile belongs to another
    circuit, whose matrices (and depth) differ."""
    from mettleq_b200.batch import CircuitBatch
    rng = np.random.default_rng(n)
    ds = [2 + c % 3 for c in range(count)]
    b = CircuitBatch([n] * count, ds, lanes=2)
    try:
        mats = [_mats("haar", d, n, rng) for d in ds]
        b.run(mats)
        for c in range(count):
            p = _oracle(n, mats[c], True)
            assert np.max(np.abs(b.probabilities(c) - p)) < 2e-6
            z = p[: 1 << (n - 1)].sum() - p[1 << (n - 1):].sum()
            assert abs(b.z0()[c] - z) < 1e-5
    finally:
        b.close()
