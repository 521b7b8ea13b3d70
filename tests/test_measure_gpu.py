"""Measurement kernels at the edges of their work split, against the oracle
(bit for bit: sums, offsets and shots are defined to the last rounding)."""
import numpy as np
import pytest

from oracle import OracleSim
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


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n,wires", [
    (1, []), (3, []), (3, [2]), (4, [3, 0]), (5, [4, 3, 2, 1]), (6, [5]), (7, [6, 5, 4, 3, 2]), (9, [8, 0, 7]),
    (10, list(range(1, 10))), (11, list(range(11))[::-1]), (12, [11, 10, 9, 8]), (12, [8, 9]), (13, [12, 3, 10]),
    (13, list(range(12))), (15, [14, 11, 12, 13, 0, 7]), (17, [3]), (20, [19, 17, 2, 9]), (21, [20]), (22, [])])
def test_marginals_over_chunk_and_sibling_edges(n, wires, dtype):
    """Chunks of 1 to 1024 entries (below and above a warp), 0 to 4 selected
    qubits on the low index bits, one level of sums to three."""
    vec = rand_state(n, 3 * n + len(wires), dtype)
    sv = _sv(n, dtype, vec)
    ref = osamp.marginal_probabilities(osamp.amp2(vec), n, wires)
    assert np.array_equal(sv.probabilities(wires), ref)
    assert np.array_equal(sv.probabilities(wires, dtype=np.float32), ref.astype(np.float32))
    if wires:
        assert np.array_equal(sv.sample_indices(50, wires, seed=4), osamp.sample_indices(ref, 4, 50))
    sv.close()


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [1, 2, 5, 11, 12, 13, 14, 18, 19, 20, 21])
def test_pauli_words_over_every_kernel_of_the_split(n, dtype):
    """Words without X and Y, words within four neighbouring index bits (in
    every window, with Z letters inside and outside it), and words spread over
    the register, more of one kind than a launch holds.  Both sides sum the
    exact float64 products of the same amplitudes: 1e-12 covers the rounding
    of 2^21 additions of a unit vector's terms."""
    vec = rand_state(n, 7 * n, dtype)
    rng = np.random.default_rng(n)
    words = [{}] + [{q: p} for q in range(n) for p in "XYZ"] + [{q: a, q + 1: b} for q in range(n - 1)
                                                               for a, b in ("XX", "YY", "ZZ", "XY")]
    for _ in range(12):
        lo = int(rng.integers(0, max(1, n - 3)))
        words.append({q: "XYZ"[int(rng.integers(3))] for q in range(lo, min(n, lo + 4))})
        words.append({int(q): "XYZ"[int(rng.integers(3))] for q in rng.permutation(n)[:int(rng.integers(1, min(n, 7) + 1))]})
    if n > 14:
        words = [words[i] for i in sorted(rng.permutation(len(words))[:60])]
    sv = _sv(n, dtype, vec)
    got = sv.expval_pauli(words)
    o = OracleSim(n, np.complex128)
    o.set_state(vec.astype(np.complex128))
    ref = np.array([o.pauli_expectation(w) for w in words])
    assert np.max(np.abs(got - ref)) < 1e-12
    assert np.array_equal(sv.expval_pauli(words), got)
    one = int(rng.integers(len(words)))
    assert sv.expval_pauli([words[one]])[0] == got[one]  # a word's bits do not depend on the others
    twice = [w for w in words for _ in range(2)]
    assert np.array_equal(sv.expval_pauli(twice), np.repeat(got, 2))
    sv.close()
