"""Packing of diagonal terms and matrices for the C ABI (CPU only)."""
import numpy as np
import pytest

from mettleq_b200.engine import _mats_array, _pack_terms


def _plain(terms):
    """The same arrays, entry by entry."""
    k = len(terms)
    kinds, wires, params = np.empty(k, np.int32), np.empty(2 * k, np.int32), np.zeros((k, 8))
    for i, (kind, a, b, p) in enumerate(terms):
        kinds[i], wires[2 * i], wires[2 * i + 1] = int(kind), int(a), int(b)
        pp = list(p)
        params[i, :len(pp)] = pp
    return kinds, wires, params


@pytest.mark.parametrize("make", [
    lambda: [(0, 0, 1, [0.3]), (0, 1, 2, (0.4,))],
    lambda: [(0, 0, 1, [0.3]), (6, 1, -1, [1, 0, 0, 1]), (5, 0, 0, [0.5])],
    lambda: [(0, 0, 1, iter([0.3])), (0, 1, 2, {0.4}), (0, 2, 3, {0.5: None})],
    lambda: [(0.0, 1.0, np.int64(2), np.array([0.3]))],
    lambda: [("0", "1", "2", [0.3])],
    lambda: [(0, np.array(1), 2, np.float32([0.25]))],
    lambda: [(0, 0, 1, [])],
])
def test_terms_are_accepted_as_written(make):
    for got, ref in zip(_pack_terms(make()), _plain(make())):
        assert got.dtype == ref.dtype and np.array_equal(got, ref)


_MANY = [(0, q, q + 1, [0.1 * q]) for q in range(9)]


@pytest.mark.parametrize("extra", [[], [(0, 0, 1, iter([0.3]))], [("1", 2.0, np.int64(3), (0.5,))], [(6, 0, -1, [1, 0, 0, 1])],
                                   [(0, 1, 2, {0.4})]])
def test_longer_lists_of_terms(extra):
    """The same by columns; an iterator among the parameters is read once."""
    ref = _plain(_MANY + [(k, a, b, [0.3]) if hasattr(p, "__next__") else (k, a, b, p) for k, a, b, p in extra])
    for got, want in zip(_pack_terms(_MANY + extra), ref):
        assert got.dtype == want.dtype and np.array_equal(got, want)


@pytest.mark.parametrize("bad", [(0, 1, 2, [0.4], 9), (0, 1, 2), (0, None, 1, [0.1]), (0, [1], 1, [0.1]), (0, 1, 2, 0.3),
                                 (0, float("nan"), 1, [0.1])])
def test_longer_lists_with_a_malformed_term(bad):
    with pytest.raises((TypeError, ValueError)):
        _pack_terms(_MANY + [bad])


@pytest.mark.parametrize("make", [
    lambda: [(0, 0, 1, [0.3]), (0, 1, 2, [0.4], 9)],
    lambda: [(0, 0, 1, [0.3]), (0, 1, 2)],
    lambda: [(0, 0, 1, 0.3)],
    lambda: [(0, 0, 1, [0.1] * 9)],
    lambda: [(0, None, 1, [0.1])],
    lambda: [(0, float("nan"), 1, [0.1])],
    lambda: [(0, float("inf"), 1, [0.1])],
    lambda: [(0, 1e12, 1, [0.1])],
    lambda: [(0, [1], 1, [0.1])],
    lambda: [(0, 1, 2, ["x"])],
])
def test_malformed_terms_are_refused(make):
    with pytest.raises(Exception) as ref:
        _plain(make())
    with pytest.raises(ref.type):
        _pack_terms(make())


def test_matrices_of_any_layout():
    rng = np.random.default_rng(0)
    m = rng.standard_normal((4, 3)) + 1j * rng.standard_normal((4, 3))
    for x in (m.T, m.T.astype(np.complex64), np.asfortranarray(m.T), m.T.tolist(), m.T[::-1], m.real.T):
        out = _mats_array(3, x)
        ref = np.asarray(x, dtype=np.complex128).reshape(3, 4)
        assert out.dtype == np.float64 and out.flags.c_contiguous and out.shape == (3, 8)
        assert np.array_equal(out[:, 0::2], ref.real) and np.array_equal(out[:, 1::2], ref.imag)
