"""mq_fuse_stream against the Python rules of fusion.py (CPU only)."""
import math

import numpy as np
import pytest

from mettleq_b200 import fusion as F
from mettleq_b200 import workloads as W


def _stream(n, count, rng):
    ops = []
    while len(ops) < count:
        u = rng.random()
        if u < 0.06 and n > 2:  # a QFT ladder or part of one, forward or inverse
            lo = int(rng.integers(0, n - 1))
            hi = int(rng.integers(lo + 2, n + 1))
            q = W.qft_ops(n, list(range(lo, hi)))
            if rng.random() < 0.5:
                q = [dict(o, parameters=[-p for p in o["parameters"]]) for o in reversed(q)]
            ops += q[: int(rng.integers(1, len(q) + 1))]
            continue
        name = F.GATE_NAMES[int(rng.integers(len(F.GATE_NAMES)))]
        k = F.ARITIES[name]
        if k > n:
            continue
        p = [float(x) for x in rng.uniform(-3, 3, F.PARAMS.get(name, 0))]
        if p and rng.random() < 0.2:
            p = [float(rng.choice([0.0, math.pi, -math.pi, math.pi / 2]))] * len(p)
        run = int(rng.integers(1, 6))
        ops += [{"name": name, "wires": [int(w) for w in rng.permutation(n)[:k]], "parameters": p} for _ in range(run)]
    return ops


def _same(a, b):
    assert a["name"] == b["name"]
    assert set(a) == set(b)
    for key in a:
        x, y = a[key], b[key]
        if key == "mats" and x is not None:
            assert np.max(np.abs(x - y)) < 1e-14
        elif key == "terms":
            assert [(t[0], t[1], t[2]) for t in x] == [(t[0], t[1], t[2]) for t in y]
            for s, t in zip(x, y):
                assert len(s[3]) == len(t[3]) and np.max(np.abs(np.subtract(s[3], t[3]))) < 1e-14
        elif key == "gates":
            assert [(list(c), t) for c, t, _ in x] == [(list(c), t) for c, t, _ in y]
            assert all(np.max(np.abs(u - v)) < 1e-15 for (_, _, u), (_, _, v) in zip(x, y))
        elif key in ("active", "rows"):
            assert (x is None and y is None) or list(x) == list(y)
        elif key == "bonds":
            assert [tuple(e) for e in x] == [tuple(e) for e in y]
        else:
            assert x == y, key


@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 20, 31])
def test_random_streams_give_the_layers_of_the_python_rules(n):
    for seed in range(40):
        rng = np.random.default_rng(1000 * n + seed)
        ops = _stream(n, int(rng.integers(1, 120)), rng)
        assert F._native_segments(ops, n) is not None
        got, ref = F.fuse(ops, n), F._fuse_python(ops, n, True)
        assert [L["name"] for L in got] == [L["name"] for L in ref]
        for a, b in zip(got, ref):
            _same(a, b)


@pytest.mark.parametrize("ops", [
    [{"name": "rx", "wires": [0], "parameters": [0.3]}],
    [{"name": "RX", "wires": ["1"], "parameters": ["0.3"]}],
    [{"name": "_M1", "wires": [0], "matrix": np.eye(2)[::-1]}],
    [{"name": "CX", "wires": (np.int64(0), 1.0), "parameters": None}, {"name": "H", "wires": [1]}],
    [{"name": "RZ", "wires": [2], "parameters": [np.float32(0.25), 7.0]}],
    [], ])
def test_other_spellings_and_values_are_accepted_as_before(ops):
    ref = F._fuse_python(ops, 3, True)
    got = F.fuse(ops, 3)
    assert len(got) == len(ref)
    for a, b in zip(got, ref):
        _same(a, b)


@pytest.mark.parametrize("name", ["H", "h"])
def test_an_iterator_of_gates_is_read_once(name):
    ops = [{"name": name, "wires": [q], "parameters": []} for q in range(3)]
    assert [L["active"] for L in F.fuse(iter(ops), 3)] == [[0, 1, 2]]


@pytest.mark.parametrize("op", [
    {"name": "RX", "wires": [0], "parameters": []}, {"name": "H", "wires": [0, 1]}, {"name": "CNOT", "wires": [1, 1]},
    {"name": "H", "wires": [3]}, {"name": "H", "wires": [-1]}, {"name": "H", "wires": [1 << 40]}, {"name": "FOO", "wires": [0]}])
def test_malformed_gates_are_refused_as_before(op):
    with pytest.raises(ValueError):
        F.fuse([{"name": "H", "wires": [0], "parameters": []}, op], 3)


def _outcome(fn):
    try:
        return fn()
    except Exception as e:
        return type(e)


@pytest.mark.parametrize("value", [None, math.inf, -math.inf, math.nan, np.timedelta64(3, "s"), np.datetime64("2020-01-01"), "x",
                                   1j, [0.5]])
@pytest.mark.parametrize("name", ["RX", "U1", "U3", "CPHASE", "CRX", "XXPHASE", "ZZPHASE", "H"])
def test_parameters_without_a_finite_value_follow_the_python_rules(name, value):
    """An unbound (None) or non-finite parameter is refused, or carried along,
    exactly as the Python rules do it: no gate becomes NaN unnoticed."""
    count = max(1, F.PARAMS.get(name, 0))  # H: a parameter it does not use is still converted
    ops = [{"name": name, "wires": list(range(F.ARITIES[name])), "parameters": [0.25] * (count - 1) + [value]}]
    ref = _outcome(lambda: F._fuse_python(ops, 3, True))
    got = _outcome(lambda: F.fuse(ops, 3))
    if isinstance(ref, type):
        assert got is ref
        return
    assert repr(got) == repr(ref)


def test_angles_whose_sum_is_not_finite_are_refused():
    with pytest.raises(ValueError):
        F.fuse([{"name": "U3", "wires": [0], "parameters": [0.1, 1e308, 1e308]}], 3)


def test_missing_keys_are_not_made_up():
    """A gate without a name is refused even where the mapping has defaults,
    and reading it adds no keys."""
    from collections import defaultdict
    op = defaultdict(lambda: "H", wires=[0])
    with pytest.raises(ValueError):
        F.fuse([op], 3)
    assert set(op) == {"wires"}


def test_a_library_that_does_not_load_leaves_the_python_rules(monkeypatch):
    """Fusion is host code: it works where libmq.so or its CUDA runtime cannot
    be loaded."""
    def broken():
        raise OSError("libcudart.so: cannot open shared object file")
    monkeypatch.setattr(F.N, "lib", broken)
    ops = [{"name": "H", "wires": [0], "parameters": []}]
    assert F.fuse(ops, 2)[0]["active"] == [0]


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan, 1e300])
def test_the_c_entry_refuses_parameters_that_are_not_finite(value):
    import ctypes as C
    from mettleq_b200 import _native as N
    i32 = C.c_int32 * 1
    out, used = (C.c_int32 * 64)(), (C.c_int64 * 2)()
    for code in (F.GATE_NAMES.index("RX"), F.GATE_NAMES.index("H")):  # H: a parameter it does not use
        rc = N.lib().mq_fuse_stream(2, 1, i32(code), i32(1), i32(0), i32(1), (C.c_double * 1)(value), out, 64,
                                    (C.c_double * 64)(), 64, used)
        assert rc == N.MQ_EINVAL
    rc = N.lib().mq_fuse_stream(2, 1, i32(F.GATE_NAMES.index("RX")), i32(1), i32(0), i32(1), None, out, 64,
                                (C.c_double * 64)(), 64, used)
    assert rc == N.MQ_EINVAL


@pytest.mark.parametrize("name", F.GATE_NAMES)
def test_short_streams_on_both_sides_of_the_rule(name):
    """One gate takes the Python rules, two the native ones: the same layers."""
    k = F.ARITIES[name]
    op = {"name": name, "wires": list(range(k)), "parameters": [0.7] * F.PARAMS.get(name, 0)}
    for ops in ([op], [op, op]):
        got, ref = F.fuse(ops, 3), F._fuse_python(ops, 3, True)
        assert [L["name"] for L in got] == [L["name"] for L in ref]
        for a, b in zip(got, ref):
            _same(a, b)
