"""The two ways a batch runs its larger circuits (in groups of one width, or
one by one with a tile plan) against each other and against 64 bits, and a
tile plan that cannot be had."""
import numpy as np
import pytest

from mettleq_b200 import _native as N
from tests.helpers import device_memory_left, haar_u2

pytestmark = pytest.mark.gpu


def _mats(d, n, seed):
    rng = np.random.default_rng([seed, d, n])
    return np.array([[haar_u2(rng).reshape(4) for _ in range(n)] for _ in range(d)])


def _run(ns, ds, ladder, **kw):
    from mettleq_b200.batch import CircuitBatch
    b = CircuitBatch(ns, ds, ladder=ladder, **kw)
    try:
        b.run([_mats(d, n, i) for i, (d, n) in enumerate(zip(ds, ns))])
        return [b.probabilities(c) for c in range(len(ns))], b.z0()
    finally:
        b.close()


@pytest.mark.parametrize("ladder", [True, False])
@pytest.mark.parametrize("n", range(14, 24))
def test_groups_give_the_bits_of_single_circuits(n, ladder):
    """The gates of an amplitude have one order and rounding on both routes;
    (12, 4, 0) is the default plan, spelled out."""
    ds = [3, 1, 2] if n < 20 else [3, 1]
    groups, z = _run([n] * len(ds), ds, ladder, lanes=2)
    single, z1 = _run([n] * len(ds), ds, ladder, lanes=2, tiles=(12, 4, 0))
    for p, q in zip(groups, single):
        assert np.array_equal(p, q)
    assert np.max(np.abs(z - z1)) < 1e-12  # the same float64 terms, added in another order


@pytest.mark.parametrize("ladder", [True, False])
def test_widest_groups_and_single_circuits_in_one_batch(ladder):
    """22 and 23 qubits in groups (three sweeps a layer), 24 one by one.  Two
    layers are 48 unitary gates, each with the rounding of its entries and of
    four operations on an amplitude: below 8 x 2^-24 of the state's norm a
    gate, 2.3e-5 in all, and the probabilities are off by twice that in sum."""
    import torch
    ns, ds = [22, 23, 24], [2, 2, 2]
    probs, z0 = _run(ns, ds, ladder, lanes=2)
    for c, n in enumerate(ns):
        x = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        x[0] = 1
        i = torch.arange(1 << n, device="cuda")
        for layer in _mats(ds[c], n, c):
            for q in range(n):
                u = torch.tensor(layer[q].reshape(2, 2), device="cuda")
                x = torch.einsum("ab,xby->xay", u, x.view(1 << q, 2, -1)).reshape(-1)
            if ladder:
                x = x[i ^ (i >> 1)]
        ref = x.abs().square()
        assert float((torch.as_tensor(probs[c], device="cuda").double() - ref).abs().sum()) < 5e-5
        half = 1 << (n - 1)
        assert abs(z0[c] - float(ref[:half].sum() - ref[half:].sum())) < 5e-5


def test_a_plan_without_memory_leaves_the_old_one():
    """Nine circuits of 21 to 23 qubits on three lanes: single circuits need
    two states per width and lane, 672 MB, the groups' buffers 384 MB.  With
    about 100 MB free the plan is refused; the batch then runs as if it had
    never been asked for, and takes the plan once there is room."""
    from mettleq_b200.batch import CircuitBatch
    ns, ds = [21, 22, 23] * 3, [2] * 9
    mats = [_mats(2, n, c) for c, n in enumerate(ns)]
    ref, zref = _run(ns, ds, True, lanes=3)
    for first in (False, True):
        b = CircuitBatch(ns, ds, lanes=3)
        try:
            if first:
                assert b._lib.mq_batch_set_tiles(b._h, 11, 4, 0) == N.MQ_OK
                assert b._lib.mq_batch_set_tiles(b._h, 0, -1, 0) == N.MQ_OK
            with device_memory_left(100 << 20):
                assert b._lib.mq_batch_set_tiles(b._h, 11, 4, 0) == N.MQ_ENOMEM
                assert "memory" in N.last_error()
                b.run(mats)  # the old plan is whole before the memory is back
                z0 = b.z0()
            assert np.array_equal(z0, zref)
            for c in range(len(ns)):
                assert np.array_equal(b.probabilities(c), ref[c])
        finally:
            b.close()
    b = CircuitBatch(ns, ds, lanes=3)
    try:
        assert b._lib.mq_batch_set_tiles(b._h, 12, 4, 0) == N.MQ_OK
        b.run(mats)
        for c in range(len(ns)):
            assert np.array_equal(b.probabilities(c), ref[c])
    finally:
        b.close()
