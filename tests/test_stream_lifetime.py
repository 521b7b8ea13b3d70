"""A state that borrows another's stream is destroyed before it (CPU only, on
a stand-in for the library)."""
import ctypes as C
import gc

import pytest

from mettleq_b200 import adjoint as A
from mettleq_b200 import engine as E


class FakeLib:
    """Handles and streams are numbers; records the order of destruction and
    any use of a stream after its owner's end."""

    def __init__(self):
        self.count, self.stream, self.dead, self.order, self.late = 0, {}, set(), [], []

    def mq_state_create(self, n, dt, device, stream, out):
        self.count += 1
        self.stream[self.count] = (stream.value or 1000 + self.count, not stream.value)
        C.cast(out, C.POINTER(C.c_void_p))[0] = self.count
        return 0

    def mq_state_stream(self, h, out):
        C.cast(out, C.POINTER(C.c_void_p))[0] = self.stream[h.value][0]
        return 0

    def mq_state_destroy(self, h):
        s, own = self.stream[h.value]
        if s in self.dead:
            self.late.append(h.value)
        if own:
            self.dead.add(s)
        self.order.append(h.value)
        return 0


@pytest.fixture
def lib(monkeypatch):
    fake = FakeLib()
    monkeypatch.setattr(E.N, "lib", lambda: fake)
    return fake


def _engine(**kw):
    return A.AdjointEngine(A.LayeredAnsatz(3, 1), A.PauliSum.ising_chain(3), **kw)


def test_an_engine_that_is_dropped(lib):
    e = _engine()
    del e
    gc.collect()
    assert sorted(lib.order) == [1, 2] and not lib.late


def test_an_engine_in_a_cycle(lib):
    e = _engine()
    e.me = e
    del e
    gc.collect()
    assert sorted(lib.order) == [1, 2] and not lib.late


def test_an_engine_that_is_closed(lib):
    e = _engine()
    e.close()
    del e
    gc.collect()
    assert lib.order == [2, 1] and not lib.late


def test_the_first_state_closed_alone(lib):
    e = _engine()
    e.psi.close()
    e.close()
    assert lib.order == [2, 1] and not lib.late


def test_a_stream_of_the_caller_is_left_to_it(lib):
    e = _engine(stream=77)
    e.psi.close()
    assert lib.order == [1]
    e.close()
    assert lib.order == [1, 2] and not lib.dead
