"""What Context.prefetch and Context.repair declare to the library, on the CPU: the library's calls
are recorded by a stand-in that takes the same arguments."""
import ctypes as C
import gc
import weakref

import numpy as np
import pytest

from scout_b200 import engine


class FakeLib:
    """scout_prefetch and scout_repair, recorded."""

    def __init__(self):
        self.declared = []
        self.fail = 0

    def scout_prefetch(self, h, edges, m):
        return 0

    def scout_repair(self, h, problem, edges, ops, m, sched, stats):
        self.declared.append(C.cast(sched, C.POINTER(engine.ScoutSched)).contents.prefetched)
        return self.fail

    def scout_last_error(self, h):
        return b"told to fail"


@pytest.fixture
def ctx(monkeypatch):
    lib = FakeLib()
    monkeypatch.setattr(engine, "LIB", lib)
    monkeypatch.setattr(engine, "_page_locked", lambda a: True)
    c = engine.Context._borrow(C.c_void_p(1))
    return c, lib


def _edges(seed, m=8):
    return np.random.default_rng(seed).integers(0, 100, (m, 2), dtype=np.int32)


def test_a_hint_is_declared_by_its_own_repair(ctx):
    c, lib = ctx
    a, b = _edges(1), _edges(2)
    c.prefetch(b)
    c.repair("bfs", a)
    c.repair("bfs", b)
    assert lib.declared == [0, 1]


@pytest.mark.parametrize("alias", ["itself", "view", "part"])
def test_a_hint_ends_with_its_batch(ctx, alias):
    """A batch hinted and repaired at once may be refilled: the next repair of the same array
    must upload it."""
    c, lib = ctx
    b = _edges(3)
    c.prefetch(b)
    c.repair("bfs", {"itself": b, "view": b[:], "part": b[:5]}[alias])
    b[:] = _edges(4)
    c.repair("bfs", b)
    assert lib.declared == [0, 0]
