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


@pytest.mark.parametrize("page_locked", [True, False])
@pytest.mark.parametrize("between", ["nothing", "repair", "refused repair", "its own repair"])
def test_the_hinted_array_outlives_the_copy(ctx, monkeypatch, page_locked, between):
    """Whether memory is page-locked the library decides by itself (an array of another library may
    be), and it may read such memory until the next hint: the array lives until then, however it
    was allocated, used or not, and also where the repair in between was refused."""
    c, lib = ctx
    monkeypatch.setattr(engine, "_page_locked", lambda a: page_locked)
    b = _edges(5)
    c.prefetch(b)
    ref = weakref.ref(b)
    if between == "its own repair":
        c.repair("bfs", _edges(6))
        c.repair("bfs", b)
    del b
    if between == "repair":
        c.repair("bfs", _edges(6))
    if between == "refused repair":
        lib.fail = -1
        with pytest.raises(engine.ScoutError):
            c.repair("bfs", _edges(6))
    gc.collect()
    assert ref() is not None
    c.prefetch(_edges(7))
    gc.collect()
    assert (ref() is None) or between in ("repair",) and page_locked   # (declared for the repair to come)


def test_a_converted_array_lives_as_long(ctx, monkeypatch):
    """as_edges may hand the library another object than the caller's."""
    c, lib = ctx
    kept = []
    monkeypatch.setattr(lib, "scout_prefetch", lambda h, e, m: kept.append(C.addressof(e.contents)) or 0, raising=False)
    b = _edges(8).astype(np.int64)
    c.prefetch(b)
    assert c._pf_keep.ctypes.data == kept[0]


def test_an_engine_has_one_context(monkeypatch):
    """A hint through MultiEngine.context is kept by the engine, not by a passing view."""
    monkeypatch.setattr(engine, "LIB", type("L", (), {"scout_multi_context": staticmethod(lambda h: 7)})())
    e = engine.MultiEngine.__new__(engine.MultiEngine)
    e._h = None
    assert e.context is e.context
