"""Batches that name one pair very often: every copy is classified against the graph before the batch,
each deletion cancels one entry while there is one, and the time of such a batch stays near that of
a batch of as many random pairs (what is done per copy must not depend on the number of copies)."""
import numpy as np
import pytest

import scout_b200 as sb
from gpu_util import assert_same_graph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _pairs(off, adj, kind, m):
    n = len(off) - 1
    rng = np.random.default_rng(7)
    big = int(np.argmax(np.diff(off)))
    mid = off[big] + (off[big + 1] - off[big]) // 2
    if kind == "random":
        return rng.integers(0, n, (m, 2)).astype(np.int32)
    if kind == "one_edge":
        return np.tile(np.array([[big, adj[mid]]], dtype=np.int32), (m, 1))
    if kind == "one_new":
        v = int(np.setdiff1d(np.arange(n), adj[off[big]:off[big + 1]])[-5])
        return np.tile(np.array([[big, v]], dtype=np.int32), (m, 1))
    few = np.concatenate([np.stack([np.full(20, big), adj[mid:mid + 20]], 1), rng.integers(0, n, (20, 2))])
    return few[rng.integers(0, len(few), m)].astype(np.int32)


@pytest.mark.parametrize("kind", ["one_edge", "one_new", "forty"])
@pytest.mark.parametrize("m", [40, 2100, 30000, 131072, 200000])
def test_repeated_pairs(rmat16, kind, m):
    _, (off, adj) = rmat16
    e = _pairs(off, adj, kind, m)
    og = orc.Graph(off, adj)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ctx.seed("bfs")
        for _ in range(3):
            ctx.repair("bfs", e)
            og.toggle_batch(e)
            assert_same_graph(ctx, og)
            o, a = ctx.graph()
            assert np.array_equal(ctx.download("bfs"), orc.gt_bfs(o, a, 0))


def _update_ms(off, adj, e):
    best = 1e9
    for _ in range(2):
        with sb.Context(0) as ctx:
            ctx.load_csr(off, adj)
            ctx.seed("mis")
            ctx.reserve_batches(len(e))
            ctx.repair("mis", e[:64])
            best = min(best, ctx.repair("mis", e)["ms_update"])
    return best


@pytest.mark.parametrize("m", [1_000_000])
def test_time_of_one_repeated_deletion(rmat16, m):
    """(10^6 copies of one edge: 0.9 s when every copy walked back over the copies before it, against
    0.5 ms for random pairs.)"""
    _, (off, adj) = rmat16
    base = _update_ms(off, adj, _pairs(off, adj, "random", m))
    assert _update_ms(off, adj, _pairs(off, adj, "one_edge", m)) < 100 * base


@pytest.mark.parametrize("kind", ["one_edge", "forty"])
@pytest.mark.parametrize("m", [9000, 300000])
def test_repeated_pairs_in_a_long_row_compacted_in_place(rmat16, kind, m):
    """Tiered store, a row past the length that one warp compacts where it lies: deletions alone, those
    that cancel an entry and the copies past them."""
    _, (off, adj) = rmat16
    e = _pairs(off, adj, kind, m)
    big = int(np.argmax(np.diff(off)))
    assert off[big + 1] - off[big] > 4096
    if kind == "forty":   # without the random pairs: entries of the long row's whole length
        at = np.random.default_rng(5).integers(off[big], off[big + 1], m)
        at[: m // 2] = off[big] + 3000
        e = np.stack([np.full(m, big), adj[at]], 1).astype(np.int32)
    og = orc.Graph(off, adj)
    with sb.Context(0) as ctx:
        ctx.load_tiered(off, adj, hbm_entries=2 * len(adj))
        ctx.seed("bfs")
        for _ in range(2):
            ctx.repair("bfs", e)
            og.toggle_batch(e)
            assert_same_graph(ctx, og)


def test_time_of_one_repeated_deletion_in_place(rmat16):
    """(10^6 copies of one edge of a row that is compacted in place, by 256 events at a time: 4 ms.)"""
    _, (off, adj) = rmat16

    def update_ms(tiered):
        best = 1e9
        for _ in range(2):
            with sb.Context(0) as ctx:
                if tiered:
                    ctx.load_tiered(off, adj, hbm_entries=4 * len(adj))
                else:
                    ctx.load_csr(off, adj)
                ctx.seed("mis")
                ctx.reserve_batches(1_000_000)
                ctx.repair("mis", _pairs(off, adj, "random", 64))
                best = min(best, ctx.repair("mis", _pairs(off, adj, "one_edge", 1_000_000))["ms_update"])
        return best

    assert update_ms(True) < 3 * update_ms(False)
