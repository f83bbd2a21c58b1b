"""Repairs at the edges of their splits: BFS candidates whose rows span one to many queue items with
the parent in the first, a middle or the last one, or in none; changed entries around the number
that comes back with the counters; component recomputes whose joining edge is the last entry
of a row around the block-wide length; classes split with and without their minimum. Levels and
labels equal the oracle's after every batch. MIS candidates whose only member neighbour is the first
entry of a row around one to many 32-entry groups, next to neighbours decided in the same round,
and batches with several candidates per warp. Colouring rounds of few and of many vertices with rows
around the lengths that go to a whole block."""
import numpy as np
import pytest

import scout_b200 as sb
from oracle import oracle as orc
from test_gpu_bfs import _run
from gpu_util import stream
from test_gpu_problems import _cc, _coloring, _mis

pytestmark = pytest.mark.gpu


def _csr(n, edges):
    e = np.unique(np.sort(np.array(edges, dtype=np.int64), axis=1), axis=0)
    e = np.concatenate([e, e[:, ::-1]])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    return np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))]).astype(np.int64), e[:, 1].astype(np.int32)


def test_bfs_candidates_of_long_rows():
    n, k = 60000, 24
    lens = (1, 7, 8, 9, 31, 32, 33, 250, 253, 254, 255, 256, 257, 509, 510, 512, 1021, 1024, 1025, 2047, 2049, 4096,
            9000, 20000)
    assert len(lens) == k
    rng = np.random.default_rng(3)
    low, hub, mid, high = 2 + np.arange(k), 100 + np.arange(k), 30000 + np.arange(k), n - 100 + np.arange(k)
    leaves = np.setdiff1d(np.arange(1000, n - 1000), mid)
    ed = [(0, 1)] + [(0, int(x)) for x in np.concatenate([low, mid, high])] + [(1, int(x)) for x in leaves]
    ed += [(1, int(x)) for x in hub[1::2]]
    for i in range(k):
        ed += [(int(hub[i]), int(p[i])) for p in (low, mid, high)]
        ed += [(int(hub[i]), int(x)) for x in rng.choice(leaves, size=lens[i], replace=False)]
    off, adj = _csr(n, ed)

    def to(p, sel=slice(None)):
        return np.stack([hub[sel], p[sel]], axis=1)

    g = np.stack([hub[1::2], np.ones(k // 2, int)], axis=1)
    batches = [np.concatenate([to(low), g]),               # parents left in the middle and last items
               to(mid),                                    # in the last only
               to(high, slice(0, None, 2)),                # half of them have none
               np.concatenate([to(low), g, to(mid), to(high, slice(0, None, 2))]),
               np.array([[0, 1]]),                         # every leaf is a candidate
               np.array([[0, 1]]),
               np.concatenate([[[0, 1]], to(low), to(mid), to(high)])]   # all at once
    _run(off, adj, [b.astype(np.int32) for b in batches], check_ref=False)


@pytest.mark.parametrize("changed", [1, 2047, 2048, 2049])
def test_changed_entries_that_come_with_the_counters(changed):
    n = 4000   # 0 - 1 - (2 .. changed): deleting (0, 1) strands `changed` vertices
    off, adj = _csr(n, [(0, 1), (0, n - 1)] + [(1, v) for v in range(2, changed + 1)])
    _run(off, adj, [np.array([[0, 1]], np.int32)] * 3, check_ref=False)
    init = orc.gt_bfs(off, adj, 0)
    with sb.Context(0) as ctx:   # entries replaced after the repair: the commit reads them as they are
        ctx.load_csr(off, adj)
        ctx.set_source(0)
        ctx.upload("bfs", init)
        ctx.repair("bfs", np.array([[0, 1]], np.int32))
        other = np.arange(n, dtype=np.int32) + 7
        ctx.upload("bfs", other)
        mirror = init.copy()
        ctx.commit("bfs", mirror)
        expected = init.copy()
        expected[1:changed + 1] = other[1:changed + 1]
        assert np.array_equal(mirror, expected)


@pytest.mark.parametrize("length", [3, 4, 129, 1023, 1024, 1025, 1500])
def test_cc_joined_by_the_last_entry_of_a_row(length):
    """Vertex h and `length` - 1 neighbours of its own form a component but for its last entry, a
    vertex of the dominant one whose own row has that edge behind its first two."""
    d, m = length, 30000                    # d: the dominant star's centre, its leaves d + 1 .. d + m
    h = d + m + 2
    ed = [(d, d + i) for i in range(1, m + 1)] + [(h, i) for i in range(length - 1)]
    x = d + m                               # the last leaf, also tied to d + 1
    ed += [(x, d + 1), (h, x)]
    off, adj = _csr(h + 3, ed)
    _cc(off, adj, [np.array([[h, 0]], np.int32), np.array([[h, 0], [h, x]], np.int32)], sched={"mode": 2},
        check_ref=False)


@pytest.mark.parametrize("mode", [0, 1])
def test_cc_splits_of_many_classes(mode):
    rng = np.random.default_rng(11)
    n, t, size = 8000, 60, 120              # 60 random trees of 120 vertices, ids shuffled
    ids = rng.permutation(n)
    ed = [(int(ids[c * size + v]), int(ids[c * size + rng.integers(max(0, v - 3), v)])) for c in range(t)
          for v in range(1, size)]
    off, adj = _csr(n, ed)
    e = np.array(ed)
    cuts = [e[rng.choice(len(e), size=s, replace=False)] for s in (1, 50, 400, 3000)]
    batches = [b.astype(np.int32) for c in cuts for b in (c, c)]   # cut, then joined again
    _cc(off, adj, batches, sched={"mode": mode}, check_ref=False)


def test_mis_candidates_of_long_rows():
    lens = (1, 2, 30, 31, 32, 33, 62, 63, 64, 65, 95, 96, 97, 1000, 3000)
    k, m = len(lens), 4000                  # ids: 0 | own members | m neighbours (held out by 0) | the hubs
    rng = np.random.default_rng(7)
    own, e, hub = 1 + np.arange(k), 1 + k + np.arange(m), 1 + k + m + np.arange(k)
    ed = [(0, int(v)) for v in e]
    for i, d in enumerate(lens):
        ed += [(int(own[i]), int(hub[i]))] + [(int(hub[i]), int(v)) for v in rng.choice(e, size=d, replace=False)]
    off, adj = _csr(1 + 2 * k + m, ed)
    first = np.array([[h, adj[off[h] + 1]] for h in hub])     # a neighbour held out: candidates stay out
    last = np.array([[h, adj[off[h + 1] - 1]] for h in hub[1:]])
    mine = np.stack([hub, own], axis=1)
    free = np.stack([np.zeros(200, int), e[-200:]], axis=1)   # neighbours of lower id, undecided as well
    batches = [first, mine, mine, np.concatenate([last, free]), np.concatenate([mine, last]), free,
               np.concatenate([mine, free])]
    _mis(off, adj, [b.astype(np.int32) for b in batches])


def test_mis_many_candidates_per_warp():
    off, adj = sb.gen_rmat(16, 8, seed=12).arrays()
    _mis(off, adj, stream(off, adj, sb.STREAM_LOWDEG, 80000, 1, seed=5, insert_ratio=0.2, lowdeg_frac=0.5))


@pytest.mark.parametrize("lens", [(0, 1, 31, 32, 33, 127, 128, 129, 1023, 1025, 4095, 4096, 4097, 5000), (126, 127, 128, 4096) * 75])
def test_coloring_rounds_of_long_rows(lens):
    k, m = len(lens), 6000                  # ids: m spokes | k hubs | k hubs with the same neighbours
    rng = np.random.default_rng(13)
    spokes = [rng.choice(m, size=d, replace=False) for d in lens]
    ed = [(i, i + 1) for i in range(0, m - 1, 3)]
    for i in range(k):
        ed += [(int(v), m + i) for v in spokes[i]] + [(int(v), m + k + i) for v in spokes[i]]
    off, adj = _csr(m + 2 * k, ed)
    twins = np.stack([m + np.arange(k), m + k + np.arange(k)], axis=1).astype(np.int32)   # of one colour
    _coloring(off, adj, orc.gt_greedy_color(off, adj), [twins, twins, twins[::2]])
