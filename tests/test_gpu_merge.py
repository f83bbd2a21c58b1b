"""The batch merge at the edges of its split: rows around one 32-entry group, the short-row limit
(128 entries, 32 half-edits), one slice (2,048 entries) and the in-place limit (4,096), whose
insertions fall before the first entry, after the last, many between the same two entries, and
next to deletions; rows that start empty or end empty; duplicates inside a batch. The adjacency
equals the oracle scratchpad's after every batch, in both stores."""
import numpy as np
import pytest

import scout_b200 as sb
from gpu_util import assert_same_graph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

N = 12000
LENS = (0, 1, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 160, 255, 256, 257, 300, 2047, 2048, 2049, 2304, 4095, 4096,
        4097, 6000)
FIRST = 1000   # hub ids are [FIRST, FIRST + len(LENS)); their neighbours lie on both sides


def _graph(seed):
    rng = np.random.default_rng(seed)
    rows = [set() for _ in range(N)]
    spokes = np.concatenate([np.arange(100, FIRST), np.arange(FIRST + len(LENS), N - 100)])
    for i, d in enumerate(LENS):
        h = FIRST + i
        for v in rng.choice(spokes, size=d, replace=False).tolist():
            rows[h].add(v)
            rows[v].add(h)
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    adj = np.concatenate([np.array(sorted(r), dtype=np.int32) for r in rows])
    return off, adj


def _edits(kind, off, adj, rng):
    """Pairs whose toggling exercises `kind` in every hub's row."""
    out = []
    for i in range(len(LENS)):
        h = FIRST + i
        row = adj[off[h]:off[h + 1]]
        absent = np.setdiff1d(np.concatenate([np.arange(0, FIRST), np.arange(FIRST + len(LENS), N)]), row)
        ins, dele = np.zeros(0, int), np.zeros(0, int)
        if kind == "ends":          # before the first entry and after the last
            ins = np.concatenate([np.arange(0, 5), np.arange(N - 5, N)])
            ins = np.setdiff1d(ins, row)
        elif kind == "one_gap":     # forty insertions between the same two entries
            at = absent[len(absent) // 2:]
            ins = at[:40]
            dele = row[:1]
        elif kind == "few":
            ins = rng.choice(absent, size=3, replace=False)
            dele = rng.choice(row, size=min(3, len(row)), replace=False)
        elif kind == "dense":       # as many edits as entries
            ins = rng.choice(absent, size=min(len(absent), len(row) + 1), replace=False)
            dele = rng.choice(row, size=len(row) // 2, replace=False)
        elif kind == "delete_all":
            dele = row
        elif kind == "delete_ends":
            dele = np.unique(np.concatenate([row[:2], row[-2:]]))
        out += [(h, int(x)) for x in ins] + [(int(x), h) for x in dele]
    e = np.array(out, dtype=np.int32)
    return e[rng.permutation(len(e))]


@pytest.mark.parametrize("tiered", [False, True])
@pytest.mark.parametrize("kind", ["ends", "one_gap", "few", "dense", "delete_all", "delete_ends"])
def test_rows_at_the_edges(kind, tiered):
    off, adj = _graph(5)
    rng = np.random.default_rng(17)
    og = orc.Graph(off, adj)
    with sb.Context(0) as ctx:
        if tiered:
            ctx.load_tiered(off, adj, hbm_entries=4 * len(adj))
        else:
            ctx.load_csr(off, adj)
        ctx.upload("bfs", orc.gt_bfs(off, adj, 0))
        for k, what in enumerate((kind, "few", kind)):
            b = _edits(what, *ctx.graph(), rng)
            st = ctx.repair("bfs", b)
            og.toggle_batch(b)
            assert st["insertions"] + st["deletions"] == len(b)
            assert_same_graph(ctx, og)
            assert ctx.info()["nnz"] == og.csr()[0][-1], f"batch {k + 1}: live entries"


@pytest.mark.parametrize("m", [1, 16, 511, 512, 513, 2047, 2048, 2049, 5121, 75776, 131071, 131072, 131073])
def test_update_sizes(rmat16, m):
    """Batch sizes around the update's pair-ranked sort (4,096 half-edits), one half-edit per
    thread (148 x 1,024), the one-launch update's limit (131,072 edits) and the separate
    launches beyond it; pairs repeated inside the batch are classified once each against the
    same state, some of them many times."""
    off, adj = rmat16[1]
    rng = np.random.default_rng(m)
    e = rng.integers(0, len(off) - 1, (m, 2)).astype(np.int32)
    e[: m // 2, 1] = adj[rng.integers(0, len(adj), m // 2)]
    at = np.searchsorted(off, rng.integers(0, len(adj), m // 4), side="right") - 1
    e[: m // 4, 0] = at
    e[: m // 4, 1] = adj[off[at]]                       # existing edges
    e[m - m // 8:] = e[: m // 8]                        # repeated pairs
    e[m // 2: m // 2 + m // 16] = e[0]                  # one pair over and over
    e[m // 3] = (-1, 5)                                 # an invalid edit
    og = orc.Graph(off, adj)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ctx.upload("cc", orc.gt_cc(off, adj))
        for _ in range(2):
            ctx.repair("cc", e)
            og.toggle_batch(e)
            assert_same_graph(ctx, og)
