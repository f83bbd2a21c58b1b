"""BFS repairs whose cascades are narrow, at most one candidate per warp and round (a path cut in its middle,
a comb, a tree, a path through rows longer than a queue item), and wide ones of the same graphs next
to them. Levels equal the oracle's after every batch."""
import numpy as np
import pytest

import scout_b200 as sb
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _csr(n, u, v):
    k = u != v
    key = np.unique(np.concatenate([u[k] * n + v[k], v[k] * n + u[k]]).astype(np.int64))
    off = np.zeros(n + 1, dtype=np.int64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.int32)


def _shape(name):
    """Edges, and the edges whose loss starts a cascade."""
    rng = np.random.default_rng(4)
    n = 3000
    a = np.arange(n - 1)
    if name == "path":
        return _csr(n, a, a + 1), [(10, 11), (1500, 1501), (2990, 2991)]
    if name == "path_shuffled":
        p = np.concatenate([[0], 1 + rng.permutation(n - 1)])
        return _csr(n, p[a], p[a + 1]), [(p[5], p[6]), (p[2000], p[2001])]
    if name == "comb":       # a spine of every third vertex, two teeth on each
        s = np.arange(0, n, 3)
        return _csr(n, np.concatenate([s[:-1], s, s]), np.concatenate([s[1:], s + 1, s + 2])), [(300, 303), (2400, 2403)]
    if name == "tree":
        c = np.arange(1, n)
        return _csr(n, (c - 1) // 2, c), [(0, 1), (6, 13)]
    # a path whose every 40th vertex has 700 leaves: its row is longer than one queue item
    h = np.arange(0, 200, 40)
    u = np.concatenate([np.arange(199), np.repeat(h, 560)])
    v = np.concatenate([np.arange(1, 200), 200 + np.arange(560 * len(h))])
    return _csr(3000, u, v), [(30, 31), (79, 80), (80, 81), (0, 1)]


@pytest.mark.parametrize("chunk_log2", [0, 8, 13])
@pytest.mark.parametrize("name", ["path", "path_shuffled", "comb", "tree", "hubs"])
def test_cascades(name, chunk_log2):
    (off, adj), cuts = _shape(name)
    n = len(off) - 1
    og = orc.Graph(off, adj)
    rng = np.random.default_rng(6)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ctx.seed("bfs")
        batches = [[c] for c in cuts for _ in (0, 1)] + [cuts, cuts]
        batches += [np.concatenate([cuts, rng.integers(0, n, (k, 2))]) for k in (3, 900)]
        batches += [[(0, n - 1)], [cuts[0]], [(0, n - 1)], [cuts[0]]]
        for k, b in enumerate(batches):
            b = np.asarray(b, dtype=np.int32)
            b = np.ascontiguousarray(b[b[:, 0] != b[:, 1]])
            ctx.repair("bfs", b, sched={"chunk_log2": chunk_log2})
            og.toggle_batch(b)
            o, a = og.csr()
            assert np.array_equal(ctx.download("bfs"), orc.gt_bfs(o, a, 0)), f"batch {k + 1}"
