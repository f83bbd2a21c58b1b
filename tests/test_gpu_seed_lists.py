"""scout_seed's greedy rules (every vertex decided from its own row's lower-id neighbours, in id
order) where the waiter lists and the scans have their edges: prefixes around one warp step
(256), the block threshold (1024) and the colour window (1024 colours), vertices without
neighbours, rows that are not symmetric (a list can be too short for its waiters), and a store
whose budget leaves no room for the lists. The oracle is the sequential rule."""
import numpy as np
import pytest

import scout_b200 as sb

pytestmark = pytest.mark.gpu


def _csr(rows):
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return off, np.concatenate([np.sort(np.asarray(r, dtype=np.int32)) for r in rows] + [np.zeros(0, np.int32)])


def _complete(n):
    return [np.delete(np.arange(n), v) for v in range(n)]


def _random(n, deg, seed, symmetric):
    rng = np.random.default_rng(seed)
    rows = [set() for _ in range(n)]
    for u, v in rng.integers(0, n, (n * deg, 2)).tolist():
        u = u * u // n   # skewed towards low ids
        if u != v:
            rows[u].add(v)
            if symmetric:
                rows[v].add(u)
    return [sorted(r) for r in rows]


def _late_hub(n, k):
    """A path on [0, k) and a last vertex joined to all of it."""
    rows = [[w for w in (v - 1, v + 1) if 0 <= w < k] if v < k else [] for v in range(n)]
    for v in range(k):
        rows[v].append(n - 1)
    rows[n - 1] = list(range(k))
    return rows


GRAPHS = {
    "one": [[]],
    "isolated": [[] for _ in range(33)],
    "complete_33": _complete(33),
    "complete_1100": _complete(1100),
    "prefix_255": _late_hub(300, 255), "prefix_256": _late_hub(300, 256), "prefix_257": _late_hub(300, 257),
    "prefix_1024": _late_hub(1100, 1024), "prefix_1025": _late_hub(1100, 1025), "prefix_9001": _late_hub(9100, 9001),
    "skewed": _random(3001, 12, 1, True),
    "one_sided": _random(3001, 12, 2, False),
}


def _greedy(problem, off, adj):
    n = len(off) - 1
    out = np.zeros(n, dtype=np.int32)
    for v in range(n):
        r = adj[off[v]:off[v + 1]]
        used = out[r[r < v]]
        if problem == "mis":
            out[v] = 0 if np.any(used == 1) else 1
        else:
            free = np.ones(len(used) + 1, dtype=bool)
            free[used[used <= len(used)]] = False
            out[v] = int(np.argmax(free))
    return out


@pytest.mark.parametrize("problem", ["mis", "coloring"])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_seed_is_the_sequential_rule(problem, name):
    off, adj = _csr(GRAPHS[name])
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        for _ in range(2):
            ctx.seed(problem)
            assert np.array_equal(ctx.download(problem), _greedy(problem, off, adj))


@pytest.mark.parametrize("problem", ["mis", "coloring"])
def test_seed_without_room_for_the_lists(problem):
    off, adj = _csr(_random(20001, 12, 3, True))
    with sb.Context(0) as ctx:
        ctx.load_tiered(off, adj, hbm_entries=len(adj) // 4)
        ctx.seed(problem)
        want, held = ctx.download(problem), ctx.held_bytes()
    assert np.array_equal(want, _greedy(problem, off, adj))
    with sb.Context(0, held + 1024) as ctx:   # the state and scratch fit, the lists do not
        ctx.load_tiered(off, adj, hbm_entries=len(adj) // 4)
        ctx.seed(problem)
        assert np.array_equal(ctx.download(problem), want)
