"""The greedy MIS seeding's two parts: rounds over all open vertices, which settle graphs of short chains
alone (R-MAT and random graphs take about ten), and the waiter lists that finish what is open
after the limit of 32 rounds (paths and grids numbered in order), from the solution as it then is."""
import numpy as np
import pytest

import scout_b200 as sb
from test_gpu_seed_lists import _csr, _greedy, _random

pytestmark = pytest.mark.gpu
LIMIT = 32


def test_short_chains_take_rounds_alone(rmat16):
    off, adj = rmat16[1]
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        assert ctx.seed("mis")["rounds"] <= LIMIT
        assert np.array_equal(ctx.download("mis"), _greedy("mis", off, adj))


def _path(n, extra=()):
    rows = [{w for w in (v - 1, v + 1) if 0 <= w < n} for v in range(n)]
    for u, v in extra:
        rows[u].add(v)
        rows[v].add(u)
    return [sorted(r) for r in rows]


def _grid(a, b):
    return [[w for w, ok in ((v - b, v >= b), (v - 1, v % b > 0), (v + 1, v % b < b - 1), (v + b, v < (a - 1) * b)) if ok]
            for v in range(a * b)]


GRAPHS = {
    "path_32": _path(32), "path_33": _path(33), "path_64": _path(64), "path_1000": _path(1000),
    "grid": _grid(61, 97),
    "hub_on_a_path": _path(3000, [(7, v) for v in range(9, 3000, 2)]),
    "late_hub": _path(3000, [(2999, v) for v in range(0, 2990, 2)]),
    "path_and_random": _path(1500) + [[w + 1500 for w in r] for r in _random(1500, 6, 5, True)],
    "one_sided_path": [[v - 1] if v else [] for v in range(2500)],
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_long_chains_are_finished_by_the_lists(name):
    off, adj = _csr(GRAPHS[name])
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        for _ in range(2):
            rounds = ctx.seed("mis")["rounds"]
            assert np.array_equal(ctx.download("mis"), _greedy("mis", off, adj))
            if name == "path_1000":
                assert rounds > LIMIT


def test_lists_without_room():
    off, adj = _csr(_grid(150, 133))
    with sb.Context(0) as ctx:
        ctx.load_tiered(off, adj, hbm_entries=len(adj) // 2)
        ctx.seed("mis")
        held = ctx.held_bytes()
        assert np.array_equal(ctx.download("mis"), _greedy("mis", off, adj))
    with sb.Context(0, held + 1024) as ctx:
        ctx.load_tiered(off, adj, hbm_entries=len(adj) // 2)
        ctx.seed("mis")
        assert np.array_equal(ctx.download("mis"), _greedy("mis", off, adj))
