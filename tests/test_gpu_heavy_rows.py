"""Rows that change by more half-edits than a warp walks (1,024): insertions placed as items of their own,
old entries by searches; on both sides of the limit, for empty, short and long rows, with the
insertions in one gap, at the end and spread, with deletions and repeated pairs among them, in the
one-launch update and beyond it, in both stores. The adjacency equals the oracle's."""
import numpy as np
import pytest

import scout_b200 as sb
from gpu_util import assert_same_graph
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
N = 30000
HUB = 15000


def _star(length):
    """Vertex HUB with `length` neighbours, every other id from 5000 on, and a ring of the rest."""
    nb = 5000 + 2 * np.arange(length)
    nb = nb[nb != HUB]
    e = [(HUB, int(v)) for v in nb]
    ring = [v for v in range(200)]
    e += [(ring[i], ring[(i + 1) % 200]) for i in range(200)]
    return nb, e


def _csr(edges):
    u = np.array([a for a, _ in edges] + [b for _, b in edges])
    v = np.array([b for _, b in edges] + [a for a, _ in edges])
    k = np.unique(u.astype(np.int64) * N + v)
    off = np.zeros(N + 1, dtype=np.int64)
    off[1:] = np.cumsum(np.bincount(k // N, minlength=N))
    return off, (k % N).astype(np.int32)


def _batch(nb, kind, many, rng):
    there = np.zeros(N, dtype=bool)
    there[nb] = True
    there[HUB] = True
    free = np.flatnonzero(~there)
    lo, hi = free[free < 5000], free[free > (nb[-1] if len(nb) else 5000)]
    half = nb[rng.permutation(len(nb))[: min(len(nb) // 2, many // 2)]]
    v = {"before": lo[:many], "after": hi[:many], "spread": rng.permutation(free)[:many],
         "both": np.concatenate([rng.permutation(free)[: many - len(half)], half]),
         "gone": nb[rng.permutation(len(nb))[: min(many, len(nb) - 1)]],
         "again": np.concatenate([rng.permutation(free)[: many // 3], half, half[: len(half) // 2],
                                  np.full(many // 3, nb[len(nb) // 2] if len(nb) else free[3])])}[kind]
    e = np.stack([np.full(len(v), HUB), v], 1)
    e = np.where(rng.random((len(v), 1)) < 0.5, e, e[:, ::-1])
    return np.ascontiguousarray(rng.permutation(e).astype(np.int32))


@pytest.mark.parametrize("tiered", [False, True])
@pytest.mark.parametrize("length", [0, 3, 129, 2049, 4097, 9000])
def test_heavy_rows(length, tiered):
    rng = np.random.default_rng(length)
    nb, edges = _star(length)
    off, adj = _csr(edges)
    for kind in ("before", "after", "spread", "both", "gone", "again"):
        if kind == "gone" and length < 129:
            continue
        for many in (1024, 1025, 4990):
            og = orc.Graph(off, adj)
            with sb.Context(0) as ctx:
                if tiered:
                    ctx.load_tiered(off, adj, hbm_entries=120000)
                else:
                    ctx.load_csr(off, adj)
                ctx.seed("bfs")
                b = _batch(nb, kind, many, rng)
                rest = np.stack([rng.integers(300, 4000, 700), rng.integers(300, 4000, 700)], 1)
                for e in (b, np.concatenate([b, rest.astype(np.int32)]), b):
                    e = np.ascontiguousarray(e[e[:, 0] != e[:, 1]])
                    ctx.repair("bfs", e)
                    og.toggle_batch(e)
                    assert_same_graph(ctx, og)
                o, a = ctx.graph()
                assert np.array_equal(ctx.download("bfs"), orc.gt_bfs(o, a, 0))


@pytest.mark.parametrize("tiered", [False, True])
def test_heavy_rows_beyond_the_one_launch_update(tiered):
    """Several heavy rows and 150,000 edits in one batch."""
    n = 200000
    rng = np.random.default_rng(3)
    k = rng.integers(0, n, (400000, 2))
    k = np.concatenate([k[k[:, 0] != k[:, 1]], np.stack([np.full(6000, 17), np.arange(1000, 7000)], 1)])
    key = np.unique(np.concatenate([k[:, 0] * n + k[:, 1], k[:, 1] * n + k[:, 0]]))
    off = np.zeros(n + 1, dtype=np.int64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    adj = (key % n).astype(np.int32)
    og = orc.Graph(off, adj)
    b = [np.stack([np.full(40000, h), rng.permutation(n)[:40000]], 1) for h in (17, 5, 199998)]
    b = np.concatenate(b + [rng.integers(0, n, (30000, 2)), np.tile([[17, 1500]], (3000, 1))])
    b = np.ascontiguousarray(b[b[:, 0] != b[:, 1]].astype(np.int32))
    with sb.Context(0) as ctx:
        if tiered:
            ctx.load_tiered(off, adj, hbm_entries=len(adj))
        else:
            ctx.load_csr(off, adj)
        ctx.seed("bfs")
        for _ in range(3):
            ctx.repair("bfs", b)
            og.toggle_batch(b)
            assert_same_graph(ctx, og)


@pytest.mark.parametrize("length,many", [(3, 20000)])
def test_time_of_a_row_that_gains_many(length, many):
    """(20,000 insertions in one gap were walked by one warp, 32 at a time: 2 ms, where an update of as
    many random pairs takes 0.1.)"""
    nb, edges = _star(length)
    off, adj = _csr(edges)
    rng = np.random.default_rng(1)

    def update_ms(e):
        best = 1e9
        for _ in range(3):
            with sb.Context(0) as ctx:
                ctx.load_csr(off, adj)
                ctx.seed("mis")
                ctx.reserve_batches(len(e))
                ctx.repair("mis", np.array([[4500, 4502]], dtype=np.int32))
                best = min(best, ctx.repair("mis", e)["ms_update"])
        return best

    # one orientation, so that the sort's sample is the same in both arms
    v = np.setdiff1d(np.arange(N), np.append(nb, HUB))[:many]
    flip = rng.random((many, 1)) < 0.5
    star = np.where(flip, np.stack([v, np.full(many, HUB)], 1), np.stack([np.full(many, HUB), v], 1))
    pairs = np.stack([rng.permutation(N)[:many], rng.permutation(N)[:many]], 1)
    pairs = pairs[pairs[:, 0] != pairs[:, 1]]
    assert update_ms(np.ascontiguousarray(star.astype(np.int32))) < 4 * update_ms(np.ascontiguousarray(pairs.astype(np.int32)))
