"""Component recomputes on graphs whose first-neighbour trees are unlike an R-MAT graph's: one long chain,
chains and grids numbered in order and at random, random graphs, many small components, stars. Labels
equal the oracle's from labels that are right, from every vertex its own, and when a batch's
deletions make a class be recomputed; the time does not grow with a chain's length."""
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


def _shape(name, n):
    rng = np.random.default_rng(n)
    a = np.arange(n - 1)
    p = rng.permutation(n)
    s = int(n ** 0.5)
    i = np.arange(s * s).reshape(s, s)
    gu, gv = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()]), np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    if name == "path":
        return _csr(n, a, a + 1)
    if name == "path_backwards":
        return _csr(n, n - 1 - a, n - 2 - a)
    if name == "path_shuffled":
        return _csr(n, p[a], p[a + 1])
    if name == "paths_of_40":
        k = a[(a + 1) % 40 != 0]
        return _csr(n, p[k], p[k + 1])
    if name == "pairs":
        k = a[::2]
        return _csr(n, p[k], p[k + 1])
    if name == "grid":
        return _csr(n, gu, gv)
    if name == "grid_shuffled":
        return _csr(n, p[gu], p[gv])
    if name == "star_low":
        return _csr(n, np.zeros(n - 1, dtype=np.int64), a + 1)
    if name == "star_high":
        return _csr(n, np.full(n - 1, n - 1), a)
    if name == "two_halves":   # odd and even ids, no edge between them; some vertices alone
        u, v = rng.integers(0, n // 2 - 50, (2, 3 * n)) * 2
        return _csr(n, np.concatenate([u, u + 1]), np.concatenate([v, v + 1]))
    d = int(name.split("_")[1])
    return _csr(n, rng.integers(0, n, n * d // 2), rng.integers(0, n, n * d // 2))


SHAPES = ["path", "path_backwards", "path_shuffled", "paths_of_40", "pairs", "grid", "grid_shuffled", "star_low",
          "star_high", "two_halves", "random_1", "random_2", "random_6", "random_40"]


@pytest.mark.parametrize("n", [2, 33, 5000, 151000])
@pytest.mark.parametrize("name", SHAPES)
def test_labels(name, n):
    if n < 33 and name in ("two_halves", "paths_of_40") or n == 33 and name == "two_halves":
        pytest.skip("too small for it")
    off, adj = _shape(name, n)
    want = orc.gt_cc(off, adj)
    og = orc.Graph(off, adj)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        for labels in (want, np.arange(n, dtype=np.int32)):
            ctx.upload("cc", labels)
            ctx.recompute_cc()
            assert np.array_equal(ctx.download("cc"), want)
        if n < 100:
            return
        rng = np.random.default_rng(5)
        e = rng.integers(0, len(adj), 400)
        u = np.searchsorted(off, e, side="right") - 1
        b = np.stack([u, adj[e]], 1).astype(np.int32)
        _, at = np.unique(np.sort(b, axis=1), axis=0, return_index=True)
        b = np.ascontiguousarray(b[at])
        for mode in (0, 1, 0):
            ctx.repair("cc", b, sched={"mode": mode, "search_limit": 1})
            og.toggle_batch(b)
            o, a = og.csr()
            assert np.array_equal(ctx.download("cc"), orc.gt_cc(o, a))


def test_time_of_a_long_chain():
    """(A path of 10^6 vertices took 111 ms where a random graph of as many takes 0.2.)"""
    ms = {}
    for name in ("path", "random_6"):
        off, adj = _shape(name, 1000000)
        with sb.Context(0) as ctx:
            ctx.load_csr(off, adj)
            ctx.seed("cc")
            ms[name] = min(ctx.recompute_cc()["ms_repair"] for _ in range(3))
    assert ms["path"] < 8 * ms["random_6"]
