"""Greedy seeding of graphs whose chains are short although they have many vertices (shuffled grids, a few
hubs that everyone is joined to), which a few rounds over the open vertices settle, and of graphs
that the rounds leave to the waiter lists (ordered grids, late hubs of long prefixes). The oracle is the
sequential rule; a colouring of short chains takes at most a few times an MIS (lists alone took 4 to 11
times as long)."""
import numpy as np
import pytest

import scout_b200 as sb
from test_gpu_seed_lists import _greedy

pytestmark = pytest.mark.gpu


def _csr(n, u, v):
    k = u != v
    key = np.unique(np.concatenate([u[k] * n + v[k], v[k] * n + u[k]]).astype(np.int64))
    off = np.zeros(n + 1, dtype=np.int64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.int32)


def _shape(name):
    rng = np.random.default_rng(2)
    s = 300
    i = np.arange(s * s).reshape(s, s)
    u, v = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()]), np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    if name == "grid":
        return _csr(s * s, u, v)
    if name == "grid_shuffled":
        p = rng.permutation(s * s)
        return _csr(s * s, p[u], p[v])
    n = 40000
    if name == "hubs":
        return _csr(n, rng.integers(0, 60, 2 * n), rng.integers(0, n, 2 * n))
    if name == "late_hubs":
        return _csr(n, n - 1 - rng.integers(0, 60, 2 * n), rng.integers(0, n, 2 * n))
    d = int(name.split("_")[1])   # every vertex past the first d is joined to the d lowest ids
    b = np.repeat(np.arange(d, n), d)
    return _csr(n, b, np.tile(np.arange(d), n - d))


@pytest.mark.parametrize("problem", ["mis", "coloring"])
@pytest.mark.parametrize("name", ["grid", "grid_shuffled", "hubs", "late_hubs", "below_8", "below_15", "below_16", "below_17"])
def test_seed_is_the_sequential_rule(problem, name):
    off, adj = _shape(name)
    want = _greedy(problem, off, adj)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        for _ in range(2):
            ctx.seed(problem)
            assert np.array_equal(ctx.download(problem), want)


@pytest.mark.parametrize("name", ["grid_shuffled", "hubs"])
def test_time_of_short_chains(name):
    off, adj = _shape(name)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ms = {p: min(ctx.seed(p)["ms_repair"] for _ in range(6)) for p in ("mis", "coloring")}
    assert ms["coloring"] < 2.5 * ms["mis"]
