"""What scout_commit hands over when other calls came between the repair and it: a classification
leaves the last repair's changed entries alone (few of them, which come with the counters, and many,
which are gathered), and a repair that is refused leaves nothing to commit."""
import numpy as np
import pytest

import scout_b200 as sb
from gpu_util import stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("problem", ["coloring", "mis"])
def test_classify_between_repair_and_commit(rmat16, problem):
    """Few changed entries."""
    g, (off, adj) = rmat16
    warm = stream(off, adj, sb.STREAM_PREFERENTIAL, 30000, 1, seed=31)[0]
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ctx.seed(problem)
        mirror = ctx.download(problem)
        ctx.repair(problem, warm)
        ctx.commit(problem, mirror)
        for k in range(3):
            o, a = ctx.graph()
            b = stream(o, a, sb.STREAM_PREFERENTIAL, 3000, 1, seed=40 + k)[0]
            assert 0 < ctx.repair(problem, b)["changed"] <= 2048
            ctx.classify(warm[:5000])
            ctx.commit(problem, mirror)
            assert np.array_equal(mirror, ctx.download(problem)), f"batch {k + 1}"


@pytest.mark.parametrize("problem", ["bfs", "cc"])
def test_classify_between_repair_and_commit_of_many(problem):
    """Many: a path cut at its first edge and joined again."""
    n = 6000
    rows = [[w for w in (v - 1, v + 1) if 0 <= w < n] for v in range(n)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    adj = np.concatenate([np.asarray(r, dtype=np.int32) for r in rows])
    cut = np.array([[0, 1]], dtype=np.int32)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ctx.seed(problem)
        mirror = ctx.download(problem)
        for k in range(4):
            assert ctx.repair(problem, cut)["changed"] == n - 1
            ctx.classify(np.array([[5, 6], [7, 9]], dtype=np.int32))
            assert ctx.commit(problem, mirror) == n - 1
            assert np.array_equal(mirror, ctx.download(problem)), f"batch {k + 1}"


def test_refused_repair_leaves_nothing_to_commit(rmat16):
    g, (off, adj) = rmat16
    small = stream(off, adj, sb.STREAM_PREFERENTIAL, 3000, 1, seed=51)[0]
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ctx.seed("mis")
        ctx.repair("mis", small)
        held = ctx.held_bytes()
    with sb.Context(0, held + (1 << 20)) as ctx:     # no room for a large batch's workspace
        ctx.load_csr(off, adj)
        ctx.seed("mis")
        mirror = ctx.download("mis")
        assert ctx.repair("mis", small)["changed"] > 0
        large = np.zeros((3_000_000, 2), dtype=np.int32)
        with pytest.raises(sb.ScoutError):
            ctx.repair("mis", large)
        before = mirror.copy()
        assert ctx.commit("mis", mirror) == 0
        assert np.array_equal(mirror, before)
