"""A repair that fails after its batch was merged: the graph is updated, and everything that follows
(a seeding, a recompute, the next batches) works on that graph. The failure here is an uploaded
component labelling that does not describe the graph."""
import numpy as np
import pytest

import scout_b200 as sb
from gpu_util import assert_same_graph, stream
from oracle import oracle as orc
from test_gpu_seed_lists import _greedy

pytestmark = pytest.mark.gpu


def _batch(o, a, m, seed):
    """m preferential edits and the deletion of forty edges to vertices of degree one (no common neighbour
    settles those, so their class is recomputed under search_limit 1), none of them at vertex 1."""
    b = stream(o, a, sb.STREAM_PREFERENTIAL, m, 1, seed=seed, insert_ratio=0.8)[0]
    leaf = np.flatnonzero(np.diff(o) == 1)
    near = a[o[leaf]]
    ok = (near != 1) & (leaf != 1) & ~np.isin(leaf, b)
    leaf, near = leaf[ok][:40], near[ok][:40]
    assert len(leaf) == 40
    b = b[(b != 1).all(axis=1)]
    return np.ascontiguousarray(np.concatenate([b, np.stack([leaf, near], 1)]).astype(np.int32))


@pytest.mark.parametrize("tiered", [False, True])
@pytest.mark.parametrize("m", [20000, 150000])
def test_the_store_after_a_failed_repair(rmat16, tiered, m):
    g, (off, adj) = rmat16
    b = _batch(off, adj, m, 61)
    og = orc.Graph(off, adj)
    with sb.Context(0) as ctx:
        if tiered:
            ctx.load_tiered(off, adj, hbm_entries=len(adj))
        else:
            ctx.load_csr(off, adj)
        for k in range(3):
            o, a = og.csr()
            labels = orc.gt_cc(o, a).copy()   # but for vertex 1, which many rows begin with
            labels[1] = 1
            ctx.upload("cc", labels)
            with pytest.raises(sb.ScoutError, match="labels"):
                ctx.repair("cc", b, sched={"search_limit": 1})
            og.toggle_batch(b)
            o, a = og.csr()
            assert ctx.info()["nnz"] == len(a)
            assert_same_graph(ctx, og)
            for problem in ("coloring", "mis"):
                ctx.seed(problem)
                so, sa = ctx.graph()
                assert np.array_equal(ctx.download(problem), _greedy(problem, so, sa))
            ctx.recompute_cc()
            assert np.array_equal(ctx.download("cc"), orc.gt_cc(o, a))
            c = stream(o, a, sb.STREAM_PREFERENTIAL, 3000, 1, seed=70 + k)[0]
            ctx.repair("cc", c)
            og.toggle_batch(c)
            o, a = og.csr()
            assert np.array_equal(ctx.download("cc"), orc.gt_cc(o, a))
            assert_same_graph(ctx, og)
            b = _batch(o, a, m, 62 + k)
