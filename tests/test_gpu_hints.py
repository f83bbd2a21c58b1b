"""Hinted batches in page-locked memory that is filled again: what a repair applies is what its array
holds when it is called."""
import numpy as np
import pytest

import scout_b200 as sb
from gpu_util import assert_same_graph, stream
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def test_refilled_after_its_own_repair(rmat16):
    """prefetch(b); repair(b); refill b; repair(b): the second repair applies the new edits."""
    g, (off, adj) = rmat16
    b = [stream(off, adj, sb.STREAM_PREFERENTIAL, 5000, 1, seed=900 + i)[0] for i in range(3)]
    og = orc.Graph(off, adj)
    with sb.Context(0) as t:
        t.load_csr(off, adj)
        t.upload("bfs", g.init_state("bfs", 0))
        t.reserve_batches(5000)
        p = sb.pinned_empty((5000, 2))
        for k, e in enumerate(b):
            p[:] = e
            if k < 2:
                t.prefetch(p)
            t.repair("bfs", p)
            og.toggle_batch(e)
            o, a = og.csr()
            assert np.array_equal(t.download("bfs"), orc.gt_bfs(o, a, 0)), f"batch {k + 1}"
        assert_same_graph(t, og)


def test_page_locked_memory_of_another_library(rmat16):
    """A hint in page-locked memory that torch allocated, dropped by the caller after prefetch() while
    more such memory is taken and written: every repair applies its own array."""
    import torch
    g, (off, adj) = rmat16
    b = [stream(off, adj, sb.STREAM_PREFERENTIAL, 20000, 1, seed=910 + i)[0] for i in range(5)]
    og = orc.Graph(off, adj)
    with sb.Context(0) as t:
        t.load_csr(off, adj)
        t.upload("bfs", g.init_state("bfs", 0))
        t.reserve_batches(20000)
        for k, e in enumerate(b):
            if k + 1 < len(b):
                t.prefetch(torch.from_numpy(b[k + 1].copy()).pin_memory().numpy())
            junk = torch.full((20000, 2), -1, dtype=torch.int32).pin_memory()
            t.repair("bfs", e)
            og.toggle_batch(e)
            o, a = og.csr()
            assert np.array_equal(t.download("bfs"), orc.gt_bfs(o, a, 0)), f"batch {k + 1}"
            del junk
        assert_same_graph(t, og)
