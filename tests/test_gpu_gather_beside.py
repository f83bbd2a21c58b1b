"""Tiered store: the gather of the next batch's rows runs beside the repair whatever the blocks_per_sm knob
says. (A BFS repair of four quarters holds all of an SM's registers, and the gather then waited for
it: it ended 127 us after the merge instead of 66.)"""
import numpy as np
import pytest

import scout_b200 as sb
from gpu_util import stream
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def test_the_knob_leaves_room_for_the_gather():
    g = sb.gen_rmat(18, 8, seed=4)
    off, adj = g.arrays()
    batches = [sb.pinned_copy(b) for b in
               g.stream(sb.STREAM_MIXED, 1000, 4, insert_ratio=0.3, lowdeg_frac=0.3, seed=9).reshape(4, 1000, 2)]
    ms = {}
    for knob in (3, 4):
        with sb.Context(0) as ctx:
            ctx.load_tiered(off, adj, hbm_entries=len(adj) * 23 // 100)
            ctx.seed("bfs")
            ctx.reserve_batches(1000)
            got = []
            for k in range(40):
                ctx.prefetch(batches[(k + 1) % 4])
                st = ctx.repair("bfs", batches[k % 4], sched={"blocks_per_sm": knob})
                if k >= 8:
                    assert st["gather_rows"] > 0
                    got.append(st["ms_gather"])
            ms[knob] = float(np.median(got))
            o, a = ctx.graph()
            assert np.array_equal(ctx.download("bfs"), orc.gt_bfs(o, a, 0))
    assert ms[4] < 1.4 * ms[3]
