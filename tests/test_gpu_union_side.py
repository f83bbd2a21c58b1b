"""Fused rounds on both sides of the line between repairs side by side and one after the other
(16,384 edits in a store's batch): two to four stores, a store without edits among them, one large
batch beside small ones. Every store's solution equals the single-stream engine's, bit for bit,
and for BFS and CC the oracle's ground truth."""
import numpy as np
import pytest

import scout_b200 as sb
from oracle import oracle as orc
from test_gpu_union import PROBLEMS, _check, _init

pytestmark = pytest.mark.gpu

LINE = 16384


@pytest.mark.parametrize("problems,rounds", [
    (PROBLEMS, [(LINE, 1, 0, 50), (LINE + 1, 1, 3, 50), (0, LINE, LINE, LINE), (2, LINE + 1, 0, 0), (0, 0, 0, 0),
                (1, 1, 1, 1), (2048, 2049, 4095, 4097)]),
    (["mis", "bfs"], [(3, LINE), (LINE + 1, 2), (0, 700), (700, 0), (5000, 5000)]),
    (["cc", "coloring", "mis"], [(LINE, 2, 1), (1, 0, LINE + 1), (300, 300, 300)]),
])
def test_rounds_around_the_line(problems, rounds):
    engines, singles, truths, data = [], [], [], []
    try:
        for pi, problem in enumerate(problems):
            h = sb.gen_rmat(13, 16, seed=70 + pi)
            off, adj = h.arrays()
            init = _init(problem, off, adj)
            me = sb.MultiEngine(problem)
            engines.append(me)
            me.add_stream(off, adj, init, 0)
            me.seal()
            ctx = sb.Context(0)
            singles.append(ctx)
            ctx.load_csr(off, adj)
            ctx.upload(problem, init)
            truths.append(orc.Graph(off, adj))
            sizes = [r[pi] for r in rounds]
            s = h.stream(sb.STREAM_LOWDEG, sum(sizes), 1, insert_ratio=0.4, lowdeg_frac=0.5, seed=80 + pi).reshape(-1, 2)
            data.append(np.split(s, np.cumsum(sizes)[:-1]))
        for j in range(len(rounds)):
            for pi, me in enumerate(engines):
                me.stage([(0, np.ascontiguousarray(data[pi][j]))])
            stats = sb.run_fused_round(engines)
            for pi, problem in enumerate(problems):
                b = np.ascontiguousarray(data[pi][j])
                singles[pi].repair(problem, b)
                got = engines[pi].download(0)
                assert np.array_equal(got, singles[pi].download(problem)), f"{problem} round {j}"
                truths[pi].toggle_batch(b)
                _check(problem, got, *truths[pi].csr())
                assert stats[pi]["ms_repair"] == stats[0]["ms_repair"] and stats[pi]["ms_update"] >= 0
    finally:
        for c in singles + engines:
            c.close()
