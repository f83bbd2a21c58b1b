"""The cost model that ships with the package is one of the present kernels: on held-out graphs and streams
its choices take less repair time than the incremental repair alone (a model of older kernels chose
nothing else for BFS)."""
import os

import numpy as np
import pytest

import scout_b200 as sb
from scout_b200 import learn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("problem", ["bfs", "cc"])
def test_shipped_model_gains_on_held_out_streams(problem):
    with np.load(os.path.join(os.path.dirname(sb.__file__), "sched_model.npz")) as d:
        params = np.asarray(d[problem], dtype=np.float32)
    specs = learn.default_specs(problem, range(300, 302), (16, 18, 20), (100, 1_000, 10_000, 100_000, 300_000),
                                graph_seeds=(400,))
    r = learn.evaluate(params, learn.collect(problem, specs), problem)
    assert r["learned_ms"] < 0.9 * r["plain_ms"], r
