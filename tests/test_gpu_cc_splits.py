"""Components of which several deletions of one batch split off sides: every class has some split records,
whose endpoints are searched against each other by different blocks at a time while any of them may
mark the class for a recompute. Labels equal the oracle's after every batch. (That every thread of
a block takes the same way past such a mark is shown by the code: one thread reads it.)"""
import os
import re

import numpy as np
import pytest

import scout_b200 as sb
from conftest import ROOT
from oracle import oracle as orc


def test_one_thread_reads_the_mark():
    """In the loop over split records nothing another block may change is read by every thread."""
    code = open(os.path.join(ROOT, "scout_b200", "csrc", "cuda", "cc_dev.cuh")).read()
    code = re.sub(r"//[^\n]*", "", code)
    loop = code[code.index("if (!grid_sync(p.bar, 40)) return;"):code.index("if (!grid_sync(p.bar, 41)) return;")]
    every = loop[loop.index("__syncthreads();"):]          # after one thread's turn
    assert "p.dirty + cls" not in every.replace("atomicExch(p.dirty + cls", "") and "p.cnt" not in every


@pytest.mark.gpu
@pytest.mark.parametrize("length,cuts", [(6, 2), (12, 3), (40, 7), (300, 20)])
@pytest.mark.parametrize("extra", [0.0, 0.5])
def test_many_splits_of_many_classes(length, cuts, extra):
    rng = np.random.default_rng(length)
    classes = 24000 // length
    n = classes * length
    p = rng.permutation(n)
    at = np.arange(n).reshape(classes, length)
    u, v = at[:, :-1].ravel(), at[:, 1:].ravel()
    x = int(extra * n)       # chords inside a class: some deletions then split nothing
    c, a, b = rng.integers(0, classes, x), rng.integers(0, length, x), rng.integers(0, length, x)
    u, v = p[np.concatenate([u, at[c, a]])], p[np.concatenate([v, at[c, b]])]
    k = u != v
    key = np.unique(np.concatenate([u[k] * n + v[k], v[k] * n + u[k]]))
    off = np.zeros(n + 1, dtype=np.int64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    adj = (key % n).astype(np.int32)
    og = orc.Graph(off, adj)
    with sb.Context(0) as ctx:
        ctx.load_csr(off, adj)
        ctx.seed("cc")
        mirror = ctx.download("cc")
        for r in range(16):
            cut = rng.permuted(np.tile(np.arange(length - 1), (classes, 1)), axis=1)[:, :cuts]
            row = np.repeat(np.arange(classes), cuts)
            b = np.stack([p[at[row, cut.ravel()]], p[at[row, cut.ravel() + 1]]], 1).astype(np.int32)
            b = np.ascontiguousarray(rng.permutation(b))
            for _ in (0, 1):                     # the cuts, then the same edges back
                ctx.repair("cc", b)
                ctx.commit("cc", mirror)
                og.toggle_batch(b)
                o, a2 = og.csr()
                assert np.array_equal(mirror, orc.gt_cc(o, a2)), f"round {r}"
