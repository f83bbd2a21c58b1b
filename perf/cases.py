"""The work a user has this engine do, as cases that can be timed and compared.

Every case holds one graph (or several) resident on the GPU with a maintained solution and puts
work through the package's public calls:

  repair     one batch of edge toggles: Context.repair + Context.commit into a host mirror.
             A program hands in batch after batch; here a short stream of batches is cycled, and
             going through it again toggles every pair back. hint: the edits lie in page-locked
             memory and the next batch is announced (Context.prefetch), as bench.py does;
             otherwise they are pageable arrays. ops: the caller classified the edits itself, as
             the MIS program does. learned: the shipped cost model picks the variant on the
             device. tiered: the graph is larger than its HBM pool and cold rows stay in host
             memory.
  multi      one round of a MultiEngine (many streams of one problem) + commit
  fused      one round of four MultiEngines, all repairs in one kernel, + commits
  recompute  a full recompute of BFS levels or component labels + commit, as at a stream's end
  seed       the initial solution computed on the device + its download, as at a stream's start

Graphs are R-MAT (a/b/c/d = .57/.19/.19/.05, symmetrised, no loops or duplicates) over any number
of vertices; batches are preferential (endpoints proportional to degree, half deletions),
uniform (random pairs) or deletion-heavy (70% deletions, 30% of those at low-degree vertices).
"""
import math
import os

import numpy as np
import torch

import scout_b200 as sb

CYCLE = 4             # batches of a stream before it repeats
BIT_ONE = 0.24        # R-MAT: probability that an endpoint's id bit is one (b + d)


def listed():
    return [
        # the smallest call: the bundled sample graph's size and batches of a few dozen edits,
        # where launches and waits are everything
        dict(name="bfs_sample_50", kind="repair", problem="bfs", n=2000, ef=8, m=50, mix="uniform"),
        # plain MIS maintenance, small: scale 16, 1,000 uniform toggles, classified by the caller
        dict(name="mis_s16_1k", kind="repair", problem="mis", n=65536, ef=16, m=1000, mix="uniform", ops=True),
        # the headline stream's small batch, run as the benchmark runs it: learned, announced
        dict(name="bfs_s22_10k", kind="repair", problem="bfs", n=1 << 22, ef=16, m=10_000, mix="preferential",
             hint=True, learned=True),
        # the headline stream's large batch, the largest case
        dict(name="bfs_s22_1m", kind="repair", problem="bfs", n=1 << 22, ef=16, m=1_000_000, mix="preferential",
             hint=True),
        # an ordinary colouring batch on a graph of ragged size, from an ordinary array
        dict(name="coloring_1500k_100k", kind="repair", problem="coloring", n=1_500_007, ef=16, m=100_003,
             mix="preferential"),
        # MIS under large batches whose edits the caller classified
        dict(name="mis_1m_300k", kind="repair", problem="mis", n=1_000_003, ef=24, m=300_007, mix="preferential",
             ops=True, hint=True),
        # components under deletions, the costly direction for them (edge factor 32 stream)
        dict(name="cc_s20_50k", kind="repair", problem="cc", n=1 << 20, ef=32, m=50_000, mix="deletions"),
        # many small streams served together, uneven batch sizes
        dict(name="multi_bfs_16", kind="multi", problem="bfs", streams=16, n_lo=1 << 12, n_hi=1 << 17, m_lo=100,
             m_hi=20_000),
        # streams of all four problems served by one kernel a round
        dict(name="fused_4x4", kind="fused", streams=4, n_lo=1 << 12, n_hi=1 << 16, m_lo=100, m_hi=10_000),
        # a graph of which 23% fits the HBM pool
        dict(name="tiered_bfs_s20_20k", kind="repair", problem="bfs", n=1 << 20, ef=16, m=20_000, mix="deletions",
             hint=True, tiered=True),
        # the components from scratch on the resident graph
        dict(name="recompute_cc_2m", kind="recompute", problem="cc", n=2_000_003, ef=16),
        # the initial colouring of a stream
        dict(name="seed_coloring_500k", kind="seed", problem="coloring", n=500_009, ef=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["repair"] * 5 + ["tiered", "multi", "fused", "recompute", "seed"])
    if kind == "multi":
        return dict(kind="multi", problem=rng.choice(["bfs", "cc", "coloring", "mis"]), streams=rng.randint(2, 16),
                    n_lo=_log(rng, 1000, 8000), n_hi=_log(rng, 10_000, 1 << 17), m_lo=rng.randint(20, 200),
                    m_hi=_log(rng, 500, 20_000))
    if kind == "fused":
        return dict(kind="fused", streams=rng.randint(1, 4), n_lo=_log(rng, 1000, 8000),
                    n_hi=_log(rng, 10_000, 1 << 16), m_lo=rng.randint(20, 200), m_hi=_log(rng, 500, 10_000))
    if kind == "recompute":
        return dict(kind="recompute", problem=rng.choice(["bfs", "cc"]), n=_log(rng, 20_000, 2_000_000),
                    ef=rng.choice([8, 16]))
    if kind == "seed":
        return dict(kind="seed", problem=rng.choice(["coloring", "mis"]), n=_log(rng, 2000, 500_000),
                    ef=rng.choice([8, 16]))
    if kind == "tiered":
        n = _log(rng, 30_000, 1 << 20)
        return dict(kind="repair", problem=rng.choice(["bfs", "cc", "coloring", "mis"]), n=n, ef=rng.choice([8, 16]),
                    m=_log(rng, 200, min(20_000, n // 4)), mix=rng.choice(["deletions", "preferential"]), hint=True,
                    tiered=True)
    problem = rng.choice(["bfs", "cc", "coloring", "mis"])
    n = _log(rng, 2000, 1 << 20 if problem == "cc" else 4_000_000)
    ef = rng.choice([8, 16, 32] if n < 2_000_000 else [8, 16])
    return dict(kind="repair", problem=problem, n=n, ef=ef,
                m=_log(rng, 50, min(50_000 if problem == "cc" else 900_000, n * ef // 16)),
                mix=rng.choice(["preferential", "uniform", "deletions"]), hint=rng.random() < 0.5,
                ops=problem == "mis" and rng.random() < 0.5)


# ---- inputs ------------------------------------------------------------------------------
def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(0x5C0 + seed)
    return g


def _keys(n, ef, g):
    """Sorted keys u * n + v of the directed entries of an R-MAT graph of n vertices."""
    e = n * ef
    u = torch.zeros(e, dtype=torch.int32, device="cuda")
    v = torch.zeros_like(u)
    for _ in range((n - 1).bit_length()):
        r = torch.rand(e, generator=g, device="cuda")
        lower = r >= 0.76
        right = ((r >= 0.57) & (r < 0.76)) | (r >= 0.95)
        u.mul_(2).add_(lower)
        v.mul_(2).add_(right)
    ok = (u < n) & (v < n) & (u != v)
    u, v = u[ok].long(), v[ok].long()
    return torch.unique(torch.cat([u * n + v, v * n + u]))


def _member(keys, x):
    at = torch.searchsorted(keys, x).clamp_(max=max(len(keys) - 1, 0))
    return keys[at] == x


def _pick(keys, k, g):
    """k random directed entries, as keys."""
    return keys[torch.randint(len(keys), (k,), generator=g, device="cuda")]


def _edits(keys, n, m, batches, mix, g):
    """batches x m pairs (fewer where a small graph has no more), no pair twice; int32."""
    total = m * batches
    over = total + total // 2 + 64
    dele = {"preferential": 0.5, "uniform": 0.5, "deletions": 0.7}[mix]

    def canon(key):
        a, b = key // n, key % n
        return torch.minimum(a, b) * n + torch.maximum(a, b)

    def some(x, k):   # k distinct values of x, in random order
        x = torch.unique(x)
        return x[torch.randperm(len(x), generator=g, device="cuda")[:k]]

    if mix == "uniform":
        # random pairs hardly ever meet an edge: half the stream are edges, as toggling a
        # pair twice makes them
        out = _pick(keys, over, g)
    elif mix == "preferential":
        out = _pick(keys, over, g)
    else:
        deg = torch.bincount(keys // n, minlength=n)
        low = keys[(deg <= 2)[keys // n]]
        out = _pick(keys, over, g)
        if len(low):
            out = torch.cat([_pick(low, over * 3 // 10, g), out[: over * 7 // 10]])
    kept = some(canon(out), int(total * dele))
    more = 2 * total + 64
    if mix == "preferential":
        a, b = _pick(keys, more, g) // n, _pick(keys, more, g) // n
    else:
        a = torch.randint(n, (more,), generator=g, device="cuda")
        b = torch.randint(n, (more,), generator=g, device="cuda")
    new = torch.minimum(a, b) * n + torch.maximum(a, b)
    new = new[(a != b) & ~_member(keys, new)]
    new = some(new, total - len(kept))
    key = torch.cat([kept, new])
    ins = torch.cat([torch.zeros(len(kept), dtype=torch.bool, device="cuda"),
                     torch.ones(len(new), dtype=torch.bool, device="cuda")])
    p = torch.randperm(len(key), generator=g, device="cuda")
    key, ins = key[p], ins[p]
    a, b = key // n, key % n
    flip = torch.rand(len(key), generator=g, device="cuda") < 0.5
    pairs = torch.stack([torch.where(flip, b, a), torch.where(flip, a, b)], 1).to(torch.int32)
    return pairs, ins


def _graph(case, seed):
    """(sorted keys, edits, insertion flags) of a one-graph case; the same for the same seed."""
    g = _rng(seed)
    keys = _keys(case["n"], case["ef"], g)
    if "m" not in case:
        return keys, None, None
    pairs, ins = _edits(keys, case["n"], case["m"], CYCLE, case["mix"], g)
    return keys, pairs, ins


def _csr(keys, n):
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(keys // n, minlength=n), 0)
    return off.cpu().numpy(), (keys % n).to(torch.int32).cpu().numpy()


def _split(pairs, batches):
    """The stream's batches as int32 arrays of nearly equal size."""
    e = pairs.cpu().numpy()
    at = [len(e) * i // batches for i in range(batches + 1)]
    return [np.ascontiguousarray(e[at[i]:at[i + 1]]) for i in range(batches)]


def _model(problem):
    with np.load(os.path.join(os.path.dirname(sb.__file__), "sched_model.npz")) as d:
        return np.asarray(d[problem], dtype=np.float32)


def _prepare_repair(case, seed):
    n, problem = case["n"], case["problem"]
    keys, pairs, ins = _graph(case, seed)
    off, adj = _csr(keys, n)
    batches = _split(pairs, CYCLE)
    ctx = sb.Context(0)
    if case.get("tiered"):
        ctx.load_tiered(off, adj, hbm_entries=max(len(adj) * 23 // 100, 4096))
    else:
        ctx.load_csr(off, adj)
    ctx.seed(problem)
    mirror = ctx.download(problem)
    sched = {}
    if case.get("learned"):
        ctx.sched_install(problem, _model(problem))
        sched["policy"] = 1
    ctx.reserve_batches(max(len(b) for b in batches))
    if case.get("hint"):
        batches = [sb.pinned_copy(b) for b in batches]
    state = dict(ctx=ctx, problem=problem, batches=batches, mirror=mirror, sched=sched, at=0,
                 hint=bool(case.get("hint")), ops=None)
    if case.get("ops"):
        flags = ins.cpu().numpy()
        at = np.cumsum([0] + [len(b) for b in batches])
        there = [np.where(flags[at[i]:at[i + 1]], sb.OP_INSERT, sb.OP_DELETE).astype(np.uint8) for i in range(CYCLE)]
        back = [(sb.OP_INSERT + sb.OP_DELETE - o).astype(np.uint8) for o in there]
        state["ops"] = there + back
    return state


def _run_repair(s):
    ctx, problem, batches, at = s["ctx"], s["problem"], s["batches"], s["at"]
    s["at"] = at + 1
    if s["hint"]:
        ctx.prefetch(batches[(at + 1) % CYCLE])
    ctx.repair(problem, batches[at % CYCLE], ops=s["ops"][at % (2 * CYCLE)] if s["ops"] else None, sched=s["sched"])
    return s["mirror"], ctx.commit(problem, s["mirror"])


def _streams(case):
    """(vertices, edge factor, edits of a batch) of each stream: sizes spread over the case's
    ranges, large graphs not always with large batches."""
    k = case["streams"]

    def between(lo, hi, i):
        return int(lo * (hi / lo) ** ((i + 0.5) / k))

    out = []
    for i in range(k):
        n, ef = between(case["n_lo"], case["n_hi"], i), (8, 16, 32)[i % 3]
        out.append((n, ef, min(between(case["m_lo"], case["m_hi"], (5 * i + 2) % k), n * ef // 16)))
    return out


def _engine(problem, case, g):
    """A MultiEngine of the case's streams, its mirrors and its rounds of batches."""
    e = sb.MultiEngine(problem)
    mirrors, arrivals = [], []
    for n, ef, m in _streams(case):
        keys = _keys(n, ef, g)
        pairs, _ = _edits(keys, n, m, CYCLE, "preferential", g)
        off, adj = _csr(keys, n)
        init = sb.HostCsr.from_arrays(off, adj).init_state(problem)
        sid = e.add_stream(off, adj, init)
        mirrors.append(init.copy())
        arrivals.append([(sid, b) for b in _split(pairs, CYCLE)])
    # the streams' batches arrive interleaved; a round takes at most one of each stream
    rounds = sb.form_rounds([a[k] for k in range(CYCLE) for a in arrivals], max_edits=1_000_000)
    most = max(sum(len(b) for _, b in r) for r in rounds)
    e.reserve_batches(most)
    return dict(engine=e, mirrors=mirrors, rounds=rounds, at=0)


def _next_round(s):
    s["at"] += 1
    return s["rounds"][(s["at"] - 1) % len(s["rounds"])]


def _run_multi(s):
    s["engine"].round(_next_round(s))
    return s["mirrors"], s["engine"].commit(s["mirrors"])


def _run_fused(states):
    for s in states:
        s["engine"].stage(_next_round(s))
    sb.run_fused_round([s["engine"] for s in states])
    return [(s["mirrors"], s["engine"].commit(s["mirrors"])) for s in states]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "repair":
        return kind, _prepare_repair(case, seed)
    if kind == "multi":
        return kind, _engine(case["problem"], case, _rng(seed))
    if kind == "fused":
        g = _rng(seed)
        return kind, [_engine(p, case, g) for p in ("bfs", "cc", "coloring", "mis")]
    n, problem = case["n"], case["problem"]
    keys, _, _ = _graph(case, seed)
    off, adj = _csr(keys, n)
    ctx = sb.Context(0)
    ctx.load_csr(off, adj)
    mirror = np.full(n, -1, dtype=np.int32)
    if kind == "recompute":
        # levels unknown, every vertex a component of its own: what the first pass corrects
        ctx.upload(problem, mirror if problem == "bfs" else np.arange(n, dtype=np.int32))
        ctx.reserve_batches(1024)
    return kind, dict(ctx=ctx, problem=problem, mirror=mirror)


def run(state):
    kind, s = state
    if kind == "repair":
        return _run_repair(s)
    if kind == "multi":
        return _run_multi(s)
    if kind == "fused":
        return _run_fused(s)
    ctx, problem = s["ctx"], s["problem"]
    if kind == "seed":
        ctx.seed(problem)
        return ctx.download(problem)
    if problem == "bfs":
        ctx.recompute_bfs(0)
    else:
        ctx.recompute_cc()
    return s["mirror"], ctx.commit(problem, s["mirror"])


# ---- work --------------------------------------------------------------------------------
def _touched(n, ef, m, mix):
    """Entries of the distinct rows that a batch of m edits changes, from R-MAT's degree law."""
    bits = (n - 1).bit_length()
    nnz = 2.0 * n * ef
    ends = 2.0 * m
    got = 0.0
    for k in range(bits + 1):
        share = BIT_ONE ** k * (1 - BIT_ONE) ** (bits - k)
        deg = min(nnz * share, float(n))
        many = math.comb(bits, k) * n / 2.0 ** bits
        by_degree, by_vertex = ends * share, ends / n
        hit = by_degree if mix == "preferential" else 0.5 * (by_degree + by_vertex)
        got += many * deg * -math.expm1(-hit)
    return min(got, nnz)


def _repair_bytes(n, ef, m, mix):
    # the edits; the changed rows read and written once; per half-edit its vertex's descriptor
    # and value, read and written
    return 8.0 * m + 8.0 * _touched(n, ef, m, mix) + 2.0 * m * 2 * (16 + 4)


def work(case):
    kind = case["kind"]
    if kind == "repair":
        b = _repair_bytes(case["n"], case["ef"], case["m"], case["mix"])
    elif kind in ("multi", "fused"):
        b = sum(_repair_bytes(n, ef, m, "preferential") for n, ef, m in _streams(case))
        b *= 4 if kind == "fused" else 1
    else:   # every row read once, every value written once
        b = 8.0 * case["n"] * case["ef"] + (8 + 4) * case["n"]
        if kind == "seed":
            b += 4.0 * case["n"]   # the solution copied to the host
    return {"bytes": b, "flops": 0}


# ---- exact values ------------------------------------------------------------------------
def _levels(src, dst, n):
    lv = torch.full((n,), -1, dtype=torch.int64, device=src.device)
    lv[0] = 0
    d = 0
    while True:
        t = dst[lv[src] == d]
        t = t[lv[t] < 0]
        if not len(t):
            return lv
        d += 1
        lv[t] = d


def _labels(src, dst, n):
    lab = torch.arange(n, device=src.device)
    while True:
        new = lab.scatter_reduce(0, src, lab[dst], "amin")
        while True:
            up = new[new]
            if torch.equal(up, new):
                break
            new = up
        if torch.equal(new, lab):
            return lab
        lab = new


def exact(case, seed):
    if case["kind"] not in ("repair", "recompute") or case["problem"] not in ("bfs", "cc"):
        return None
    n = case["n"]
    keys, pairs, _ = _graph(case, seed)
    if pairs is not None:
        first = pairs[: len(pairs) // CYCLE].long()
        t = torch.cat([first[:, 0] * n + first[:, 1], first[:, 1] * n + first[:, 0]])
        gone = torch.sort(t[_member(keys, t)]).values
        keep = keys[~_member(gone, keys)] if len(gone) else keys
        keys = torch.cat([keep, t[~_member(keys, t)]])
    src, dst = keys // n, keys % n
    sol = _levels(src, dst, n) if case["problem"] == "bfs" else _labels(src, dst, n)
    return sol.to(torch.int32).cpu().numpy(), None
