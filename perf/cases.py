"""What a user of the library has it do, as cases that can be measured.

Five kinds of call:

  run      a whole merge run on a resident engine (reset, 20 iterations, the
           partition and the work counters read back); `batch` is
           group_batch_size: 64 is the reference's block size and the library's
           default (plain form), 1 << 30 one block per iteration (batched form),
           and the block-size tuner picks sizes in between
  fresh    a whole summary of a graph in hand: engine created from the host
           CSR, 20 iterations, encoding metrics, partition, engine closed
  encode   the encoding metrics and the exact partition cost of a summary
  pairs    the exact-gain service for explicit pairs of a resident quotient
           graph (host arrays in and out)
  flat     the legacy-objective scoring service of one block (host arrays in
           and out)

Graphs are the seeded generators of the library with its tests' and
benchmark's parameters; the case's seed is the generator's.
"""

import numpy as np

from beam_gb300 import Engine, FlatScorer, Graph

ALL = 1 << 30  # one block of every group of an iteration

# the work counters that do not depend on how the kernels do the work
COUNTERS = ("merge_group_count", "merge_group_max_size", "merge_raw_pair_count", "merge_candidate_pairs_after_prune",
            "candidate_proxy_pairs_examined", "merge_exact_gain_calls", "exact_gain_input_nnz",
            "exact_raw_entries_a", "exact_raw_entries_b", "exact_union_neighbors", "exact_overlap_neighbors",
            "merge_positive_gain_pairs", "merge_rejected_by_threshold", "merge_rejected_by_overlap",
            "merge_candidate_pairs", "merge_selected_pairs", "merge_total_local_gain", "isolated_gain_sum",
            "selected_merges_for_validation", "validation_exact_calls", "validation_exact_row_entry_work",
            "accepted_merges_after_validation", "rejected_nonpositive", "update_touched_quotient_entries",
            "divide_max_group_size", "divide_fallback_splits")


def listed():
    return [
        # the reference's mode on its smallest kind of input: latency of the block chain
        {"name": "plain_rmat12", "kind": "run", "graph": "rmat", "scale": 12, "ef": 4, "batch": 64},
        # the reference's mode on a graph with planted twins: many merges, groups that depend on each other
        {"name": "plain_chunglu20k", "kind": "run", "graph": "chunglu", "n": 20000, "deg": 8, "twins": 1500,
         "batch": 64},
        # the reference's mode on a mid-sized skewed graph (hub rows of thousands of entries)
        {"name": "plain_rmat16", "kind": "run", "graph": "rmat", "scale": 16, "ef": 8, "batch": 64},
        # the block size that the tuner picks for a road-like and a skewed component together
        {"name": "blocks16k_union", "kind": "run", "graph": "union", "side": 1400, "n": 1100000, "batch": 16384},
        # the batched form on a sparse graph: short kernels, launches and host round trips count
        {"name": "batched_rmat19", "kind": "run", "graph": "rmat", "scale": 19, "ef": 2, "batch": ALL},
        # the batched form on a graph of planted twins
        {"name": "batched_chunglu1m", "kind": "run", "graph": "chunglu", "n": 1000001, "deg": 17, "twins": 50000,
         "batch": ALL},
        # the largest: the batched form at edge factor 16, tens of GB resident
        {"name": "batched_rmat23", "kind": "run", "graph": "rmat", "scale": 23, "ef": 16, "batch": ALL},
        # the batched form with the learned candidate ranker
        {"name": "ranker_rmat20", "kind": "run", "graph": "rmat", "scale": 20, "ef": 16, "batch": ALL,
         "ranker": True},
        # one small graph summarised from scratch, engine creation and all
        {"name": "fresh_dcsbm4096", "kind": "fresh", "graph": "dcsbm", "n": 4096, "blocks": 32, "deg": 43,
         "batch": ALL},
        # encoding metrics of a finished summary
        {"name": "encode_rmat20", "kind": "encode", "graph": "rmat", "scale": 20, "ef": 16, "batch": ALL},
        # pairs inside the groups of a half-merged quotient graph, as an embedding host asks for them
        {"name": "pairs_rmat20", "kind": "pairs", "graph": "rmat", "scale": 20, "ef": 16, "batch": ALL,
         "pairs": 262144},
        # one 64-group block of the reference's own CUDA mode, through the adapter's service
        {"name": "flat_block", "kind": "flat", "rows": 701, "deg": 40, "pairs": 6007},
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def _draw_graph(rng, largest):
    """Graph parameters with at most about `largest` edges."""
    graph = rng.choice(("rmat", "rmat", "chunglu", "union", "dcsbm"))
    if graph == "rmat":
        ef = rng.choice((2, 3, 4, 8, 11, 16))
        top = 10
        while top < 23 and (ef << (top + 1)) <= largest:
            top += 1
        return {"graph": graph, "scale": rng.randint(min(10, top), top), "ef": ef}
    if graph == "chunglu":
        deg = rng.choice((5, 8, 17))
        n = _spread(rng, 2000, max(2001, largest // (2 * deg)))
        return {"graph": graph, "n": n, "deg": deg, "twins": n // rng.choice((10, 20, 50))}
    if graph == "union":
        side = _spread(rng, 30, max(31, min(1400, int((largest / 5) ** 0.5))))
        return {"graph": graph, "side": side, "n": max(500, side * side // 2 + 1)}
    deg = rng.choice((16, 31, 43))
    return {"graph": graph, "n": _spread(rng, 1000, max(1001, min(300000, largest // deg))), "blocks": 32, "deg": deg}


def draw(rng):
    kind = rng.choice(("plain", "plain", "plain", "blocks", "batched", "batched", "batched", "ranker", "fresh",
                       "encode", "pairs", "flat"))
    if kind == "flat":
        return {"kind": "flat", "rows": _spread(rng, 65, 6000), "deg": _spread(rng, 4, 200),
                "pairs": _spread(rng, 100, 60000)}
    if kind == "plain":
        return {"kind": "run", **_draw_graph(rng, 400000), "batch": rng.choice((64, 64, 64, 33, 100))}
    if kind == "blocks":
        return {"kind": "run", **_draw_graph(rng, 3000000), "batch": rng.choice((4096, 10000, 16384, 65536))}
    if kind in ("batched", "ranker"):
        c = {"kind": "run", **_draw_graph(rng, 32000000), "batch": ALL}
        return {**c, "ranker": True} if kind == "ranker" else c
    if kind == "fresh":
        return {"kind": "fresh", **_draw_graph(rng, 2000000), "batch": ALL}
    c = {"kind": kind, **_draw_graph(rng, 16000000), "batch": ALL}
    return {**c, "pairs": _spread(rng, 1000, 400000)} if kind == "pairs" else c


def _nodes(case):
    if case["graph"] == "rmat":
        return 1 << case["scale"]
    return case["n"] + (case["side"] ** 2 if case["graph"] == "union" else 0)


def _graph(case, seed):
    kind = case["graph"]
    if kind == "rmat":
        spec = f"rmat:scale={case['scale']},ef={case['ef']},a=0.57,b=0.19,c=0.19,seed={seed}"
    elif kind == "chunglu":
        spec = f"chunglu:n={case['n']},gamma=2.3,deg={case['deg']},twins={case['twins']},seed={seed}"
    elif kind == "union":
        spec = (f"union:side={case['side']},del=0.10,diag=0.02,n={case['n']},gamma=2.1,deg=5.4,"
                f"maxdeg={max(50, case['n'] // 40)},seed={seed}")
    else:
        spec = f"dcsbm:n={case['n']},blocks={case['blocks']},ratio=40,gamma=2.5,deg={case['deg']},seed={seed}"
    g = Graph.generate(spec)
    # ids up to the generator's own number of nodes: the last ones may be
    # isolated, which the edge list alone does not show
    extra = _nodes(case) - g.n
    if extra > 0:
        g.row_ptr = np.concatenate([g.row_ptr, np.full(extra, g.arcs, g.row_ptr.dtype)])
        g.n += extra
    return g


def _engine(case, g):
    return Engine(g, group_batch_size=case["batch"], ea_use_threshold=True, ranker=bool(case.get("ranker", False)))


def _flat_block(case, rng):
    """A block's rows as the reference aggregates them: sorted neighbours, some
    rows listing their own representative, a hub row here and there."""
    rows, ids = case["rows"], 40 * case["rows"]
    reps = np.sort(rng.choice(ids, size=rows, replace=False)).astype(np.int32)
    size_of = rng.integers(1, 50, size=ids)
    nb, offsets = [], [0]
    for i in range(rows):
        deg = min(ids // 2, 40 * case["deg"] if i % 97 == 0 else int(rng.integers(0, 2 * case["deg"])))
        row = np.unique(rng.integers(0, ids, size=deg))
        if i % 3 == 0:
            row = np.union1d(row, reps[i:i + 1])
        nb.append(row)
        offsets.append(offsets[-1] + len(row))
    nb = np.concatenate(nb).astype(np.int32)
    rsz = size_of[reps]
    owner = np.repeat(np.arange(rows), np.diff(offsets))
    cap = np.where(nb == reps[owner], rsz[owner] * (rsz[owner] - 1) // 2, rsz[owner] * size_of[nb])
    flat = {"offsets": np.asarray(offsets, np.int32), "reps": reps, "rsz": rsz.astype(np.int64),
            "self": (rsz * (rsz - 1) // 6).astype(np.int64), "nb": nb,
            "wt": 1 + rng.integers(0, 1 << 30, size=len(nb)) % np.maximum(cap, 1),
            "nsz": size_of[nb].astype(np.int64)}
    a = rng.integers(0, rows, size=case["pairs"])
    b = (a + rng.integers(1, 20, size=case["pairs"])) % rows
    return flat, np.stack([np.minimum(a, b), np.maximum(a, b)], axis=1).astype(np.int32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "flat":
        flat, pairs = _flat_block(case, np.random.default_rng(seed))
        return {"case": case, "scorer": FlatScorer(), "flat": flat, "pairs": pairs}
    g = _graph(case, seed)
    if kind == "fresh":
        return {"case": case, "graph": g}
    e = _engine(case, g)
    state = {"case": case, "engine": e}
    if kind == "encode":
        e.run(20)
    elif kind == "pairs":
        e.run(5)
        e.divide(6)
        order, starts, lengths = e.groups()
        real = np.flatnonzero(lengths >= 2)
        rng = np.random.default_rng(seed)
        gi = rng.choice(real, size=case["pairs"])
        i = rng.integers(0, lengths[gi])
        j = (i + 1 + rng.integers(0, lengths[gi] - 1)) % lengths[gi]
        state["a"], state["b"] = order[starts[gi] + i], order[starts[gi] + j]
    return state


def _summary(e):
    labels, head, nxt = e.partition()
    st = e.stats()
    return {"labels": labels, "head": head, "next": nxt, **{k: st[k] for k in COUNTERS}}


def run(state):
    kind = state["case"]["kind"]
    if kind == "run":
        e = state["engine"]
        e.reset()
        e.run(20)
        return _summary(e)
    if kind == "fresh":
        with _engine(state["case"], state["graph"]) as e:
            e.run(20)
            return {**_summary(e), **e.encode()}
    if kind == "encode":
        return {**state["engine"].encode(), "cost": state["engine"].exact_partition_cost()}
    if kind == "pairs":
        gain, before = state["engine"].score_pairs(state["a"], state["b"])
    else:
        gain, before = state["scorer"].score(state["flat"], state["pairs"])
    return {"gain": gain, "before": before}


def _edges(case):
    if case["graph"] == "rmat":
        return case["ef"] << case["scale"]
    if case["graph"] == "union":
        return 2 * case["side"] ** 2 + 3 * case["n"]
    return case["n"] * case["deg"] // 2


def work(case):
    if case["kind"] == "flat":
        # 20 B per entry, 24 B per row and 24 B per pair
        entries = case["rows"] * case["deg"] * 1.4
        return {"bytes": 20 * entries + 24 * case["rows"] + 24 * case["pairs"], "flops": 0}
    nodes = _nodes(case)
    csr = 8 * _edges(case) + 8 * nodes
    if case["kind"] == "pairs":
        # both rows of every pair (8 B an entry, the mean row), ids in and results out
        return {"bytes": case["pairs"] * (24 + 16 * (1 + 2 * _edges(case) / nodes)), "flops": 0}
    if case["kind"] == "encode":
        return {"bytes": csr + 4 * nodes, "flops": 0}
    # the graph in, three words per node out
    return {"bytes": csr + 12 * nodes, "flops": 0}
