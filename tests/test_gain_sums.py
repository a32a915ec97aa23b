"""The exact gain made from sums (RowSums, the pair words and GainFromSums in
beam_gb300/csrc/merge.cu) against the sum over the union of the two rows
(QuotientGraph::ExactMergeGainPersistentImpl): restated in Python on rows with
light entries, dense entries of one and of several size limits, and counts
beyond their block; and the kernels against the oracle on graphs whose
supernodes turn dense. Integer work: every value must be equal."""

import random

import pytest


def f(s, sx, c):
    return min(c, 1 + s * sx - c)


def row_sums(row, s, size):
    r = {"before": 0, "light": 0, "hsx": 0, "hc": 0, "n": 0, "smin": 1 << 40, "smax": 0, "sbad": 0}
    for x, c in row.items():
        sx = size[x]
        r["before"] += f(s, sx, c)
        if 1 + (s + 1) * sx < 2 * c:
            lim = (2 * c - 2) // sx
            r["hsx"] += sx
            r["hc"] += c
            r["n"] += 1
            r["smin"], r["smax"] = min(r["smin"], lim), max(r["smax"], lim)
            r["sbad"] = max(r["sbad"], -(-c // sx))
        else:
            r["light"] += c
    return r


def row_after(r, s, row, size, seen):
    if r["n"] == 0:
        seen.add("light")
        return r["light"]
    if s <= r["smin"]:
        seen.add("dense")
        return r["light"] + r["n"] + s * r["hsx"] - r["hc"]
    if s > r["smax"]:
        seen.add("past")
        return r["light"] + r["hc"]
    seen.add("read")
    return sum(f(s, size[x], c) for x, c in row.items())


def test_gain_from_sums_equals_the_sum_over_the_union():
    rng = random.Random(5)
    seen = set()
    for trial in range(4000):
        size = {x: rng.choice((1, 1, 1, 2, 3, 7, 40)) for x in range(12)}
        a, b = 0, 1
        top = rng.choice((1.0, 1.0, 0.3, 1.4))  # 1.4: counts beyond the capacity
        rows = {}
        for r in (a, b):
            rows[r] = {x: max(1, int(size[r] * size[x] * rng.uniform(0, top)))
                       for x in range(2, 12) if rng.random() < 0.6}
        eab = rng.randint(0, size[a] * size[b])
        if eab:
            rows[a][b] = rows[b][a] = eab
        sa, sb = size[a], size[b]
        s = sa + sb
        # the sum over the union
        before = after = 0
        bad = False
        for x in set(rows[a]) | set(rows[b]):
            if x in (a, b):
                continue
            ca, cb = rows[a].get(x, 0), rows[b].get(x, 0)
            before += (f(sa, size[x], ca) if ca else 0) + (f(sb, size[x], cb) if cb else 0)
            after += f(s, size[x], ca + cb)
            bad |= ca > sa * size[x] or cb > sb * size[x]
        before += f(sa, sb, eab)
        # from the sums
        ra, rb = row_sums(rows[a], sa, size), row_sums(rows[b], sb, size)
        proxy = corr = ovl = 0
        for x in set(rows[a]) & set(rows[b]):
            ca, cb, sx = rows[a][x], rows[b][x], size[x]
            d = max(0, f(sa, sx, ca) + f(sb, sx, cb) - f(s, sx, ca + cb))
            t = f(s, sx, ca + cb) - f(s, sx, ca) - f(s, sx, cb) + d
            if 2 * ca <= 1 + sa * sx and 2 * cb <= 1 + sb * sx:
                assert t == 0  # no second atomic where both entries are sparse
            proxy, corr, ovl = proxy + d, corr + t, ovl + 1
        shared = corr - proxy
        got_before = ra["before"] + rb["before"] - f(sb, sa, eab)
        got_after = (row_after(ra, s, rows[a], size, seen) + row_after(rb, s, rows[b], size, seen) -
                     f(s, sb, eab) - f(s, sa, eab) + shared)
        assert (got_before, got_after) == (before, after)
        assert (sa < ra["sbad"] or sb < rb["sbad"]) == bad
        assert ovl == len((set(rows[a]) & set(rows[b])) - {a, b})
    assert seen == {"light", "dense", "past", "read"}


def test_pair_words_hold_their_range():
    """Field bounds of the pair words for graphs of fewer than 2^30 arcs."""
    arcs = (1 << 30) - 1
    edges = arcs // 2
    assert 2 * edges + edges < 1 << 34          # two rows' counts and the direct edges
    assert arcs // 4 < 1 << 28                  # targets two rows share (both list them, both are listed)
    assert 6 * edges < 1 << 35                  # |corr| stays below half of the mark of a bad target
    assert all((k << 36) % (1 << 64) for k in (1, 7, (1 << 28) - 1))


def planted(kind, seed):
    """Edges of groups of near twins (same neighbours, a few missing) over a
    random background: merged supernodes have rows of dense entries, with one
    or several size limits."""
    rng = random.Random(seed)
    n, edges = 1200, set()
    for g in range(30):
        members = rng.sample(range(600), 2 + g % 9)
        targets = rng.sample(range(600, n), 4 if kind == "short" else 60)
        for u in members:
            for v in targets:
                if rng.random() < (1.0 if g % 2 else 0.9):
                    edges.add((u, v))
        if g % 3 == 0:
            edges |= {(min(u, v), max(u, v)) for u in members for v in members if u != v}
    for _ in range(2500):
        u, v = rng.sample(range(n), 2)
        edges.add((min(u, v), max(u, v)))
    u, v = zip(*sorted(edges))
    return list(u), list(v)


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [64, 300, 1 << 30])
@pytest.mark.parametrize("kind,max_group", [("short", 512), ("long", 512), ("long", 30), ("long", 1024)])
def test_dense_supernodes_match_the_oracle(kind, max_group, batch):
    from beam_gb300 import Engine, Graph, partition_hash
    from oracle import Oracle
    g = Graph.from_edges(*planted(kind, 3))
    kw = dict(group_batch_size=batch, divide_max_group=max_group, ea_use_threshold=True)
    o = Oracle.from_graph(g, **kw)
    o.run(20)
    with Engine(g, **kw) as e:
        e.run(20)
        assert partition_hash(e.partition()[0]) == o.partition_hash()
        st, ost = e.stats(), o.stats()
    for k in ("accepted_merges_after_validation", "merge_exact_gain_calls", "candidate_proxy_pairs_examined",
              "merge_positive_gain_pairs", "merge_total_local_gain", "exact_gain_input_nnz", "exact_union_neighbors",
              "exact_overlap_neighbors", "update_touched_quotient_entries"):
        assert st[k] == ost[k], k
