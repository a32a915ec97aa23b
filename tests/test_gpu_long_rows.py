"""Neighbour rows longer than the rewrite kernels stage in shared memory
(beam_gb300/csrc/merge.cu, ScanHugeRows and RewriteHugeKernel): a hub's row
after an explicit batch of merges of its neighbours, against the row made from
the merged ids. Lengths around the row limit and the chunk size; entries that
fold into one already there, that move left, that move right, and more
insertions than a chunk holds."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def hub_graph(length, outside, low):
    """Hub with `length` neighbours and as many nodes as `outside` not listed by
    it (tied to one another), with ids below (low) or above the neighbours."""
    a, b = (1, 1 + outside) if low else (1 + length, 1)
    out, nbr = np.arange(a, a + outside), np.arange(b, b + length)
    u = np.concatenate([np.zeros(length, np.int32), out[:-1]]).astype(np.int32)
    v = np.concatenate([nbr, out[1:]]).astype(np.int32)
    return u, v, out, nbr


@pytest.mark.parametrize("length", [2048, 2049, 8191, 8192, 8193, 16384, 20011])
@pytest.mark.parametrize("kind", ["fold", "left", "right", "mixed", "all_right"])
def test_hub_row_after_merges(length, kind):
    from beam_gb300 import Engine, Graph
    rng = np.random.default_rng(length)
    count = {"all_right": length, "fold": length // 2}.get(kind, min(length, 97))
    u, v, out, nbr = hub_graph(length, max(2, count), kind in ("right", "all_right", "mixed"))
    g = Graph.from_edges(u, v)
    picked = rng.permutation(nbr)
    if kind == "fold":      # both ends are listed by the hub
        keep, rem = picked[:count], picked[count:2 * count]
    else:                   # the kept end is not
        keep, rem = rng.permutation(out)[:count], picked[:count]
        if kind == "mixed":
            keep, rem = np.concatenate([keep, picked[count:count + 40]]), np.concatenate([rem, picked[count + 40:count + 80]])
    into = np.arange(g.n)
    into[rem] = keep
    with Engine(g) as e:
        e.merge_pairs(keep, rem)
        got_nb, got_cnt, _, _ = e.row(0)
        ids, counts = np.unique(into[nbr], return_counts=True)
        assert np.array_equal(got_nb, ids)
        assert np.array_equal(got_cnt, counts)
        e.validate_quotient()


@pytest.mark.parametrize("longer,shorter,tied", [(1024, 1024, False), (1025, 1024, True), (2048, 1, False),
                                                 (2049, 0, False), (3072, 3072, True), (3073, 700, True),
                                                 (9001, 5000, True)])
def test_scores_of_long_pairs(longer, shorter, tied):
    """ScorePairsKernel's pairs in units (ScoreLongPairsKernel) against the
    oracle, around the length limit and the unit; some neighbours merged."""
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    rng = np.random.default_rng(longer + shorter)
    n = 3 + longer + shorter
    u = [np.full(longer, 0), np.full(shorter, 1), [2]]
    v = [3 + rng.choice(n - 3, longer, replace=False), 3 + rng.choice(n - 3, shorter, replace=False), [3]]
    if tied:
        u.append([0])
        v.append([1])
    g = Graph.from_edges(np.concatenate(u).astype(np.int32), np.concatenate(v).astype(np.int32))
    o = Oracle.from_graph(g)
    with Engine(g) as e:
        ends = 3 + rng.permutation(g.n - 3)[:40]
        for k, r in zip(ends[:20].tolist(), ends[20:].tolist()):
            o.merge_pair(k, r)
        e.merge_pairs(ends[:20], ends[20:])
        pairs = [(0, 1), (1, 0), (0, 2), (2, 1), (0, int(ends[0])), (int(ends[3]), 1)]
        gain, before = e.score_pairs([a for a, _ in pairs], [b for _, b in pairs])
        for i, (a, b) in enumerate(pairs):
            assert (gain[i], before[i]) == o.exact_gain(a, b), (a, b)


def test_first_rows_of_long_adjacency_lists():
    """The rows that InitRowsKernel and InitLongRowsKernel make: lengths around
    the row limit and the tile, arcs given twice and more (also across a tile's
    border), several long rows to a block of the grid."""
    from beam_gb300 import Engine, Graph
    rng = np.random.default_rng(8)
    lengths = [511, 512, 513, 4095, 4096, 4097, 8192, 8193, 20001] + [600] * 700
    hubs = len(lengths)
    u, v = [], []
    for i, length in enumerate(lengths):
        nb = hubs + np.sort(rng.choice(21000, length, replace=False))
        if i % 2:  # some arcs repeated, in all as many as the length says
            nb = np.sort(np.concatenate([nb[:length - length // 3], nb[:length // 3]]))
        if i == 7:
            nb[4000:4200] = nb[4000]
        u.append(np.full(length, i)), v.append(nb)
    g = Graph.from_edges(np.concatenate(u), np.concatenate(v))
    with Engine(g) as e:
        for i in range(hubs):
            if i > 12 and i % 50:
                continue
            nbrs, cnts, _, _ = e.row(i)
            ids, counts = np.unique(v[i], return_counts=True)
            assert np.array_equal(nbrs, ids) and np.array_equal(cnts, counts)


@pytest.mark.parametrize("scale", [9, 10, 11, 12, 13, 14, 15])
@pytest.mark.parametrize("limit", [48, 512])
def test_sort_slots_of_large_groups(scale, limit):
    """Groups whose shared targets are found by a sort: target widths and numbers
    of groups that leave out from none to several bits of the group index."""
    from beam_gb300 import Engine, Graph, partition_hash
    from oracle import Oracle
    g = Graph.generate(f"rmat:scale={scale},ef=24,a=0.57,b=0.19,c=0.19,seed={scale}")
    kw = {"ea_use_threshold": True, "group_batch_size": 1 << 30, "divide_max_group": limit}
    o = Oracle.from_graph(g, **kw)
    o.run(3)
    with Engine(g, **kw) as e:
        e.run(3)
        assert partition_hash(e.partition()[0]) == o.partition_hash()
        st, ost = e.stats(), o.stats()
        for k in ("candidate_proxy_pairs_examined", "exact_gain_input_nnz", "merge_total_local_gain"):
            assert st[k] == ost[k], k


@pytest.mark.parametrize("length", [1, 127, 128, 129, 383, 1000])
def test_divide_over_rows_of_whole_steps(length):
    """MinHashKernel's steps that lie in one row: hubs whose rows begin and end
    on, before and behind a step, the last row of the graph among them."""
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    rng = np.random.default_rng(length)
    hubs, leaves = 40, 3000
    u = np.repeat(np.arange(hubs), length)
    v = np.concatenate([hubs + rng.choice(leaves, length, replace=False) for _ in range(hubs)])
    last = np.full(1024, hubs + leaves)
    g = Graph.from_edges(np.concatenate([u, last]), np.concatenate([v, hubs + np.arange(1024)]))
    o = Oracle.from_graph(g, divide_max_group=16)
    with Engine(g, divide_max_group=16) as e:
        for it in (1, 2, 3):
            e.divide(it), o.divide(it)
            for a, b in zip(e.groups(), o.groups()):
                assert np.array_equal(a, b)
            e.merge(it), o.merge(it)
