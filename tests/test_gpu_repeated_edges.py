"""Prepare of a small group in a graph with repeated edges, whose counts are beyond
their block's capacity: such an entry's approximate old cost is negative, and a
member's sum may pass through zero on the way (AddRowEntry in
beam_gb300/csrc/merge.cu). Against the oracle, which sums in 64 bits."""

import numpy as np
import pytest


def edges(copies, targets):
    """Member 0 lists `targets` nodes, the first of them `copies` times. Members
    1 and 2 share ten targets, and one each with member 0; so does member 3."""
    x, y, z = 4, 4 + targets, 4 + targets + 10
    e = [(0, x)] * copies + [(0, x + k) for k in range(1, targets)]
    e += [(m, x + targets - m) for m in (1, 2, 3)]
    e += [(m, y + k) for m in (1, 2) for k in range(10)] + [(3, z + k) for k in range(6)]
    return zip(*e)


CASES = [(40, 64), (33, 33), (200, 220), (36, 40), (1, 64), (5, 20)]


def test_oracle_pairs_the_members_that_share_most():
    from beam_gb300 import Graph
    from oracle import Oracle
    for copies, targets in CASES[:2]:
        o = Oracle.from_graph(Graph.from_edges(*map(list, edges(copies, targets))), top_k=1)
        assert [1, 2] in o.prepare_group([0, 1, 2, 3]).tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("copies,targets", CASES)
@pytest.mark.parametrize("q", [[0, 1, 2, 3], [3, 0, 2, 1], [2, 1, 0]])
def test_small_groups_match_the_oracle(copies, targets, q):
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    g = Graph.from_edges(*map(list, edges(copies, targets)))
    o = Oracle.from_graph(g, top_k=1)
    with Engine(g, top_k=1) as e:
        assert np.array_equal(e.prepare_group(q), o.prepare_group(q))


def twins_with_leaves(clusters):
    """Pairs of twins with six targets of their own; the first twin has a leaf too.
    Edges and the leaf edges, one of each a cluster."""
    c = 9 * np.arange(clusters)
    e = [(c + m, c + 2 + t) for m in (0, 1) for t in range(6)]
    u, v = (np.concatenate(x) for x in zip(*e))
    return u, v, np.stack([c, c + 8], 1)


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [700, 1024, 1025, 4096, 1 << 30])
def test_large_blocks_check_counts_at_the_merged_size(batch):
    """A leaf edge given twice is beyond the capacity of two single nodes, but
    not beyond that of the merged twins and the leaf. Blocks of more than 256
    groups of two members or more accept the merge (smaller ones report the
    state, as the reference does). The leaf, alone in its group, takes part in
    no pair, and the twins' gain of 5 for 6 decides nothing: the partition is the
    one of the graph without repeated edges."""
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    u, v, leaf = twins_with_leaves(2000)
    once = Graph.from_edges(np.concatenate([u, leaf[:, 0]]).astype(np.int32),
                            np.concatenate([v, leaf[:, 1]]).astype(np.int32))
    kw = {"ea_use_threshold": True, "group_batch_size": batch}
    o = Oracle.from_graph(once, **kw)
    o.divide(4)
    order, starts, lengths = o.groups()
    real = np.array([(lengths[i:i + batch] >= 2).sum() for i in range(0, len(lengths), batch)])
    group = np.zeros(once.n, int)
    group[order] = np.repeat(np.arange(len(starts)), lengths)
    first, alone = group[leaf[:, 0]], lengths[group[leaf[:, 1]]] == 1
    twice = leaf[(first == group[leaf[:, 0] + 1]) & alone & (real[first // batch] > 256)]
    assert len(twice) > 100
    g = Graph.from_edges(np.concatenate([u, leaf[:, 0], twice[:, 0]]).astype(np.int32),
                         np.concatenate([v, leaf[:, 1], twice[:, 1]]).astype(np.int32))
    o.merge(4)
    assert (o.labels()[twice[:, 0] + 1] == twice[:, 0]).sum() > 100
    with Engine(g, **kw) as e:
        e.divide(4)
        e.merge(4)
        assert np.array_equal(e.partition()[0], o.labels())
        e.validate_quotient()
