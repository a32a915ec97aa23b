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
