"""Encoding metrics without files (counts from the quotient rows) and with them
(lists), and the exact partition cost from the input graph, against the host
versions: singletons, a merged state, complete and missing blocks, rows on both
sides of the long-row limit, node counts at powers of two (the bits of the
packed sort keys)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def star(leaves):
    return np.zeros(leaves, np.int32), np.arange(1, leaves + 1, dtype=np.int32)


def bicliques():
    """K(5, 7) complete and K(6, 6) without two edges, tied by one edge."""
    e = [(i, 5 + j) for i in range(5) for j in range(7)]
    e += [(12 + i, 18 + j) for i in range(6) for j in range(6) if (i, j) not in ((0, 0), (3, 4))]
    u, v = zip(*(e + [(0, 12)]))
    return np.array(u, np.int32), np.array(v, np.int32)


CASES = {"edge": star(1), "star1024": star(1024), "star1025": star(1025), "star5000": star(5000), "pow2": star(4095),
         "bicliques": bicliques()}


@pytest.mark.parametrize("case", [*CASES, "rmat:scale=13,ef=6,a=0.57,b=0.19,c=0.19,seed=9",
                                  "dcsbm:n=3000,blocks=32,ratio=40,gamma=2.5,deg=31,seed=2"])
def test_counts_match_the_lists_and_the_host(case, tmp_path):
    from beam_gb300 import Engine, Graph
    g = Graph.from_edges(*CASES[case]) if case in CASES else Graph.generate(case)
    with Engine(g, group_batch_size=1 << 30) as e:
        for step in range(3):
            labels, head, nxt = e.partition()
            want = g.encode(head, nxt)
            assert e.encode() == want
            assert e.encode(tmp_path) == want
            assert e.exact_partition_cost() == g.exact_partition_cost(labels)
            if step == 0 and case == "bicliques":
                e.merge_pairs([0, 5, 12, 18], [1, 6, 13, 19])
            else:
                e.divide(step + 1)
                e.merge(step + 1, 20)
