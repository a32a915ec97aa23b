"""prepare_group of a group that lists a supernode more than once: its copies tie
with each other as partners, so more pairs are kept than the members' top_k make
room for otherwise (cand_off in PrepareIterationBuffers)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def groups(order, rng):
    yield np.repeat(order[-1:], 6)                   # one warp (240 entries at most)
    yield np.repeat(order[:1], 32)                   # one block, many entries
    yield np.repeat(order[:2], 24)                   # one block, 48 members
    yield np.repeat(order[:9], 60)                   # sorted, 540 members
    yield np.repeat(order[:1], 1024)                 # the largest
    yield rng.permutation(np.concatenate([order[:200], order[:150], order[:20]]))


@pytest.mark.parametrize("top_k", [1, 3])
def test_every_kept_pair_has_its_place(top_k):
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    g = Graph.generate("rmat:scale=12,ef=8,a=0.57,b=0.19,c=0.19,seed=9")
    o = Oracle.from_graph(g, top_k=top_k, ea_use_threshold=True)
    rng = np.random.default_rng(4)
    order = np.argsort(-np.diff(g.row_ptr))[:300].astype(np.int32)
    assert np.diff(g.row_ptr)[order[-1]] <= 40
    with Engine(g, top_k=top_k, ea_use_threshold=True) as e:
        for q in groups(order[30:], rng):
            pairs = e.prepare_group(q)
            assert len(pairs) and (pairs[:, 0] < pairs[:, 1]).all() and pairs.max() < len(q) and pairs.min() >= 0
            key = pairs[:, 0].astype(np.int64) * len(q) + pairs[:, 1]
            assert (np.diff(key) > 0).all()
        # what lies beside the candidates is as it was
        e.run(5)
        o.run(5)
        assert np.array_equal(e.partition()[0], o.labels())
        e.validate_quotient()


def test_all_pairs_are_the_oracles():
    """With top_k beyond the group every positive pair is kept, copies or not."""
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    g = Graph.generate("rmat:scale=12,ef=8,a=0.57,b=0.19,c=0.19,seed=9")
    order = np.argsort(-np.diff(g.row_ptr))[:300].astype(np.int32)
    o = Oracle.from_graph(g, top_k=64)
    with Engine(g, top_k=64) as e:
        for q in (np.repeat(order[40:44], 8), np.repeat(order[50:75], 2), np.repeat(order[10:12], 25)):
            assert np.array_equal(e.prepare_group(q), o.prepare_group(q))
