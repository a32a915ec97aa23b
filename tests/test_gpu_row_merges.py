"""Graphs beyond the limit of the row and pair sums (2^30 arcs): every pair is
scored by the merge of its two rows, the prepare kernels leave no sums behind
and no block goes through a window. The engine's limit, lowered to one arc,
takes small graphs there. Against the oracle, in every form."""

import numpy as np
import pytest

from test_gain_sums import planted

pytestmark = pytest.mark.gpu

COUNTERS = ["merge_group_count", "merge_group_max_size", "merge_raw_pair_count",
            "merge_candidate_pairs_after_prune", "candidate_proxy_pairs_examined", "merge_exact_gain_calls",
            "exact_gain_input_nnz", "exact_raw_entries_a", "exact_raw_entries_b", "exact_union_neighbors",
            "exact_overlap_neighbors", "merge_positive_gain_pairs", "merge_rejected_by_threshold",
            "merge_rejected_by_overlap", "merge_candidate_pairs", "merge_selected_pairs", "merge_total_local_gain",
            "isolated_gain_sum", "validation_exact_calls", "accepted_merges_after_validation",
            "update_touched_quotient_entries"]


def graph(name):
    from beam_gb300 import Graph
    if name == "rmat":
        return Graph.generate("rmat:scale=13,ef=6,a=0.57,b=0.19,c=0.19,seed=9")
    if name == "twins":
        return Graph.generate("chunglu:n=20000,gamma=2.3,deg=8,twins=1000,seed=2")
    return Graph.from_edges(*planted(name, 3))


@pytest.mark.parametrize("name,batch,kw", [
    ("rmat", 64, {}), ("rmat", 7, {"top_k": 4}), ("rmat", 300, {}), ("rmat", 1 << 30, {}),
    ("rmat", 64, {"verify_cuda_gain": True}), ("rmat", 64, {"ea_use_threshold": False}), ("twins", 64, {}),
    ("twins", 4500, {}), ("twins", 1 << 30, {"divide_max_group": 1024}), ("long", 64, {}), ("long", 1 << 30, {}),
    ("short", 64, {"divide_max_group": 30})])
def test_row_merges_match_the_oracle(name, batch, kw):
    from beam_gb300 import Engine, partition_hash
    from beam_gb300._native import LIMIT_ROW_SUM_ARCS
    from oracle import Oracle
    g = graph(name)
    kw = {"ea_use_threshold": True, **kw, "group_batch_size": batch}
    o = Oracle.from_graph(g, **{k: v for k, v in kw.items() if k != "verify_cuda_gain"})
    o.run(8)
    with Engine(g, **kw) as e:
        e.set_limit(LIMIT_ROW_SUM_ARCS, 1)
        e.run(8)
        labels, head, nxt = e.partition()
        assert partition_hash(labels) == o.partition_hash()
        oh, on = o.member_lists()
        assert np.array_equal(head, oh) and np.array_equal(nxt, on)
        st, ost = e.stats(), o.stats()
        assert {k: st[k] for k in COUNTERS} == {k: ost[k] for k in COUNTERS}
        e.validate_quotient()
        # the same engine with sums again
        e.set_limit(LIMIT_ROW_SUM_ARCS, 1 << 30)
        e.reset()
        e.run(8)
        assert np.array_equal(e.partition()[0], labels)


def test_prepare_group_without_sums():
    from beam_gb300 import Engine
    from beam_gb300._native import LIMIT_ROW_SUM_ARCS
    from oracle import Oracle
    g = graph("rmat")
    o = Oracle.from_graph(g)
    with Engine(g) as e:
        e.set_limit(LIMIT_ROW_SUM_ARCS, 1)
        e.divide(1)
        o.divide(1)
        order, starts, lengths = e.groups()
        for k in np.argsort(-lengths)[[0, 1, 5, 50]]:
            q = order[starts[k]:starts[k] + lengths[k]]
            assert np.array_equal(e.prepare_group(q), o.prepare_group(q))


def test_ranker_without_sums_is_the_ranker_with_them():
    """The ranker decides from candidates and exact gains, the same either way."""
    from beam_gb300 import Engine
    from beam_gb300._native import LIMIT_ROW_SUM_ARCS
    labels = []
    with Engine(graph("twins"), ea_use_threshold=True, group_batch_size=1 << 30, ranker=True) as e:
        for arcs in (1 << 30, 1):
            e.set_limit(LIMIT_ROW_SUM_ARCS, arcs)
            e.reset()
            e.run(10)
            labels.append(e.partition()[0])
    assert np.array_equal(*labels)


def test_the_limit_is_not_above_what_the_fields_hold():
    from beam_gb300 import Engine
    from beam_gb300._native import LIMIT_ROW_SUM_ARCS, BeamError
    with Engine(graph("short")) as e:
        for value in (0, -1, (1 << 30) + 1):
            with pytest.raises(BeamError):
                e.set_limit(LIMIT_ROW_SUM_ARCS, value)
