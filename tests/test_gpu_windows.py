"""Windows of blocks (beam_gb300/csrc/window.cuh) against the oracle, which
takes the blocks one after another: the partition and every counter. Block
sizes up to the largest that goes through windows and the first that does not;
graphs whose groups touch each other often (twins), hold hub rows beyond every
row limit, and need no, some and long rankings; ranking limits on both sides of
the lists kept per lane."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTERS = ["merge_group_count", "merge_group_max_size", "merge_raw_pair_count",
            "merge_candidate_pairs_after_prune", "candidate_proxy_pairs_examined", "merge_exact_gain_calls",
            "exact_gain_input_nnz", "exact_raw_entries_a", "exact_raw_entries_b", "exact_union_neighbors",
            "exact_overlap_neighbors", "merge_positive_gain_pairs", "merge_rejected_by_threshold",
            "merge_rejected_by_overlap", "merge_candidate_pairs", "merge_selected_pairs", "merge_total_local_gain",
            "isolated_gain_sum", "selected_merges_for_validation", "validation_exact_calls",
            "validation_exact_row_entry_work", "accepted_merges_after_validation", "update_touched_quotient_entries"]


def hubs(seed):
    """Three hubs of thousands of neighbours over a sparse background, leaves
    with the same few neighbours in numbers."""
    rng = np.random.default_rng(seed)
    n = 12000
    u = [np.full(9000, 0), np.full(5000, 1), np.full(2500, 2), rng.integers(0, n, 9000)]
    v = [np.arange(3, 9003), 3 + rng.choice(n - 3, 5000, replace=False), 3 + rng.choice(n - 3, 2500, replace=False),
         rng.integers(0, n, 9000)]
    a, b = np.concatenate(u), np.concatenate(v)
    e = np.unique(np.stack([np.minimum(a, b), np.maximum(a, b)], 1)[a != b], axis=0)
    return e[:, 0], e[:, 1]


GRAPHS = {"hubs": None, "rmat": "rmat:scale=13,ef=6,a=0.57,b=0.19,c=0.19,seed=9",
          "twins": "chunglu:n=6000,gamma=2.3,deg=8,twins=600,seed=2", "grid": "grid:side=90,del=0.1,diag=0.02,seed=4"}


@pytest.mark.parametrize("graph,batch,kw", [
    ("hubs", 64, {}), ("hubs", 7, {}), ("hubs", 256, {}), ("rmat", 33, {}), ("rmat", 256, {}), ("rmat", 257, {}),
    ("rmat", 64, {"top_k": 1}), ("rmat", 64, {"top_k": 33}), ("rmat", 64, {"ea_use_threshold": False}),
    ("rmat", 64, {"divide_max_group": 1024}), ("rmat", 64, {"verify_cuda_gain": True}), ("twins", 64, {}),
    ("twins", 1, {}), ("twins", 100, {"top_k": 4}), ("grid", 64, {}), ("grid", 10, {"seed": 7}),
    ("rmat", 1024, {}), ("rmat", 1025, {}), ("hubs", 700, {}), ("twins", 1024, {}), ("grid", 1024, {}),
    ("grid", 1025, {})])
def test_windows_match_the_blocks_in_order(graph, batch, kw):
    from beam_gb300 import Engine, Graph, partition_hash
    from oracle import Oracle
    g = Graph.generate(GRAPHS[graph]) if GRAPHS[graph] else Graph.from_edges(*hubs(3))
    kw = {"ea_use_threshold": True, **kw, "group_batch_size": batch}
    o = Oracle.from_graph(g, **{k: v for k, v in kw.items() if k != "verify_cuda_gain"})
    o.run(12)
    with Engine(g, **kw) as e:
        for _ in range(2):  # a second run meets the buffers and controls of the first
            e.reset()
            e.run(12)
            labels, head, nxt = e.partition()
            assert partition_hash(labels) == o.partition_hash()
            oh, on = o.member_lists()
            assert np.array_equal(head, oh) and np.array_equal(nxt, on)
            st, ost = e.stats(), o.stats()
            assert {k: st[k] for k in COUNTERS if k in ost} == {k: ost[k] for k in COUNTERS if k in ost}
        e.validate_quotient()


def test_windows_leave_the_other_entry_points_usable():
    """divide, prepare_group and merge_pairs between windowed iterations."""
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    g = Graph.generate(GRAPHS["rmat"])
    o = Oracle.from_graph(g)
    with Engine(g) as e:
        for it in (1, 2, 3):
            e.divide(it)
            o.divide(it)
            order, starts, lengths = e.groups()
            k = int(np.argmax(lengths))
            q = order[starts[k]:starts[k] + lengths[k]]
            assert np.array_equal(e.prepare_group(q), o.prepare_group(q))
            e.divide(it)
            e.merge(it, 3)
            o.merge(it, 3)
            assert np.array_equal(e.partition()[0], o.labels())
