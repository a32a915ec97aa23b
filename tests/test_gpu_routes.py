"""The ways that an iteration's groups can go, each reached for certain (the
engine counts them) and checked against the oracle: MediumKernel
(beam_gb300/csrc/medium.cuh) in blocks planned on the host and on the device, at
the limits of its groups; iterations of one and of several blocks planned on the
device, with groups of every preparation class, small and large, and a last block
of a few groups, whose tables are not cleared by one memset; the block sizes on
both sides of each line between windows, host plan and device plan."""

import numpy as np
import pytest

from test_medium_groups import clusters

COUNTERS = ("merge_group_count", "merge_group_max_size", "merge_raw_pair_count", "merge_candidate_pairs_after_prune",
            "candidate_proxy_pairs_examined", "merge_exact_gain_calls", "exact_gain_input_nnz",
            "exact_union_neighbors", "exact_overlap_neighbors", "merge_positive_gain_pairs",
            "merge_rejected_by_threshold", "merge_rejected_by_overlap", "merge_selected_pairs",
            "merge_total_local_gain", "accepted_merges_after_validation", "update_touched_quotient_entries")

MEDIUM = [(9, 40, {}), (17, 16, {}), (18, 15, {}), (33, 8, {}), (46, 44, {}), (48, 43, {}), (63, 32, {}), (64, 32, {}),
          (65, 31, {}), (64, 33, {}), (40, 20, {"top_k": 1}), (40, 20, {"top_k": 33}),
          (64, 20, {"ea_use_threshold": False})]


def medium_groups(o, g, batch):
    """Medium groups of iteration 1 (rows are the graph's) per block."""
    order, starts, lengths = o.groups()
    entries = np.add.reduceat(np.diff(g.row_ptr)[order], starts)
    medium = (lengths >= 2) & ~((lengths <= 32) & (entries <= 256)) & (lengths <= 64) & (entries <= 2048)
    return [int(medium[i:i + batch].sum()) for i in range(0, len(medium), batch)]


def padded(u, v, pairs):
    """The same graph and `pairs` edges of two nodes each beside it."""
    n = int(max(u.max(), v.max())) + 1
    p = n + 2 * np.arange(pairs)
    return np.concatenate([u, p]).astype(np.int32), np.concatenate([v, p + 1]).astype(np.int32)


def compare(e, o):
    labels, head, nxt = e.partition()
    assert np.array_equal(labels, o.labels())
    oh, on = o.member_lists()
    assert np.array_equal(head, oh) and np.array_equal(nxt, on)
    st, ost = e.stats(), o.stats()
    assert {k: st[k] for k in COUNTERS} == {k: ost[k] for k in COUNTERS}
    e.validate_quotient()


def check(g, kw, iterations, wanted):
    """Runs against the oracle; wanted(engine) is asked after the first iteration."""
    from beam_gb300 import Engine
    from oracle import Oracle
    o = Oracle.from_graph(g, **kw)
    with Engine(g, **kw) as e:
        e.run(1)
        wanted(e)
        o.run(1)
        compare(e, o)
        o = Oracle.from_graph(g, **kw)
        o.run(iterations)
        e.reset()
        e.run(iterations)
        compare(e, o)


@pytest.mark.gpu
@pytest.mark.parametrize("members,targets,kw", MEDIUM)
def test_medium_groups_of_host_planned_blocks(members, targets, kw):
    """Blocks of 2,000 groups, planned on the host: the kernel takes the medium
    groups of blocks with at least 304 of them."""
    from beam_gb300 import Graph
    from beam_gb300._native import ROUTE_HOST_PLANS, ROUTE_MEDIUM_GROUPS
    from oracle import Oracle
    g = Graph.from_edges(*clusters(members, targets, 1200, members))
    kw = {"ea_use_threshold": True, **kw, "group_batch_size": 2000}
    o = Oracle.from_graph(g, **kw)
    o.divide(1)
    want = sum(m for m in medium_groups(o, g, 2000) if m >= 304)
    assert want >= 304 and o.group_count() > 2000

    def wanted(e):
        assert e.route_count(ROUTE_HOST_PLANS) == 1 and e.route_count(ROUTE_MEDIUM_GROUPS) == want
    check(g, kw, 3, wanted)


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1 << 30, 65536, 66000])
@pytest.mark.parametrize("members,targets,kw", [(9, 40, {}), (46, 44, {}), (64, 32, {}), (65, 31, {}), (40, 20, {"top_k": 1}),
                                                (40, 20, {"top_k": 33})])
def test_medium_groups_of_device_planned_blocks(members, targets, kw, batch):
    """More than 65,536 groups: every medium group of the iteration."""
    from beam_gb300 import Graph
    from beam_gb300._native import ROUTE_DEVICE_PLANS, ROUTE_MEDIUM_GROUPS
    from oracle import Oracle
    g = Graph.from_edges(*padded(*clusters(members, targets, 300, members), 68000))
    kw = {"ea_use_threshold": True, **kw, "group_batch_size": batch}
    o = Oracle.from_graph(g, **kw)
    o.divide(1)
    want = sum(medium_groups(o, g, batch))
    assert want > 0 and o.group_count() > 66000

    def wanted(e):
        assert e.route_count(ROUTE_DEVICE_PLANS) == 1 and e.route_count(ROUTE_MEDIUM_GROUPS) == want
    check(g, kw, 2, wanted)


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [1, 2, 3])
@pytest.mark.parametrize("kw", [{}, {"top_k": 2}, {"top_k": 40}, {"divide_max_group": 40}, {"divide_max_group": 1024}])
def test_blocks_of_a_skewed_graph_planned_on_the_device(kw, blocks):
    """Blocks of over 4,096 groups and a last one of 100 (for blocks > 1)."""
    from beam_gb300 import Graph
    from beam_gb300._native import ROUTE_DEVICE_PLANS
    from oracle import Oracle
    g = Graph.generate("rmat:scale=16,ef=6,a=0.57,b=0.19,c=0.19,seed=9")
    kw = {"ea_use_threshold": True, **kw}
    o = Oracle.from_graph(g, **kw)
    o.divide(1)
    groups = o.group_count()
    batch = groups if blocks == 1 else (groups - 100) // (blocks - 1)
    assert batch >= 4096 and (blocks == 1 or 100 <= groups % batch < 256)

    def wanted(e):
        assert e.route_count(ROUTE_DEVICE_PLANS) == 1
    check(g, {**kw, "group_batch_size": batch}, 4, wanted)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,ranker,route", [
    (1024, False, "ROUTE_WINDOW_ROUNDS"), (1025, False, "ROUTE_HOST_PLANS"), (4095, False, "ROUTE_HOST_PLANS"),
    (4096, False, "ROUTE_DEVICE_PLANS"), (64, True, "ROUTE_HOST_PLANS"), (4096, True, "ROUTE_DEVICE_PLANS")])
def test_the_lines_between_the_ways(batch, ranker, route):
    from beam_gb300 import Engine, Graph
    from beam_gb300 import _native as N
    g = Graph.generate("grid:side=110,del=0.1,diag=0.02,seed=4")
    with Engine(g, ea_use_threshold=True, group_batch_size=batch, ranker=ranker) as e:
        e.divide(1)
        assert len(e.groups()[1]) > 4096
        e.merge(1)
        taken = {r for r in ("ROUTE_WINDOW_ROUNDS", "ROUTE_HOST_PLANS", "ROUTE_DEVICE_PLANS")
                 if e.route_count(getattr(N, r)) > 0}
    assert taken == {route}
