"""Iterations of several blocks planned on the device (blocks of 4096 groups
and more) against the oracle: a border at the first size planned there, one
that no tile of the plan ends on, blocks of more than one tile and a last block
of a few groups; groups of every preparation class; the ranker, which has no
oracle of this form, twice to the same partition."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


COUNTERS = ["merge_group_count", "merge_raw_pair_count", "candidate_proxy_pairs_examined", "exact_gain_input_nnz",
            "exact_overlap_neighbors", "merge_selected_pairs", "merge_total_local_gain",
            "accepted_merges_after_validation"]


@pytest.mark.parametrize("spec,batch,kw", [
    ("rmat:scale=14,ef=6,a=0.57,b=0.19,c=0.19,seed=9", 1023, {}),
    ("rmat:scale=14,ef=6,a=0.57,b=0.19,c=0.19,seed=9", 1024, {}),
    ("rmat:scale=14,ef=6,a=0.57,b=0.19,c=0.19,seed=9", 1025, {"top_k": 2}),
    ("chunglu:n=20000,gamma=2.3,deg=8,twins=1000,seed=2", 1500, {}),
    ("chunglu:n=20000,gamma=2.3,deg=8,twins=1000,seed=2", 2048, {"ranker": True}),
    ("grid:side=120,del=0.1,diag=0.02,seed=4", 1111, {"divide_max_group": 40}),
    ("grid:side=300,del=0.1,diag=0.02,seed=4", 4095, {}), ("grid:side=300,del=0.1,diag=0.02,seed=4", 4096, {}),
    ("chunglu:n=150000,gamma=2.3,deg=8,twins=7500,seed=2", 4097, {}),
    ("chunglu:n=150000,gamma=2.3,deg=8,twins=7500,seed=2", 5000, {"ranker": True})])
def test_blocks_planned_on_the_device(spec, batch, kw):
    from beam_gb300 import Engine, Graph, partition_hash
    from oracle import Oracle
    g = Graph.generate(spec)
    kw = {"ea_use_threshold": True, "group_batch_size": batch, **kw}
    ranker = "ranker" in kw
    if not ranker:
        o = Oracle.from_graph(g, **kw)
        o.run(8)
    hashes = set()
    with Engine(g, **kw) as e:
        for _ in range(2):
            e.reset()
            e.run(8)
            labels, head, nxt = e.partition()
            hashes.add(partition_hash(labels))
            if not ranker:
                oh, on = o.member_lists()
                assert np.array_equal(head, oh) and np.array_equal(nxt, on)
                st, ost = e.stats(), o.stats()
                assert {k: st[k] for k in COUNTERS} == {k: ost[k] for k in COUNTERS}
        e.validate_quotient()
    assert len(hashes) == 1
    assert ranker or hashes == {o.partition_hash()}
