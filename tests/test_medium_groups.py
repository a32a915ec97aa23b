"""Groups handled from rows to selected pairs by one CTA
(beam_gb300/csrc/medium.cuh) against the oracle, around the limits of that path
(members, row entries, ranking), and the order of proxy ratios by cross products
(ExactRanks in beam_gb300/csrc/merge.cu) against the rounded double quotients
that the reference compares."""

import random

import numpy as np
import pytest


def test_cross_products_order_like_the_rounded_quotients():
    rng = random.Random(11)
    top = (1 << 26) - 1
    for trial in range(200000):
        d1 = rng.randint(1, top) if trial % 2 else rng.randint(top - 5000, top)
        p1 = rng.randint(1, top) if trial % 3 else rng.randint(max(1, d1 - 3), min(top, d1 + 3))
        if trial % 4 == 0:  # a neighbour in the Farey sense: p1 d2 - p2 d1 = +-1 where one exists
            d2 = rng.randint(1, top)
            p2 = min(top, max(1, (p1 * d2 + rng.choice((-1, 0, 1))) // d1))
        else:
            p2, d2 = rng.randint(1, top), rng.randint(1, top)
        l, r = p1 * d2, p2 * d1
        q1, q2 = p1 / d1, p2 / d2
        assert (l > r) == (q1 > q2) and (l == r) == (q1 == q2)


def clusters(members, targets, count, seed):
    """Groups of members with the same targets but a few, tied to a sparse
    background of single edges."""
    rng = np.random.default_rng(seed)
    u, v = [], []
    step = members + targets
    for c in range(count):
        m, t = np.meshgrid(c * step + np.arange(members), c * step + members + np.arange(targets), indexing="ij")
        # one edge in a hundred missing in every third cluster
        on = rng.random(m.shape) >= (0.01 if c % 3 == 0 else 0.0)
        u.append(m[on])
        v.append(t[on])
        if c % 5 == 0:
            u.append(np.full(members - 1, c * step))
            v.append(c * step + 1 + np.arange(members - 1))
    n = count * step
    x, y = rng.integers(0, n, n // 2), rng.integers(0, n, n // 2)
    u, v = np.concatenate([*u, x[x != y]]), np.concatenate([*v, y[x != y]])
    e = np.unique(np.stack([np.minimum(u, v), np.maximum(u, v)], 1), axis=0)
    return e[:, 0].astype(np.int32), e[:, 1].astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("members,targets,kw", [
    (9, 40, {}), (17, 16, {}), (18, 15, {}), (33, 8, {}), (48, 43, {}), (63, 32, {}), (64, 32, {}), (65, 31, {}),
    (64, 33, {}), (40, 20, {"top_k": 1}), (40, 20, {"top_k": 33}), (64, 20, {"ea_use_threshold": False})])
def test_medium_groups_match_the_oracle(members, targets, kw):
    from beam_gb300 import Engine, Graph, partition_hash
    from oracle import Oracle
    g = Graph.from_edges(*clusters(members, targets, 700, members))
    kw = {"ea_use_threshold": True, **kw, "group_batch_size": 6000}
    o = Oracle.from_graph(g, **kw)
    o.run(3)
    with Engine(g, **kw) as e:
        e.run(3)
        assert partition_hash(e.partition()[0]) == o.partition_hash()
        st, ost = e.stats(), o.stats()
        e.validate_quotient()
    for k in ("merge_group_count", "merge_candidate_pairs_after_prune", "candidate_proxy_pairs_examined",
              "merge_exact_gain_calls", "exact_gain_input_nnz", "exact_union_neighbors", "exact_overlap_neighbors",
              "merge_positive_gain_pairs", "merge_rejected_by_threshold", "merge_total_local_gain",
              "accepted_merges_after_validation", "update_touched_quotient_entries"):
        assert st[k] == ost[k], k
