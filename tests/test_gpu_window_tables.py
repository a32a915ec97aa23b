"""Memory of the plain form (beam_gb300/csrc/window.cuh): the pair tables of the
groups evaluated at once stay within their limit, whatever the graph, and no
limit changes a result."""

import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

COUNTERS = ["merge_group_count", "merge_raw_pair_count", "candidate_proxy_pairs_examined", "merge_exact_gain_calls",
            "exact_gain_input_nnz", "exact_union_neighbors", "exact_overlap_neighbors", "merge_positive_gain_pairs",
            "merge_rejected_by_threshold", "merge_selected_pairs", "merge_total_local_gain",
            "accepted_merges_after_validation", "update_touched_quotient_entries"]


def twin_groups(count, members, targets):
    """Groups of nodes with the same few neighbours."""
    step = members + targets
    c = np.arange(count)[:, None, None] * step
    u = c + np.arange(members)[None, :, None] + np.zeros((1, 1, targets), int)
    v = c + members + np.arange(targets)[None, None, :] + np.zeros((1, members, 1), int)
    return u.ravel().astype(np.int32), v.ravel().astype(np.int32)


# one byte: a block at a time; then windows of a few of the lengths in between
@pytest.mark.parametrize("limit", [1, 1 << 20, 5 << 20, 40 << 20, 1 << 40])
@pytest.mark.parametrize("graph,batch", [("rmat", 64), ("rmat", 7), ("rmat", 1024), ("twins", 64)])
def test_no_limit_changes_a_result(graph, batch, limit):
    from beam_gb300 import Engine, Graph, partition_hash
    from beam_gb300._native import LIMIT_WINDOW_TABLES
    from oracle import Oracle
    if graph == "rmat":
        g = Graph.generate("rmat:scale=13,ef=6,a=0.57,b=0.19,c=0.19,seed=9")
    else:
        g = Graph.from_edges(*twin_groups(60, 150, 3))
    kw = {"ea_use_threshold": True, "group_batch_size": batch}
    o = Oracle.from_graph(g, **kw)
    o.run(6)
    with Engine(g, **kw) as e:
        e.set_limit(LIMIT_WINDOW_TABLES, limit)
        e.run(6)
        assert partition_hash(e.partition()[0]) == o.partition_hash()
        st, ost = e.stats(), o.stats()
        assert {k: st[k] for k in COUNTERS} == {k: ost[k] for k in COUNTERS}
        e.validate_quotient()


def test_limits_out_of_range_are_refused():
    from beam_gb300 import Engine, Graph
    from beam_gb300._native import LIMIT_WINDOW_TABLES, BeamError
    with Engine(Graph.generate("gnm:n=50,m=120,seed=2")) as e:
        with pytest.raises(BeamError):
            e.set_limit(LIMIT_WINDOW_TABLES, 0)
        with pytest.raises(BeamError):
            e.set_limit(99, 1)


CHILD = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import torch
from beam_gb300 import Engine, Graph
from test_gpu_window_tables import twin_groups
g = Graph.from_edges(*twin_groups(4000, 500, 4))
torch.cuda.init()
free = torch.cuda.mem_get_info(0)[0]
with Engine(g, ea_use_threshold=True) as e:
    e.run(1)
    print("used", free - torch.cuda.mem_get_info(0)[0], "merged", e.stats()["accepted_merges_after_validation"])
"""


def test_tables_of_two_million_nodes_in_groups_of_500():
    """4,000 groups of 500 members are 9 GB of pair tables. The tables may take 4
    GiB; what else the run holds is below 3.5 GB: entry pools 16 B x (3 x 16 M
    arcs + 2 x 2 M nodes) = 0.8, scratch 32 B x 18 M = 0.6, selection keys 16 B x
    16 per node = 0.5, row sums 0.13, CSR and per-node arrays 0.5, the rest and
    the context below 1."""
    child = CHILD.format(root=str(ROOT), tests=str(ROOT / "tests"))
    out = subprocess.run([sys.executable, "-c", child], capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert out.returncode == 0, out.stderr[-2000:]
    words = out.stdout.split()
    used, merged = int(words[1]), int(words[3])
    assert merged > 0
    assert used < (4 << 30) + 3_500_000_000
