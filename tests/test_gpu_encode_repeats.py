"""Encoding of graphs that list edges more than once, at the start, after merges by
hand and after runs, also with counts beyond a block's capacity: the lists and
their lengths are the host encoder's and the oracle's, which look the member
pairs up one by one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FILES = ("G.txt", "P.txt", "Cp.txt", "Cm.txt")


def repeated(n, m, copies, seed):
    """A random graph whose edges are listed up to `copies` times."""
    rng = np.random.default_rng(seed)
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    e = np.unique(np.stack([np.minimum(u, v), np.maximum(u, v)], 1)[u != v], axis=0)
    e = np.repeat(e, rng.integers(1, copies + 1, len(e)), axis=0)
    return e[:, 0].astype(np.int32), e[:, 1].astype(np.int32)


def star(copies):
    """One node joined to 300 others, and again to some of them."""
    leaf = np.concatenate([np.arange(1, 301), np.repeat(np.arange(3, 40), copies)])
    return np.zeros(len(leaf), np.int32), leaf.astype(np.int32)


def compare(e, g, o, tmp):
    """Files and counts of the engine, the host encoder and the oracle."""
    keys = ("p", "cp", "cm", "encoding_cost_mags_x2", "cost_ratio_mags_compatible")
    for d in ("a", "b", "c"):
        (tmp / d).mkdir(exist_ok=True)
    _, head, nxt = e.partition()
    files, host, ref = e.encode(tmp / "a"), g.encode(head, nxt, tmp / "b"), o.encode(tmp / "c")
    assert {k: files[k] for k in keys} == {k: host[k] for k in keys} == {k: ref[k] for k in keys}
    assert e.encode() == files == host
    for f in FILES:
        want = (tmp / "c" / f).read_bytes()
        assert (tmp / "a" / f).read_bytes() == want and (tmp / "b" / f).read_bytes() == want, f


@pytest.mark.parametrize("edges", [(40, 60, 2), (40, 300, 2), (40, 300, 5), (300, 900, 3), (300, 20000, 2), (2000, 3000, 4)])
def test_repeated_edges_encode_like_the_oracle(edges, tmp_path):
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    g = Graph.from_edges(*repeated(*edges, seed=sum(edges)))
    o = Oracle.from_graph(g)
    rng = np.random.default_rng(1)
    with Engine(g) as e:
        compare(e, g, o, tmp_path)
        for _ in range(3):  # merges whatever they cost: dense blocks with missing pairs
            act = np.unique(e.partition()[0])
            p = rng.permutation(act)[:2 * (len(act) // 3)]
            e.merge_pairs(p[0::2], p[1::2])
            for keep, remove in zip(p[0::2], p[1::2]):
                o.merge_pair(keep, remove)
            compare(e, g, o, tmp_path)


@pytest.mark.parametrize("copies", [1, 2, 9])
def test_star_with_repeated_edges(copies, tmp_path):
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    g = Graph.from_edges(*star(copies))
    o = Oracle.from_graph(g)
    with Engine(g) as e:
        for merges in ([], [(5, 6), (7, 50)], [(5, 60), (8, 61), (0, 9)], [(0, 70), (100, 101)]):
            if merges:
                e.merge_pairs(*zip(*merges))
                for k, r in merges:
                    o.merge_pair(k, r)
            compare(e, g, o, tmp_path)


def test_repeats_of_one_graph_are_not_the_next_ones(tmp_path):
    """The flag is an engine's, and set anew by every reset."""
    from beam_gb300 import Engine, Graph
    from oracle import Oracle
    for copies in (3, 1, 3):
        g = Graph.from_edges(*repeated(300, 2000, copies, 5))
        o = Oracle.from_graph(g)
        with Engine(g) as e:
            for _ in range(2):
                compare(e, g, o, tmp_path)
                e.reset()


@pytest.mark.parametrize("n", [1, 4, 300])
def test_graph_without_edges(n, tmp_path):
    from beam_gb300 import Engine
    from oracle import Oracle

    class Edgeless:
        def __init__(self):
            self.n, self.arcs = n, 0
            self.row_ptr, self.col_idx = np.zeros(n + 1, np.int64), np.zeros(0, np.int32)

    o = Oracle(np.zeros(n + 1, np.int64), np.zeros(0, np.int32))
    (tmp_path / "a").mkdir()
    (tmp_path / "c").mkdir()
    with Engine(Edgeless()) as e:
        for merged in (False, True):
            files, ref = e.encode(tmp_path / "a"), o.encode(tmp_path / "c")
            assert files == e.encode() and files["supernodes"] == ref["n_supernodes"]
            assert files["encoding_cost_mags_x2"] == ref["encoding_cost_mags_x2"] == 0
            for f in FILES:
                assert (tmp_path / "a" / f).read_bytes() == (tmp_path / "c" / f).read_bytes(), f
            if n > 2 and not merged:
                e.merge_pairs([0], [2])
                o.merge_pair(0, 2)
        e.run(2)
