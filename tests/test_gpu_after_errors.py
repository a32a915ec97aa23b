"""A CUDA call that failed is reported by the call that made it and by no other."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_after_a_wrong_device_ordinal():
    from beam_gb300 import Engine, FlatScorer, Graph
    from beam_gb300._native import BeamError
    from oracle import Oracle
    g = Graph.generate("gnm:n=200,m=700,seed=2")
    o = Oracle.from_graph(g, ea_use_threshold=True)
    o.run(3)
    flat = {"offsets": [0, 1, 2], "reps": [0, 1], "rsz": [1, 1], "self": [0, 0], "nb": [5, 5], "wt": [1, 1],
            "nsz": [1, 1]}
    with Engine(g, ea_use_threshold=True) as e, FlatScorer() as s:
        want = s.score(flat, [[0, 1]])
        for again in (lambda: e.run(3), lambda: s.score(flat, [[0, 1]]), lambda: e.encode(), lambda: e.quotient_nnz()):
            with pytest.raises(BeamError, match="invalid device ordinal"):
                Engine(g, device=99)
            again()
        assert np.array_equal(e.partition()[0], o.labels())
        assert np.array_equal(s.score(flat, [[0, 1]]), want)
