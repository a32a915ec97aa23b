"""A pair-scoring call that fails on the device leaves the caller's result arrays
as they were."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b", [([0, 1, 5], [2, 3, 6]),    # 1 was merged into 0
                                 ([0, 4, 5], [2, 4, 6])])   # a pair of one supernode
def test_failing_call_leaves_the_results_alone(a, b):
    from beam_gb300 import Engine, Graph
    from beam_gb300 import _native as N
    a, b = np.array(a, np.int32), np.array(b, np.int32)
    gain, before = np.full(3, -77, np.int64), np.full(3, -78, np.int64)
    with Engine(Graph.generate("gnm:n=50,m=120,seed=2")) as e:
        e.merge_pairs([0], [1])
        rc = N.lib().beam_engine_score_pairs(
            e._h, a.ctypes.data_as(N.P_i32), b.ctypes.data_as(N.P_i32), 3,
            gain.ctypes.data_as(N.P_i64), before.ctypes.data_as(N.P_i64))
        assert rc != 0 and b"inactive" in N.lib().beam_engine_last_error()
    assert gain.tolist() == [-77] * 3 and before.tolist() == [-78] * 3
