"""The emission of the beam pieces: leaf boxes of at most 32 pieces are reduced across lanes, larger ones
from the pieces' boxes in memory.  The smallest and largest leaf of each, over piece counts that fill
neither the last leaf nor the last warp, against the oracle (candidate counts and hashes, no tolerance)."""
import numpy as np
import pytest

from smallupbp_b200 import engine
from smallupbp_b200 import workload as W


@pytest.mark.gpu
@pytest.mark.parametrize("leaf", [1, 32, 64])
@pytest.mark.parametrize("light_paths", [3, 601])
def test_leaf_boxes_hold_the_oracle_candidates(leaf, light_paths):
    from oracle import port

    w = W.generate(W.cube_scene("leaves", 21, 13, light_paths, 5, 0.05, techniques=W.BPT | W.BB1D), 0)
    want = port.run(w)
    assert want["count_bb1d"].sum() > 0
    for mode in (engine.MODE_PLAIN, engine.MODE_MIXED):
        with engine.EstimatorStage(0, mode) as st:
            st.set_tuning(bb1d_leaf=leaf)
            st.run(w)
            got = st.query_stats()
        np.testing.assert_array_equal(got["count_bb1d"], want["count_bb1d"])
        np.testing.assert_array_equal(got["hash_bb1d"], want["hash_bb1d"])
