"""KNN photon radii from the reference's kd-tree search at sizes whose top levels are split by whole
blocks (more than 4096 points) and whose walks prune by cells: the PB2D candidate sets depend on every
radius, and must equal the oracle's (counts and hashes, no tolerance)."""
import numpy as np
import pytest

from smallupbp_b200 import engine
from smallupbp_b200 import workload as W


@pytest.mark.gpu
@pytest.mark.parametrize("light_paths,k", [(8800, 1), (17500, 6), (70000, 8), (150000, 3)])
def test_photon_radii_give_the_oracle_candidates(light_paths, k):
    from oracle import port

    # radius 0.4 x 2 x (distance to the k-th nearest): of the size of the photons' spacing
    w = W.generate(W.cube_scene("k", 48, 40, light_paths, 6, 0.4, techniques=W.BPT | W.PB2D, pb2d_knn=k), 0)
    assert (w["lv_flags"] & W.LV_IN_MEDIUM).astype(bool).sum() > 4096
    want = port.run(w)
    with engine.EstimatorStage(0, engine.MODE_PLAIN) as st:
        st.run(w)
        got = st.query_stats()
    assert got["count_pb2d"].sum() > 5000
    np.testing.assert_array_equal(got["count_pb2d"], want["count_pb2d"])
    np.testing.assert_array_equal(got["hash_pb2d"], want["hash_pb2d"])
