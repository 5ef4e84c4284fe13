"""The grid gather's first checks, on 16-byte lines with bounds wider than the rounding: no pair that the
predicate takes may be lost.  The candidates over the grid and over the beam pieces (the oracle's) are the
same pairs but for closest points on a cell's face, and pairs that the predicate takes through rounding and
the oracle's reach rule drops: at most 1e-3 of them fewer and 1e-2 more.

Cells with many whole batches and with single entries, KNN radii (a bound per entry), coordinates far from
the origin (rounding 30 times larger), and directions off the unit length, whose lines pass every check."""
import numpy as np
import pytest

from smallupbp_b200 import engine
from smallupbp_b200 import workload as W


@pytest.mark.gpu
@pytest.mark.parametrize("res,knn,shift,beam,query", [
    (1, 0, 0.0, 1.0, 1.0), (64, 0, 0.0, 1.0, 1.0), (7, 4, 0.0, 1.0, 1.0), (7, 0, 32.0, 1.0, 1.0),
    (7, 0, 0.0, 1.0 + 4e-6, 1.0), (7, 0, 0.0, 1.0, 1.0 + 4e-6)])
def test_no_candidate_of_the_predicate_is_lost(res, knn, shift, beam, query):
    from oracle import port

    w = W.generate(W.cube_scene("lines", 40, 30, 400, 6, 0.4 if knn else 0.04, techniques=W.BPT | W.BB1D, bb1d_knn=knn), 0)
    for k in ("lv_position", "beam_origin", "sq_origin"):
        w[k] = (w[k] + np.float32(shift)).astype(np.float32)
    w["beam_direction"] = (w["beam_direction"] * np.float32(beam)).astype(np.float32)
    w["sq_direction"] = (w["sq_direction"] * np.float32(query)).astype(np.float32)
    want = port.run(w)["count_bb1d"].astype(np.int64).sum()
    assert want > 10000
    for mode in (engine.MODE_PLAIN, engine.MODE_MIXED):
        with engine.EstimatorStage(0, mode) as st:
            st.set_bb1d_grid(res)
            st.run(w)
            got = st.query_stats()["count_bb1d"].astype(np.int64).sum()
        assert want * (1 - 1e-3) <= got <= want * (1 + 1e-2), (want, got)
