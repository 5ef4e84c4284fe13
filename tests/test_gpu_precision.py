"""Precision of the mixed mode's BB1D contributions: pdfs below the normal FP32 range, and packets of camera rays
(upbp_packet.cu) against one warp per query (query_order 0, which forms no packets)."""
import numpy as np
import pytest

import golden_io as G
from smallupbp_b200 import engine
from smallupbp_b200 import workload as W


def run(w, mode, **tuning):
    with engine.EstimatorStage(0, mode) as st:
        st.set_tuning(**tuning)
        st.run(w)
        return st.segment_results()[1].astype(np.float64), st.query_stats(), st.tested_counts()["bb1d"]


@pytest.mark.gpu
@pytest.mark.parametrize("query", [W.LONG_BEAM, W.SHORT_BEAM], ids=["long", "short"])
def test_beam_pdfs_below_the_normal_range(query):
    # the beam's pdf at the pair is subnormal (3e-39 to 1e-38); its reciprocal is a number.  Against the gather with a
    # thread per query, which evaluates the same pairs' closest points by the general form of the contribution
    cfg = W.cube_scene("pdf", 64, 48, 500, 6, 0.05, query_beam_type=query, photon_beam_type=W.LONG_BEAM,
                       beam_length_cap=2.0)
    w = W.generate(cfg, 0)
    w["beam_ray_sample_pdf"][:] = 1.7e-38
    # (these keep the products with that reciprocal below the largest float)
    w["beam_last_pdf_w_inv"] = w["beam_last_pdf_w_inv"] * np.float32(1e-3)
    w["params"]["mis_factor_bb1d"] = 1e-3
    want, s0, _ = run(w, engine.MODE_MIXED, bb1d_kernel=0)
    got, s, _ = run(w, engine.MODE_MIXED)
    np.testing.assert_array_equal(s["count_bb1d"], s0["count_bb1d"])
    assert (want.max(axis=1) > 0).sum() > 500
    G.assert_close(got, want, "BB1D")


SCENES = {
    "boxes_short": W.nested_boxes_scene("p", 457, 331, 60000, 6, 0.01, query_beam_type=W.SHORT_BEAM),
    "cube_long": W.cube_scene("q", 419, 317, 60000, 6, 0.01, photon_beam_type=W.LONG_BEAM, beam_length_cap=2.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(SCENES))
def test_packets_are_as_close_to_fp64(name):
    # the same pairs and terms of a sum; the packets' sums over the rounds are in FP64.  Over the 138,000 queries
    # here the two errors differ by 0.5 % at most
    w = W.generate(SCENES[name], 0)
    got, _, tested = run(w, engine.MODE_MIXED, query_order=1)
    want, _, tested0 = run(w, engine.MODE_MIXED, query_order=0)
    ref = run(w, engine.MODE_FP64)[0]
    assert tested != tested0  # the packets ran
    err, err0 = np.linalg.norm(got - ref), np.linalg.norm(want - ref)
    rel = np.abs(ref).max(axis=1) + 1e-30
    e, e0 = np.abs(got - ref).max(axis=1) / rel, np.abs(want - ref).max(axis=1) / rel
    assert err <= 1.005 * err0
    assert np.median(e[e0 > 0]) <= 1.005 * np.median(e0[e0 > 0])
