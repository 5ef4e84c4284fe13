"""Precision of the mixed mode's BB1D contributions."""
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
