"""BB1D over packets of camera rays (8 x 4 pixel blocks of one pinhole, upbp_packet.cu; iterations of
100,000 segment queries and more) against one warp per query: the order along the midpoints
(query_order 0) forms no packets, so it is the general path.  Both take the same pairs, so counts and
hashes are equal.  In plain mode the pairs' values are the same and only the order of the sums
differs: the relative error of a sum of n terms of one sign is below n 2^-24 in any order, 2e-5 for the
few hundred pairs of a query here.  In mixed mode the closest approach comes from another FP32 formula
for well-conditioned pairs: a query is held to the fixtures' 1e-4, the root mean square over all to 1e-5."""
import dataclasses

import numpy as np
import pytest

import golden_io as G
from smallupbp_b200 import engine
from smallupbp_b200 import workload as W

# images whose edges cut the pixel blocks, SHORT and LONG beams, nested media (several segments per ray),
# radii that vary along the beam, a camera inside the medium, rejects by path length and distance
CASES = {
    "ragged": W.cube_scene("a", 419, 317, 3000, 6, 0.01),
    "flat_long_beams": W.cube_scene("b", 1301, 101, 3000, 6, 0.01, photon_beam_type=W.LONG_BEAM, beam_length_cap=2.0),
    "boxes_short_query_beams": W.nested_boxes_scene("c", 457, 331, 3000, 6, 0.01, query_beam_type=W.SHORT_BEAM),
    "knn": W.cube_scene("d", 419, 317, 3000, 6, 0.02, bb1d_knn=4, pb2d_knn=4),
    "inside_min_dist": W.cube_scene("e", 331, 310, 3000, 6, 0.01, camera_pos=(0.5, 0.45, 0.3), min_dist_to_med=0.2,
                                    min_path_length=3),
}
_made = {}


def workload(name):
    if name not in _made:
        _made[name] = W.generate(CASES[name], 0)
        assert len(_made[name]["sq_flags"]) >= 100000
    return dict(_made[name])


def results(w, mode, **tuning):
    with engine.EstimatorStage(0, mode) as st:
        st.set_tuning(**tuning)
        st.run(w)
        return st.segment_results()[1], st.query_stats(), st.tested_counts()["bb1d"]


def compare(w, mode, **tuning):
    got, s, tested = results(w, mode, query_order=1, **tuning)
    want, s0, tested0 = results(w, mode, query_order=0, **tuning)
    assert tested != tested0  # the packets ran
    for k in ("count_bb1d", "hash_bb1d"):
        np.testing.assert_array_equal(s[k], s0[k], err_msg=k)
    err = G.rel_errors(got.astype(np.float64), want.astype(np.float64))
    assert err.max() <= (2e-5 if mode == engine.MODE_PLAIN else G.RTOL), (float(err.max()), int(err.argmax()))
    assert G.image_rel_l2(got, want) <= 1e-5
    return got, s


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [engine.MODE_PLAIN, engine.MODE_MIXED], ids=["plain", "mixed"])
@pytest.mark.parametrize("name", list(CASES))
def test_packets_match_one_warp_per_query(name, mode):
    compare(workload(name), mode)


@pytest.mark.gpu
@pytest.mark.parametrize("leaf,radii", [(1, 3.0), (64, 6.0), (8, 1024.0)])
def test_packets_match_for_other_trees(leaf, radii):
    compare(workload("ragged"), engine.MODE_PLAIN, bb1d_leaf=leaf, beam_piece_radii=radii)


@pytest.mark.gpu
def test_packets_without_mis():
    compare(W.without_mis(workload("ragged")), engine.MODE_PLAIN)


@pytest.mark.gpu
def test_rays_that_make_no_packet_and_beams_that_are_no_unit_vectors():
    # per some block of pixels: a ray with another origin, a direction that is no unit vector, 40 queries
    # on one pixel; and beams whose direction is no unit vector, which no approximate test may judge
    w = workload("ragged")
    first = np.nonzero(w["sq_path_length"] == 1)[0]
    for k in ("sq_origin", "sq_direction", "sq_pixel", "beam_direction"):
        w[k] = w[k].copy()
    w["sq_origin"][first[::160], 0] += np.float32(1e-3)
    w["sq_direction"][first[40::160]] *= np.float32(1.00001)
    w["sq_pixel"][first[1000:1040]] = w["sq_pixel"][first[1000]]
    w["beam_direction"][::7] *= np.float32(0.9999)
    compare(w, engine.MODE_PLAIN)


@pytest.mark.gpu
def test_one_piece_and_rays_flagged_off():
    w = workload("flat_long_beams")
    for k in [k for k in w if k.startswith("beam_")]:
        w[k] = np.ascontiguousarray(w[k][:1])
    w["beam_length"][:] = 0.05
    w["beam_origin"][:] = (0.5, 0.5, 0.5)
    w["beam_direction"][:] = (0.6, 0.8, 0.0)
    off = np.nonzero(w["sq_path_length"] == 1)[0][::3]
    w["sq_flags"] = w["sq_flags"].copy()
    w["sq_flags"][off] &= ~np.uint32(W.Q_BB1D)
    got, s = compare(w, engine.MODE_MIXED)
    assert s["count_bb1d"].sum() > 0 and not got[off].any() and not s["count_bb1d"][off].any()
