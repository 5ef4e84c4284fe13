"""BB1D over packets of camera rays (upbp_packet.cu), for ray records that a caller supplies: rays whose
transmittance beyond their last segment is no number, wide fans of short rays, and coordinates far
from the origin.  As in test_gpu_packets.py the order along the midpoints (query_order 0), which forms no
packets, is the general path: both take the same pairs, so counts and hashes are equal."""
import numpy as np
import pytest

import golden_io as G
from smallupbp_b200 import engine
from smallupbp_b200 import workload as W

_made = {}


def workload(**kw):
    key = tuple(sorted(kw.items()))
    if key not in _made:
        _made[key] = W.generate(W.cube_scene("rays", 419, 317, 3000, 6, 0.01, **kw), 0)
        assert len(_made[key]["sq_flags"]) >= 100000
    return {k: v.copy() for k, v in _made[key].items()}


def results(w, mode, **tuning):
    with engine.EstimatorStage(0, mode) as st:
        st.set_tuning(**tuning)
        st.run(w)
        return st.segment_results()[1], st.query_stats(), st.tested_counts()["bb1d"]


def both(w, mode, **tuning):
    got, s, tested = results(w, mode, query_order=1, **tuning)
    want, s0, tested0 = results(w, mode, query_order=0, **tuning)
    assert tested != tested0  # the packets ran
    return got, s, want, s0


def same_pairs(s, s0):
    for k in ("count_bb1d", "hash_bb1d"):
        np.testing.assert_array_equal(s[k], s0[k], err_msg=k)


def set_segments(w, q, segments, flags=None):
    """The segments (dmin, dmax, medium, pdf, attenuation) of query q, appended to the arrays' lists."""
    w["sq_seg_begin"][q] = len(w["seg_dist_min"])
    w["sq_seg_count"][q] = len(segments)
    for k, i in (("seg_dist_min", 0), ("seg_dist_max", 1), ("seg_medium", 2), ("seg_pdf", 3), ("seg_rev_pdf", 3),
                 ("seg_attenuation", 4)):
        w[k].extend(s[i] for s in segments)
    if flags is not None:
        w["sq_flags"][q] = flags


def segment_lists(w):
    for k in ("seg_dist_min", "seg_dist_max", "seg_pdf", "seg_rev_pdf", "seg_attenuation", "seg_medium"):
        w[k] = list(w[k])


def segment_arrays(w):
    for k in ("seg_dist_min", "seg_dist_max", "seg_pdf", "seg_rev_pdf"):
        w[k] = np.asarray(w[k], np.float32)
    w["seg_attenuation"] = np.asarray(w["seg_attenuation"], np.float32).reshape(-1, 3)
    w["seg_medium"] = np.asarray(w["seg_medium"], np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [engine.MODE_PLAIN, engine.MODE_MIXED], ids=["plain", "mixed"])
@pytest.mark.parametrize("case", ["infinite_clear_segment", "zero_over_zero"])
def test_rays_that_end_before_their_neighbours(case, mode):
    # every other ray has a last segment that passes on no number (exp(-0 inf) in a clear medium, or 0 / 0 of a
    # SHORT query beam), while its neighbours in the packet have another scattering segment
    lite = case == "infinite_clear_segment"
    w = workload(**({} if lite else {"query_beam_type": W.SHORT_BEAM}))
    segment_lists(w)
    inside = 0
    for q in np.nonzero((w["sq_path_length"] == 1) & (w["sq_seg_count"] == 2))[0]:
        b = int(w["sq_seg_begin"][q])
        seg = [(w["seg_dist_min"][b + i], w["seg_dist_max"][b + i], int(w["seg_medium"][b + i]), w["seg_pdf"][b + i],
                w["seg_attenuation"][b + i]) for i in range(2)]
        assert seg[0][2] == 0 and seg[1][2] == 1
        t0, t1 = seg[1][0], seg[1][1]
        flags = int(w["sq_flags"][q]) | W.Q_LITE if lite else int(w["sq_flags"][q]) & ~W.Q_LITE
        if inside % 2:
            last = (t1, np.float32(np.inf), 0, 1.0, (1.0, 1.0, 1.0)) if lite else (t1, t1 + 1, 0, 0.0, (0.0, 0.0, 0.0))
            set_segments(w, q, seg + [last], flags)
        else:
            tm = np.float32(0.5) * (t0 + t1)
            set_segments(w, q, [seg[0], (t0, tm) + seg[1][2:], (tm, t1) + seg[1][2:]], flags)
        inside += 1
    assert inside > 50000
    segment_arrays(w)
    got, s, want, s0 = both(w, mode)
    same_pairs(s, s0)
    assert np.isfinite(want).all() and np.isfinite(got).all()
    err = G.rel_errors(got.astype(np.float64), want.astype(np.float64))
    assert err.max() <= (2e-5 if mode == engine.MODE_PLAIN else G.RTOL)


def morton_lanes():
    """The pixels (x, y) of an 8 x 4 block in the pixel order: bits x0 y0 x1 y1 x2 of the lane."""
    lane = np.arange(32)
    return (lane & 1) | (lane >> 1 & 2) | (lane >> 2 & 4), (lane >> 1 & 1) | (lane >> 2 & 2)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [engine.MODE_PLAIN, engine.MODE_MIXED], ids=["plain", "mixed"])
def test_wide_fans_of_short_rays(mode):
    # a dozen pixel blocks hold fans of rays about (1, 1, 1) from one origin; no other query makes a packet
    # (each has its own origin), so every fan is split into runs of 4 rays.  All advance along the first
    # ray's main axis x, but the lead of a run has its main axis y, along which its neighbours hardly advance
    w = workload()
    rng = np.random.default_rng(3)
    n = len(w["sq_flags"])
    w["sq_origin"] += rng.uniform(-1e-3, 1e-3, (n, 3)).astype(np.float32)
    by_pixel = {int(w["sq_pixel"][q]): q for q in np.nonzero(w["sq_path_length"] == 1)[0]}
    blocks = [[by_pixel.get((y0 + int(y)) * 419 + x0 + int(x)) for x, y in zip(*morton_lanes())]
              for y0 in range(0, 316, 4) for x0 in range(0, 416, 8)]
    blocks = [b for b in blocks if None not in b][::100][:12]
    segment_lists(w)
    fans = []
    for k, block in enumerate(blocks):
        for lane, q in enumerate(block):
            d = np.array((0.62, 0.55, 0.56) if lane < 4 else ((0.55, 0.62, 0.56) if lane % 4 == 0 else (0.8, 0.33, 0.5)))
            d = d + rng.uniform(-0.01, 0.01, 3)
            w["sq_direction"][q] = d / np.linalg.norm(d)
            w["sq_origin"][q] = (0.4, 0.45 + 0.002 * k, 0.35)
            set_segments(w, q, [(0.0, 0.3, 1, 0.9, (0.9, 0.9, 0.9))],
                         W.Q_ORIGIN_IN_MEDIUM | int(w["sq_flags"][q]))
            fans.append(q)
    segment_arrays(w)
    got, s, want, s0 = both(w, mode)
    assert s0["count_bb1d"][fans].sum() > 1000
    same_pairs(s, s0)
    err = G.rel_errors(got.astype(np.float64), want.astype(np.float64))
    assert err.max() <= (2e-5 if mode == engine.MODE_PLAIN else G.RTOL)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [engine.MODE_PLAIN, engine.MODE_MIXED], ids=["plain", "mixed"])
def test_segment_ends_at_piece_boundaries_far_from_the_origin(mode):
    # at coordinates of 4000 the predicate's t1 is off by about 1e-3: it takes pairs whose lines are closest
    # just beyond the ray's end, and the beam piece that owns such a pair is the one opposite that end, not the
    # one that holds the lines' closest point.  One beam of three pieces per ray, the end of the middle one close
    # to both points
    w = workload()
    rng = np.random.default_rng(5)
    for k in ("lv_position", "sq_origin", "pq_position", "beam_origin"):
        w[k] += np.float32(4000.0)
    rays = np.nonzero((w["sq_path_length"] == 1) & (w["sq_seg_count"] == 2))[0]
    n, r, length = len(rays), 0.01, 0.0899
    o, d = w["sq_origin"][rays].astype(np.float64), w["sq_direction"][rays].astype(np.float64)
    last = w["sq_seg_begin"][rays] + 1
    t0, t1 = w["seg_dist_min"][last], w["seg_dist_max"][last]
    t = t0 + (t1 - t0) * rng.uniform(0.3, 0.9, n)
    # directions at 30 to 60 degrees from the ray's
    c = rng.uniform(0.5, 0.87, n)
    v = np.cross(d, rng.normal(size=(n, 3)))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    d2 = (c[:, None] * d + np.sqrt(1 - c * c)[:, None] * v)
    d2 = (d2 / np.linalg.norm(d2, axis=1, keepdims=True)).astype(np.float32)
    side = np.cross(d, d2)
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    u = length * 2 / 3 + rng.uniform(-1e-3, 1e-3, n)
    o2 = (o + t[:, None] * d + 0.3 * r * side - u[:, None] * d2.astype(np.float64)).astype(np.float32)
    # the lines' closest point for the rounded inputs, and the rays' ends just before it
    b64, w64 = d2.astype(np.float64), o - o2.astype(np.float64)
    aa, cc, bb = (d * d).sum(1), (b64 * b64).sum(1), (d * b64).sum(1)
    dd, ee = (d * w64).sum(1), (b64 * w64).sum(1)
    t = (bb * ee - cc * dd) / (aa * cc - bb * bb)
    w["seg_dist_max"][last] = t - rng.uniform(0.0, 1e-3, n)
    old = len(w["beam_length"])
    for k in [k for k in w if k.startswith("beam_")]:
        w[k] = w[k][np.arange(n) % old].copy()
    w["beam_origin"], w["beam_direction"] = o2, d2
    w["beam_length"][:] = length
    w["beam_medium_id"][:] = 1
    got, s, want, s0 = both(w, mode, beam_piece_radii=3.0)
    assert s0["count_bb1d"][rays].sum() > n // 10
    same_pairs(s, s0)


@pytest.mark.gpu
def test_few_camera_queries_among_many_make_no_packets():
    # 40,000 camera queries on a pixel among 138,000 segment queries: too few to keep the packets' blocks busy
    w = workload()
    first = np.nonzero(w["sq_path_length"] == 1)[0]
    w["sq_pixel"][first[40000:]] = -1
    _, s, tested = results(w, engine.MODE_MIXED, query_order=1)
    _, s0, tested0 = results(w, engine.MODE_MIXED, query_order=0)
    assert tested == tested0
    same_pairs(s, s0)


@pytest.mark.gpu
def test_packets_of_a_crop_take_memory_by_the_queries():
    # the queries of 419 x 317 pixels in an image of 8192 x 8192: the packets' lists, at most 100 bytes per query
    w = workload()
    x, y = w["sq_pixel"] % 419, w["sq_pixel"] // 419
    w["sq_pixel"] = np.where(w["sq_pixel"] < 0, -1, (y + 4000) * 8192 + x + 4001).astype(np.int32)
    w["pq_pixel"][:] = -1
    w["params"]["image_width"], w["params"]["image_height"] = 8192, 8192
    made = []
    for order in (0, 1):
        with engine.EstimatorStage(0, engine.MODE_PLAIN) as st:
            st.set_tuning(query_order=order)
            st.run(w)
            made.append((st.device_bytes(), st.query_stats(), st.tested_counts()["bb1d"], st.segment_results()[1]))
    (bytes0, s0, tested0, want), (bytes1, s, tested, got) = made
    assert tested != tested0  # the packets ran
    same_pairs(s, s0)
    assert G.rel_errors(got.astype(np.float64), want.astype(np.float64)).max() <= 2e-5
    assert bytes1 - bytes0 <= 100 * len(w["sq_pixel"])
